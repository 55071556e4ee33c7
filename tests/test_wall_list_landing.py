"""More particles near a wall than the wall list has room for, inside one call.

A layer of some 20,000 spheres (above 16,384 the list does not start with room
for all) stays out of the floor's reach when the call begins and lands in it at
once, while every twentieth sphere rests on the floor from the start and slides
(so there is wall memory to carry over).  No wall contact may be left out: every
evaluation sees all of them, or is put off until the list has grown.  The
trajectory is, to the byte, that of the same spheres with room for everybody,
through replayed graphs and plain launches, in calls shorter and longer than the
interval between two looks at the lists, with ended contacts forgotten or kept;
and it is the CPU FP64 restatement's.

The same for spheres inserted on the floor between two calls."""
import numpy as np
import pytest

from pacific_b200 import FP32_SPLIT, FP64, Grains, scenarios
from tests.helpers import oracle_for

pytestmark = pytest.mark.gpu

R = 1.0e-3
NX, NY = 143, 140
N = NX * NY
ROOM = 4 * N          # a quarter of the capacity is what the list starts with


def _layer(speed=1.0):
    spacing = 2.05e-3
    box = (spacing * (NX + 1e-6), spacing * (NY + 1e-6), 6.0e-3)
    sc = scenarios.settling_box(n=N, seed=11, box=box, spacing=spacing, jitter=1.0e-9, vmax=1.0e-3,
                                etat=None)
    resting = np.arange(N) % 20 == 0
    # (resting: the overlap that carries the weight)
    sag = 2500.0 * 4.0 / 3.0 * np.pi * R ** 3 * 9.81 / 1.0e4
    sc.x[:, 2] = np.where(resting, R - sag, 2.0 * R)
    sc.v[:] = (0.002, 0.001, 0.0)
    sc.v[~resting, 2] = -speed
    return sc, resting


def _run(xml, sc, precision, calls, room=0, graphs=True, prune=True):
    g = Grains(xml, precision)
    g.use_graphs(graphs)
    g.set_contact_memory_pruning(prune)
    if room:
        g.reserve(room)
    g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
    g.do_before_time_stepping()
    for k in calls:
        assert g.Simulation(k) == 0
    s, h, counts = g.download_state(), g.download_history(), g.step_counts()
    g.close()
    return s, h, counts


def _on_the_floor(h):
    """Spheres that remember a contact with the floor (wall 4)."""
    return len(np.unique(h["owner"][h["partner"] == -6]))


def _same(a, b):
    for k in ("x", "v", "w", "q", "F", "T"):
        assert np.array_equal(a[0][k], b[0][k]), k
    for k in a[1]:
        assert np.array_equal(a[1][k], b[1][k]), k
    assert a[2] == b[2]


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
@pytest.mark.parametrize("graphs,prune", [(True, True), (False, True), (True, False)])
def test_layer_lands_within_a_call(tmp_path, lib, precision, graphs, prune):
    sc, resting = _layer()
    xml = str(sc.write_xml(tmp_path / "layer.xml"))
    got = _run(xml, sc, precision, (101,), graphs=graphs, prune=prune)
    _same(got, _run(xml, sc, precision, (101,), room=ROOM, graphs=graphs, prune=prune))
    assert got[2][0] == 102                             # every evaluation once
    assert _on_the_floor(got[1]) == N


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
def test_layer_lands_in_long_and_split_calls(tmp_path, lib, precision):
    # 0.16 m/s: contact after 537 steps, past the first look at the lists
    sc, resting = _layer(speed=0.16)
    xml = str(sc.write_xml(tmp_path / "slow.xml"))
    ref = _run(xml, sc, precision, (542,), room=ROOM)
    assert _on_the_floor(ref[1]) == N
    _same(_run(xml, sc, precision, (542,)), ref)


def test_landed_layer_matches_the_oracle(tmp_path, lib, oracle_lib):
    sc, resting = _layer()
    xml = str(sc.write_xml(tmp_path / "layer.xml"))
    o = oracle_for(sc, xml)
    o.init()
    o.step(101)
    ref = o.state()
    got, h, _ = _run(xml, sc, FP64, (101,))
    scale = np.abs(ref["F"]).max()
    assert np.abs(got["F"] - ref["F"]).max() <= 101 * 1e-10 * scale
    assert _on_the_floor(h) == N


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
def test_spheres_inserted_on_the_floor(tmp_path, lib, precision):
    sc, _ = _layer()
    sc.x[:, 2] = 4.0 * R                                # out of reach of floor and lid
    sc.v[:] = 0.0
    keep = 17000                                        # the others come in on the floor
    xml = str(sc.write_xml(tmp_path / "empty.xml"))
    g = Grains(xml, precision)
    g.reserve(N - keep + 3000)
    g.upload_state(sc.type[:keep], sc.x[:keep], sc.v[:keep], sc.w[:keep], sc.q[:keep])
    g.do_before_time_stepping()
    assert g.Simulation(2) == 0
    spots = [(sc.x[k, 0], sc.x[k, 1], R - 1.0e-7) for k in range(6000)]
    for p in spots:
        assert g.insert_particle(0, p, v=(0.02, 0.0, 0.0), force=True) is not None
    assert g.Simulation(2) == 0
    F = g.download_state()["F"]
    assert len(F) == keep + 6000
    assert (F[keep:, 2] > 0.0).all() and (F[:keep, 2] <= 0.0).all()
    g.close()


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
def test_convex_layer_lands_within_a_call(tmp_path, lib, precision):
    """17,161 cubes, tetrahedra and cylinders (walls of a particle in turn, support
    vertices carried on) thrown onto the floor."""
    tet = scenarios.write_tetrahedron(tmp_path / "tet.insert")
    sc = scenarios.convex_pour(n=131 * 131, seed=4, poly_path=tet, box=(0.4915, 0.4915, 0.02),
                               cylinders=True)
    sc.x[:, 2] += 0.6e-3                                # out of the floor's reach
    sc.v[:, 2] = -5.0
    xml = str(sc.write_xml(tmp_path / "convex.xml"))
    got = _run(xml, sc, precision, (110,))
    assert (got[1]["partner"] == -6).sum() > 1000
    _same(got, _run(xml, sc, precision, (110,), room=4 * sc.n))
