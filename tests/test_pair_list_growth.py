"""The pair list outgrows its allocation inside a call: a cubic lattice of 512
spheres that contracts from a spacing beyond the skin (no pair listed) to one
where the list needs more than the 16 entries per particle and 4,096 that it
starts with, before the first look at the allocation (every 512 steps).  No pair
may be left out: the trajectory, through the first contacts, is to the byte that
of the same spheres with room for 5,000 more, whose list never runs short."""
import numpy as np
import pytest

from pacific_b200 import FP32_SPLIT, FP64, Grains, scenarios

pytestmark = pytest.mark.gpu

R, SIDE, SKIN = 1.0e-3, 8, 4.0
STEPS = 274


def _contracting():
    spacing = 6.3 * R
    box = (spacing * (SIDE + 1e-6),) * 3
    sc = scenarios.settling_box(n=SIDE ** 3, seed=31, box=box, spacing=spacing, jitter=1.0e-6,
                                vmax=1.0e-3, etat=None)
    # from a spacing of 6.3 radii to 1.998 in STEPS steps
    sc.v += (sc.x - 0.5 * np.array(box)) * ((1.998 - 6.3) / 6.3 / (STEPS * sc.dt))
    return sc


def _run(xml, sc, precision, calls, reserve, graphs):
    g = Grains(xml, precision)
    g.use_graphs(graphs)
    if reserve:
        g.reserve(reserve)
    g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
    g.set_tuning(SKIN)
    g.do_before_time_stepping()
    first = g.pair_counts()[0]
    for k in calls:
        assert g.Simulation(k) == 0
    out = g.download_state(), g.download_history(), g.step_counts()
    entries, contacts = g.pair_counts()
    g.close()
    return out, first, entries, contacts


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
@pytest.mark.parametrize("graphs", [True, False], ids=["graphs", "plain"])
def test_list_runs_short_within_a_call(tmp_path, lib, precision, graphs):
    sc = _contracting()
    xml = str(sc.write_xml(tmp_path / "lattice.xml"))
    room, _, _, contacts = _run(xml, sc, precision, (STEPS,), 5000, graphs)
    assert contacts > 500
    got, first, entries, _ = _run(xml, sc, precision, (STEPS,), 0, graphs)
    assert first < 0.8 * (16 * sc.n + 4096) < 16 * sc.n + 4096 < entries
    for k in ("x", "v", "w", "q", "F", "T"):
        assert np.array_equal(got[0][k], room[0][k]), k
    for k in got[1]:
        assert np.array_equal(got[1][k], room[1][k]), k
    assert got[2] == room[2] and got[2][0] == STEPS + 1
