"""Obstacles that do not span a periodic direction: a sphere that leaves through
one face of the box meets, right behind the opposite face, an obstacle that was
a whole period away when the lists were built.  No particle moves half the skin
on the way, so the lists are not rebuilt in between.

Blocks near the low and the high face of every periodic direction, spheres
crossing in both senses, in one direction and in all three, against the CPU FP64
restatement at every step (its wall contacts have no lists).  FP64 agrees to
rounding, FP32-split to its force law; before contact the force is the weight."""
import numpy as np
import pytest

from pacific_b200 import FP32_SPLIT, FP64, Grains
from pacific_b200.scenarios import Scenario
from tests.helpers import oracle_for

pytestmark = pytest.mark.gpu

L, R = 0.02, 1.0e-3
STEPS = 10


def _scene(axis, periodic):
    """Two spheres crossing the faces of one axis, 1 m/s and 1e-5 s a step: 60
    um before the face, in contact 20 um behind it, after eight steps (half the
    skin is 125 um)."""
    x = np.full((2, 3), 0.5 * L)
    v = np.zeros((2, 3))
    x[0, axis], v[0, axis] = L - 60.0e-6, 1.0
    x[1, axis], v[1, axis] = 60.0e-6, -1.0
    side = (axis + 1) % 3
    x[0, side], x[1, side] = 0.25 * L, 0.75 * L
    v[:, side] = 0.05
    walls = []
    for k in range(2):
        c, s = x[k].copy(), np.full(3, 6.0e-3)
        s[axis] = 2.0e-3
        gap = R + 20.0e-6 + 0.5 * s[axis]
        c[axis] = gap if k == 0 else L - gap
        walls.append(dict(centre=tuple(c), size=tuple(s), crust=1.0e-4, material="matW"))
    law = dict(kn=1.0e4, en=0.7, etat=None, muc=0.5, kt=2.0e3)
    q = np.zeros((2, 4))
    q[:, 3] = 1.0
    return Scenario("crossing", (0.0, 0.0, 0.0), (L, L, L), periodic, (0.0, 0.0, 0.0), 1.0e-5,
                    [dict(radius=R, crust=1.0e-4, density=2500.0, material="matP")], walls,
                    [dict(matA="matP", matB="matP", **law), dict(matA="matP", matB="matW", **law)],
                    np.zeros(2, np.int32), x, v, np.zeros((2, 3)), q)


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-10), (FP32_SPLIT, 1e-5)],
                         ids=["fp64", "fp32split"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("every", [False, True], ids=["one", "all"])
def test_crossing_spheres_meet_the_obstacle(tmp_path, lib, oracle_lib, axis, every, precision, tol):
    periodic = tuple(1 if every or d == axis else 0 for d in range(3))
    sc = _scene(axis, periodic)
    xml = str(sc.write_xml(tmp_path / "crossing.xml"))
    o = oracle_for(sc, xml)
    o.init()
    g = Grains(xml, precision)
    g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
    g.do_before_time_stepping()
    touched = 0
    for _ in range(STEPS):
        o.step(1)
        assert g.Simulation(1) == 0
        ref, got = o.state(), g.download_state()
        scale = max(np.abs(ref["F"]).max(), 1e-300)
        touched += int(np.abs(ref["F"]).max() > 0.0)
        assert np.abs(got["F"] - ref["F"]).max() <= STEPS * tol * scale
        assert np.abs(got["x"] - ref["x"]).max() <= STEPS * tol * R
    assert touched >= 2 and g.step_counts()[1] == 1     # in contact, on the first lists
    assert (np.abs(ref["F"][:, axis]) > 0.0).all()
    g.close()
