"""The wall list and the contact memory beside the lists at sizes where their
allocations and launches change: a packed slab two layers high, whose spheres
all touch a wall and their neighbours, just below and above the particle count
up to which the wall list starts with two slots per particle (16,384; above, a
slot per two particles, so that it has to grow before or, started from forces,
at the first evaluation), one evaluation per warp lane and several.

Against the CPU FP64 restatement over three steps (the memory of the first is
used by the next two), started by the leapfrog start and from uploaded forces
(the way a reload does, without it).  FP64 agrees to the order of the sums,
FP32-split to its force law: 1e-10 and 1e-5 of the largest force per step."""
import numpy as np
import pytest

from pacific_b200 import FP32_SPLIT, FP64, Grains, scenarios
from tests.helpers import oracle_for

pytestmark = pytest.mark.gpu

STEPS = 3


def _slab(nx, ny, mur):
    spacing = 2.0e-3 - 4.0e-7
    box = (spacing * (nx + 1e-6), spacing * (ny + 1e-6), spacing * (2 + 1e-6))
    sc = scenarios.settling_box(n=2 * nx * ny, seed=3, box=box, spacing=spacing, jitter=2.0e-8,
                                vmax=1.0e-3, etat=None)
    for m in sc.models:
        m["mur"] = mur
    return sc


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-10), (FP32_SPLIT, 1e-5)])
@pytest.mark.parametrize("nx,ny,mur", [(3, 2, 0.02), (90, 91, 0.0), (91, 91, 0.02)])
def test_slab_matches_the_oracle(tmp_path, lib, oracle_lib, nx, ny, mur, precision, tol):
    sc = _slab(nx, ny, mur)
    xml = str(sc.write_xml(tmp_path / "slab.xml"))
    o = oracle_for(sc, xml)
    o.init()
    start = o.state()
    o.step(STEPS)
    ref = o.state()
    scale = {k: np.abs(ref[k]).max() for k in ("F", "T")}
    for reload in (False, True):
        g = Grains(xml, precision)
        g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
        if reload:
            g.upload_forces(start["F"], start["T"])
        else:
            g.do_before_time_stepping()
        assert g.Simulation(STEPS) == 0
        got = g.download_state()
        n, contacts = sc.n, g.pair_counts()[1]
        h = g.download_history()
        # every sphere remembers its wall below or above it
        assert len(np.unique(h["owner"][h["partner"] < 0])) == n
        assert contacts >= 2 * n
        g.close()
        for k in ("F", "T"):
            assert np.abs(got[k] - ref[k]).max() <= STEPS * tol * scale[k], (reload, k)
        assert np.abs(got["x"] - ref["x"]).max() <= STEPS * tol * 1e-7
