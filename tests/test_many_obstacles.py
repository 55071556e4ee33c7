"""Systems of many obstacles: spheres resting in the gaps of a floor of 810 short
bars, on two of them or, across a seam, on four.

The wall list holds the (particle, wall) pairs within reach, so its memory goes
with those and not with particles times walls, and it grows when the few slots
per particle that it starts with do not do.  Forces against the CPU FP64
restatement over three steps (the memory of the first is used by the next two):
FP64 agrees to the order of the sums, FP32-split to its force law."""
import numpy as np
import pytest
import torch

from pacific_b200 import FP32_SPLIT, FP64, Grains, scenarios
from tests.helpers import oracle_for

pytestmark = pytest.mark.gpu

R = 1.0e-3
BARS, PIECES = 81, 10
STEPS = 3


def _scene(mur=0.02):
    """Bars 0.8 R wide at a pitch of 1.6 R; a sphere over every second gap sits
    on the two edges beside it, 1e-7 m into them."""
    pitch, length = 1.6 * R, 10.0 * R
    nx, ny = BARS // 2, int(PIECES * length / (2.5 * R)) - 1
    n = nx * ny
    box = (BARS * pitch, PIECES * length, 8.0 * R)
    j, i = np.divmod(np.arange(n), nx)
    rng = np.random.default_rng(21)
    x = np.empty((n, 3))
    x[:, 0] = (2 * i + 1.0) * pitch                     # the middle of a gap
    x[:, 1] = (j + 1.0) * 2.5 * R                   # every fourth on a seam
    x[:, 2] = 2.0 * R + np.sqrt((R - 1.0e-7) ** 2 - (0.4 * R) ** 2)
    walls = [dict(centre=((b + 0.5) * pitch, (k + 0.5) * length, 1.0 * R),
                  size=(0.8 * R, length, 2.0 * R), crust=0.1 * R, material="matW")
             for b in range(BARS) for k in range(PIECES)]
    law = dict(kn=1.0e4, en=0.7, etat=None, muc=0.5, kt=2.0e3, mur=mur)
    q = np.zeros((n, 4))
    q[:, 3] = 1.0
    return scenarios.Scenario(
        "bars", (0.0, 0.0, 0.0), box, (0, 0, 0), (0.0, 0.0, -9.81), 1.0e-5,
        [dict(radius=R, crust=0.1 * R, density=2500.0, material="matP")], walls,
        [dict(matA="matP", matB="matP", **law), dict(matA="matP", matB="matW", **law)],
        np.zeros(n, np.int32), x, rng.uniform(-1.0e-3, 1.0e-3, (n, 3)), np.zeros((n, 3)), q)


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-10), (FP32_SPLIT, 1e-5)],
                         ids=["fp64", "fp32split"])
def test_spheres_between_bars(tmp_path, lib, oracle_lib, precision, tol):
    sc = _scene()
    xml = str(sc.write_xml(tmp_path / "bars.xml"))
    o = oracle_for(sc, xml)
    o.init()
    o.step(STEPS)
    ref = o.state()
    g = Grains(xml, precision)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
    g.do_before_time_stepping()
    assert g.Simulation(STEPS) == 0
    taken = free - torch.cuda.mem_get_info()[0]
    got, h = g.download_state(), g.download_history()
    g.close()
    # a slot takes 188 bytes, a sphere's other arrays some 5 KB
    assert taken < 10_000 * sc.n + (32 << 20)
    own, par = o.history()[:2]
    assert set(zip(h["owner"].tolist(), h["partner"].tolist())) == set(zip(own.tolist(), par.tolist()))
    hits = np.bincount(own[par < 0], minlength=sc.n)
    assert hits.max() == 4 and hits.sum() > 2 * sc.n + 64   # more than the list starts with
    for k in ("F", "T"):
        assert np.abs(got[k] - ref[k]).max() <= STEPS * tol * np.abs(ref[k]).max(), k
