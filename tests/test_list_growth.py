"""A small system whose pair list outgrows its first allocation: the lists then
move to an allocation of their own, and every other array of the system stays
where it was.  110 packed FP64 spheres with a skin of four radii need more
entries than 16 per particle and 4,096 (the first lists open a block that later
arrays share); the skin changes no result, so the trajectory is that of the same
spheres at the default skin and of the same spheres with room for 5,000 more,
whose first lists hold them all, to the byte."""
import numpy as np
import pytest

from pacific_b200 import FP32_SPLIT, FP64, Grains, scenarios

pytestmark = pytest.mark.gpu


def _packed():
    spacing = 2.0e-3 - 4.0e-7
    box = (spacing * (5 + 1e-6), spacing * (5 + 1e-6), spacing * (5 + 1e-6))
    return scenarios.settling_box(n=110, seed=9, box=box, spacing=spacing, jitter=2.0e-8,
                                  vmax=1.0e-3, etat=None)


def _run(xml, sc, precision, skin, reserve):
    g = Grains(xml, precision)
    if reserve:
        g.reserve(reserve)
    g.upload_state(sc.type, sc.x, sc.v, sc.w, sc.q)
    if skin is not None:
        g.set_tuning(skin)
    g.do_before_time_stepping()
    for steps in (1, 20, 30):
        assert g.Simulation(steps) == 0
    s, entries, h = g.download_state(), g.pair_counts()[0], g.download_history()
    g.close()
    return s, entries, h


@pytest.mark.parametrize("precision", [FP64, FP32_SPLIT], ids=["fp64", "fp32split"])
def test_small_system_outgrows_its_first_lists(tmp_path, lib, precision):
    sc = _packed()
    xml = str(sc.write_xml(tmp_path / "packed.xml"))
    ref, _, href = _run(xml, sc, precision, None, 0)
    for reserve in (0, 5000):
        s, entries, h = _run(xml, sc, precision, 4.0, reserve)
        assert (entries > 0.8 * (16 * (sc.n + reserve) + 4096)) == (reserve == 0)
        for k in ("x", "v", "w", "q", "F", "T"):
            assert np.array_equal(s[k], ref[k]), (reserve, k)
        for k in ("owner", "partner", "kdelta"):
            assert np.array_equal(h[k], href[k]), (reserve, k)
