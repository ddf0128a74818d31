"""Sweeps that take more than one launch of the split sweep (its surface planes hold a part
of the sectors): the same bits as sectors added in turn, one by one.  Every decision and
every addition is the same, so no tolerance applies."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("precision", ["exact32", "fp32", "mixed64", "fp64"])
def test_surfaces_over_several_launches(tvs, synth, precision):
    """601 x 601 points of view: 38 x 76 tiles of 128, 3.0 MB of 32-bit planes a sector, of
    which 256 MB hold 90: 180 sectors take two launches (64-bit planes: four)."""
    z = np.round(synth.fbm(1801, 1801, 0.75, 7, 0.0, 1500.0))
    with tvs.Engine(z, 1801, 30.0, 18000, observer_height=1.65, precision=precision) as eng:
        assert eng.geometry.tvs_width == 601
        eng.device_reset()
        eng.device_run_sectors(0, 180)
        eng.device_finish()
        assert eng.last_launch_count() == 1 + (4 if precision in ("mixed64", "fp64") else 2)
        planes = eng.read_surfaces()
        eng.set_queue_wait(held_tile=0xFFFFFFFE)  # no such tile: added in turn, in one launch
        eng.device_reset()
        eng.device_run_sectors(0, 180)
        eng.device_finish()
        assert eng.last_launch_count() == 2
        turn = eng.read_surfaces()
    for a, b in zip(planes, turn):
        assert np.array_equal(bits(a), bits(b))
    assert planes[0].any()


def test_ring_records_over_several_launches(tvs, synth):
    """46 sectors in one call: 5.9 MB of planes each, of which 256 MB hold 45."""
    z = np.round(synth.fbm(1801, 1801, 0.95, 7, 0.0, 300.0))
    first, n = 60, 46
    with tvs.Engine(z, 1801, 30.0, 18000, observer_height=1.65, precision="mixed64") as eng:
        cum = np.zeros(eng.count, np.float32)
        eng.compute_sectors_rings(first, n, cum)  # (allocates, and computes the shapes)
        before = eng.last_launch_count()
        cum[:] = 0.0
        offsets, ids = eng.compute_sectors_rings(first, n, cum)[:2]
        assert eng.last_launch_count() - before == 2 + 2  # sweeps, count and gather
        per = eng.geometry.total_bands
        for s in range(n):
            one = np.zeros(eng.count, np.float32)
            o, i, _ = eng.compute_sector_rings(first + s, one)
            span = offsets[s * per:(s + 1) * per + 1]
            assert np.array_equal(np.diff(span), np.diff(o)), s
            assert np.array_equal(ids[span[0]:span[-1]], i), s
        eng.set_queue_wait(held_tile=0xFFFFFFFE)
        eng.device_reset()
        eng.device_run_sectors(first, n)
        eng.device_finish()
        want, _ = eng.read_surfaces()
    assert np.array_equal(bits(cum), bits(want))
