"""Sectors whose steps move a point of view more than the line of sight sideways:
the reference's linear sample ids wrap into a neighbouring row (kernel.rs:259-292), so
a bound of a segment's samples by a patch of the DEM says nothing about them.  Bit for
bit against the oracle: every decision and every addition is the same, so no tolerance
applies."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, SCALE, LOS = 801, 1.0, 100
ANGLES = (60, 88, 89, 91, 92)  # 90 is not wide; past these a band leaves the DEM
ORACLE_MODE = {"exact32": "exact32", "mixed64": "fp64", "fp32": "fp32", "fp64": "fp64"}


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def f32(c):
    return c.astype(np.float32) if c.dtype == np.float64 else c


def walls():
    """Points of view at the left edge look over a ridge of 300 m, past which their
    samples wrap to a wall of 5000 m at the right edge, 60 steps (two segments) away."""
    z = np.zeros((W, W), np.float32)
    z[:, 60:98] = 300.0
    z[:, 721:] = 5000.0
    return z


@pytest.fixture(scope="module")
def expected(oracle):
    """{(mode, angle): (surfaces, counts, ids)} of the oracle, made once."""
    made = {}

    def get(mode, angle):
        if (mode, angle) not in made:
            g = oracle.geometry(W, SCALE, LOS)
            d, x, n = oracle.compile_band_data(g, float(angle))
            rows = np.cumsum(d[:n].astype(np.int64)) + W // 2
            assert np.abs(rows % W - W // 2).max() > LOS and n > 32  # wide, several segments
            made[mode, angle] = oracle.sweep_sector(g, walls(), 1.65, d, x, mode=mode, compact=True)
        return made[mode, angle]

    return get


@pytest.mark.parametrize("precision,layout", [(p, k) for p in ("exact32", "mixed64", "fp32")
                                              for k in range(1, 10)] + [("fp64", None)])
def test_no_segment_of_a_wide_sector_is_skipped(tvs, expected, precision, layout):
    mode = ORACLE_MODE[precision]
    with tvs.Engine(walls(), W, SCALE, LOS, observer_height=1.65, precision=precision) as eng:
        if layout:
            eng.set_sweep_config(4, 1, layout=layout)
        for angle in ANGLES:
            c0, n0, ids0 = expected(mode, angle)
            cum = np.zeros(eng.count, np.float32)
            eng.compute_sector(angle, cum)
            assert np.array_equal(bits(cum), bits(f32(c0))), angle
            cum[:] = 0.0
            offsets, ids, _ = eng.compute_sector_rings(angle, cum)
            assert np.array_equal(bits(cum), bits(f32(c0))), angle
            assert np.array_equal(np.diff(offsets).astype(np.uint32), n0), angle
            assert np.array_equal(ids, ids0), angle


@pytest.mark.parametrize("precision", ["mixed64", "fp64"])
def test_a_run_over_wide_and_other_sectors(tvs, oracle, precision):
    """Sectors 70 to 109 in one sweep (90 alone is not wide)."""
    g = oracle.geometry(W, SCALE, LOS)
    want = np.zeros(g.computable_points_count, np.float64)
    for angle in range(70, 110):
        d, x, _ = oracle.compile_band_data(g, float(angle))
        oracle.sweep_sector(g, walls(), 1.65, d, x, mode="fp64", cumulative=want)
    with tvs.Engine(walls(), W, SCALE, LOS, observer_height=1.65, precision=precision) as eng:
        eng.device_reset()
        eng.device_run_sectors(70, 40)
        eng.device_finish()
        got, _ = eng.read_surfaces()
    assert np.array_equal(bits(got), bits(want.astype(np.float32)))
