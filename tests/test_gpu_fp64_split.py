"""FP64's split form: what it skips on a grid whose last tiles are cut, and its step
loop's remainders, bit for bit against the oracle (no tolerance applies)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def swept_steps(tvs, z, w, los, precision):
    with tvs.Engine(z, w, 30.0, los * 30, observer_height=1.65, precision=precision) as eng:
        eng.sweep_counters(True)
        eng.run()
        swept, _, steps, _ = eng.sweep_counters()
    return swept, steps


def test_cut_tiles_skip_segments(tvs, synth):
    """33 x 33 points of view: 8 of the 15 tiles of 16 x 8 are whole.  FP64 and EXACT32
    skip by the same bound against thresholds that differ by 2^-19 of the angle, so the
    steps that they sweep differ by less than a thousandth (a segment differs when its
    bound lies in that part: about one in 10^5)."""
    w, los = 833, 400
    z = synth.fbm(w, w, 0.8, 11, 0.0, 1500.0)
    exact, steps = swept_steps(tvs, z, w, los, "exact32")
    fp64, steps64 = swept_steps(tvs, z, w, los, "fp64")
    assert steps == steps64 and 0.1 * steps < exact < 0.9 * steps
    assert abs(fp64 - exact) <= exact // 1000


@pytest.mark.parametrize("los", [8, 11, 54, 56, 58, 60, 110, 112])
def test_step_loop_remainders(tvs, oracle, synth, los):
    """Step counts around the loop's unit (2) and a segment (32), on a grid whose last
    tiles are cut in both axes."""
    w = 3 * los + 5
    z = synth.fbm(w, w, 0.7, los, 0.0, 800.0)
    g = oracle.geometry(w, 30.0, los * 30)
    with tvs.Engine(z, w, 30.0, los * 30, observer_height=1.65, precision="fp64") as eng:
        for angle in (0, 38, 90, 141):
            d, x, _ = oracle.compile_band_data(g, float(angle))
            want = oracle.sweep_sector(g, z, 1.65, d, x, mode="fp64")[0]
            cum = np.zeros(eng.count, np.float32)
            eng.compute_sector(angle, cum)
            assert np.array_equal(bits(cum), bits(want.astype(np.float32))), angle
