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


def swept(eng):
    """Whether the split form ran: it counts its steps, the row kernel does not."""
    eng.sweep_counters(True)
    out = eng.run()[:2]
    steps = eng.sweep_counters()[2]
    eng.sweep_counters(False)
    return steps > 0, out


def set_again(eng, c):
    eng.set_sweep_config(c.points_x, c.points_y, bool(c.packed), bool(c.prefetch), c.layout)


def fields(c):
    return c.points_x, c.points_y, c.packed, c.prefetch, c.layout


def test_configuration_read_and_set_back(tvs, synth):
    """What is read, or chosen by the autotuner, names what runs: setting it changes
    nothing.  The row kernel stays within reach and agrees bit for bit."""
    z = np.round(synth.fbm(301, 301, 0.7, 9, 0.0, 1500.0))
    with tvs.Engine(z, 301, 30.0, 3000, observer_height=1.65, precision="fp64") as eng:
        split, want = swept(eng)
        assert split
        before = eng.sweep_config()
        set_again(eng, before)
        assert fields(eng.sweep_config()) == fields(before) and swept(eng)[0]
        for px, py, prefetch in ((1, 1, False), (4, 1, False), (2, 2, False), (2, 1, True)):
            eng.set_sweep_config(px, py, prefetch=prefetch)
            split, got = swept(eng)
            assert not split
            for a, b in zip(got, want):
                assert np.array_equal(bits(a), bits(b))
        chosen = eng.autotune(4)
        tuned = swept(eng)[0]
        set_again(eng, chosen)
        assert fields(eng.sweep_config()) == fields(chosen) and swept(eng)[0] == tuned
        set_again(eng, before)
        assert swept(eng)[0]
        with pytest.raises(tvs.TvsError):
            eng.set_sweep_config(4, 1, layout=9)


def test_batch_configuration_read_and_set_back(tvs, synth):
    import ctypes

    z = np.round(synth.fbm(257, 261, 0.7, 5, 0.0, 900.0))
    with tvs.Batch([(z, 30.0, 2550)], observer_height=1.65, precision="fp64") as b:
        def config():
            c = tvs.SweepConfig()
            assert tvs.lib().tvs_batch_get_sweep_config(b.b, ctypes.byref(c)) == tvs.OK
            return c

        def run():
            b.run()
            b.finish()
            return b.read(0)

        want, held = run(), b.device_bytes()  # (the split form's surface planes are in it)
        before = config()
        set_again(b, before)
        assert fields(config()) == fields(before) and b.device_bytes() == held
        for c in (b.autotune(4), before):
            set_again(b, c)
            assert fields(config()) == fields(c)
            for x, y in zip(run(), want):
                assert np.array_equal(bits(x), bits(y))
