"""The split sweep's two ways of adding surfaces (a plane per sector and
direction, or in turn behind a wait) and its step loop's remainders, against
each other and the oracle, bit for bit: every decision and every addition is
the same, so no tolerance applies."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORACLE_MODE = {"exact32": "exact32", "mixed64": "fp64", "fp32": "fp32"}
IN_TURN = 0xFFFFFFFE  # no such tile: nothing is held, but the surfaces are added in turn


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("precision", ["exact32", "mixed64", "fp32"])
@pytest.mark.parametrize("w,h,los,rows", [(301, 301, 100, None), (340, 262, 87, (11, 77)),
                                          (1201, 1201, 400, None)])
def test_planes_equal_surfaces_added_in_turn(tvs, synth, precision, w, h, los, rows):
    """1201^2 takes its 180 sectors in more than one launch."""
    z = np.round(synth.fbm(w, h, 0.75, 3, 0.0, 1500.0))
    with tvs.Engine(z, w, 30.0, los * 30, height=h, observer_height=1.65, precision=precision,
                    rows=rows) as eng:
        planes = eng.run()[:2]
        eng.set_queue_wait(held_tile=IN_TURN)
        turn = eng.run()[:2]
    for a, b in zip(planes, turn):
        assert np.array_equal(bits(a), bits(b))
    assert planes[0].any()


@pytest.mark.parametrize("precision", ["exact32", "mixed64", "fp32"])
@pytest.mark.parametrize("los", [8, 11, 54, 56, 58, 60, 110, 112])
def test_step_loop_remainders(tvs, oracle, synth, precision, los):
    """Step counts around the loop's unit (2 or 4) and a segment (32), on a grid
    whose last tiles are cut in both axes."""
    w = 3 * los + 5
    z = synth.fbm(w, w, 0.7, los, 0.0, 800.0)
    g = oracle.geometry(w, 30.0, los * 30)
    with tvs.Engine(z, w, 30.0, los * 30, observer_height=1.65, precision=precision) as eng:
        for angle in (0, 38, 90, 141):
            d, x, _ = oracle.compile_band_data(g, float(angle))
            want = oracle.sweep_sector(g, z, 1.65, d, x, mode=ORACLE_MODE[precision])[0]
            cum = np.zeros(eng.count, np.float32)
            eng.compute_sector(angle, cum)
            assert np.array_equal(bits(cum), bits(want.astype(np.float32))), angle


@pytest.mark.parametrize("observer", [0.0, 1e-6, -2.0, 1.65, 300.0])
def test_mixed64_guard_band_observer_heights(tvs, oracle, synth, observer):
    """The guard band's part of the observer height, with the ties that it must
    re-decide: a plane (every sample's angle the same but for the curvature),
    whole-metre terrain and a flat sea."""
    w, los = 160, 50
    yy, xx = np.mgrid[0:w, 0:w].astype(np.float32)
    plane = 3000.0 + 12.0 * xx + 7.0 * yy
    metres = np.round(synth.fbm(w, w, 0.8, 5, 0.0, 90.0))
    metres[:60] = 0.0
    g = oracle.geometry(w, 30.0, los * 30)
    for z in (plane, metres):
        z = np.ascontiguousarray(z, np.float32)
        with tvs.Engine(z, w, 30.0, los * 30, observer_height=observer, precision="mixed64") as eng:
            for angle in (0, 27, 45, 90, 120):
                d, x, _ = oracle.compile_band_data(g, float(angle))
                want = oracle.sweep_sector(g, z, observer, d, x, mode="fp64")[0]
                cum = np.zeros(eng.count, np.float32)
                eng.compute_sector(angle, cum)
                assert np.array_equal(bits(cum), bits(want.astype(np.float32))), (observer, angle)


@pytest.mark.parametrize("w,h,los,rows,observer,relief", [
    (301, 301, 100, None, 1.65, 1500.0), (340, 262, 87, (11, 77), 0.0, 40.0),
    (173, 173, 57, None, -3.0, 9000.0)])
def test_fp64_split_form_equals_the_rows_and_the_oracle(tvs, oracle, synth, w, h, los, rows, observer,
                                                        relief):
    """FP64 by default evaluates angles where its first test passes; the row
    kernel (a configuration set by hand) evaluates every step.  Whole metres and a
    flat sea give exact ties."""
    z = np.round(synth.fbm(w, h, 0.7, 9, 0.0, relief))
    z[:h // 4] = 0.0
    with tvs.Engine(z, w, 30.0, los * 30, height=h, observer_height=observer, precision="fp64",
                    rows=rows) as eng:
        c0 = eng.sweep_config()
        assert (c0.points_x, c0.points_y, c0.layout) == (2, 1, 0)
        split = eng.run()[:2]
        eng.set_queue_wait(held_tile=IN_TURN)
        turn = eng.run()[:2]
        eng.set_queue_wait()
        eng.set_sweep_config(2, 1)
        row = eng.run()[:2]
        cfg = eng.autotune(2)
        assert cfg.layout == 0
        tuned = eng.run()[:2]
    for other in (turn, row, tuned):
        for a, b in zip(split, other):
            assert np.array_equal(bits(a), bits(b))
    if rows is None:
        g = oracle.geometry(w, 30.0, los * 30, height=h)
        want = oracle.run_f64(g, z, observer)[0].astype(np.float32)
        assert np.array_equal(bits(split[0]), bits(want))


def test_fp64_batch_equals_engines(tvs, synth):
    tiles = [(np.round(synth.fbm(w, h, 0.7, w, 0.0, 900.0)), 30.0, min(w, h) // 3 * 30)
             for w, h in ((257, 261), (330, 258))]
    with tvs.Batch(tiles, observer_height=1.65, precision="fp64") as b:
        b.run()
        b.finish()
        got = [b.read(i) for i in range(2)]
    for (z, s, los), g in zip(tiles, got):
        with tvs.Engine(z, z.shape[1], s, los, height=z.shape[0], observer_height=1.65,
                        precision="fp64") as eng:
            eng.set_sweep_config(4, 1)
            want = eng.run()[:2]
        for a, b in zip(g, want):
            assert np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("precision", ["exact32", "mixed64", "fp32"])
@pytest.mark.parametrize("los", [8, 54, 58, 112])
def test_ring_records_where_segments_are_skipped(tvs, oracle, synth, precision, los):
    """A ring open before a skipped segment or step closes at its first step: a ridge
    in front of low ground, where whole segments lie below every horizon, and a
    flat sea; several sectors per call and one."""
    w = 3 * los + 5
    z = synth.fbm(w, w, 0.7, los, 0.0, 30.0)
    z[::max(los // 2, 3), :] += 900.0
    z[:, ::max(los // 3, 3)] += 500.0
    z[: w // 4] = 0.0
    g = oracle.geometry(w, 30.0, los * 30)
    mode = ORACLE_MODE[precision]
    with tvs.Engine(z, w, 30.0, los * 30, observer_height=1.65, precision=precision) as eng:
        cum = np.zeros(eng.count, np.float32)
        offsets, ids, _ = eng.compute_sectors_rings(88, 4, cum)
        per = eng.geometry.total_bands
        for s in range(4):
            d, x, _ = oracle.compile_band_data(g, float(88 + s))
            c0, n0, ids0 = oracle.sweep_sector(g, z, 1.65, d, x, mode=mode, compact=True)
            one = np.zeros(eng.count, np.float32)
            o1, i1, _ = eng.compute_sector_rings(88 + s, one)
            assert np.array_equal(bits(one), bits(c0.astype(np.float32)))
            assert np.array_equal(np.diff(o1).astype(np.uint32), n0)
            assert np.array_equal(i1, ids0)
            span = offsets[s * per:(s + 1) * per + 1]
            assert np.array_equal(np.diff(span).astype(np.uint32), n0)
            assert np.array_equal(ids[span[0]:span[-1]], ids0)


@pytest.mark.parametrize("precision", ["exact32", "mixed64", "fp64"])
@pytest.mark.parametrize("planes_before", [0, 1, 20])
def test_sweeps_in_a_callers_capture(tvs, synth, precision, planes_before):
    """A caller's graph of a sweep computes the sweep whatever planes there were when it
    was captured (none, one sector's, all), and after the context's planes have grown."""
    import torch

    z = synth.fbm(301, 301, 0.8, 5, 0.0, 1500.0)
    with tvs.Engine(z, 301, 30.0, 3000, observer_height=1.65, precision=precision) as eng, \
            tvs.Engine(z, 301, 30.0, 3000, observer_height=1.65, precision=precision) as other:
        other.device_reset()
        other.device_run_sectors(40, 20)
        other.device_finish()
        want, _ = other.read_surfaces()
        if planes_before:
            eng.device_run_sectors(40, planes_before)
        else:  # (uploads what a first sweep uploads; a held tile takes no planes)
            eng.set_queue_wait(0, 1 << 30)
            eng.device_run_sectors(40, 1)
            eng.set_queue_wait()
        eng.device_finish()
        graph = torch.cuda.CUDAGraph()
        stream = torch.cuda.ExternalStream(eng.stream())
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            eng.device_reset()
            eng.device_run_sectors(40, 20)
            graph.capture_end()
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            eng.device_finish()
            got, _ = eng.read_surfaces()
            assert np.array_equal(bits(got), bits(want))
            eng.run()  # 180 sectors: more planes
        del graph
