"""Surface planes are only speed: with little device memory left, calls that need some
take the planes', and the sweeps that then find no room for planes give the same bits."""

import contextlib
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, LOS = 1201, 400  # 245 MB of planes for EXACT32's 180 sectors
MB = 1 << 20


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def engine(tvs, z, precision="exact32"):
    return tvs.Engine(z, W, 30.0, LOS * 30, observer_height=1.65, precision=precision)


@contextlib.contextmanager
def leave(free):
    """Holds the device's memory but for `free` bytes (in allocations of 2 MB).  What the
    device reports as free cannot all be had, so `free` bytes are taken first, then all
    that there is, and the first are given back."""
    import torch

    torch.empty(1, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cuda, held = ctypes.CDLL("libcuda.so.1"), []

    def take(n):
        p = ctypes.c_uint64()
        rc = cuda.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n))
        assert rc in (0, 2), rc  # (2: out of memory)
        if rc == 0:
            held.append(p)
        return rc == 0

    try:
        assert take(free)
        n = torch.cuda.mem_get_info()[0] // (2 * MB) * 2 * MB
        while n >= 2 * MB:
            if not take(n):
                n = n // (4 * MB) * 2 * MB
        cuda.cuMemFree_v2(held.pop(0))
        yield
    finally:
        for p in held:
            cuda.cuMemFree_v2(p)


@pytest.fixture(scope="module")
def terrain(synth):
    return synth.fbm(W, W, 0.75, 3, 0.0, 1500.0)


def test_ring_records_take_the_planes_memory(tvs, terrain):
    """One sector's ring records need 82 MB of slots and a 64 MB list: neither is left
    beside the planes of a whole run (100 MB), both are without them (345 MB)."""
    with engine(tvs, terrain) as eng:
        cum = np.zeros(eng.count, np.float32)
        want = eng.compute_sector_rings(46, cum)
    with engine(tvs, terrain) as eng:
        run = eng.run()[:2]
        before = eng.device_bytes()
        with leave(100 * MB):
            got = np.zeros(eng.count, np.float32)
            offsets, ids, _ = eng.compute_sector_rings(46, got)
            assert np.array_equal(bits(got), bits(cum))
            assert np.array_equal(offsets, want[0]) and np.array_equal(ids, want[1])
            after = eng.device_bytes()
            again = eng.run()[:2]
        assert after < before + 200 * MB  # the planes' 245 MB are not counted any more
        for a, b in zip(again, run):
            assert np.array_equal(bits(a), bits(b))


def test_a_context_takes_the_memory_of_freed_planes(tvs, terrain):
    """The pool keeps freed planes while any context lives; a new context's own buffers (the
    DEM's 5.8 MB, its copies' 23 MB and more, beside 6 MB left) come first."""
    with engine(tvs, terrain) as first:
        want = first.run()[:2]
        with engine(tvs, terrain) as second:
            second.run()
        with leave(6 * MB), engine(tvs, terrain) as third:
            got = third.run()[:2]
    for a, b in zip(got, want):
        assert np.array_equal(bits(a), bits(b))


def test_plain_kernel_scratch_in_part(tvs, synth):
    """The plain kernel's two scratch buffers (2.6 MB each): where only one fits the call
    fails, also when it is made again, and the context computes once there is room."""
    z = synth.fbm(2401, 2401, 0.75, 3, 0.0, 1500.0)
    with tvs.Engine(z, 2401, 30.0, 800 * 30, observer_height=1.65, sweep_kernel="plain") as eng:
        failed = 0
        for free in (2, 3, 4, 5, 6):
            with leave(free * MB):
                for _ in range(2):
                    try:
                        eng.device_run_sectors(46, 1)
                        eng.device_finish()
                        break
                    except tvs.TvsError as e:
                        assert "out of memory" in str(e)
                        failed += 1
        assert failed >= 2
        cum = np.zeros(eng.count, np.float32)
        eng.compute_sector(46, cum)
    with tvs.Engine(z, 2401, 30.0, 800 * 30, observer_height=1.65) as eng:
        want = np.zeros(eng.count, np.float32)
        eng.compute_sector(46, want)
    assert np.array_equal(bits(cum), bits(want))


@pytest.mark.parametrize("precision", ["exact32", "fp64"])
def test_a_context_without_memory_for_the_copies(tvs, terrain, precision):
    """The DEM's row-interleaved copies (23 MB, with the DEM in one allocation) are only
    speed too: where they do not fit beside a context's other buffers (15 MB), it runs
    from the plain DEM, and adds the surfaces in turn."""
    with engine(tvs, terrain, precision) as eng:
        want = eng.run()[:2]
    with leave(22 * MB), engine(tvs, terrain, precision) as eng:
        assert eng.device_bytes() < 22 * MB
        got = eng.run()[:2]
    for a, b in zip(got, want):
        assert np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("precision", ["exact32", "mixed64", "fp64"])
def test_planes_of_fewer_sectors_where_memory_is_short(tvs, terrain, precision):
    """70 MB hold a quarter or an eighth of the 180 sectors' planes (245, 489 MB): the sweep
    takes launches of those, and neither asks again nor adds the surfaces in turn."""
    with engine(tvs, terrain, precision) as eng:
        want = eng.run()[:2]
    with engine(tvs, terrain, precision) as eng:
        before = eng.device_bytes()
        with leave(70 * MB):
            eng.device_reset()
            eng.device_run_sectors(0, 180)
            eng.device_finish()
            held = eng.device_bytes()
            assert 30 * MB <= held - before <= 70 * MB
            assert 1 + 4 <= eng.last_launch_count() <= 1 + 9
            got = eng.read_surfaces()
            again = eng.run()[:2]
        once_more = eng.run()[:2]  # (with memory to spare)
        assert eng.device_bytes() == held
    for r in (got, again, once_more):
        for a, b in zip(r, want):
            assert np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("sectors_before", [0, 1])
def test_a_callers_capture_allocates_planes(tvs, synth, sectors_before):
    """A sweep that is captured takes planes for all its sectors, whatever there were."""
    import torch

    z = synth.fbm(601, 601, 0.8, 5, 0.0, 1500.0)
    with tvs.Engine(z, 601, 30.0, 6000, observer_height=1.65) as eng:
        want = eng.run()[:2]
    with tvs.Engine(z, 601, 30.0, 6000, observer_height=1.65) as eng:
        eng.set_queue_wait(0, 1 << 30)  # (uploads what a first sweep uploads, without planes)
        eng.device_run_sectors(0, 1)
        eng.set_queue_wait()
        if sectors_before:
            eng.device_run_sectors(0, sectors_before)
        eng.device_finish()
        before = eng.device_bytes()
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.ExternalStream(eng.stream())
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="thread_local")
            eng.device_reset()
            eng.device_run_sectors(0, 180)
            graph.capture_end()
        assert eng.last_launch_count() == 2  # 338 tiles: 62 MB of planes
        assert eng.device_bytes() - before >= 180 * 2 * 338 * 128 * 4
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            eng.device_finish()
            for a, b in zip(eng.read_surfaces(), want):
                assert np.array_equal(bits(a), bits(b))
        del graph
        eng.run()
