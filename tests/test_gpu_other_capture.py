"""A program that captures a graph on a stream of its own may call a context meanwhile: the
context's first planes, or larger ones, are allocated without breaking that capture."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("sectors_before", [0, 1])
@pytest.mark.parametrize("beside", [False, True])
def test_sweep_while_another_stream_is_captured(tvs, synth, mode, sectors_before, beside):
    import torch

    z = synth.fbm(601, 601, 0.8, 5, 0.0, 1500.0)

    def engine():
        return tvs.Engine(z, 601, 30.0, 6000, observer_height=1.65, precision="mixed64")

    with engine() as eng:
        eng.device_reset()
        eng.device_run_sectors(10, 40)
        eng.device_finish()
        want, _ = eng.read_surfaces()
    x = torch.zeros(1000, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with engine() as eng, engine() as other:
        if beside:  # another context with planes: freed ones are kept
            other.run()
        if sectors_before:
            eng.device_run_sectors(0, sectors_before)
            eng.device_finish()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
            x += 1
            eng.device_reset()
            eng.device_run_sectors(10, 40)
            x += 1
        eng.device_finish()
        got, _ = eng.read_surfaces()
        graph.replay()
        torch.cuda.synchronize()
    assert float(x.min()) == float(x.max()) == 2.0
    assert np.array_equal(bits(got), bits(want))
