"""The host's side of results (csrc/host_stage.cu) on the CPU: it holds no device code, so
it compiles with the C++ compiler, here against a runtime that does nothing."""

import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import PKG_DIR

RUNTIME = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
extern "C" {
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
}
#include "host_stage.hpp"
"""


def run(tmp_path, source):
    """Compiles source with host_stage.cu and returns the program's exit code."""
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(RUNTIME + source)
    csrc = PKG_DIR / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(csrc), "-I",
                    str(Path(nvcc).resolve().parent.parent / "include"), "-x", "c++",
                    str(csrc / "host_stage.cu"), str(main), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], timeout=60).returncode


def test_contexts_come_and_go_while_the_block_is_lent(tmp_path):
    """A call holds the block until the GPU has finished: a context that another thread
    creates or destroys meanwhile (on another GPU, say) does not wait for it, and one that
    finds the block lent goes without."""
    assert run(tmp_path, r"""
#include <atomic>
#include <chrono>
#include <thread>
int main() {
    tvs_host::stage_ref(true);
    std::atomic<bool> done{false}, without{false};
    std::thread other;
    {
        tvs_host::SmallStage waits_for_the_gpu(nullptr);
        if (!waits_for_the_gpu.p) return 2;
        other = std::thread([&] {
            tvs_host::stage_ref(true);
            without = tvs_host::SmallStage(nullptr).p == nullptr;
            tvs_host::stage_unref();
            done = true;
        });
        for (int i = 0; i < 500 && !done; i++) std::this_thread::sleep_for(std::chrono::milliseconds(10));
        if (!done || !without) std::_Exit(1);
    }
    other.join();
    if (!tvs_host::SmallStage(nullptr).p) return 3;
    tvs_host::stage_unref();
    return 0;
}
""") == 0
