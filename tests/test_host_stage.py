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


def test_slots_without_memory_for_threads(tmp_path):
    """The slots are laid out whatever memory there is for threads: none, or for the first
    few alone.  (A single-core machine starts none.)"""
    assert run(tmp_path, r"""
#include <new>
#include <vector>
long left = -1;  // allocations until the first that fails (-1: none fails)
void *operator new(size_t n) {
    if (left == 0) throw std::bad_alloc();
    if (left > 0) left--;
    void *p = std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
int main() {
    const uint32_t bands = 40000, reserved = 200;  // 32 MB
    std::vector<uint64_t> offsets(bands + 1);
    for (uint32_t k = 0; k < bands; k++) offsets[k + 1] = offsets[k] + 1 + k % 7 + (k == 11) * 300;
    std::vector<uint32_t> ids(offsets[bands]), rings((size_t)bands * reserved);
    for (size_t i = 0; i < ids.size(); i++) ids[i] = (uint32_t)i + 1;
    for (long memory : {0l, 2l, -1l}) {
        rings.assign(rings.size(), 0xABCDABCDu);
        left = memory;
        tvs_host::expand_records(rings.data(), bands, reserved, offsets.data(), ids.data());
        left = -1;
        for (uint32_t k = 0; k < bands; k++) {
            const uint32_t *row = &rings[(size_t)k * reserved];
            const uint64_t n = offsets[k + 1] - offsets[k];
            if (row[0] != n) return 1;
            for (uint32_t i = 1; i < reserved; i++)
                if (row[i] != (i <= n ? (uint32_t)(offsets[k] + i) : 0)) return 2;
        }
    }
    return 0;
}
""") == 0
