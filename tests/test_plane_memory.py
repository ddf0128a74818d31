"""The memory of the surface planes (csrc/planes.cu) on the CPU: host code alone, compiled
with the C++ compiler against a runtime that counts allocations."""

import shutil
import subprocess
from pathlib import Path

from conftest import PKG_DIR

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "tvs_internal.cuh"

// the runtime: `room` bytes a device, allocations counted
static std::mutex mu;
static std::map<void *, size_t> live[80];
static size_t room = (size_t)-1;
static int made = 0;
static thread_local int device = 0;
static thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
static size_t used(int d) {
    size_t n = 0;
    for (auto &b : live[d]) n += b.second;
    return n;
}
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
    std::swap(*m, mode);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    std::lock_guard<std::mutex> l(mu);
    *p = nullptr;
    if (used(device) + n > room) return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    live[device][*p] = n;
    made++;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::mutex> l(mu);
    if (!live[device].erase(p)) std::_Exit(99);  // not of this device, or freed before
    std::free(p);
    return cudaSuccess;
}
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
const size_t MB = 1 << 20;

static void *take(size_t want, size_t *got = nullptr, size_t one = 0) {
    void *p;
    size_t n = want;
    if (tvs::plane_alloc(&p, &n, one) != cudaSuccess) return nullptr;
    if (got) *got = n;
    return p;
}

int main() {
    size_t got;
    // one piece per context; the only context's end gives it back
    void *a = take(245 * MB, &got);
    CHECK(a && got == 245 * MB && made == 1);
    tvs::plane_free(a, got);
    CHECK(used(0) == 0);
    // beside another context the next one takes what was freed, if it is not twice the need
    void *other = take(10 * MB);
    a = take(100 * MB);
    tvs::plane_free(a, 100 * MB);
    CHECK(used(0) == 110 * MB);
    made = 0;
    CHECK(take(60 * MB, &got) == a && got == 100 * MB && made == 0);
    tvs::plane_free(a, got);
    void *b = take(49 * MB, &got);
    CHECK(b != a && got == 49 * MB && made == 1);
    // the smallest that serves
    tvs::plane_free(b, got);
    CHECK(take(48 * MB, &got) == b && got == 49 * MB);
    tvs::plane_free(b, got);
    // at most kPlanesKept of them
    void *c = take(200 * MB);
    tvs::plane_free(c, 200 * MB);
    CHECK(used(0) == (10 + 100 + 49) * MB);
    for (int i = 0; i < 20; i++) {
        void *p[20];
        for (int k = 0; k < 20; k++) p[k] = take(MB);
        for (int k = 0; k < 20; k++) tvs::plane_free(p[k], MB);
        CHECK(used(0) <= 10 * MB + tvs::kPlanesKept);
    }
    // another device has its own
    device = 1;
    void *d1 = take(100 * MB);
    CHECK(used(1) == 100 * MB);
    tvs::plane_free(d1, 100 * MB);
    CHECK(used(1) == 0);
    device = 70;
    d1 = take(MB);
    tvs::plane_free(d1, MB);
    CHECK(d1 && used(70) == 0);
    device = 0;
    // where memory runs out the kept ones go first, for any buffer of the library
    room = used(0) + 5 * MB;
    void *buffer = nullptr;
    CHECK(tvs::device_malloc(&buffer, 20 * MB) == cudaSuccess && used(0) == 30 * MB);
    CHECK(take(1000 * MB) == nullptr && used(0) == 30 * MB);
    cudaFree(buffer);
    // where memory is short, the planes of fewer sectors: 180 of 1 MB, 90, 45, 22
    room = used(0) + 40 * MB;
    a = take(180 * MB, &got, MB);
    CHECK(a && got == 22 * MB);
    tvs::plane_free(a, got);
    tvs::plane_trim();
    room = used(0) + MB / 2;
    CHECK(take(180 * MB, nullptr, MB) == nullptr);
    // the last one's end gives everything back
    room = (size_t)-1;
    a = take(100 * MB);
    tvs::plane_free(a, 100 * MB);
    CHECK(used(0) == 110 * MB);
    tvs::plane_free(other, 10 * MB);
    CHECK(used(0) == 0);
    // a request that fails beside nothing leaves nothing
    room = MB;
    CHECK(take(2 * MB) == nullptr && used(0) == 0);
    room = (size_t)-1;
    CHECK(mode == cudaStreamCaptureModeGlobal);
    // threads
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; t++)
        ts.emplace_back([t] {
            device = t & 1;
            for (int i = 0; i < 2000; i++) {
                size_t n;
                void *p = take((1 + (i * 7 + t) % 90) * MB, &n);
                tvs::plane_free(p, n);
            }
        });
    for (auto &t : ts) t.join();
    CHECK(used(0) == 0 && used(1) == 0);
    return 0;
}
"""


def test_planes_are_kept_within_bounds_and_given_back(tmp_path):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(PROGRAM)
    csrc = PKG_DIR / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-pthread", "-I", str(csrc), "-I",
                    str(PKG_DIR.parent / "include"), "-I",
                    str(Path(nvcc).resolve().parent.parent / "include"), "-x", "c++",
                    str(csrc / "planes.cu"), str(main), "-o", str(exe)], check=True)
    got = subprocess.run([str(exe)], timeout=60, capture_output=True, text=True)
    assert got.returncode == 0, got.stdout
