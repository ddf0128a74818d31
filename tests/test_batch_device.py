"""A batch's host code (csrc/batch.cu) on the CPU, against a runtime that only keeps the
current device: its planes come from its own device, whatever the caller's thread has
current."""

import shutil
import subprocess
from pathlib import Path

from conftest import PKG_DIR

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>
#include "tvs.h"
#include "tvs_context.hpp"
#include "tvs_internal.cuh"

static int device = 0;
static std::vector<std::pair<int, size_t>> planes;  // {device, bytes} of every allocation
static char some[1];
extern "C" {
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaEventCreate(cudaEvent_t *) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
int tvs_create(const tvs_params *p, const float *, uint64_t, tvs_context **out) {
    device = p->device;
    tvs_context *c = new tvs_context();
    c->p = *p;
    c->g.tvs_width = 33;
    c->g.tvs_height = c->row_end = 257;
    c->done_cap = 1 << 20;
    *out = c;
    return TVS_OK;
}
void tvs_destroy(tvs_context *c) { delete c; }
}
namespace tvs {
cudaError_t plane_alloc(void **p, size_t *bytes, size_t) {
    planes.push_back({device, *bytes});
    *p = some;
    return cudaSuccess;
}
void plane_free(void *, size_t) {}
cudaError_t device_malloc(void **p, size_t) { *p = some; return cudaSuccess; }
cudaError_t launch_shape_batch(const ShapeArgs *, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
}  // namespace tvs

int main() {
    tvs_params p{};
    p.width = p.height = 300;
    p.precision = TVS_PRECISION_FP32;
    p.device = 3;
    const float *z = nullptr;
    tvs_batch *b = nullptr;
    if (tvs_batch_create(&p, &z, 1, &b) != TVS_OK || planes.size() != 1) return 1;
    device = 0;  // the caller goes on with another device
    tvs_sweep_config c{4, 1, 0, 0, 3};  // 1 x 257 tiles in place of 3 x 33: larger planes
    if (tvs_batch_set_sweep_config(b, &c) != TVS_OK) return 2;
    if (planes.size() != 2 || planes[1].second <= planes[0].second) return 3;
    for (auto &a : planes)
        if (a.first != 3) return 4;
    tvs_batch_destroy(b);
    return 0;
}
"""


def test_planes_come_from_the_batchs_device(tmp_path):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    main, exe = tmp_path / "main.cpp", tmp_path / "main"
    main.write_text(PROGRAM)
    csrc = PKG_DIR / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-I", str(csrc), "-I", str(PKG_DIR.parent / "include"),
                    "-I", str(Path(nvcc).resolve().parent.parent / "include"), "-x", "c++",
                    str(csrc / "batch.cu"), str(main), "-x", "none", "-L", str(PKG_DIR), "-ltvs_cuda",
                    f"-Wl,-rpath,{PKG_DIR}", "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
