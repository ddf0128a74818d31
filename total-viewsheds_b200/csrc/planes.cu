// planes.cu -- device memory of the surface planes (host code; tvs_internal.cuh says
// what they are and how many bytes a sweep wants).
#include <cstdint>
#include <mutex>
#include <utility>

#include "tvs_internal.cuh"

namespace tvs {
namespace {

// A device's freed planes, kept for the next context of a program that opens one DEM
// after another while it has any.
struct FreedPlanes {
    static constexpr int kMost = 8;
    uint32_t held = 0;  // planes not yet freed
    size_t bytes = 0;
    int n = 0;
    struct { void *p; size_t bytes; } block[kMost];

    void *take(int i) {
        void *p = block[i].p;
        bytes -= block[i].bytes;
        block[i] = block[--n];
        return p;
    }
};
std::mutex mutex;
constexpr int kDevices = 64;  // devices past these keep none
FreedPlanes freed[kDevices];

FreedPlanes *freed_of_current_device() {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && dev < kDevices ? &freed[dev] : nullptr;
}

// Frees (outside the lock: cudaFree waits for the device) what f keeps, and p.
void give_back(FreedPlanes *f, std::unique_lock<std::mutex> lock, void *p = nullptr) {
    void *ps[FreedPlanes::kMost + 1] = {p};
    int n = 1;
    while (f && f->n) ps[n++] = f->take(f->n - 1);
    lock.unlock();
    const AnyCapture any;
    for (int i = 0; i < n; i++)
        if (ps[i]) cudaFree(ps[i]);
}

}  // namespace

cudaError_t plane_alloc(void **p, size_t *bytes, size_t one) {
    *p = nullptr;
    FreedPlanes *f = freed_of_current_device();
    if (f) {
        const std::lock_guard<std::mutex> lock(mutex);
        f->held++;
        int best = -1;
        for (int i = 0; i < f->n; i++)
            if (f->block[i].bytes >= *bytes && f->block[i].bytes / 2 <= *bytes &&
                (best < 0 || f->block[i].bytes < f->block[best].bytes))
                best = i;
        if (best >= 0) {
            *bytes = f->block[best].bytes;
            *p = f->take(best);
            return cudaSuccess;
        }
    }
    const AnyCapture any;
    cudaError_t e = device_malloc(p, *bytes);
    while (e == cudaErrorMemoryAllocation && one != 0 && *bytes >= 2 * one) {
        cudaGetLastError();
        *bytes = *bytes / one / 2 * one;
        e = device_malloc(p, *bytes);
    }
    if (e != cudaSuccess && f) {
        std::unique_lock<std::mutex> lock(mutex);
        if (--f->held == 0) give_back(f, std::move(lock));
    }
    return e;
}

void plane_free(void *p, size_t bytes) {
    if (!p) return;
    FreedPlanes *f = freed_of_current_device();
    std::unique_lock<std::mutex> lock(mutex);
    if (f && --f->held != 0) {
        if (f->n < FreedPlanes::kMost && f->bytes + bytes <= kPlanesKept) {
            f->block[f->n].p = p;
            f->block[f->n++].bytes = bytes;
            f->bytes += bytes;
            return;
        }
        f = nullptr;  // (the kept ones stay)
    }
    give_back(f, std::move(lock), p);
}

void plane_trim() { give_back(freed_of_current_device(), std::unique_lock<std::mutex>(mutex)); }

cudaError_t device_malloc(void **p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    plane_trim();
    return cudaMalloc(p, bytes);
}

}  // namespace tvs
