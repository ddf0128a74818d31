// host_stage.cu -- see host_stage.hpp.
#include "host_stage.hpp"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace tvs_host {
namespace {

struct Stage {
    std::mutex refs;  // users, and who makes the block
    int users = 0;
    std::mutex lent;  // held by the call that uses the block, for as long as it waits for the GPU
    std::atomic<unsigned char *> block{nullptr};  // made once, never freed
    std::mutex records_lent;  // the same for the record buffer
    unsigned char *records = nullptr;
    size_t records_cap = 0;
};

Stage &stage() {
    static Stage *s = new Stage;  // contexts may outlive static destruction
    return *s;
}

}  // namespace

void stage_ref(bool device_set) {
    Stage &st = stage();
    std::lock_guard<std::mutex> lock(st.refs);
    st.users++;
    if (st.block || !device_set) return;
    void *p = nullptr;
    if (posix_memalign(&p, 4096, kSmall) != 0) return;
    if (cudaHostRegister(p, kSmall, cudaHostRegisterPortable) != cudaSuccess) {
        cudaGetLastError();
        std::free(p);
        return;
    }
    st.block = (unsigned char *)p;  // (a call that looked before takes the driver's path)
}

void stage_unref() {
    Stage &st = stage();
    std::lock_guard<std::mutex> lock(st.refs);
    if (--st.users > 0) return;
    std::lock_guard<std::mutex> records(st.records_lent);
    if (st.records) cudaFreeHost(st.records);
    st.records = nullptr;
    st.records_cap = 0;
}

SmallStage::SmallStage(cudaStream_t stream, size_t bytes) : stream_(stream) {
    Stage &st = stage();
    if (bytes > kSmall || !st.lent.try_lock()) return;
    p = st.block;
    if (!p) st.lent.unlock();
}

SmallStage::~SmallStage() {
    if (!p) return;
    if (stream_) cudaStreamSynchronize(stream_);
    stage().lent.unlock();
}

RecordBuffer::RecordBuffer(cudaStream_t stream)
    : stream_(stream), lent_(stage().records_lent.try_lock()) {}

RecordBuffer::~RecordBuffer() {
    if (stream_) cudaStreamSynchronize(stream_);
    if (lent_) stage().records_lent.unlock();
    std::free(own_);
}

unsigned char *RecordBuffer::get(size_t bytes) {
    Stage &st = stage();
    if (lent_ && bytes <= kPinnedMost) {
        if (bytes > st.records_cap) {
            const size_t cap = std::min(bytes + bytes / 2, kPinnedMost);
            if (st.records) cudaFreeHost(st.records);
            st.records_cap = 0;
            if (cudaHostAlloc((void **)&st.records, cap, cudaHostAllocPortable) == cudaSuccess) {
                st.records_cap = cap;
            } else {
                cudaGetLastError();
                st.records = nullptr;
            }
        }
        if (st.records) return st.records;
    }
    own_ = (unsigned char *)std::malloc(bytes);
    return own_;
}

void expand_records(uint32_t *rings, uint64_t bands, uint32_t reserved, const uint64_t *offsets,
                    const uint32_t *ids) {
    auto rows = [&](uint64_t from, uint64_t to) {
        for (uint64_t k = from; k < to; k++) {
            uint32_t *row = rings + k * reserved;
            const uint64_t n = offsets[k + 1] - offsets[k];
            const size_t kept = (size_t)std::min<uint64_t>(n, reserved - 1);
            row[0] = (uint32_t)n;
            std::memcpy(row + 1, ids + offsets[k], kept * sizeof(uint32_t));
            std::memset(row + 1 + kept, 0, (reserved - 1 - kept) * sizeof(uint32_t));
        }
    };
    // a thread for every 4 MB, up to three quarters of the machine's (39 MB: 4.2 ms on
    // one thread, 0.6 on 8, 0.4 on 12)
    constexpr int kMost = 16;
    const uint64_t bytes = bands * reserved * sizeof(uint32_t);
    const int n = (int)std::max<uint64_t>(
        1, std::min<uint64_t>({(uint64_t)kMost, std::thread::hardware_concurrency() * 3 / 4, bytes >> 22}));
    std::thread helpers[kMost];
    int started = 0;
    uint64_t at = 0;
    const uint64_t each = (bands + n - 1) / n;
    try {
        for (; started < n - 1; started++) {
            const uint64_t to = std::min(at + each, bands);
            helpers[started] = std::thread(rows, at, to);
            at = to;
        }
    } catch (const std::exception &) {  // no more threads, or no memory for one: the rest is done here
    }
    rows(at, bands);
    for (int t = 0; t < started; t++) helpers[t].join();
}

void complete_records(uint32_t *rings, uint64_t bands, uint32_t reserved, const uint32_t *counts) {
    for (uint64_t k = 0; k < bands; k++) {
        uint32_t *row = rings + k * reserved;
        const size_t kept = std::min(counts[k], reserved - 1);
        row[0] = counts[k];
        std::memset(row + 1 + kept, 0, (reserved - 1 - kept) * sizeof(uint32_t));
    }
}

}  // namespace tvs_host
