// host_stage.hpp -- the host's side of results that come back to pageable memory
// (internal to the library).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace tvs_host {

// A copy to pageable memory waits by itself and goes through the driver's own pinned
// buffer.  The small results of a call share a pinned block instead, so that one
// wait serves all.  The block is ordinary memory of the process, pinned with its first
// context and left so (pinning and unpinning it with every only context of a program
// took 2.6 ms of a 301^2 context's 3.5), and is lent to one call at a time; a call that
// finds it lent (another thread's) takes the driver's path.
constexpr size_t kSmall = 256 << 10;

void stage_ref(bool device_set);  // a context exists, its device current
void stage_unref();

// The block, for as long as this lives; p is null when it is lent, missing or smaller
// than bytes.  No call waits for a lent block, nor does a context's creation or end.  The
// copies between it and the device run on stream; unless done() has said that they
// were waited for, the end of this waits for them (error paths).
class SmallStage {
public:
    explicit SmallStage(cudaStream_t stream, size_t bytes = 0);
    void done() { stream_ = nullptr; }
    ~SmallStage();
    SmallStage(const SmallStage &) = delete;
    SmallStage &operator=(const SmallStage &) = delete;
    unsigned char *p = nullptr;

private:
    cudaStream_t stream_;
};

// Host memory for the compact records of one call, for as long as this lives: the
// process's pinned buffer (grown up to kPinnedMost, lent as the block above is, done()
// included, and freed with the last context), or memory of its own where that is lent or too small.
class RecordBuffer {
public:
    explicit RecordBuffer(cudaStream_t stream);
    void done() { stream_ = nullptr; }
    ~RecordBuffer();
    RecordBuffer(const RecordBuffer &) = delete;
    RecordBuffer &operator=(const RecordBuffer &) = delete;
    unsigned char *get(size_t bytes);  // once; null: out of memory

private:
    static constexpr size_t kPinnedMost = (size_t)64 << 20;
    cudaStream_t stream_;
    bool lent_ = false;
    unsigned char *own_ = nullptr;
};

// The reference's ring layout from compact records: band k's reserved u32 slots get
// its count, its ids (the first reserved - 1 of them) and zeros, by several threads
// where there is much to write.
void expand_records(uint32_t *rings, uint64_t bands, uint32_t reserved, const uint64_t *offsets,
                    const uint32_t *ids);

// The same where the ids are in their slots already (and what follows them is not zero).
void complete_records(uint32_t *rings, uint64_t bands, uint32_t reserved, const uint32_t *counts);

}  // namespace tvs_host
