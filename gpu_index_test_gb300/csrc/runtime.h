// runtime.h — host-side runtime of the C-ABI: error reporting, device buffers,
// temporary workspaces and launch accounting.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <functional>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "gbsa.h"

namespace gbsa {

// Exceptions never cross the C-ABI: every entry point catches Error and returns its
// code, with the message stored for gbsa_last_error().
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void set_last_error(const std::string& msg);

#define GBSA_CUDA(call)                                                                                      \
    do {                                                                                                     \
        cudaError_t _e = (call);                                                                             \
        if (_e != cudaSuccess) {                                                                             \
            throw ::gbsa::Error(_e == cudaErrorMemoryAllocation ? GBSA_ERR_NOMEM : GBSA_ERR_CUDA,            \
                                std::string(#call " failed: ") + cudaGetErrorString(_e) + " at " __FILE__ ":" \
                                    + std::to_string(__LINE__));                                             \
        }                                                                                                    \
    } while (0)

// Counts kernel launches issued by this library (reported by gbsa_launch_count).
extern std::atomic<uint64_t> g_launches;
#define GBSA_LAUNCHED()                                                                                     \
    do {                                                                                                    \
        ::gbsa::g_launches.fetch_add(1, std::memory_order_relaxed);                                         \
        GBSA_CUDA(cudaGetLastError());                                                                      \
    } while (0)

// Scratch of a call, in the order of the stream that uses it, from a memory pool that the
// library keeps for each device.  The pool holds on to at most kScratchKept bytes, and only
// while an index lives (ScratchLease): with the last index its memory goes back, and
// without one it returns whatever is free at each synchronisation, as CUDA's default pool
// does.  (An allocation from memory that the pool holds takes 1 us; mapping new memory and
// giving it back 70 + 50 us for a status word, 130 + 60 us and a wait for the whole device
// with cudaMalloc and cudaFree.)  Safe with several threads and streams: CUDA hands a
// block on only when the stream that freed it has passed that point.
constexpr uint64_t kScratchKept = 256ull << 20;
void* scratch_alloc(size_t bytes, cudaStream_t st);
void scratch_free(void* p, cudaStream_t st) noexcept;

struct ScratchLease {
    ScratchLease();
    ~ScratchLease();
    ScratchLease(const ScratchLease&) = delete;
    ScratchLease& operator=(const ScratchLease&) = delete;
};

// Owning device buffer: memory of its own, or with a stream scratch that only this stream's
// work uses.
class DeviceBuffer {
public:
    DeviceBuffer() = default;
    explicit DeviceBuffer(size_t bytes) { resize(bytes); }
    DeviceBuffer(size_t bytes, cudaStream_t st) : st_(st), scratch_(true) { resize(bytes); }
    ~DeviceBuffer() { release(); }
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    DeviceBuffer(DeviceBuffer&& o) noexcept : p_(o.p_), n_(o.n_), st_(o.st_), scratch_(o.scratch_) {
        o.p_ = nullptr;
        o.n_ = 0;
    }
    DeviceBuffer& operator=(DeviceBuffer&& o) noexcept {
        if (this != &o) {
            release();
            p_ = o.p_;
            n_ = o.n_;
            st_ = o.st_;
            scratch_ = o.scratch_;
            o.p_ = nullptr;
            o.n_ = 0;
        }
        return *this;
    }
    void resize(size_t bytes) {
        if (bytes <= n_) return;
        release();
        void* p = nullptr;
        if (scratch_) p = scratch_alloc(bytes, st_);
        else GBSA_CUDA(cudaMalloc(&p, bytes ? bytes : 16));
        p_ = p;
        n_ = bytes;
    }
    void release() {
        if (p_ && scratch_) scratch_free(p_, st_);
        else if (p_) cudaFree(p_);
        p_ = nullptr;
        n_ = 0;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p_);
    }
    size_t size() const { return n_; }

private:
    void* p_ = nullptr;
    size_t n_ = 0;
    cudaStream_t st_ = nullptr;
    bool scratch_ = false;
};

// Pinned host buffer.
class PinnedBuffer {
public:
    PinnedBuffer() = default;
    ~PinnedBuffer() {
        if (p_) cudaFreeHost(p_);
    }
    PinnedBuffer(const PinnedBuffer&) = delete;
    PinnedBuffer& operator=(const PinnedBuffer&) = delete;
    void resize(size_t bytes) {
        if (bytes <= n_) return;
        if (p_) cudaFreeHost(p_);
        p_ = nullptr;
        n_ = 0;
        GBSA_CUDA(cudaMallocHost(&p_, bytes ? bytes : 16));
        n_ = bytes;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p_);
    }
    size_t size() const { return n_; }

private:
    void* p_ = nullptr;
    size_t n_ = 0;
};

// Grow-only pool of temporary device buffers, handed out in order and recycled by
// reset().  Not thread-safe; one per handle, or with a stream one per call (scratch).
class Workspace {
public:
    Workspace() = default;
    explicit Workspace(cudaStream_t st) : st_(st), scratch_(true) {}
    void* get(size_t bytes) {
        bytes = (bytes + 255) & ~size_t(255);
        if (next_ == bufs_.size()) bufs_.push_back(scratch_ ? DeviceBuffer(0, st_) : DeviceBuffer());
        DeviceBuffer& b = bufs_[next_++];
        b.resize(bytes);
        return b.as<void>();
    }
    template <class T>
    T* get(size_t n) {
        return static_cast<T*>(get(n * sizeof(T)));
    }
    void reset() { next_ = 0; }
    // Buffers handed out after mark() are handed out again after rewind(): for scratch of
    // steps that follow each other in one stream.
    size_t mark() const { return next_; }
    void rewind(size_t mark) { next_ = mark; }

private:
    std::vector<DeviceBuffer> bufs_;
    size_t next_ = 0;
    cudaStream_t st_ = nullptr;
    bool scratch_ = false;
};

inline unsigned grid_for(size_t n, unsigned block, unsigned max_blocks = 1u << 30) {
    size_t g = (n + block - 1) / block;
    if (g == 0) g = 1;
    if (g > max_blocks) g = max_blocks;
    return (unsigned)g;
}

int device_sm_count();

// Runs fn(begin, end) over [0, n) in chunks on a process-wide pool of host threads
// (the calling thread takes part); small ranges run inline.  For the per-read host
// loops of the C-ABI (staging offsets, rebasing results).
void host_parallel_for(size_t n, const std::function<void(size_t, size_t)>& fn);

// Runs fn(i) for i in [0, n) as separate tasks on the same pool (one task per
// thread at a time); for a few coarse tasks.
void host_parallel_tasks(size_t n, const std::function<void(size_t)>& fn);

}  // namespace gbsa
