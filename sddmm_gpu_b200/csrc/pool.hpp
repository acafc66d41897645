// Device memory that plans and calls give back is kept by the handle for the next ones: cudaMalloc and cudaFree of a few
// megabytes cost up to 1.5 ms a pair and wait for the whole device, more than planning a small matrix.
//
// The pool belongs to one handle.  The handle is used by one host thread at a time, but its plans may be destroyed by others
// (a garbage collector's), so the pool locks.  It keeps at most LIMIT bytes that nobody uses; more go back to CUDA at
// once, all of it when the handle is trimmed or destroyed or an allocation fails.  A
// block given back while work on a stream may still touch it carries that stream and is handed out again only to work
// on the same stream, until wait() has waited for that stream.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <new>
#include <unordered_map>

namespace sddmm {

class DevicePool {
public:
    static constexpr size_t LIMIT = 2ull << 30;

    ~DevicePool() { release(); }
    // for work on the stream
    cudaError_t alloc(void **ptr, size_t bytes, cudaStream_t stream)
    {
        std::lock_guard<std::mutex> hold(lock_);
        const size_t n = rounded(bytes);
        // a quarter more than asked for at most, so that a small request does not take a large block away
        for (auto it = free_.lower_bound(n); it != free_.end() && it->first <= n + n / 4; ++it) {
            if (it->second.busy && it->second.stream != stream) continue;
            *ptr = it->second.ptr;
            kept_ -= it->first;
            free_.erase(it);
            return cudaSuccess;
        }
        cudaError_t e = cudaMalloc(ptr, n);
        if (e == cudaErrorMemoryAllocation && kept_ > 0) {
            (void)cudaGetLastError();
            release_all();
            e = cudaMalloc(ptr, n);
        }
        if (e != cudaSuccess) {
            *ptr = nullptr;
            return e;
        }
        try {
            size_[*ptr] = n;
        } catch (const std::bad_alloc &) {
            cudaFree(*ptr);
            *ptr = nullptr;
            return cudaErrorMemoryAllocation;
        }
        return cudaSuccess;
    }
    // busy: work enqueued on the stream may still use the block
    void free(void *ptr, cudaStream_t stream, bool busy)
    {
        if (!ptr) return;
        std::lock_guard<std::mutex> hold(lock_);
        auto it = size_.find(ptr);
        if (it == size_.end() || it->second > LIMIT / 2) {
            if (it != size_.end()) size_.erase(it);
            cudaFree(ptr);  // waits for the device
            return;
        }
        // the blocks that have been idle longest make room
        while (kept_ + it->second > LIMIT) {
            auto old = free_.begin();
            for (auto f = free_.begin(); f != free_.end(); ++f)
                if (f->second.since < old->second.since) old = f;
            kept_ -= old->first;
            size_.erase(old->second.ptr);
            cudaFree(old->second.ptr);
            free_.erase(old);
        }
        try {
            free_.emplace(it->second, Block{ptr, stream, busy, ++clock_});
            kept_ += it->second;
        } catch (const std::bad_alloc &) {
            size_.erase(it);
            cudaFree(ptr);
        }
    }
    // Waits for the stream; what was given back on it is idle then.
    cudaError_t wait(cudaStream_t s)
    {
        // only what was given back before the wait began: another thread may give more back meanwhile
        unsigned long long before;
        {
            std::lock_guard<std::mutex> hold(lock_);
            before = clock_;
        }
        const cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> hold(lock_);
        for (auto &f : free_)
            if (f.second.stream == s && f.second.since <= before) f.second.busy = false;
        return cudaSuccess;
    }
    // everything that nobody uses goes back to CUDA
    void release()
    {
        std::lock_guard<std::mutex> hold(lock_);
        release_all();
    }

private:
    void release_all()
    {
        for (auto &f : free_) {
            size_.erase(f.second.ptr);
            cudaFree(f.second.ptr);
        }
        free_.clear();
        kept_ = 0;
    }

    struct Block {
        void *ptr;
        cudaStream_t stream;
        bool busy;
        unsigned long long since;
    };
    std::multimap<size_t, Block> free_;
    std::unordered_map<void *, size_t> size_;  // every block taken from CUDA and not given back to it
    size_t kept_ = 0;
    unsigned long long clock_ = 0;
    std::mutex lock_;

    // sizes with three bits of mantissa, so that similar requests share blocks
    static size_t rounded(size_t n)
    {
        if (n <= 4096) return 4096;
        size_t step = 512;
        while (step * 16 < n) step *= 2;
        return (n + step - 1) / step * step;
    }
};

// The pool and stream that pool_alloc / pool_free use on this thread while a PoolScope lives; without one they are cudaMalloc /
// cudaFree.
struct PoolScope {
    DevicePool &pool;
    const cudaStream_t stream;
    PoolScope *const before;
    PoolScope(DevicePool &p, cudaStream_t s) : pool(p), stream(s), before(current()) { current() = this; }
    ~PoolScope() { current() = before; }
    PoolScope(const PoolScope &) = delete;
    PoolScope &operator=(const PoolScope &) = delete;
    static PoolScope *&current();
};
cudaError_t pool_alloc(void **ptr, size_t bytes);
void pool_free(void *ptr);  // after the last use on the call's stream has been enqueued

template <class T>
cudaError_t pool_alloc(T **ptr, size_t count)
{
    return pool_alloc(reinterpret_cast<void **>(ptr), sizeof(T) * (count ? count : 1));
}

}  // namespace sddmm
