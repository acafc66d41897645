// The handle's memory pool (csrc/pool.hpp) over a fake of the CUDA calls it makes.
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "pool.hpp"

static std::mutex fake;
static std::set<void *> live;
static std::set<cudaStream_t> waited;
static bool stream_fails = false;

extern "C" cudaError_t cudaMalloc(void **p, size_t n)
{
    std::lock_guard<std::mutex> hold(fake);
    *p = std::malloc(n);
    live.insert(*p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::mutex> hold(fake);
    live.erase(p);
    std::free(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    if (stream_fails) return cudaErrorLaunchFailure;
    std::lock_guard<std::mutex> hold(fake);
    waited.insert(s);
    return cudaSuccess;
}

using sddmm::DevicePool;

static int failures = 0;
static void check(bool holds, const char *what)
{
    printf("%s: %s\n", holds ? "ok" : "FAILED", what);
    failures += !holds;
}

int main()
{
    const cudaStream_t A = (cudaStream_t)0x10, B = (cudaStream_t)0x20;
    {
        DevicePool pool;
        void *a = nullptr, *b = nullptr, *c = nullptr;
        pool.alloc(&a, 1 << 20, A);
        pool.free(a, A, true);  // work on A may still use it
        pool.alloc(&b, 1 << 20, B);
        check(b != a, "a block that work on another stream may use is not handed out");
        pool.wait(B);
        pool.alloc(&c, 1 << 20, B);
        check(c != a, "nor after a wait for some other stream");
        pool.free(c, B, false);
        stream_fails = true;
        check(pool.wait(A) != cudaSuccess, "a failed wait is reported");
        stream_fails = false;
        void *d = nullptr;
        pool.alloc(&d, 1 << 20, A);
        check(d == a || d == c, "the same stream takes it at once");
        pool.free(d, A, true);
        waited.clear();
        check(pool.wait(A) == cudaSuccess && waited.count(A) == 1, "wait() waits");
        void *e = nullptr, *f = nullptr;
        pool.alloc(&e, 1 << 20, B);
        pool.alloc(&f, 1 << 20, B);
        check((e == a && f == c) || (e == c && f == a), "after the wait any stream takes it");
        pool.free(b, B, false);
        pool.free(e, B, false);
        pool.free(f, B, false);
    }
    check(live.empty(), "everything goes back to CUDA with the pool");
    {
        // a block is never in two hands: every thread writes its number all over its blocks and finds it again
        DevicePool pool;
        std::vector<std::thread> threads;
        std::vector<int> wrong(4, 0);
        for (int t = 0; t < 4; ++t)
            threads.emplace_back([&, t] {
                const cudaStream_t s = (cudaStream_t)(size_t)(0x100 * (t + 1));
                for (int i = 0; i < 3000; ++i) {
                    void *p = nullptr;
                    const size_t n = 4096 + 512 * ((i * 7 + t) % 40);
                    pool.alloc(&p, n, s);
                    for (size_t k = 0; k < n; k += 64) static_cast<volatile unsigned char *>(p)[k] = (unsigned char)t;
                    for (size_t k = 0; k < n; k += 64) wrong[t] += static_cast<volatile unsigned char *>(p)[k] != (unsigned char)t;
                    pool.free(p, s, i % 3 != 0);
                    if (i % 50 == 0) pool.wait(s);
                    if (i % 997 == 0) pool.release();
                }
            });
        for (std::thread &t : threads) t.join();
        int sum = 0;
        for (int w : wrong) sum += w;
        check(sum == 0, "threads share the pool");
        pool.release();
        check(live.empty(), "release() gives everything back");
    }
    return failures;
}
