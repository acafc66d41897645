// The handle's memory pool (csrc/pool.hpp) over a fake of the CUDA calls it makes.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "pool.hpp"

static std::set<void *> live;
static std::set<cudaStream_t> waited;
static bool stream_fails = false;

extern "C" cudaError_t cudaMalloc(void **p, size_t n)
{
    *p = std::malloc(n);
    live.insert(*p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void *p)
{
    live.erase(p);
    std::free(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    if (stream_fails) return cudaErrorLaunchFailure;
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
        pool.stream = A;
        pool.alloc(&a, 1 << 20);
        pool.free(a, true);  // work on A may still use it
        pool.stream = B;
        pool.alloc(&b, 1 << 20);
        check(b != a, "a block that work on another stream may use is not handed out");
        pool.wait(B);
        pool.alloc(&c, 1 << 20);
        check(c != a, "nor after a wait for some other stream");
        pool.free(c, false);
        stream_fails = true;
        check(pool.wait(A) != cudaSuccess, "a failed wait is reported");
        stream_fails = false;
        pool.stream = A;
        void *d = nullptr;
        pool.alloc(&d, 1 << 20);
        check(d == a || d == c, "the same stream takes it at once");
        pool.free(d, true);
        pool.stream = B;
        waited.clear();
        check(pool.wait(A) == cudaSuccess && waited.count(A) == 1, "wait() waits");
        void *e = nullptr, *f = nullptr;
        pool.alloc(&e, 1 << 20);
        pool.alloc(&f, 1 << 20);
        check((e == a && f == c) || (e == c && f == a), "after the wait any stream takes it");
        pool.free(b, false);
        pool.free(e, false);
        pool.free(f, false);
    }
    check(live.empty(), "everything goes back to CUDA with the pool");
    return failures;
}
