// C ABI of the engine: handle, plan (GPU binning pass), execute.
// Replaces the host driver sddmm_GPU of the reference (HiPC18/src/sddmm.cu:32-151):
// device memory for the pattern is owned by a reusable plan instead of being
// allocated and freed per call, errors come back as status codes instead of
// assert(), and an execute with device operands is one kernel launch (two where S
// has dense cells and a remainder).
#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <algorithm>
#include <string>
#include <vector>

#include "binning.cuh"
#include "common.cuh"
#include "gather_index.hpp"
#include "sddmm_b200.h"

using namespace sddmm;

#include "engine_internal.hpp"

namespace {

int fail_cuda(sddmm_handle_s *h, cudaError_t e, const char *what)
{
    if (h) {
        h->last_error = std::string(what) + ": " + cudaGetErrorString(e);
    }
    (void)cudaGetLastError();  // clear the sticky-free error state
    return e == cudaErrorMemoryAllocation ? SDDMM_OUT_OF_MEMORY : SDDMM_CUDA_ERROR;
}

#define CUDA_TRY(h, expr)                                   \
    do {                                                    \
        cudaError_t _e = (expr);                            \
        if (_e != cudaSuccess) return fail_cuda((h), _e, #expr); \
    } while (0)

// A kernel launch: counted per handle (sddmm_kernel_launches).
#define LAUNCH_TRY(h, expr)   \
    do {                      \
        CUDA_TRY(h, expr);    \
        ++(h)->n_launches;    \
    } while (0)

bool is_device_ptr(const void *p)
{
    if (!p) return false;
    cudaPointerAttributes a;
    cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Device-side address of a page-locked host allocation that is mapped into the
// device's address space, or null (pageable memory, device memory, unknown).
const float *mapped_host_ptr(const float *p, unsigned align = 16)
{
    if (!p) return nullptr;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer) return nullptr;
    if (((uintptr_t)a.devicePointer & (align - 1)) != 0) return nullptr;  // the row upload moves 16-byte vectors
    return static_cast<const float *>(a.devicePointer);
}

// Behind SDDMM_PLAN_SKIP_VALIDATION: what works on whole rows has no row pointer to go by.
int needs_sorted(sddmm_handle_s *h)
{
    h->last_error = "the plan's nonzeros are not sorted by row";
    return SDDMM_UNSORTED_INPUT;
}

int check_k(int K)
{
    if (K <= 0 || (K % 4) != 0 || K > SDDMM_MAX_K) return SDDMM_K_UNSUPPORTED;
    return SDDMM_OK;
}

template <class T>
cudaError_t dev_alloc(sddmm_plan_s *p, T **ptr, size_t count)
{
    size_t bytes = sizeof(T) * (count ? count : 1);
    cudaError_t e = pool_alloc((void **)ptr, bytes);
    if (e == cudaSuccess) p->device_bytes += (int64_t)bytes;
    return e;
}

// Device copies that live for one call.
struct CallTmp {
    void *p[6] = {};
    ~CallTmp() { for (void *q : p) pool_free(q); }
};

// What destroying a plan has to wait for: everything enqueued since the last wait, on whatever stream.
void mark_pending(sddmm_plan_s *p, bool async, cudaStream_t s)
{
    p->pending = true;
    if (!async) return;
    if (p->async_pending && p->async_stream != s) p->async_mixed = true;
    p->async_pending = true;
    p->async_stream = s;
}
void waited_for(sddmm_plan_s *p, cudaStream_t s)
{
    if (p->async_mixed || (p->async_pending && p->async_stream != s)) return;
    p->pending = p->async_pending = p->setup_unwaited = false;
}

// Gives the plan's memory back to the handle's pool.  Work that was enqueued and not waited for may still use it: wait
// for the device then, as cudaFree would.
void free_plan_memory(sddmm_plan_s *p)
{
    sddmm_handle_s *h = p->h;
    PoolScope scope(h->pool, h->stream);
    if (p->pending) cudaDeviceSynchronize();
    if (p->owns_rows) pool_free(p->d_rows);
    if (p->owns_cols) pool_free(p->d_cols);
    for (void *q : {(void *)p->d_rows_t, (void *)p->d_cols_t, (void *)p->d_perm, (void *)p->d_row_ptr, (void *)p->d_items, (void *)p->d_item_rows,
                    (void *)p->d_cols_hint, (void *)p->d_col_used, (void *)p->d_used_rows, (void *)p->d_used_cols, (void *)p->d_spmm_scratch,
                    (void *)p->d_Wt, (void *)p->d_Ht, (void *)p->d_W, (void *)p->d_H, (void *)p->d_S, (void *)p->d_P})
        pool_free(q);
    p->dense.release();
}

// Streams and events of the host-operand pipeline, created on first use.
cudaError_t ensure_pipeline(sddmm_handle_s *h)
{
    if (h->pipe_joined) return cudaSuccess;
    cudaError_t e = cudaStreamCreateWithFlags(&h->pipe_compute, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->pipe_download, cudaStreamNonBlocking);
    for (int i = 0; i < SDDMM_PIPE_MAX_CHUNKS && e == cudaSuccess; ++i) {
        e = cudaEventCreateWithFlags(&h->pipe_uploaded[i], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreate(&h->pipe_started[i]);
        if (e == cudaSuccess) e = cudaEventCreate(&h->pipe_computed[i]);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&h->pipe_joined, cudaEventDisableTiming);
    return e;
}

// ---- kernel time of synchronous calls (sddmm_last_kernel_ms) ----

// Brings the last call's kernel time into p->last_ms.
cudaError_t resolve_ms(sddmm_plan_s *p)
{
    sddmm_handle_s *h = p->h;
    cudaError_t e = cudaSuccess;
    if (p->ms_state == sddmm_plan_s::MS_IN_EVENTS) {
        e = cudaEventElapsedTime(&p->last_ms, h->ev_begin[p->ev_pair], h->ev_end[p->ev_pair]);
    } else if (p->ms_state == sddmm_plan_s::MS_IN_PIPE) {
        // kernel time only: the chunks' kernels, not the waits for uploads between them
        p->last_ms = 0.f;
        for (int i = 0; i < p->n_pipe && e == cudaSuccess; i += p->pipe_step) {
            float ms = 0.f;
            e = cudaEventElapsedTime(&ms, h->pipe_started[i], h->pipe_computed[i]);
            p->last_ms += ms;
        }
    } else if (p->ms_state == sddmm_plan_s::MS_IN_CLOCK) {
        unsigned long long t[2] = {0, 0};
        e = cudaMemcpyAsync(t, h->d_clocks + 2 * p->clock, sizeof(t), cudaMemcpyDeviceToHost, h->own_stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->own_stream);
        p->last_ms = t[1] > t[0] ? (float)((double)(t[1] - t[0]) * 1e-6) : 0.f;
    }
    p->ms_state = sddmm_plan_s::MS_KNOWN;
    return e;
}

// Times the kernels of one call: by the kernel's own clock when the call is one launch of a kernel that has one
// (clock() is then non-null and is passed to it), else by an event pair.  Nothing for an asynchronous call.
struct CallTimer {
    sddmm_plan_s *p;
    bool async;
    unsigned long long *clk = nullptr;
    int pair = -1;
    CallTimer(sddmm_plan_s *plan, bool is_async) : p(plan), async(is_async)
    {
        p->last_ms = -1.f;
        p->ms_state = sddmm_plan_s::MS_KNOWN;
    }
    cudaError_t begin(bool kernel_has_clock, cudaStream_t s)
    {
        if (async) return cudaSuccess;
        sddmm_handle_s *h = p->h;
        std::lock_guard<std::mutex> hold(h->owners);
        if (kernel_has_clock && p->clock < 0 && !h->free_clocks.empty()) {
            p->clock = h->free_clocks.back();
            h->free_clocks.pop_back();
        }
        if (kernel_has_clock && p->clock >= 0) {
            clk = h->d_clocks + 2 * p->clock;
            return cudaSuccess;
        }
        pair = h->next_pair;
        h->next_pair = (pair + 1) % SDDMM_EVENT_PAIRS;
        sddmm_plan_s *before = h->ev_owner[pair];
        if (before && before != p && before->ms_state == sddmm_plan_s::MS_IN_EVENTS && before->ev_pair == pair) {
            cudaError_t e = resolve_ms(before);
            if (e != cudaSuccess) return e;
        }
        h->ev_owner[pair] = p;
        return cudaEventRecord(h->ev_begin[pair], s);
    }
    cudaError_t end(cudaStream_t s) { return pair >= 0 ? cudaEventRecord(p->h->ev_end[pair], s) : cudaSuccess; }
    // after the synchronisation
    void done()
    {
        p->ms_state = clk ? sddmm_plan_s::MS_IN_CLOCK : sddmm_plan_s::MS_IN_EVENTS;
        p->ev_pair = pair;
    }
};

// After a synchronising point: turn the device status word into a status code.
int check_device_status(sddmm_handle_s *h)
{
    volatile int *status = h->h_status;
    if (*status != DEV_OK) {
        h->last_error = "a bounded device-side wait (mbarrier) gave up";
        *status = DEV_OK;
        return SDDMM_DEVICE_TIMEOUT;
    }
    return SDDMM_OK;
}

// Plan data that is built when a call first needs it.  It is built on the handle's own stream, whose pattern is complete
// since planning, and waited for: calls of the plan on any stream find it complete.  The calling thread may be capturing a
// stream meanwhile; allocating and waiting for another stream are allowed then in the relaxed mode only.
template <class Fn>
cudaError_t build_now(sddmm_handle_s *h, Fn build)
{
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    {
        PoolScope scope(h->pool, h->own_stream);
        e = build(h->own_stream);
        const cudaError_t w = h->pool.wait(h->own_stream);  // after an error too: its temporaries have gone back to the pool
        if (e == cudaSuccess) e = w;
    }
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    return e;
}

// Row pointer over all rows (empty rows included).
cudaError_t build_plan_row_ptr(sddmm_plan_s *p, cudaStream_t s)
{
    int64_t *row_ptr = nullptr;
    cudaError_t e = dev_alloc(p, &row_ptr, (size_t)p->M + 1);
    if (e != cudaSuccess) return e;
    e = build_row_ptr(p->d_rows, p->nnz, p->M, row_ptr, s);
    if (e == cudaSuccess) p->d_row_ptr = row_ptr;
    else pool_free(row_ptr);
    return e;
}
// Set-up that a call enqueued in front of itself, and that nothing has waited for since, has to be complete for another call.
cudaError_t wait_for_setup(sddmm_plan_s *p)
{
    if (!p->setup_unwaited) return cudaSuccess;
    const cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) p->setup_unwaited = false;
    return e;
}
cudaError_t ensure_row_ptr(sddmm_plan_s *p)
{
    if (p->d_row_ptr) return wait_for_setup(p);
    return build_now(p->h, [&](cudaStream_t s) { return build_plan_row_ptr(p, s); });
}

// The rows of W (0) or H (1) that are read at all.
cudaError_t ensure_used_rows(sddmm_plan_s *p)
{
    if (p->d_used_rows || p->nnz == 0) return cudaSuccess;
    cudaError_t e = ensure_row_ptr(p);
    if (e != cudaSuccess) return e;
    e = build_now(p->h, [&](cudaStream_t s) { return build_used_row_list(p->d_row_ptr, p->M, &p->d_used_rows, &p->n_used_rows, s); });
    p->device_bytes += (int64_t)sizeof(int32_t) * p->n_used_rows;
    return e;
}
cudaError_t ensure_used_cols(sddmm_plan_s *p)
{
    if (p->d_used_cols || p->nnz == 0) return cudaSuccess;
    const cudaError_t e = build_now(p->h, [&](cudaStream_t s) { return build_used_col_list(p->d_cols, p->nnz, p->N, &p->d_used_cols, &p->n_used_cols, s); });
    p->device_bytes += (int64_t)sizeof(int32_t) * p->n_used_cols;
    return e;
}

// What the upload of used rows looks at: the row pointer and a mark per column.  Enqueued in front of the call, which waits
// for all of it.
cudaError_t ensure_upload_marks(sddmm_plan_s *p, bool rows, bool cols, cudaStream_t s)
{
    cudaError_t e = wait_for_setup(p);
    rows = rows && !p->d_row_ptr;
    cols = cols && !p->d_col_used;
    if (e != cudaSuccess || (!rows && !cols)) return e;
    p->setup_unwaited = true;
    mark_pending(p, true, s);
    if (rows) e = build_plan_row_ptr(p, s);
    if (e != cudaSuccess || !cols) return e;
    unsigned char *used = nullptr;
    e = dev_alloc(p, &used, (size_t)p->N);
    if (e != cudaSuccess) return e;
    e = mark_used_cols(p->d_cols, p->nnz, p->N, used, s);
    if (e == cudaSuccess) p->d_col_used = used;
    else pool_free(used);
    return e;
}

// Host-operand pipeline (sddmm_execute with W in host memory): S is cut into chunks of consecutive nonzeros, about 32 MB
// of W rows each.  Rows are sorted, so a chunk needs one contiguous block of W rows, and W rows between two chunks
// that no nonzero touches are never uploaded.  Here: the first and last row of every chunk.
cudaError_t ensure_pipe(sddmm_plan_s *p)
{
    if (p->pipe_ready) return cudaSuccess;
    sddmm_handle_s *h = p->h;
    const int chunks = p->n_pipe;
    PickAt at{};
    for (int i = 0; i < chunks; ++i) {
        p->pipe_nnz[i] = (p->nnz * i / chunks) & ~(int64_t)31;
        at.v[2 * i] = p->pipe_nnz[i];
        if (i > 0) at.v[2 * i - 1] = p->pipe_nnz[i] - 1;
    }
    p->pipe_nnz[chunks] = p->nnz;
    at.v[2 * chunks - 1] = p->nnz - 1;
    // on the call's stream, which waits anyway: work on one stream more slows the call's overlap of upload, kernel and download
    // (1 M vertices, K = 128: 13.17 -> 13.36 ms)
    cudaError_t e = pick_values(p->d_rows, at, 2 * chunks, h->d_words, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return e;
    int64_t next_row = 0;  // first row of W no earlier chunk uploads
    for (int i = 0; i < chunks; ++i) {
        const int64_t first = (int64_t)h->h_words[2 * i], r1 = (int64_t)h->h_words[2 * i + 1] + 1;
        p->pipe_w_begin[i] = first > next_row ? first : next_row;
        p->pipe_w_end[i] = r1 > p->pipe_w_begin[i] ? r1 : p->pipe_w_begin[i];
        if (r1 > next_row) next_row = r1;
    }
    p->pipe_ready = true;
    return cudaSuccess;
}

// Work items of the row-panel kernel, built when the kernel is forced or their number is asked for.
cudaError_t ensure_items(sddmm_plan_s *p)
{
    if (p->n_items >= 0) return cudaSuccess;
    const bool tiled = p->d_perm != nullptr;
    int64_t n = 0;
    const cudaError_t e = build_now(p->h, [&](cudaStream_t s) {
        return build_work_items(tiled ? p->d_rows_t : p->d_rows, tiled ? p->d_cols_t : p->d_cols, p->nnz, p->cfg.panel_rows, p->col_tile,
                                p->cfg.item_nnz, &p->d_items, &n, &p->d_item_rows, &p->n_item_rows, s);
    });
    if (e != cudaSuccess) return e;
    p->n_items = n;
    p->device_bytes += (int64_t)(sizeof(WorkItem) * (size_t)n + sizeof(int32_t) * (size_t)p->n_item_rows);
    return cudaSuccess;
}

// Hub-column marks for the ring kernel, when H is too large to live in L2 as a whole.
cudaError_t build_hints(sddmm_plan_s *p, cudaStream_t s)
{
    const int64_t row_bytes = (int64_t)p->K * 4;
    if (p->nnz > 0 && ring_supports(p->K) && p->hub_budget > 0 && p->N * row_bytes > p->hub_budget) {
        int32_t *marked = nullptr;
        cudaError_t e = dev_alloc(p, &marked, (size_t)p->nnz);
        if (e != cudaSuccess) return e;
        int thr = 0;
        e = build_hub_column_hints(p->d_perm ? p->d_cols_t : p->d_cols, p->nnz, p->N, row_bytes, p->hub_budget, marked, &p->n_hub_cols, &thr, s);
        if (e != cudaSuccess) {
            pool_free(marked);
            return e;
        }
        p->d_cols_hint = marked;
    }
    p->hints_built = true;
    return cudaSuccess;
}
cudaError_t ensure_hints(sddmm_plan_s *p)
{
    if (p->hints_built) return cudaSuccess;
    return build_now(p->h, [&](cudaStream_t s) { return build_hints(p, s); });
}

}  // namespace

namespace sddmm {

bool rows_on_ring(const sddmm_plan_s *p, bool force_ring, bool permuted)
{
    return ring_supports(p->K) && (force_ring || (ring_preferred(p->N, p->K) && (permuted || ring_few(p->nnz, p->K * 4))));
}

cudaError_t launch_rows(sddmm_plan_s *p, const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                        const float *W, const float *H, float *P, int64_t first, int64_t count, bool force_ring,
                        unsigned long long *clock, cudaStream_t stream, bool beside, bool awaited)
{
    sddmm_handle_s *h = p->h;
    p->pending = true;  // (sddmm_execute clears it again when it waits)
    // the split of the whole matrix: a chunk of it is summed in the order that the whole would be
    const int64_t whole = rows == p->dense.rows_s ? p->dense.n_sparse : p->nnz;
    GatherPasses passes = gather_passes(whole, p->N, p->K, p->d_perm && !perm, sval, P);
    passes.awaited = awaited;
    rows += first;
    if (perm) {
        perm += first;
    } else {
        P += first;
        if (sval) sval += first;
    }
    if (rows_on_ring(p, force_ring, perm != nullptr)) {
        // the marks are in the plan's processing order: not for the dense-cell remainder
        const bool hinted = p->d_cols_hint && cols == (p->d_perm ? p->d_cols_t : p->d_cols);
        return launch_ring(rows, (hinted ? p->d_cols_hint : cols) + first, perm, sval, W, H, P, count, p->K, hinted, h->sm_count,
                           h->work_counter(), h->d_status, stream);
    }
    if (!perm) h->n_launches += passes.n - 1;
    return launch_gather(rows, cols + first, perm, sval, W, H, P, count, p->K, passes, h->sm_count, clock, stream, beside);
}

}  // namespace sddmm

extern "C" {

const char *sddmm_status_string(int s)
{
    switch (s) {
    case SDDMM_OK: return "ok";
    case SDDMM_INVALID_ARG: return "invalid argument";
    case SDDMM_UNSORTED_INPUT: return "input is not sorted by row";
    case SDDMM_INDEX_OUT_OF_RANGE: return "row or column index out of range";
    case SDDMM_K_UNSUPPORTED: return "K must be a positive multiple of 4 not larger than SDDMM_MAX_K";
    case SDDMM_CUDA_ERROR: return "CUDA error";
    case SDDMM_NCCL_ERROR: return "NCCL error";
    case SDDMM_OUT_OF_MEMORY: return "out of device memory";
    case SDDMM_DEVICE_TIMEOUT: return "device-side wait timed out";
    case SDDMM_IO_ERROR: return "I/O error";
    case SDDMM_PARSE_ERROR: return "Matrix Market parse error";
    case SDDMM_NO_DEVICE: return "no usable CUDA device (this engine has no CPU fallback)";
    default: return "unknown status";
    }
}

int sddmm_create(sddmm_handle_t *out, int device)
{
    if (!out) return SDDMM_INVALID_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        return SDDMM_NO_DEVICE;
    }
    if (device < 0 || device >= n) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = new (std::nothrow) sddmm_handle_s;
    if (!h) return SDDMM_OUT_OF_MEMORY;
    h->device = device;
    cudaError_t e = cudaSetDevice(device);
    cudaDeviceProp prop;
    if (e == cudaSuccess) e = cudaGetDeviceProperties(&prop, device);
    if (e == cudaSuccess && prop.major < 10) {
        delete h;
        return SDDMM_NO_DEVICE;  // kernels are built for sm_100a only
    }
    if (e == cudaSuccess) {
        h->sm_count = prop.multiProcessorCount;
        h->smem_optin = prop.sharedMemPerBlockOptin;
        e = cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking);
    }
    for (int i = 0; i < SDDMM_EVENT_PAIRS && e == cudaSuccess; ++i) {
        e = cudaEventCreate(&h->ev_begin[i]);
        if (e == cudaSuccess) e = cudaEventCreate(&h->ev_end[i]);
    }
    if (e == cudaSuccess) e = cudaMalloc((void **)&h->d_clocks, 2 * sizeof(unsigned long long) * N_KERNEL_CLOCKS);
    if (e == cudaSuccess) e = cudaMemset(h->d_clocks, 0, 2 * sizeof(unsigned long long) * N_KERNEL_CLOCKS);
    if (e == cudaSuccess) e = cudaMalloc((void **)&h->d_work_counters, sizeof(unsigned long long) * SDDMM_WORK_COUNTERS);
    // mapped host memory: the status word, and at 64 bytes the words that plan-time kernels answer in
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&h->h_status, 64 + sizeof(unsigned long long) * PICK_MAX, cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&h->d_status, h->h_status, 0);
    if (e == cudaSuccess) e = cudaMalloc((void **)&h->d_plan_words, sizeof(unsigned long long) * PLAN_WORDS);
    if (e == cudaSuccess) e = init_plan_words(h->d_plan_words);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = cudaEventCreate(&h->ev_plan[i]);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        sddmm_destroy(h);
        return SDDMM_CUDA_ERROR;
    }
    *h->h_status = DEV_OK;
    h->h_words = reinterpret_cast<volatile unsigned long long *>(h->h_status + 16);
    h->d_words = reinterpret_cast<unsigned long long *>(h->d_status + 16);
    h->free_clocks.reserve(N_KERNEL_CLOCKS);
    for (int i = N_KERNEL_CLOCKS - 1; i >= 0; --i) h->free_clocks.push_back(i);
    h->stream = h->own_stream;
    if (const char *env = std::getenv("SDDMM_DENSE_TENSOR")) {
        const int v = std::atoi(env);
        if (v >= 0 && v <= 2) h->dense_mode = v;
    }
    if (const char *env = std::getenv("SDDMM_PIPELINE")) h->pipeline = std::atoi(env) != 0;
    if (const char *env = std::getenv("SDDMM_SPARSE_UPLOAD")) h->sparse_upload = std::atoi(env) != 0;
    h->upload_ctas = h->sm_count / 2 > 0 ? h->sm_count / 2 : 1;
    if (const char *env = std::getenv("SDDMM_UPLOAD_CTAS")) {
        const int v = std::atoi(env);
        if (v > 0 && v <= 4096) h->upload_ctas = v;
    }
    *out = h;
    return SDDMM_OK;
}

int sddmm_destroy(sddmm_handle_t h)
{
    if (!h) return SDDMM_OK;
    cudaSetDevice(h->device);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    for (cudaEvent_t e : h->ev_begin) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : h->ev_end) if (e) cudaEventDestroy(e);
    if (h->d_clocks) cudaFree(h->d_clocks);
    if (h->d_plan_words) cudaFree(h->d_plan_words);
    for (cudaEvent_t e : h->ev_plan) if (e) cudaEventDestroy(e);
    h->pool.release();
    if (h->d_work_counters) cudaFree(h->d_work_counters);
    if (h->h_status) cudaFreeHost(h->h_status);
    if (h->pipe_compute) cudaStreamDestroy(h->pipe_compute);
    if (h->pipe_download) cudaStreamDestroy(h->pipe_download);
    for (cudaEvent_t e : h->pipe_uploaded) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : h->pipe_started) if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : h->pipe_computed) if (e) cudaEventDestroy(e);
    if (h->pipe_joined) cudaEventDestroy(h->pipe_joined);
    (void)cudaGetLastError();
    delete h;
    return SDDMM_OK;
}

int sddmm_trim(sddmm_handle_t h)
{
    if (!h) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    h->pool.release();
    return SDDMM_OK;
}

const char *sddmm_last_error(sddmm_handle_t h) { return h ? h->last_error.c_str() : ""; }

int sddmm_set_stream(sddmm_handle_t h, void *cuda_stream)
{
    if (!h) return SDDMM_INVALID_ARG;
    h->stream = cuda_stream ? (cudaStream_t)cuda_stream : h->own_stream;
    return SDDMM_OK;
}

int sddmm_plan_coo(sddmm_handle_t h, int64_t M, int64_t N, int64_t nnz, const int32_t *rows,
                   const int32_t *cols, int K, int panel_rows_hint, int col_tile_hint, uint32_t flags,
                   sddmm_plan_t *out)
{
    if (!h || !out) return SDDMM_INVALID_ARG;
    *out = nullptr;
    if (M < 0 || N < 0 || nnz < 0 || (nnz > 0 && (!rows || !cols))) return SDDMM_INVALID_ARG;
    if (M > INT32_MAX || N > INT32_MAX || nnz >= INT32_MAX) return SDDMM_INVALID_ARG;  // int32 indices, as the reference
    if (nnz > 0 && (M == 0 || N == 0)) return SDDMM_INDEX_OUT_OF_RANGE;
    int st = check_k(K);
    if (st != SDDMM_OK) return st;
    CUDA_TRY(h, cudaSetDevice(h->device));

    sddmm_plan_s *p = new (std::nothrow) sddmm_plan_s;
    if (!p) return SDDMM_OUT_OF_MEMORY;
    p->h = h;
    p->M = M; p->N = N; p->nnz = nnz; p->K = K;
    cudaStream_t s = h->stream;
    PoolScope scope(h->pool, s);

    auto drop = [&](int st) {
        free_plan_memory(p);
        delete p;
        return st;
    };
#define PLAN_TRY(expr)                                                      \
    do {                                                                    \
        cudaError_t _e = (expr);                                            \
        if (_e != cudaSuccess) return drop(fail_cuda(h, _e, #expr));        \
    } while (0)

    const bool dev_idx = (flags & SDDMM_PLAN_DEVICE_INDICES) != 0;
    if (dev_idx) {
        p->d_rows = const_cast<int32_t *>(rows);
        p->owns_rows = false;
        if (((uintptr_t)cols & 15u) == 0) {
            p->d_cols = const_cast<int32_t *>(cols);
            p->owns_cols = false;
        } else {
            // the kernels read column indices with 16-byte vector loads: realign a borrowed array
            PLAN_TRY(dev_alloc(p, &p->d_cols, (size_t)nnz));
            if (nnz > 0) PLAN_TRY(cudaMemcpyAsync(p->d_cols, cols, sizeof(int32_t) * nnz, cudaMemcpyDeviceToDevice, s));
        }
    } else {
        PLAN_TRY(dev_alloc(p, &p->d_rows, (size_t)nnz));
        PLAN_TRY(dev_alloc(p, &p->d_cols, (size_t)nnz));
        if (nnz > 0) {
            PLAN_TRY(cudaMemcpyAsync(p->d_rows, rows, sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, s));
            PLAN_TRY(cudaMemcpyAsync(p->d_cols, cols, sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, s));
        }
    }
    if (nnz > 0) {
        PLAN_TRY(scan_coo(p->d_rows, p->d_cols, nnz, M, N, h->d_plan_words, h->d_words, s));
        PLAN_TRY(h->pool.wait(s));
        const unsigned long long unsorted = h->h_words[0], oob = h->h_words[1];
        if (!(flags & SDDMM_PLAN_SKIP_VALIDATION) && (unsorted != ULLONG_MAX || oob != ULLONG_MAX)) {
            char buf[160];
            snprintf(buf, sizeof(buf), "%s at nonzero %llu", oob != ULLONG_MAX ? "index out of range" : "rows not sorted",
                     oob != ULLONG_MAX ? oob : unsorted);
            h->last_error = buf;
            return drop(oob != ULLONG_MAX ? SDDMM_INDEX_OUT_OF_RANGE : SDDMM_UNSORTED_INPUT);
        }
        p->sorted = unsorted == ULLONG_MAX;
        p->n_nonempty_rows = (int64_t)h->h_words[2];
        p->plan_ms = (float)((double)h->h_words[3] * 1e-6);
    }
    // everything after the first look is timed by events, and only if there is anything
    bool more = false;
    auto begin_more = [&]() -> cudaError_t {
        if (more) return cudaSuccess;
        more = true;
        return cudaEventRecord(h->ev_plan[0], s);
    };

    // column tiles: a hint >= N (or <= 0) means one tile, the identity order
    p->cfg = choose_panel_config(K, panel_rows_hint, h->sm_count, h->smem_optin);
    int64_t ct = (col_tile_hint <= 0 || col_tile_hint >= N) ? (N > 0 ? N : 1) : col_tile_hint;
    p->col_tile = (int)ct;
    p->n_col_tiles = (int)((N + ct - 1) / ct);
    if (p->n_col_tiles < 1) p->n_col_tiles = 1;
    if (p->n_col_tiles > 1 && nnz > 0) {
        PLAN_TRY(begin_more());
        PLAN_TRY(dev_alloc(p, &p->d_perm, (size_t)nnz));
        PLAN_TRY(dev_alloc(p, &p->d_rows_t, (size_t)nnz));
        PLAN_TRY(dev_alloc(p, &p->d_cols_t, (size_t)nnz));
        PLAN_TRY(build_tiled_order(p->d_rows, p->d_cols, nnz, N, p->col_tile, p->d_perm, p->d_rows_t, p->d_cols_t, s));
    }
    // Locally dense matrices (many nonzeros per row): cells that are at least a
    // quarter full go to the dense-cell kernel, if they hold half of S or more
    // (below that the second launch and the permuted remainder cost more than they save).
    // From 2^26 multiplications on.  The line is a compromise between the call and the plan, to which the classification adds
    // 300 us.  Up to 2^25.2 the cells save a call nothing; from there to the line 1 to 6 us of 14 to 20, which a mask pays that
    // is kept for more than some fifty calls; above it 6 us and more.  (us per call, band + global masks, gather / cells:
    // 2^24.3 multiplications: 0.33 M nonzeros, K = 64 10.4 / 10.7;  2^25.1: 0.57 M, K = 64 12.4 / 11.6, 1.1 M, K = 32 14.5 / 13.9,
    // 0.14 M, K = 256 12.5 / 16.4;  2^25.3: 0.33 M, K = 128 15.5 / 13.0, 0.67 M, K = 64 14.4 / 12.4;  2^25.7: 0.57 M, K = 96 16.5 /
    // 12.4, 1.7 M, K = 32 18.6 / 14.3;  2^25.9: 0.67 M, K = 96 20.4 / 14.4;  2^26.1: 0.57 M, K = 128 22.4 / 13.3, 2.2 M, K = 32
    // 22.7 / 16.5, 0.14 M, K = 512 22.7 / 22.7;  planned, called and closed: 0.36 M, K = 64 42 / 365.)
    // SDDMM_DENSE_CELLS=0 switches the classification off, 1 takes it at every size: the choice for a mask of that size that is kept.
    {
        const char *env = std::getenv("SDDMM_DENSE_CELLS");
        const bool enabled = !(env && std::atoi(env) == 0), always = env && std::atoi(env) == 1;
        const bool candidate = enabled && p->sorted && p->n_col_tiles == 1 && p->n_nonempty_rows > 0 && nnz / p->n_nonempty_rows >= 32;
        if (candidate && (always || nnz * K >= (1ll << 26))) {
            PLAN_TRY(begin_more());
            PLAN_TRY(build_plan_row_ptr(p, s));
            PLAN_TRY(build_dense_cells(p->d_rows, p->d_cols, p->d_row_ptr, nnz, M, N, DENSE_MIN_FILL, DENSE_MIN_SHARE, &p->dense, s));
            if (p->dense.n_cells > 0)
                p->device_bytes += (int64_t)((sizeof(DenseCell) + 20 * DENSE_CELL_ROWS) * p->dense.n_cells + sizeof(DenseUnit) * p->dense.n_units +
                                             sizeof(int32_t) * DENSE_CELL_ROWS * DENSE_CELL_COLS * p->dense.n_table_cells + 12 * p->dense.n_sparse);
        }
    }
    // Hub-column marks are for the ring kernel: now if the order is permuted and it will run by default, else if it is forced.
    // SDDMM_L2_HUB_MB overrides the share of L2 set aside for hub rows (0 = off).
    {
        int64_t budget_mb = 64;  // best of a 16..128 MB sweep on the scale-22 R-MAT matrix at K = 256
        if (const char *env = std::getenv("SDDMM_L2_HUB_MB")) budget_mb = std::atoll(env);
        p->hub_budget = budget_mb > 0 ? budget_mb * (1ll << 20) : 0;
        if (p->d_perm && ring_preferred(N, K)) {
            PLAN_TRY(begin_more());
            PLAN_TRY(build_hints(p, s));
        }
    }
    // chunks of the host-operand pipeline; what they need is built by the first call with host operands
    if (p->sorted && p->n_col_tiles == 1 && p->dense.n_cells == 0 && nnz >= (1 << 17)) {
        const int64_t chunks = std::min<int64_t>((int64_t)sizeof(float) * M * K / (32ll << 20), SDDMM_PIPE_MAX_CHUNKS);
        if (chunks >= 2) p->n_pipe = (int)chunks;
    }
    if (more) {
        PLAN_TRY(cudaEventRecord(h->ev_plan[1], s));
        PLAN_TRY(h->pool.wait(s));
        float ms = 0.f;
        PLAN_TRY(cudaEventElapsedTime(&ms, h->ev_plan[0], h->ev_plan[1]));
        p->plan_ms += ms;
    }
#undef PLAN_TRY
    *out = p;
    return SDDMM_OK;
}

int sddmm_destroy_plan(sddmm_plan_t p)
{
    if (!p) return SDDMM_OK;
    cudaSetDevice(p->h->device);
    free_plan_memory(p);
    if (p->spmm_done) cudaEventDestroy(p->spmm_done);
    {
        std::lock_guard<std::mutex> hold(p->h->owners);
        if (p->clock >= 0) p->h->free_clocks.push_back(p->clock);
        for (sddmm_plan_s *&owner : p->h->ev_owner) if (owner == p) owner = nullptr;
        if (p->h->pipe_owner == p) p->h->pipe_owner = nullptr;
    }
    (void)cudaGetLastError();
    delete p;
    return SDDMM_OK;
}

int sddmm_execute(sddmm_plan_t p, const float *W, const float *H, const float *Sval, float *P, uint32_t flags)
{
    if (!p) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    if (p->nnz == 0) { p->last_ms = 0.f; p->ms_state = sddmm_plan_s::MS_KNOWN; return SDDMM_OK; }
    if (!W || !H || !P) return SDDMM_INVALID_ARG;
    const bool use_gather = (flags & SDDMM_FLAG_KERNEL_GATHER) != 0;
    const bool tiled_out = (flags & SDDMM_FLAG_TILED_ORDER) != 0;
    const uint32_t forced = flags & (SDDMM_FLAG_KERNEL_GATHER | SDDMM_FLAG_KERNEL_PANEL | SDDMM_FLAG_KERNEL_RING);
    if (forced & (forced - 1)) return SDDMM_INVALID_ARG;  // at most one kernel may be forced
    const bool use_ring = (flags & SDDMM_FLAG_KERNEL_RING) != 0, use_panel = (flags & SDDMM_FLAG_KERNEL_PANEL) != 0;
    if (use_ring && !rows_path_supports(p->K)) return SDDMM_K_UNSUPPORTED;
    if (use_gather && tiled_out && p->d_perm) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    PoolScope scope(h->pool, s);

    const bool w_dev = is_device_ptr(W), h_dev = is_device_ptr(H), p_dev = is_device_ptr(P);
    const bool s_dev = Sval ? is_device_ptr(Sval) : true;
    const bool all_dev = w_dev && h_dev && p_dev && s_dev;
    const bool async = (flags & SDDMM_FLAG_ASYNC) != 0;
    if (async && !all_dev) return SDDMM_INVALID_ARG;
    mark_pending(p, async, s);

    if (flags & SDDMM_FLAG_OPERANDS_BF16) {
        // W and H hold bfloat16: rows of 2K bytes, products and sums in fp32.  Opt-in and
        // outside the fp32 tolerance contract; device arrays only, no other layout or kernel flag.
        if (!ring_bf16_supports(p->K)) return SDDMM_K_UNSUPPORTED;
        if (!all_dev || (flags & ~(uint32_t)(SDDMM_FLAG_OPERANDS_BF16 | SDDMM_FLAG_ASYNC | SDDMM_FLAG_KERNEL_RING))) {
            h->last_error = "SDDMM_FLAG_OPERANDS_BF16 takes device arrays and no flag but ASYNC / KERNEL_RING";
            return SDDMM_INVALID_ARG;
        }
        if ((((uintptr_t)W | (uintptr_t)H) & 15u) != 0) {
            h->last_error = "W and H must be 16-byte aligned on the device";
            return SDDMM_INVALID_ARG;
        }
        const bool tiled = p->d_perm != nullptr;
        const int32_t *rows_p = tiled ? p->d_rows_t : p->d_rows, *cols_p = tiled ? p->d_cols_t : p->d_cols;
        const int32_t *perm_p = tiled ? p->d_perm : nullptr;
        // rows of half the bytes: the same line between the two kernels as for fp32 rows of K / 2
        const bool few = !tiled && !(flags & SDDMM_FLAG_KERNEL_RING) && ring_few(p->nnz, p->K * 2);
        const bool gather = gather_bf16_supports(p->K) && !(flags & SDDMM_FLAG_KERNEL_RING) && !(ring_preferred(p->N / 2, p->K) && (tiled || few));
        const int passes = gather && !tiled ? gather_passes_bf16(p->nnz, p->N, p->K, Sval, P).n : 1;
        if (!gather && !few) CUDA_TRY(h, ensure_hints(p));
        p->last_kernel = gather ? "gather (bf16 operands)" : "ring (bf16 operands)";
        p->last_h2d_bytes = p->last_d2h_bytes = 0;
        CallTimer timer(p, async);
        CUDA_TRY(h, timer.begin(gather && passes == 1, s));
        h->n_launches += passes - 1;
        if (gather)
            LAUNCH_TRY(h, launch_gather_bf16(rows_p, cols_p, perm_p, Sval, W, H, P, p->nnz, p->N, p->K, h->sm_count, timer.clk, s));
        else
            LAUNCH_TRY(h, launch_ring_bf16(rows_p, p->d_cols_hint ? p->d_cols_hint : cols_p, perm_p, Sval, W, H, P, p->nnz, p->K,
                                           p->d_cols_hint != nullptr, h->sm_count, h->work_counter(), h->d_status, s));
        CUDA_TRY(h, timer.end(s));
        if (async) return SDDMM_OK;
        CUDA_TRY(h, cudaStreamSynchronize(s));
        waited_for(p, s);
        timer.done();
        return check_device_status(h);
    }
    const float *dW = W, *dH = H, *dS = Sval;
    float *dP = P;
    const size_t wbytes = sizeof(float) * (size_t)p->M * p->K, hbytes = sizeof(float) * (size_t)p->N * p->K;
    const size_t nbytes = sizeof(float) * (size_t)p->nnz;
    const bool w_t = (flags & SDDMM_FLAG_W_TRANSPOSED) != 0, h_t = (flags & SDDMM_FLAG_H_TRANSPOSED) != 0;
    // W in host memory and the row path: upload W (and S) chunk by chunk and let every chunk's kernel and download run
    // behind the later uploads
    const bool pipelined = h->pipeline && p->n_pipe > 0 && !w_dev && !use_gather && !use_panel && !tiled_out && !p->d_perm &&
                           p->dense.n_cells == 0 && !w_t && !h_t;
    if (pipelined) CUDA_TRY(h, ensure_pipe(p));
    // page-locked, mapped host arrays are read by the GPU: one launch for all of them instead of a copy each, and of W and
    // H only the rows that a nonzero touches travel (short rows all do: reads below 128 bytes waste the link)
    const float *W_mapped = h->sparse_upload && p->sorted && !w_dev && !w_t ? mapped_host_ptr(W) : nullptr;
    const float *H_mapped = h->sparse_upload && !h_dev && !h_t ? mapped_host_ptr(H) : nullptr;
    // a large array with nearly all rows used: the copy engine moves whole arrays at 56 GB/s, the kernel rows at 45 to 50
    constexpr size_t LARGE = 4 << 20;
    if (W_mapped && wbytes >= LARGE && p->n_nonempty_rows > p->M * 7 / 8) W_mapped = nullptr;
    if (H_mapped && hbytes >= LARGE) {
        int64_t used = 0;  // counted once per plan
        const int st = sddmm_plan_count_cols(p, &used);
        if (st != SDDMM_OK) return st;
        if (used > p->N * 7 / 8) H_mapped = nullptr;
    }
    const float *S_mapped = h->sparse_upload && Sval && !s_dev ? mapped_host_ptr(Sval) : nullptr;
    const bool used_rows_only = p->K >= 32;
    if (used_rows_only) CUDA_TRY(h, ensure_upload_marks(p, W_mapped != nullptr, H_mapped != nullptr, s));
    UploadRows up_w, up_h;
    up_w.row_bytes = up_h.row_bytes = p->K * (int)sizeof(float);
    const float *up_s = nullptr;
    p->last_h2d_bytes = p->last_d2h_bytes = 0;
    p->last_h2d_used_cols = false;
    // K-major operands (the layout make_HTasH builds, util.h:68-73): brought to the device if need be and
    // transposed there into the plan's row-major staging copy
    if (h_t) {
        const float *src = H;
        if (!h_dev) {
            if (!p->d_Ht) CUDA_TRY(h, dev_alloc(p, &p->d_Ht, (size_t)p->N * p->K));
            CUDA_TRY(h, cudaMemcpyAsync(p->d_Ht, H, hbytes, cudaMemcpyHostToDevice, s));
            p->last_h2d_bytes += (int64_t)hbytes;
            src = p->d_Ht;
        }
        if (!p->d_H) CUDA_TRY(h, dev_alloc(p, &p->d_H, (size_t)p->N * p->K));
        LAUNCH_TRY(h, launch_transpose_operand(src, p->d_H, p->N, p->K, s));
        dH = p->d_H;
    } else if (!h_dev) {
        if (!p->d_H) CUDA_TRY(h, dev_alloc(p, &p->d_H, (size_t)p->N * p->K));
        if (H_mapped) {
            up_h.src = reinterpret_cast<const char *>(H_mapped);
            up_h.dst = reinterpret_cast<char *>(p->d_H);
            up_h.col_used = used_rows_only ? p->d_col_used : nullptr;
            up_h.end = p->N;
            p->last_h2d_used_cols = used_rows_only;
            if (!used_rows_only) p->last_h2d_bytes += (int64_t)hbytes;
        } else {
            CUDA_TRY(h, cudaMemcpyAsync(p->d_H, H, hbytes, cudaMemcpyHostToDevice, s));
            p->last_h2d_bytes += (int64_t)hbytes;
        }
        dH = p->d_H;
    }
    if (w_t) {
        const float *src = W;
        if (!w_dev) {
            if (!p->d_Wt) CUDA_TRY(h, dev_alloc(p, &p->d_Wt, (size_t)p->M * p->K));
            CUDA_TRY(h, cudaMemcpyAsync(p->d_Wt, W, wbytes, cudaMemcpyHostToDevice, s));
            p->last_h2d_bytes += (int64_t)wbytes;
            src = p->d_Wt;
        }
        if (!p->d_W) CUDA_TRY(h, dev_alloc(p, &p->d_W, (size_t)p->M * p->K));
        LAUNCH_TRY(h, launch_transpose_operand(src, p->d_W, p->M, p->K, s));
        dW = p->d_W;
    } else if (!w_dev) {
        if (!p->d_W) CUDA_TRY(h, dev_alloc(p, &p->d_W, (size_t)p->M * p->K));
        if (W_mapped) {
            up_w.src = reinterpret_cast<const char *>(W_mapped);
            up_w.dst = reinterpret_cast<char *>(p->d_W);
            up_w.row_ptr = used_rows_only ? p->d_row_ptr : nullptr;
            up_w.end = p->M;
            p->last_h2d_bytes += used_rows_only ? (int64_t)sizeof(float) * p->n_nonempty_rows * p->K : (int64_t)wbytes;
        } else if (!pipelined) {
            CUDA_TRY(h, cudaMemcpyAsync(p->d_W, W, wbytes, cudaMemcpyHostToDevice, s));
            p->last_h2d_bytes += (int64_t)wbytes;
        }
        dW = p->d_W;
    }
    if (Sval && !s_dev) {
        if (!p->d_S) CUDA_TRY(h, dev_alloc(p, &p->d_S, (size_t)p->nnz));
        if (S_mapped) up_s = S_mapped;
        else if (!pipelined) CUDA_TRY(h, cudaMemcpyAsync(p->d_S, Sval, nbytes, cudaMemcpyHostToDevice, s));
        p->last_h2d_bytes += (int64_t)nbytes;
        dS = p->d_S;
    }
    const bool use_dense = !forced && !tiled_out && p->dense.n_cells > 0;
    // a call that is one gather launch is timed by the kernel itself, everything else by events
    const bool permuted = p->d_perm && !tiled_out;
    const bool one_gather = !use_dense && !use_panel && (use_gather || !rows_on_ring(p, use_ring, permuted)) &&
                            (permuted || use_gather || gather_passes(p->nnz, p->N, p->K, p->d_perm != nullptr, dS, P).n == 1);
    bool p_copy = false;
    bool awaited = !async;  // the kernel for few nonzeros stores in smaller pieces, which counts over PCIe (mapped P, us, before / with it: K = 32, 30,000 nonzeros 18.8 / 20.4, K = 128, 16,777 18.7 / 21.1)
    if (!p_dev) {
        // a small P is written to mapped host memory by the kernel: its 32-byte stores over PCIe cost less than a copy
        float *P_mapped = one_gather && !pipelined && h->sparse_upload && nbytes <= (256 << 10) ? const_cast<float *>(mapped_host_ptr(P, 4)) : nullptr;
        p_copy = !P_mapped;
        awaited &= p_copy;
        if (p_copy && !p->d_P) CUDA_TRY(h, dev_alloc(p, &p->d_P, (size_t)p->nnz));
        dP = P_mapped ? P_mapped : p->d_P;
        p->last_d2h_bytes = (int64_t)nbytes;
    }

    // every kernel moves 16-byte vectors
    if ((((uintptr_t)dW | (uintptr_t)dH) & 15u) != 0) {
        h->last_error = "W and H must be 16-byte aligned on the device";
        return SDDMM_INVALID_ARG;
    }
    if (use_panel) CUDA_TRY(h, ensure_items(p));
    if (use_ring && ring_supports(p->K)) CUDA_TRY(h, ensure_hints(p));
    if (pipelined) {
        p->last_kernel = rows_on_ring(p, use_ring, false) ? "ring (pipelined chunks)" : "gather (pipelined chunks)";
        CUDA_TRY(h, ensure_pipeline(h));
        {
            std::lock_guard<std::mutex> hold(h->owners);
            if (h->pipe_owner && h->pipe_owner != p && h->pipe_owner->ms_state == sddmm_plan_s::MS_IN_PIPE)
                CUDA_TRY(h, resolve_ms(h->pipe_owner));
            h->pipe_owner = p;
        }
        // A copy into pageable memory holds the host until it is done, and with it the next upload: nothing overlaps and chunks
        // only cost, so about 128 MB of W go together (R-MAT, H on the device, W, S and P pageable, ms: 128 MB of W 14.4 -> 14.2,
        // 537 MB 58.6 -> 58.0;  W page-locked, 537 MB: 10.4 -> 10.1).
        p->pipe_step = 1;
        if (!p_dev && !mapped_host_ptr(P, 4)) p->pipe_step = (int)std::max<int64_t>(1, (128ll << 20) * p->n_pipe / (int64_t)wbytes);
        for (int i = 0; i < p->n_pipe; i += p->pipe_step) {
            const int next = std::min(i + p->pipe_step, p->n_pipe);
            const int64_t n0 = p->pipe_nnz[i], cnt = p->pipe_nnz[next] - n0, r0 = p->pipe_w_begin[i], r1 = p->pipe_w_end[next - 1];
            up_w.begin = r0;
            up_w.end = W_mapped ? r1 : r0;
            if (W_mapped || up_s || (i == 0 && up_h.src))
                LAUNCH_TRY(h, launch_upload_operands(i == 0 ? up_h : UploadRows(), up_w, up_s ? up_s + n0 : nullptr,
                                                     up_s ? p->d_S + n0 : nullptr, up_s ? cnt : 0, h->upload_ctas, s));
            if (!W_mapped && r1 > r0) {
                CUDA_TRY(h, cudaMemcpyAsync(p->d_W + r0 * p->K, W + r0 * p->K, sizeof(float) * (size_t)(r1 - r0) * p->K,
                                            cudaMemcpyHostToDevice, s));
                p->last_h2d_bytes += (int64_t)sizeof(float) * (r1 - r0) * p->K;
            }
            if (Sval && !s_dev && !up_s)
                CUDA_TRY(h, cudaMemcpyAsync(p->d_S + n0, Sval + n0, sizeof(float) * (size_t)cnt, cudaMemcpyHostToDevice, s));
            CUDA_TRY(h, cudaEventRecord(h->pipe_uploaded[i], s));
            CUDA_TRY(h, cudaStreamWaitEvent(h->pipe_compute, h->pipe_uploaded[i], 0));
            CUDA_TRY(h, cudaEventRecord(h->pipe_started[i], h->pipe_compute));
            LAUNCH_TRY(h, launch_rows(p, p->d_rows, p->d_cols, nullptr, dS, dW, dH, dP, n0, cnt, use_ring, nullptr,
                                      h->pipe_compute));
            CUDA_TRY(h, cudaEventRecord(h->pipe_computed[i], h->pipe_compute));
            if (!p_dev) {
                CUDA_TRY(h, cudaStreamWaitEvent(h->pipe_download, h->pipe_computed[i], 0));
                CUDA_TRY(h, cudaMemcpyAsync(P + n0, dP + n0, sizeof(float) * (size_t)cnt, cudaMemcpyDeviceToHost,
                                            h->pipe_download));
            }
        }
        // the caller's stream continues only after the last kernel and the last download
        cudaStream_t last = p_dev ? h->pipe_compute : h->pipe_download;
        CUDA_TRY(h, cudaEventRecord(h->pipe_joined, last));
        CUDA_TRY(h, cudaStreamWaitEvent(s, h->pipe_joined, 0));
        CUDA_TRY(h, cudaStreamSynchronize(s));
        waited_for(p, s);
        p->ms_state = sddmm_plan_s::MS_IN_PIPE;
        return check_device_status(h);
    }
    if (up_w.src || up_h.src || up_s)
        LAUNCH_TRY(h, launch_upload_operands(up_h, up_w, up_s, p->d_S, up_s ? p->nnz : 0, h->upload_ctas, s));
    CallTimer timer(p, async);
    CUDA_TRY(h, timer.begin(one_gather && p->nnz <= GATHER_SLICE, s));
    if (use_dense) {
        // locally dense plan: dense cells as small dense products, the rest gathered
        {
            static const char *const names[3][3] = {{"dense_fma", "dense_fma+gather", "dense_fma+ring"},
                                                    {"dense_mma_sync", "dense_mma_sync+gather", "dense_mma_sync+ring"},
                                                    {"dense_tc", "dense_tc+gather", "dense_tc+ring"}};
            p->last_kernel = names[h->dense_mode][p->dense.n_sparse == 0 ? 0 : rows_on_ring(p, false, true) ? 2 : 1];
        }
        if (h->dense_mode == 2)
            LAUNCH_TRY(h, launch_dense_cells_tc(p->dense, dS, dW, dH, dP, p->M, p->N, p->K, h->sm_count, h->d_status, s));
        else
            LAUNCH_TRY(h, launch_dense_cells(p->dense, dS, dW, dH, dP, p->M, p->N, p->K, h->dense_mode == 1, h->sm_count, s));
        // the remainder runs beside the cells (other entries of P; 12 us of 180 on a 65,536-token mask when it ran after them)
        if (p->dense.n_sparse > 0)
            LAUNCH_TRY(h, launch_rows(p, p->dense.rows_s, p->dense.cols_s, p->dense.perm_s, dS, dW, dH, dP, 0, p->dense.n_sparse,
                                      false, nullptr, s, h->dense_mode == 2));
    } else if (use_gather) {
        p->last_kernel = "gather";
        GatherPasses whole = gather_whole(p->nnz, p->N, p->K);
        whole.awaited = awaited;
        LAUNCH_TRY(h, launch_gather(p->d_rows, p->d_cols, nullptr, dS, dW, dH, dP, p->nnz, p->K, whole, h->sm_count, timer.clk, s));
    } else {
        const bool tiled = p->d_perm != nullptr;
        const int32_t *rows_p = tiled ? p->d_rows_t : p->d_rows;
        const int32_t *cols_p = tiled ? p->d_cols_t : p->d_cols;
        // tiled processing order: results go back to input order through the
        // permutation unless the caller asked for the tiled order itself
        const int32_t *perm = (tiled && !tiled_out) ? p->d_perm : nullptr;
        if (tiled && tiled_out && dS) {
            // S values are in input order; the tiled-order result is produced
            // unscaled only (what the reference's kernel leaves in d_val)
            h->last_error = "SDDMM_FLAG_TILED_ORDER with S values is not supported on a multi-tile plan";
            return SDDMM_INVALID_ARG;
        }
        p->last_kernel = use_panel ? "panel" : rows_on_ring(p, use_ring, perm != nullptr) ? "ring" : "gather";
        if (use_panel)
            LAUNCH_TRY(h, launch_panel(p->d_items, p->n_items, p->d_item_rows, rows_p, cols_p, perm, dS, dW, dH, dP, p->K,
                                     p->cfg, h->sm_count, h->d_status, s));
        else
            LAUNCH_TRY(h, launch_rows(p, rows_p, cols_p, perm, dS, dW, dH, dP, 0, p->nnz, use_ring, timer.clk, s, false, awaited));
    }
    CUDA_TRY(h, timer.end(s));
    if (p_copy) CUDA_TRY(h, cudaMemcpyAsync(P, dP, nbytes, cudaMemcpyDeviceToHost, s));
    if (async) return SDDMM_OK;
    CUDA_TRY(h, cudaStreamSynchronize(s));
    waited_for(p, s);
    timer.done();
    return check_device_status(h);
}

int sddmm_coo_sort_rows_gpu(sddmm_handle_t h, int64_t *M, int64_t *N, int64_t nnz, int32_t *rows, int32_t *cols,
                            float *vals, int transpose)
{
    if (!h || !M || !N || nnz < 0 || nnz >= INT32_MAX || (nnz > 0 && (!rows || !cols || !vals))) return SDDMM_INVALID_ARG;
    if (nnz > 0) {
        CUDA_TRY(h, cudaSetDevice(h->device));
        cudaStream_t s = h->stream;
        PoolScope scope(h->pool, s);
        const bool idx_dev = is_device_ptr(rows), val_dev = is_device_ptr(vals);
        if (idx_dev != is_device_ptr(cols)) {
            h->last_error = "sddmm_coo_sort_rows_gpu: rows and cols must both be host or both be device arrays";
            return SDDMM_INVALID_ARG;
        }
        CallTmp tmp;
        const size_t bytes = 4 * (size_t)nnz;
        int32_t *d_rows = rows, *d_cols = cols;
        float *d_vals = vals;
        if (!idx_dev) {
            CUDA_TRY(h, pool_alloc(&tmp.p[0], bytes));
            CUDA_TRY(h, pool_alloc(&tmp.p[1], bytes));
            d_rows = (int32_t *)tmp.p[0];
            d_cols = (int32_t *)tmp.p[1];
            CUDA_TRY(h, cudaMemcpyAsync(d_rows, rows, bytes, cudaMemcpyHostToDevice, s));
            CUDA_TRY(h, cudaMemcpyAsync(d_cols, cols, bytes, cudaMemcpyHostToDevice, s));
        }
        if (!val_dev) {
            CUDA_TRY(h, pool_alloc(&tmp.p[2], bytes));
            d_vals = (float *)tmp.p[2];
            CUDA_TRY(h, cudaMemcpyAsync(d_vals, vals, bytes, cudaMemcpyHostToDevice, s));
        }
        // transposing: the reference sorts whole (col, row, val) tuples and then swaps the roles
        // (util.h:88-104): the old columns become the rows of the result
        if (transpose) CUDA_TRY(h, sort_coo(d_cols, d_rows, d_vals, nnz, true, s));
        else CUDA_TRY(h, sort_coo(d_rows, d_cols, d_vals, nnz, false, s));
        const int32_t *new_rows = transpose ? d_cols : d_rows, *new_cols = transpose ? d_rows : d_cols;
        if (!idx_dev) {
            CUDA_TRY(h, cudaMemcpyAsync(rows, new_rows, bytes, cudaMemcpyDeviceToHost, s));
            CUDA_TRY(h, cudaMemcpyAsync(cols, new_cols, bytes, cudaMemcpyDeviceToHost, s));
        } else if (transpose) {
            // device arrays: exchange the contents of rows and cols through a scratch copy
            CUDA_TRY(h, pool_alloc(&tmp.p[0], bytes));
            CUDA_TRY(h, cudaMemcpyAsync(tmp.p[0], rows, bytes, cudaMemcpyDeviceToDevice, s));
            CUDA_TRY(h, cudaMemcpyAsync(rows, cols, bytes, cudaMemcpyDeviceToDevice, s));
            CUDA_TRY(h, cudaMemcpyAsync(cols, tmp.p[0], bytes, cudaMemcpyDeviceToDevice, s));
        }
        if (!val_dev) CUDA_TRY(h, cudaMemcpyAsync(vals, d_vals, bytes, cudaMemcpyDeviceToHost, s));
        CUDA_TRY(h, cudaStreamSynchronize(s));
    }
    if (transpose) std::swap(*M, *N);
    return SDDMM_OK;
}

int sddmm_plan_used_lines(sddmm_plan_t p, int which, const int32_t **d_ids, int64_t *n)
{
    if (!p || !d_ids || !n || (which != 0 && which != 1)) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    *d_ids = nullptr;
    *n = 0;
    if (p->nnz == 0) return SDDMM_OK;
    if (which == 0 && !p->sorted) return needs_sorted(h);
    CUDA_TRY(h, cudaSetDevice(h->device));
    PoolScope scope(h->pool, h->stream);
    if (which == 0) {
        CUDA_TRY(h, ensure_used_rows(p));
        *d_ids = p->d_used_rows;
        *n = p->n_used_rows;
    } else {
        CUDA_TRY(h, ensure_used_cols(p));
        *d_ids = p->d_used_cols;
        *n = p->n_used_cols;
    }
    // whoever reads the list does so on streams that the plan never hears of: destroying it waits for the device
    p->pending = p->async_pending = p->async_mixed = true;
    return SDDMM_OK;
}

int sddmm_upload_rows(sddmm_handle_t h, const float *host, float *dev, const int32_t *d_row_ids, int64_t n_rows, int K,
                      void *cuda_stream)
{
    if (!h || n_rows < 0) return SDDMM_INVALID_ARG;
    int st = check_k(K);
    if (st != SDDMM_OK) return st;
    if (n_rows == 0) return SDDMM_OK;
    if (!host || !dev || !d_row_ids) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    const float *mapped = mapped_host_ptr(host);
    if (!mapped) {
        h->last_error = "sddmm_upload_rows needs page-locked, mapped host memory (cudaHostAlloc / cudaHostRegister)";
        return SDDMM_INVALID_ARG;
    }
    if (!is_device_ptr(dev) || !is_device_ptr(d_row_ids) || (((uintptr_t)mapped | (uintptr_t)dev) & 15u) != 0) {
        h->last_error = "sddmm_upload_rows: dev and d_row_ids must be device memory, both arrays 16-byte aligned";
        return SDDMM_INVALID_ARG;
    }
    LAUNCH_TRY(h, launch_upload_rows(mapped, dev, d_row_ids, n_rows, K, h->upload_ctas,
                                   cuda_stream ? (cudaStream_t)cuda_stream : h->stream));
    return SDDMM_OK;
}

int sddmm_last_transfer_bytes(sddmm_plan_t p, int64_t *h2d_bytes, int64_t *d2h_bytes)
{
    if (!p) return SDDMM_INVALID_ARG;
    int64_t cols = 0;
    if (h2d_bytes && p->last_h2d_used_cols) {
        const int st = sddmm_plan_count_cols(p, &cols);
        if (st != SDDMM_OK) return st;
    }
    if (h2d_bytes) *h2d_bytes = p->last_h2d_bytes + (int64_t)sizeof(float) * cols * p->K;
    if (d2h_bytes) *d2h_bytes = p->last_d2h_bytes;
    return SDDMM_OK;
}

int sddmm_kernel_launches(sddmm_handle_t h, int64_t *n)
{
    if (!h || !n) return SDDMM_INVALID_ARG;
    *n = h->n_launches;
    return SDDMM_OK;
}

const char *sddmm_last_kernel_name(sddmm_plan_t p) { return p ? p->last_kernel : ""; }

int sddmm_sync(sddmm_handle_t h)
{
    if (!h) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return check_device_status(h);
}

int sddmm_check_result(sddmm_plan_t p, const float *W, const float *H, const float *Sval, const float *P,
                       int64_t stride, double tol, double *max_scaled_err, int64_t *n_checked, int64_t *n_bad)
{
    if (!p || stride < 1 || !(tol > 0)) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    if (max_scaled_err) *max_scaled_err = 0.0;
    if (n_checked) *n_checked = 0;
    if (n_bad) *n_bad = 0;
    if (p->nnz == 0) return SDDMM_OK;
    if (!W || !H || !P) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    PoolScope scope(h->pool, h->stream);
    // host arrays are staged for this call only
    CallTmp tmp;
    auto stage = [&](int slot, const float *src, size_t count, const float **dst) -> cudaError_t {
        if (!src || is_device_ptr(src)) { *dst = src; return cudaSuccess; }
        cudaError_t e = pool_alloc(&tmp.p[slot], sizeof(float) * (count ? count : 1));
        if (e != cudaSuccess) return e;
        *dst = (const float *)tmp.p[slot];
        return cudaMemcpyAsync(tmp.p[slot], src, sizeof(float) * count, cudaMemcpyHostToDevice, h->stream);
    };
    const float *dW, *dH, *dS, *dP;
    CUDA_TRY(h, stage(0, W, (size_t)p->M * p->K, &dW));
    CUDA_TRY(h, stage(1, H, (size_t)p->N * p->K, &dH));
    CUDA_TRY(h, stage(2, Sval, (size_t)p->nnz, &dS));
    CUDA_TRY(h, stage(3, P, (size_t)p->nnz, &dP));
    CheckResult host{};
    CUDA_TRY(h, pool_alloc(&tmp.p[4], sizeof(CheckResult)));
    CheckResult *d_out = (CheckResult *)tmp.p[4];
    cudaError_t e = launch_check_result(p->d_rows, p->d_cols, dS, dW, dH, dP, p->nnz, p->K, stride, tol, d_out, h->sm_count,
                                        h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host, d_out, sizeof(host), cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return fail_cuda(h, e, "sddmm_check_result");
    if (max_scaled_err) *max_scaled_err = host.max_scaled_err;
    if (n_checked) *n_checked = (int64_t)host.n_checked;
    if (n_bad) *n_bad = (int64_t)host.n_bad;
    return SDDMM_OK;
}

namespace {

// What SpMM needs of the plan: the row pointer, and scratch for partial rows behind their counters, which every call leaves at
// zero.  Enqueued in front of the first call, as part of it: what orders the later calls behind that one (spmm_behind_last)
// orders them behind this too, and a pattern that is planned for one call does not wait for it (20 us of 65).  Under capture it is
// built at once.
cudaError_t ensure_spmm_data(sddmm_plan_s *p, cudaStream_t s)
{
    if (p->d_row_ptr && (p->d_spmm_scratch || p->nnz == 0)) return cudaSuccess;
    auto build = [&](cudaStream_t on) {
        cudaError_t e = p->d_row_ptr ? cudaSuccess : build_plan_row_ptr(p, on);
        if (e != cudaSuccess || p->d_spmm_scratch || p->nnz == 0) return e;
        float *scratch = nullptr;
        e = dev_alloc(p, &scratch, spmm_scratch_floats(p->nnz, p->N, p->K, p->h->sm_count));
        if (e != cudaSuccess) return e;
        e = cudaMemsetAsync(scratch, 0, sizeof(float) * spmm_counter_floats(p->nnz, p->N, p->K, p->h->sm_count), on);
        if (e == cudaSuccess) p->d_spmm_scratch = scratch;
        else pool_free(scratch);
        return e;
    };
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const cudaError_t e = cudaStreamIsCapturing(s, &capture);
    if (e != cudaSuccess) return e;
    if (capture != cudaStreamCaptureStatusNone) return build_now(p->h, build);
    p->setup_unwaited = p->setup_unwaited || !p->d_row_ptr;
    mark_pending(p, true, s);
    p->spmm_running = true;
    p->spmm_stream = s;
    return build(s);
}

// The scratch is the plan's, so a call on another stream starts behind the one before it.  A plan whose calls stay on one
// stream keeps no event for that (one behind every call costs 2 us of a call of 24): the first change of stream waits for
// the device, the later ones for the event.  A captured call waits for nothing: what its replays overlap is decided where they
// are launched.
cudaError_t spmm_behind_last(sddmm_plan_s *p, cudaStream_t s, bool *captured)
{
    *captured = false;
    const bool other = p->spmm_running && p->spmm_stream != s;
    if (!other && !p->spmm_event_kept) return cudaSuccess;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(s, &capture);
    *captured = capture != cudaStreamCaptureStatusNone;  // (an event recorded under capture could not be waited for)
    if (e != cudaSuccess || *captured || !other) return e;
    if (p->spmm_event_kept) return cudaStreamWaitEvent(s, p->spmm_done, 0);
    e = cudaEventCreateWithFlags(&p->spmm_done, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
    p->spmm_event_kept = true;
    return cudaDeviceSynchronize();
}
cudaError_t spmm_enqueued(sddmm_plan_s *p, cudaStream_t s, bool captured)
{
    if (captured) return cudaSuccess;
    p->spmm_running = true;
    p->spmm_stream = s;
    return p->spmm_event_kept ? cudaEventRecord(p->spmm_done, s) : cudaSuccess;
}

// Y = P H (fused: P = S o (W H^T) on the fly).  Host arrays are staged for the call.
int run_spmm(sddmm_plan_s *p, bool fused, const float *W, const float *H, const float *pval, float *P_out, float *Y,
             uint32_t flags)
{
    sddmm_handle_s *h = p->h;
    if (!spmm_supports(p->K)) return SDDMM_K_UNSUPPORTED;
    if (!H || !Y || (fused && !W)) return SDDMM_INVALID_ARG;
    if (flags & ~(uint32_t)SDDMM_FLAG_ASYNC) return SDDMM_INVALID_ARG;
    if (!p->sorted) return needs_sorted(h);
    CUDA_TRY(h, cudaSetDevice(h->device));
    PoolScope scope(h->pool, h->stream);
    const bool y_dev = is_device_ptr(Y), p_dev = P_out ? is_device_ptr(P_out) : true;
    auto on_host = [](const float *a) { return a && !is_device_ptr(a); };
    if ((flags & SDDMM_FLAG_ASYNC) && (!y_dev || !p_dev || on_host(W) || on_host(H) || on_host(pval))) return SDDMM_INVALID_ARG;
    const bool async = (flags & SDDMM_FLAG_ASYNC) != 0;
    cudaStream_t s = h->stream;
    mark_pending(p, async, s);
    bool captured = false;
    CUDA_TRY(h, spmm_behind_last(p, s, &captured));
    CUDA_TRY(h, ensure_spmm_data(p, s));
    CallTmp tmp;
    auto stage_in = [&](int slot, const float *src, size_t count, const float **dst) -> cudaError_t {
        if (!src || is_device_ptr(src)) { *dst = src; return cudaSuccess; }
        cudaError_t e = pool_alloc(&tmp.p[slot], sizeof(float) * (count ? count : 1));
        if (e != cudaSuccess) return e;
        *dst = (const float *)tmp.p[slot];
        return cudaMemcpyAsync(tmp.p[slot], src, sizeof(float) * count, cudaMemcpyHostToDevice, s);
    };
    const size_t mk = (size_t)p->M * p->K, nk = (size_t)p->N * p->K, nz = (size_t)p->nnz;
    const float *dW = nullptr, *dH = nullptr, *dV = nullptr;
    CUDA_TRY(h, stage_in(0, W, mk, &dW));
    CUDA_TRY(h, stage_in(1, H, nk, &dH));
    CUDA_TRY(h, stage_in(2, pval, nz, &dV));
    float *dY = Y, *dP = P_out;
    if (!y_dev) {
        CUDA_TRY(h, pool_alloc(&tmp.p[3], sizeof(float) * (mk ? mk : 1)));
        dY = (float *)tmp.p[3];
    }
    if (P_out && !p_dev) {
        CUDA_TRY(h, pool_alloc(&tmp.p[4], sizeof(float) * (nz ? nz : 1)));
        dP = (float *)tmp.p[4];
    }
    if ((((uintptr_t)dW | (uintptr_t)dH | (uintptr_t)dY) & 15u) != 0) {
        h->last_error = "W, H and Y must be 16-byte aligned on the device";
        return SDDMM_INVALID_ARG;
    }
    CallTimer timer(p, async);
    CUDA_TRY(h, timer.begin(p->M > 0 && (fused || spmm_passes(p->nnz, p->N, p->K) == 1), s));
    SpmmCall call{p->d_rows, p->d_cols, p->d_row_ptr, dV, fused ? dW : nullptr, dH, dP, dY, p->d_spmm_scratch, p->M, p->N, p->nnz, p->K,
                  timer.clk};
    CUDA_TRY(h, launch_spmm(call, h->sm_count, &h->n_launches, s));
    CUDA_TRY(h, timer.end(s));
    p->last_kernel = fused ? "fused_sddmm_spmm" : "spmm";
    if (!y_dev) CUDA_TRY(h, cudaMemcpyAsync(Y, dY, sizeof(float) * mk, cudaMemcpyDeviceToHost, s));
    if (P_out && !p_dev) CUDA_TRY(h, cudaMemcpyAsync(P_out, dP, sizeof(float) * nz, cudaMemcpyDeviceToHost, s));
    if (async) {
        CUDA_TRY(h, spmm_enqueued(p, s, captured));
        return SDDMM_OK;
    }
    CUDA_TRY(h, cudaStreamSynchronize(s));
    p->spmm_running = false;  // (this call was behind all of them)
    waited_for(p, s);
    timer.done();
    return check_device_status(h);
}

}  // namespace

int sddmm_spmm_execute(sddmm_plan_t p, const float *Pval, const float *H, float *Y, uint32_t flags)
{
    if (!p) return SDDMM_INVALID_ARG;
    return run_spmm(p, false, nullptr, H, Pval, nullptr, Y, flags);
}

int sddmm_fused_execute(sddmm_plan_t p, const float *W, const float *H, const float *Sval, float *P_out, float *Y,
                        uint32_t flags)
{
    if (!p) return SDDMM_INVALID_ARG;
    return run_spmm(p, true, W, H, Sval, P_out, Y, flags);
}

int sddmm_selftest_optin_cache(void)
{
    // host-only: the shared-memory opt-in cache must be keyed by device ordinal
    SmemOptinCache c;
    if (!c.needs(0, 1024) || !c.needs(1, 1024)) return SDDMM_INVALID_ARG;
    c.record(0, 4096);
    if (c.needs(0, 4096) || c.needs(0, 1024)) return SDDMM_INVALID_ARG;   // device 0 holds it
    if (!c.needs(1, 1024) || !c.needs(0, 8192)) return SDDMM_INVALID_ARG;  // device 1 does not; larger sizes do not either
    if (!c.needs(-1, 1) || !c.needs(SmemOptinCache::MAX_DEVICES, 1)) return SDDMM_INVALID_ARG;
    c.record(SmemOptinCache::MAX_DEVICES, 1);                               // out of table: never cached
    if (!c.needs(SmemOptinCache::MAX_DEVICES, 1)) return SDDMM_INVALID_ARG;
    return SDDMM_OK;
}

int sddmm_last_kernel_ms(sddmm_plan_t p, float *ms)
{
    if (!p || !ms) return SDDMM_INVALID_ARG;
    CUDA_TRY(p->h, resolve_ms(p));
    *ms = p->last_ms;
    return SDDMM_OK;
}

int sddmm_coo(sddmm_handle_t h, int64_t M, int64_t N, int64_t nnz, const int32_t *rows, const int32_t *cols,
              const float *Sval, const float *W, const float *H, int K, float *P)
{
    if (!h) return SDDMM_INVALID_ARG;
    if (M < 0 || N < 0 || nnz < 0) return SDDMM_INVALID_ARG;
    int st = check_k(K);
    if (st != SDDMM_OK) return st;
    if (nnz == 0) return SDDMM_OK;
    if (!rows || !cols || !W || !H || !P) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    PoolScope scope(h->pool, s);
    // Everything that is not already on the device is staged for this call only,
    // as the reference does (sddmm.cu:38-73,147-150).
    CallTmp tmp;
    auto stage = [&](int slot, const void *src, size_t bytes, const void **dst) -> cudaError_t {
        if (is_device_ptr(src)) { *dst = src; return cudaSuccess; }
        cudaError_t e = pool_alloc(&tmp.p[slot], bytes);
        if (e != cudaSuccess) return e;
        *dst = tmp.p[slot];
        return cudaMemcpyAsync(tmp.p[slot], src, bytes, cudaMemcpyHostToDevice, s);
    };
    const void *dr, *dc, *dw, *dh, *ds = nullptr;
    CUDA_TRY(h, stage(0, rows, sizeof(int32_t) * nnz, &dr));
    CUDA_TRY(h, stage(1, cols, sizeof(int32_t) * nnz, &dc));
    CUDA_TRY(h, stage(2, W, sizeof(float) * (size_t)M * K, &dw));
    CUDA_TRY(h, stage(3, H, sizeof(float) * (size_t)N * K, &dh));
    if (Sval) CUDA_TRY(h, stage(4, Sval, sizeof(float) * nnz, &ds));
    float *dp = P;
    const bool p_dev = is_device_ptr(P);
    if (!p_dev) {
        CUDA_TRY(h, pool_alloc(&tmp.p[5], sizeof(float) * nnz));
        dp = (float *)tmp.p[5];
    }
    GatherPasses passes = gather_passes(nnz, N, K, false, (const float *)ds, dp);
    passes.awaited = true;
    CUDA_TRY(h, launch_gather((const int32_t *)dr, (const int32_t *)dc, nullptr, (const float *)ds, (const float *)dw,
                              (const float *)dh, dp, nnz, K, passes, h->sm_count, nullptr, s));
    if (!p_dev) CUDA_TRY(h, cudaMemcpyAsync(P, dp, sizeof(float) * nnz, cudaMemcpyDeviceToHost, s));
    CUDA_TRY(h, cudaStreamSynchronize(s));
    return SDDMM_OK;
}

int sddmm_selftest_wait_timeout(sddmm_handle_t h)
{
    if (!h) return SDDMM_INVALID_ARG;
    CUDA_TRY(h, cudaSetDevice(h->device));
    cudaStream_t s = h->stream;
    CUDA_TRY(h, launch_wait_timeout_probe(h->d_status, s));
    CUDA_TRY(h, cudaStreamSynchronize(s));
    return check_device_status(h);
}

int sddmm_plan_get_info(sddmm_plan_t p, sddmm_plan_info *info)
{
    if (!p || !info) return SDDMM_INVALID_ARG;
    info->M = p->M; info->N = p->N; info->nnz = p->nnz; info->K = p->K;
    info->panel_rows = p->cfg.panel_rows;
    info->col_tile = p->col_tile;
    info->n_col_tiles = p->n_col_tiles;
    info->n_work_items = p->n_items < 0 ? 0 : p->n_items;
    info->n_nonempty_rows = p->n_nonempty_rows;
    info->n_nonempty_cols = p->n_nonempty_cols;
    info->device_bytes = p->device_bytes;
    info->plan_ms = p->plan_ms;
    info->n_dense_cells = p->dense.n_cells;
    info->n_dense_nnz = p->dense.n_dense_nnz;
    info->n_hub_cols = p->n_hub_cols;
    return SDDMM_OK;
}

int sddmm_plan_count_cols(sddmm_plan_t p, int64_t *out)
{
    if (!p || !out) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    if (p->n_nonempty_cols < 0) {
        CUDA_TRY(h, cudaSetDevice(h->device));
        PoolScope scope(h->pool, h->stream);
        int64_t c = 0;
        CUDA_TRY(h, count_distinct_cols(p->d_cols, p->nnz, p->N, &c, h->stream));
        p->n_nonempty_cols = c;
    }
    *out = p->n_nonempty_cols;
    return SDDMM_OK;
}

int sddmm_plan_export_row_ptr(sddmm_plan_t p, int64_t *row_ptr)
{
    if (!p || !row_ptr) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    if (!p->sorted) return needs_sorted(h);
    CUDA_TRY(h, cudaSetDevice(h->device));
    PoolScope scope(h->pool, h->stream);
    CUDA_TRY(h, ensure_row_ptr(p));
    CUDA_TRY(h, cudaMemcpyAsync(row_ptr, p->d_row_ptr, sizeof(int64_t) * (size_t)(p->M + 1), cudaMemcpyDeviceToHost,
                                h->stream));
    CUDA_TRY(h, cudaStreamSynchronize(h->stream));
    return SDDMM_OK;
}

int sddmm_plan_export_tiling(sddmm_plan_t p, int panel_rows, int col_tile, int32_t *t_rows, int32_t *t_cols,
                             int32_t *tiled_ind, int32_t *lastIdx_tile, int32_t *lastIdx_block_tile,
                             int32_t *active_row, int32_t *n_actv_row, int32_t *max_active_row)
{
    if (!p || panel_rows <= 0 || col_tile <= 0) return SDDMM_INVALID_ARG;
    sddmm_handle_s *h = p->h;
    CUDA_TRY(h, cudaSetDevice(h->device));
    PoolScope scope(h->pool, h->stream);
    TilingTables t{t_rows, t_cols, tiled_ind, lastIdx_tile, lastIdx_block_tile, active_row, n_actv_row, max_active_row};
    CUDA_TRY(h, export_reference_tiling(p->d_rows, p->d_cols, p->nnz, p->M, p->N, panel_rows, col_tile, t, h->stream));
    return SDDMM_OK;
}

}  // extern "C"
