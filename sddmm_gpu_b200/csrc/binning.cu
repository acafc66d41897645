// GPU binning pass (see binning.cuh).  Plan-time code: runs once per sparsity
// pattern, outside the timed SDDMM region, exactly like the host preprocessing it
// replaces (HiPC18/src/sddmm.cu:203-233 is untimed in the reference too).
// Scans, selections and the stable tile sort use CUB device primitives; the
// passes that are specific to this engine are the kernels below.
#include "binning.cuh"
#include "device_utils.cuh"

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <climits>
#include <vector>

namespace sddmm {

PoolScope *&PoolScope::current()
{
    static thread_local PoolScope *scope = nullptr;
    return scope;
}
cudaError_t pool_alloc(void **ptr, size_t bytes)
{
    if (PoolScope *at = PoolScope::current()) return at->pool.alloc(ptr, bytes, at->stream);
    return cudaMalloc(ptr, bytes);
}
void pool_free(void *ptr)
{
    if (!ptr) return;
    if (PoolScope *at = PoolScope::current()) at->pool.free(ptr, at->stream, true);
    else cudaFree(ptr);
}

cudaError_t Scratch::reserve(size_t n)
{
    if (n <= bytes) return cudaSuccess;
    release();
    cudaError_t e = pool_alloc(&ptr, n);
    if (e == cudaSuccess) bytes = n;
    else ptr = nullptr;
    return e;
}
void Scratch::release()
{
    pool_free(ptr);
    ptr = nullptr;
    bytes = 0;
}

namespace {

constexpr int TPB = 256;
inline unsigned grid_for(int64_t n, int64_t cap = 148 * 32)
{
    int64_t b = (n + TPB - 1) / TPB;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

// One pass over the indices for everything a plan has to know before it decides anything: the first unsorted and the
// first out-of-range nonzero and the number of rows that hold one.  words[0..3] are kept by the handle in their initial
// state (ULLONG_MAX, ULLONG_MAX, 0, 0) between calls: the last block takes them out, resets them and writes the result
// and the time since block 0 began to mapped host memory, so that one launch and one wait are the whole plan of an
// ordinary matrix.  VEC: both arrays are 16-byte aligned.
template <bool VEC>
__global__ void __launch_bounds__(TPB)
plan_scan_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, int64_t nnz, int64_t M, int64_t N,
                 unsigned long long *words, unsigned long long *out /* [4], mapped */)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) words[4] = dev::globaltimer_ns();
    unsigned long long bad_sort = ULLONG_MAX, bad_range = ULLONG_MAX;
    unsigned heads = 0;
    auto visit = [&](int64_t i, int before, int r, int c) {
        if (r < 0 || r >= M || c < 0 || c >= N) bad_range = min(bad_range, (unsigned long long)i);
        if (i > 0 && before > r) bad_sort = min(bad_sort, (unsigned long long)i);
        heads += (i == 0 || before != r) ? 1 : 0;
    };
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if (VEC) {
        for (int64_t q = t0; q < nnz / 4; q += step) {
            const int4 r = __ldg(reinterpret_cast<const int4 *>(rows) + q), c = __ldg(reinterpret_cast<const int4 *>(cols) + q);
            const int before = q > 0 ? __ldg(rows + 4 * q - 1) : 0;
            visit(4 * q, before, r.x, c.x);
            visit(4 * q + 1, r.x, r.y, c.y);
            visit(4 * q + 2, r.y, r.z, c.z);
            visit(4 * q + 3, r.z, r.w, c.w);
        }
    }
    for (int64_t i = (VEC ? nnz / 4 * 4 : 0) + t0; i < nnz; i += step) visit(i, i > 0 ? __ldg(rows + i - 1) : 0, __ldg(rows + i), __ldg(cols + i));
    if (bad_sort != ULLONG_MAX) atomicMin(&words[0], bad_sort);
    if (bad_range != ULLONG_MAX) atomicMin(&words[1], bad_range);
    __shared__ unsigned block_heads;
    if (threadIdx.x == 0) block_heads = 0;
    __syncthreads();
    heads = __reduce_add_sync(0xffffffffu, heads);
    if ((threadIdx.x & 31) == 0 && heads) atomicAdd(&block_heads, heads);
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (block_heads) atomicAdd(&words[2], (unsigned long long)block_heads);
    __threadfence();
    if (atomicAdd(&words[3], 1ull) + 1 < gridDim.x) return;
    __threadfence();
    out[0] = atomicExch(&words[0], ULLONG_MAX);
    out[1] = atomicExch(&words[1], ULLONG_MAX);
    out[2] = atomicExch(&words[2], 0ull);
    words[3] = 0;
    const unsigned long long now = dev::globaltimer_ns();
    out[3] = now - min(now, *reinterpret_cast<volatile unsigned long long *>(&words[4]));
    __threadfence_system();
}

// One thread per boundary i in [0, nnz]: rows (rows[i-1], rows[i]] start at i.
__global__ void row_ptr_kernel(const int32_t *__restrict__ rows, int64_t nnz, int64_t M, int64_t *__restrict__ row_ptr)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t prev = (i == 0) ? -1 : rows[i - 1];
        const int64_t cur = (i == nnz) ? M : rows[i];
        for (int64_t r = prev + 1; r <= cur; ++r) row_ptr[r] = i;
    }
}

__global__ void mark_cols_kernel(const int32_t *__restrict__ cols, int64_t nnz, unsigned char *mark)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x)
        mark[cols[i]] = 1;
}
__global__ void count_marks_kernel(const unsigned char *__restrict__ mark, int64_t n, unsigned long long *out)
{
    unsigned long long c = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        c += mark[i];
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void tile_key_kernel(const int32_t *__restrict__ cols, int64_t nnz, int col_tile, uint32_t *keys,
                                int32_t *idx)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = (uint32_t)(cols[i] / col_tile);
        idx[i] = (int32_t)i;
    }
}
__global__ void gather2_kernel(const int32_t *__restrict__ perm, const int32_t *__restrict__ a,
                               const int32_t *__restrict__ b, int64_t nnz, int32_t *a_out, int32_t *b_out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t p = perm[i];
        a_out[i] = a[p];
        b_out[i] = b[p];
    }
}

// A nonzero opens a run when it is the first one or when its column tile or its
// row panel differs from its predecessor's.
struct RunHead {
    const int32_t *rows, *cols;
    int panel_rows, col_tile;
    __device__ __forceinline__ bool operator()(int j) const
    {
        if (j == 0) return true;
        return (rows[j] / panel_rows != rows[j - 1] / panel_rows) || (cols[j] / col_tile != cols[j - 1] / col_tile);
    }
};
struct RunHeadCount {
    RunHead h;
    __device__ __forceinline__ int operator()(int j) const { return h(j) ? 1 : 0; }
};

__global__ void pieces_per_run_kernel(const int32_t *__restrict__ run_start, int n_runs, int item_nnz,
                                      int64_t *pieces)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n_runs; i += gridDim.x * blockDim.x) {
        if (i == n_runs) { pieces[i] = 0; continue; }
        const int len = run_start[i + 1] - run_start[i];
        pieces[i] = (len + item_nnz - 1) / item_nnz;
    }
}

// One thread per work item: find its run, cut the run into equal pieces.
__global__ void fill_items_kernel(const int32_t *__restrict__ run_start, const int64_t *__restrict__ item_off,
                                  int n_runs, int64_t n_items, const int32_t *__restrict__ rows, WorkItem *items)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_items; t += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = n_runs;  // last run with item_off[run] <= t
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_off[mid] <= t) lo = mid; else hi = mid;
        }
        const int64_t c = t - item_off[lo];
        const int64_t n_i = item_off[lo + 1] - item_off[lo];
        const int64_t s = run_start[lo], len = run_start[lo + 1] - s;
        const int64_t b = s + (len * c) / n_i, e = s + (len * (c + 1)) / n_i;
        WorkItem w;
        w.nnz_begin = b;
        w.nnz_count = (int32_t)(e - b);
        w.row_begin = rows[b];
        w.n_rows = 0;      // filled by count_item_rows_kernel
        w.list_begin = 0;  // filled by set_list_begin_kernel
        w.reserved = 0;
        items[t] = w;
    }
}

// A nonzero heads a (work item, row) group when it opens an item or its row
// differs from its predecessor's.
struct ItemRowHead {
    const int32_t *rows;
    const unsigned char *item_start;
    __device__ __forceinline__ bool operator()(int j) const
    {
        return item_start[j] || rows[j] != rows[j - 1];  // item_start[0] is always set
    }
};

__global__ void mark_item_starts_kernel(const WorkItem *__restrict__ items, int64_t n_items, unsigned char *flag)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_items; t += (int64_t)gridDim.x * blockDim.x)
        flag[items[t].nnz_begin] = 1;
}

// One warp per item: number of distinct rows among its nonzeros.
__global__ void count_item_rows_kernel(WorkItem *items, int64_t n_items, const int32_t *__restrict__ rows,
                                       int64_t *n_rows_out)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = warp; t < n_items; t += n_warps) {
        const int64_t b = items[t].nnz_begin;
        const int n = items[t].nnz_count;
        int heads = 0;
        for (int o = lane; o < n; o += 32) heads += (o == 0 || rows[b + o] != rows[b + o - 1]) ? 1 : 0;
        for (int s = 16; s; s >>= 1) heads += __shfl_xor_sync(0xffffffffu, heads, s);
        if (lane == 0) {
            items[t].n_rows = heads;
            n_rows_out[t] = heads;
        }
    }
}

__global__ void set_list_begin_kernel(WorkItem *items, int64_t n_items, const int64_t *__restrict__ list_off)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_items; t += (int64_t)gridDim.x * blockDim.x)
        items[t].list_begin = list_off[t];
}

#define CK(x)                         \
    do {                              \
        cudaError_t _e = (x);         \
        if (_e != cudaSuccess) return _e; \
    } while (0)

}  // namespace

cudaError_t init_plan_words(unsigned long long *words)
{
    const unsigned long long init[PLAN_WORDS] = {ULLONG_MAX, ULLONG_MAX, 0, 0, 0};
    return cudaMemcpy(words, init, sizeof(init), cudaMemcpyHostToDevice);
}

cudaError_t scan_coo(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t M, int64_t N, unsigned long long *words,
                     unsigned long long *out_mapped, cudaStream_t stream)
{
    const bool vec = (((uintptr_t)d_rows | (uintptr_t)d_cols) & 15u) == 0;
    const unsigned grid = grid_for((nnz + 3) / 4, 148 * 8);
    if (vec) plan_scan_kernel<true><<<grid, TPB, 0, stream>>>(d_rows, d_cols, nnz, M, N, words, out_mapped);
    else plan_scan_kernel<false><<<grid, TPB, 0, stream>>>(d_rows, d_cols, nnz, M, N, words, out_mapped);
    return cudaGetLastError();
}

cudaError_t build_row_ptr(const int32_t *d_rows, int64_t nnz, int64_t M, int64_t *d_row_ptr, cudaStream_t stream)
{
    row_ptr_kernel<<<grid_for(nnz + 1), TPB, 0, stream>>>(d_rows, nnz, M, d_row_ptr);
    return cudaGetLastError();
}

cudaError_t count_distinct_cols(const int32_t *d_cols, int64_t nnz, int64_t N, int64_t *host_out,
                                cudaStream_t stream)
{
    Scratch s;
    const size_t mark_bytes = ((size_t)N + 15) & ~(size_t)15;
    CK(s.reserve(mark_bytes + 16));
    CK(cudaMemsetAsync(s.ptr, 0, mark_bytes + 16, stream));
    unsigned char *mark = (unsigned char *)s.ptr;
    unsigned long long *cnt = (unsigned long long *)(mark + mark_bytes);
    if (nnz > 0) mark_cols_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols, nnz, mark);
    count_marks_kernel<<<grid_for(N), TPB, 0, stream>>>(mark, N, cnt);
    CK(cudaGetLastError());
    unsigned long long h = 0;
    CK(cudaMemcpyAsync(&h, cnt, sizeof(h), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    *host_out = (int64_t)h;
    return cudaSuccess;
}

namespace {

__global__ void row_used_flags_kernel(const int64_t *__restrict__ row_ptr, int64_t M, unsigned char *flag)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < M; r += (int64_t)gridDim.x * blockDim.x)
        flag[r] = row_ptr[r + 1] > row_ptr[r];
}

// ids of the flagged positions of [0, n), ascending, into a fresh allocation
cudaError_t select_flagged_ids(const unsigned char *flag, int64_t n, int32_t **d_list, int64_t *n_list,
                               cudaStream_t stream)
{
    *d_list = nullptr;
    *n_list = 0;
    if (n == 0) return cudaSuccess;
    Scratch out;  // n ids | selected count
    CK(out.reserve(sizeof(int32_t) * (size_t)n + 16));
    int32_t *ids = (int32_t *)out.ptr;
    int *d_n_sel = (int *)((char *)out.ptr + sizeof(int32_t) * (size_t)((n + 3) & ~(int64_t)3));
    thrust::counting_iterator<int32_t> counting(0);
    size_t tb = 0;
    CK(cub::DeviceSelect::Flagged(nullptr, tb, counting, flag, ids, d_n_sel, (int)n, stream));
    Scratch tmp;
    CK(tmp.reserve(tb));
    CK(cub::DeviceSelect::Flagged(tmp.ptr, tb, counting, flag, ids, d_n_sel, (int)n, stream));
    int n_sel = 0;
    CK(cudaMemcpyAsync(&n_sel, d_n_sel, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    if (n_sel > 0) {
        CK(pool_alloc(d_list, (size_t)n_sel));
        CK(cudaMemcpyAsync(*d_list, ids, sizeof(int32_t) * (size_t)n_sel, cudaMemcpyDeviceToDevice, stream));
        CK(cudaStreamSynchronize(stream));
    }
    *n_list = n_sel;
    return cudaSuccess;
}

}  // namespace

namespace {

__global__ void iota_kernel(int32_t *idx, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        idx[i] = (int32_t)i;
}
// floats -> unsigned keys with the same order
__global__ void value_keys_kernel(const float *__restrict__ v, int64_t n, uint32_t *keys)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t u = __float_as_uint(v[i]);
        keys[i] = u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u);
    }
}
__global__ void pair_keys_kernel(const int32_t *__restrict__ a, const int32_t *__restrict__ b,
                                 const int32_t *__restrict__ idx, int64_t n, unsigned long long *keys)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t j = idx[i];
        keys[i] = ((unsigned long long)(uint32_t)a[j] << 32) | (uint32_t)b[j];
    }
}
__global__ void gather_triples_kernel(const int32_t *__restrict__ idx, const int32_t *__restrict__ a,
                                      const int32_t *__restrict__ b, const float *__restrict__ v, int64_t n,
                                      int32_t *a_out, int32_t *b_out, float *v_out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t j = idx[i];
        a_out[i] = a[j];
        b_out[i] = b[j];
        v_out[i] = v[j];
    }
}

}  // namespace

cudaError_t sort_coo(int32_t *d_a, int32_t *d_b, float *d_v, int64_t nnz, bool tie_by_value, cudaStream_t stream)
{
    if (nnz <= 1) return cudaSuccess;
    const size_t n = (size_t)nnz;
    Scratch buf;  // keys64 in | keys64 out | idx A | idx B | sorted a, b, v
    CK(buf.reserve(n * (8 + 8 + 4 + 4 + 4 + 4 + 4) + 64));
    unsigned long long *k_in = (unsigned long long *)buf.ptr, *k_out = k_in + n;
    int32_t *idx_a = (int32_t *)(k_out + n), *idx_b = idx_a + n;
    int32_t *a_s = idx_b + n, *b_s = a_s + n;
    float *v_s = (float *)(b_s + n);
    iota_kernel<<<grid_for(nnz), TPB, 0, stream>>>(idx_a, nnz);
    CK(cudaGetLastError());
    Scratch tmp;
    if (tie_by_value) {
        // first by value; the stable sort by (a, b) that follows keeps that order inside equal pairs
        uint32_t *vk_in = (uint32_t *)k_in, *vk_out = vk_in + n;
        value_keys_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_v, nnz, vk_in);
        CK(cudaGetLastError());
        size_t tb = 0;
        CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, vk_in, vk_out, idx_a, idx_b, (int)nnz, 0, 32, stream));
        CK(tmp.reserve(tb));
        CK(cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, vk_in, vk_out, idx_a, idx_b, (int)nnz, 0, 32, stream));
        std::swap(idx_a, idx_b);
    }
    pair_keys_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_a, d_b, idx_a, nnz, k_in);
    CK(cudaGetLastError());
    size_t tb = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k_in, k_out, idx_a, idx_b, (int)nnz, 0, 64, stream));
    if (tb > tmp.bytes) {
        tmp.release();
        CK(tmp.reserve(tb));
    }
    CK(cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, k_in, k_out, idx_a, idx_b, (int)nnz, 0, 64, stream));
    gather_triples_kernel<<<grid_for(nnz), TPB, 0, stream>>>(idx_b, d_a, d_b, d_v, nnz, a_s, b_s, v_s);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(d_a, a_s, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, stream));
    CK(cudaMemcpyAsync(d_b, b_s, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, stream));
    CK(cudaMemcpyAsync(d_v, v_s, sizeof(float) * n, cudaMemcpyDeviceToDevice, stream));
    return cudaStreamSynchronize(stream);
}

namespace {
__global__ void pick_kernel(const int32_t *__restrict__ a, PickAt at, int n, unsigned long long *out /* mapped */)
{
    const int i = threadIdx.x;
    if (i < n) out[i] = (unsigned long long)a[at.v[i]];
    __threadfence_system();
}
}  // namespace

cudaError_t pick_values(const int32_t *d_array, const PickAt &at, int n, unsigned long long *out_mapped, cudaStream_t stream)
{
    pick_kernel<<<1, PICK_MAX, 0, stream>>>(d_array, at, n, out_mapped);
    return cudaGetLastError();
}
cudaError_t mark_used_cols(const int32_t *d_cols, int64_t nnz, int64_t N, unsigned char *d_used, cudaStream_t stream)
{
    CK(cudaMemsetAsync(d_used, 0, (size_t)N, stream));
    mark_cols_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols, nnz, d_used);
    return cudaGetLastError();
}

cudaError_t build_used_row_list(const int64_t *d_row_ptr, int64_t M, int32_t **d_list, int64_t *n_list,
                                cudaStream_t stream)
{
    Scratch flag;
    CK(flag.reserve((size_t)M + 16));
    if (M > 0) row_used_flags_kernel<<<grid_for(M), TPB, 0, stream>>>(d_row_ptr, M, (unsigned char *)flag.ptr);
    CK(cudaGetLastError());
    return select_flagged_ids((const unsigned char *)flag.ptr, M, d_list, n_list, stream);
}

cudaError_t build_used_col_list(const int32_t *d_cols, int64_t nnz, int64_t N, int32_t **d_list, int64_t *n_list,
                                cudaStream_t stream)
{
    Scratch flag;
    CK(flag.reserve((size_t)N + 16));
    CK(cudaMemsetAsync(flag.ptr, 0, (size_t)N + 16, stream));
    if (nnz > 0) mark_cols_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols, nnz, (unsigned char *)flag.ptr);
    CK(cudaGetLastError());
    return select_flagged_ids((const unsigned char *)flag.ptr, N, d_list, n_list, stream);
}

cudaError_t build_tiled_order(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t N, int col_tile,
                              int32_t *d_perm, int32_t *d_rows_t, int32_t *d_cols_t, cudaStream_t stream)
{
    if (nnz == 0) return cudaSuccess;
    const int64_t n_tiles = N / col_tile + 1;
    int bits = 1;
    while (((int64_t)1 << bits) < n_tiles) ++bits;
    Scratch keys;  // keys_in | keys_out | idx_in
    CK(keys.reserve(sizeof(uint32_t) * 3 * (size_t)nnz));
    uint32_t *k_in = (uint32_t *)keys.ptr, *k_out = k_in + nnz;
    int32_t *i_in = (int32_t *)(k_out + nnz);
    tile_key_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols, nnz, col_tile, k_in, i_in);
    CK(cudaGetLastError());
    size_t tmp_bytes = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, k_in, k_out, i_in, d_perm, (int)nnz, 0, bits, stream));
    Scratch tmp;
    CK(tmp.reserve(tmp_bytes));
    CK(cub::DeviceRadixSort::SortPairs(tmp.ptr, tmp_bytes, k_in, k_out, i_in, d_perm, (int)nnz, 0, bits, stream));
    gather2_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_perm, d_rows, d_cols, nnz, d_rows_t, d_cols_t);
    CK(cudaGetLastError());
    return cudaStreamSynchronize(stream);
}

cudaError_t build_work_items(const int32_t *d_rows_p, const int32_t *d_cols_p, int64_t nnz, int panel_rows,
                             int col_tile, int item_nnz, WorkItem **d_items, int64_t *n_items,
                             int32_t **d_item_rows, int64_t *n_item_rows, cudaStream_t stream)
{
    *d_items = nullptr;
    *n_items = 0;
    *d_item_rows = nullptr;
    *n_item_rows = 0;
    if (nnz == 0) return cudaSuccess;
    const int n = (int)nnz;
    RunHead head{d_rows_p, d_cols_p, panel_rows, col_tile};
    thrust::counting_iterator<int> counting(0);

    // 1. number of runs
    auto ones = thrust::make_transform_iterator(counting, RunHeadCount{head});
    Scratch small;  // [0] n_runs (int), [8] select count (int)
    CK(small.reserve(64));
    int *d_n_runs = (int *)small.ptr, *d_n_sel = d_n_runs + 2;
    size_t tmp_bytes = 0;
    CK(cub::DeviceReduce::Sum(nullptr, tmp_bytes, ones, d_n_runs, n, stream));
    Scratch tmp;
    CK(tmp.reserve(tmp_bytes));
    CK(cub::DeviceReduce::Sum(tmp.ptr, tmp_bytes, ones, d_n_runs, n, stream));
    int n_runs = 0;
    CK(cudaMemcpyAsync(&n_runs, d_n_runs, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));

    // 2. run starts (+ sentinel nnz)
    Scratch runs;  // run_start int32[n_runs+1] | pieces int64[n_runs+1] | item_off int64[n_runs+1]
    const size_t rs_bytes = (sizeof(int32_t) * ((size_t)n_runs + 1) + 15) & ~(size_t)15;
    const size_t pc_bytes = sizeof(int64_t) * ((size_t)n_runs + 1);
    CK(runs.reserve(rs_bytes + 2 * pc_bytes));
    int32_t *run_start = (int32_t *)runs.ptr;
    int64_t *pieces = (int64_t *)((char *)runs.ptr + rs_bytes);
    int64_t *item_off = pieces + (n_runs + 1);
    tmp_bytes = 0;
    CK(cub::DeviceSelect::If(nullptr, tmp_bytes, counting, run_start, d_n_sel, n, head, stream));
    CK(tmp.reserve(tmp_bytes));
    CK(cub::DeviceSelect::If(tmp.ptr, tmp_bytes, counting, run_start, d_n_sel, n, head, stream));
    CK(cudaMemcpyAsync(run_start + n_runs, &n, sizeof(int), cudaMemcpyHostToDevice, stream));

    // 3. pieces per run -> item offsets
    pieces_per_run_kernel<<<grid_for(n_runs + 1), TPB, 0, stream>>>(run_start, n_runs, item_nnz, pieces);
    CK(cudaGetLastError());
    tmp_bytes = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, pieces, item_off, n_runs + 1, stream));
    CK(tmp.reserve(tmp_bytes));
    CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tmp_bytes, pieces, item_off, n_runs + 1, stream));
    int64_t total = 0;
    CK(cudaMemcpyAsync(&total, item_off + n_runs, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));

    // 4. the items
    WorkItem *items = nullptr;
    CK(pool_alloc(&items, (size_t)total));
    fill_items_kernel<<<grid_for(total), TPB, 0, stream>>>(run_start, item_off, n_runs, total, d_rows_p, items);
    cudaError_t e = cudaGetLastError();

    // 5. the distinct rows of every item, concatenated in item order
    int32_t *item_rows = nullptr;
    int64_t n_list = 0;
    auto body = [&]() -> cudaError_t {
        Scratch per_item;  // n_rows int64[total+1] | list_off int64[total+1]
        CK(per_item.reserve(sizeof(int64_t) * 2 * ((size_t)total + 1)));
        int64_t *cnt = (int64_t *)per_item.ptr, *list_off = cnt + (total + 1);
        CK(cudaMemsetAsync(cnt + total, 0, sizeof(int64_t), stream));
        Scratch flags;
        CK(flags.reserve((size_t)nnz));
        CK(cudaMemsetAsync(flags.ptr, 0, (size_t)nnz, stream));
        mark_item_starts_kernel<<<grid_for(total), TPB, 0, stream>>>(items, total, (unsigned char *)flags.ptr);
        count_item_rows_kernel<<<grid_for(total * 32), TPB, 0, stream>>>(items, total, d_rows_p, cnt);
        CK(cudaGetLastError());
        size_t tb = 0;
        CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, list_off, (int)(total + 1), stream));
        CK(tmp.reserve(tb));
        CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, cnt, list_off, (int)(total + 1), stream));
        set_list_begin_kernel<<<grid_for(total), TPB, 0, stream>>>(items, total, list_off);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(&n_list, list_off + total, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        CK(pool_alloc(&item_rows, (size_t)(n_list > 0 ? n_list : 1)));
        auto head_flags = thrust::make_transform_iterator(counting, ItemRowHead{d_rows_p, (const unsigned char *)flags.ptr});
        tb = 0;
        CK(cub::DeviceSelect::Flagged(nullptr, tb, d_rows_p, head_flags, item_rows, d_n_sel, n, stream));
        CK(tmp.reserve(tb));
        CK(cub::DeviceSelect::Flagged(tmp.ptr, tb, d_rows_p, head_flags, item_rows, d_n_sel, n, stream));
        return cudaStreamSynchronize(stream);
    };
    if (e == cudaSuccess) e = body();
    if (e != cudaSuccess) {
        pool_free(items);
        pool_free(item_rows);
        return e;
    }
    *d_items = items;
    *n_items = total;
    *d_item_rows = item_rows;
    *n_item_rows = n_list;
    return cudaSuccess;
}


// ---------------------------------------------------------------------------
// Hub-column hints for the ring kernel
// ---------------------------------------------------------------------------
namespace {

constexpr int DEG_CAP = 1 << 16;  // degrees are histogrammed exactly up to here

__global__ void col_degree_kernel(const int32_t *__restrict__ cols, int64_t nnz, int32_t *deg)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&deg[cols[i]], 1);
}
__global__ void degree_histogram_kernel(const int32_t *__restrict__ deg, int64_t N, unsigned long long *hist)
{
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < N; c += (int64_t)gridDim.x * blockDim.x) {
        const int d = deg[c];
        if (d > 0) atomicAdd(&hist[d < DEG_CAP ? d : DEG_CAP - 1], 1ull);
    }
}
__global__ void flag_cols_kernel(const int32_t *__restrict__ cols, const int32_t *__restrict__ deg, int64_t nnz,
                                 int threshold, int32_t *cols_out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = cols[i];
        cols_out[i] = deg[c] >= threshold ? (int32_t)((uint32_t)c | 0x80000000u) : c;
    }
}

}  // namespace

cudaError_t build_hub_column_hints(const int32_t *d_cols_p, int64_t nnz, int64_t N, int64_t row_bytes,
                                   int64_t budget_bytes, int32_t *d_cols_hinted, int64_t *n_hub_cols,
                                   int *degree_threshold, cudaStream_t stream)
{
    *n_hub_cols = 0;
    *degree_threshold = 0;
    if (nnz == 0 || N == 0) return cudaSuccess;
    Scratch deg, hist;
    CK(deg.reserve(sizeof(int32_t) * (size_t)N));
    CK(hist.reserve(sizeof(unsigned long long) * DEG_CAP));
    CK(cudaMemsetAsync(deg.ptr, 0, sizeof(int32_t) * (size_t)N, stream));
    CK(cudaMemsetAsync(hist.ptr, 0, sizeof(unsigned long long) * DEG_CAP, stream));
    col_degree_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols_p, nnz, (int32_t *)deg.ptr);
    degree_histogram_kernel<<<grid_for(N), TPB, 0, stream>>>((const int32_t *)deg.ptr, N, (unsigned long long *)hist.ptr);
    CK(cudaGetLastError());
    std::vector<unsigned long long> h(DEG_CAP);
    CK(cudaMemcpyAsync(h.data(), hist.ptr, sizeof(unsigned long long) * DEG_CAP, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    // the most popular columns first, until their rows of H fill the budget; a
    // column used once gains nothing from staying in L2
    const int64_t max_cols = budget_bytes / row_bytes;
    int64_t taken = 0;
    int t = DEG_CAP;
    for (int d = DEG_CAP - 1; d >= 2; --d) {
        if (taken + (int64_t)h[d] > max_cols) break;
        taken += (int64_t)h[d];
        t = d;
    }
    if (t == DEG_CAP) t = INT32_MAX;  // nothing fits: no column is marked
    flag_cols_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols_p, (const int32_t *)deg.ptr, nnz, t, d_cols_hinted);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream));
    *n_hub_cols = taken;
    *degree_threshold = t;
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Dense-cell classification
//
// Three classes of cells, each 128 rows x 64 columns:
//   class 0  rows that are (nearly) full -- "global" rows -- are compacted into
//            virtual row panels (row r -> its rank among the dense rows);
//   class 1  likewise for (nearly) full columns of the remaining nonzeros;
//   class 2  the regular grid over everything else (bands, dense blocks).
// A cell is handed to the dense-cell kernel when it holds at least min_density
// of its 8192 positions.
// ---------------------------------------------------------------------------
namespace {

__global__ void dense_line_flags_kernel(const int64_t *__restrict__ row_ptr, int64_t M, int64_t min_row_deg,
                                        const int32_t *__restrict__ col_deg, int64_t N, int64_t min_col_deg,
                                        int32_t *row_flag, int32_t *col_flag)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = t; r <= M; r += step) row_flag[r] = (r < M && row_ptr[r + 1] - row_ptr[r] >= min_row_deg) ? 1 : 0;
    for (int64_t c = t; c <= N; c += step) col_flag[c] = (c < N && col_deg[c] >= min_col_deg) ? 1 : 0;
}
// flag + exclusive scan -> virtual id (or -1) and the compacted list
__global__ void dense_line_ids_kernel(const int32_t *__restrict__ flag, const int32_t *__restrict__ rank, int64_t n,
                                      int32_t *vid, int32_t *list)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (flag[i]) {
            vid[i] = rank[i];
            list[rank[i]] = (int32_t)i;
        } else {
            vid[i] = -1;
        }
    }
}

// An upper bound of the nonzeros that dense cells can hold, without sorting anything: those in (nearly) full rows and
// columns, and those in cells of the regular grid with min_count or more of the others.  A block per panel of 128 rows,
// the panel's cell counts in shared memory, a warp per row (full rows are not read at all), four column loads per lane in
// flight, one atomic per run of nonzeros in one cell (15.9 M nonzeros of an attention mask: 225 us nonzero by nonzero).
__global__ void __launch_bounds__(1024)
dense_bound_kernel(const int32_t *__restrict__ cols, const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ col_deg,
                   int64_t M, int n_cell_cols, int64_t min_row_deg, int64_t min_col_deg, int min_count, unsigned long long *bound)
{
    extern __shared__ int cell_count[];
    const int64_t r0 = (int64_t)blockIdx.x * DENSE_CELL_ROWS, r1 = min(M, r0 + DENSE_CELL_ROWS);
    if (row_ptr[r0] == row_ptr[r1]) return;
    for (int i = threadIdx.x; i < n_cell_cols; i += blockDim.x) cell_count[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    unsigned long long total = 0;
    for (int64_t r = r0 + (threadIdx.x >> 5); r < r1; r += blockDim.x >> 5) {
        const int64_t j0 = row_ptr[r], j1 = row_ptr[r + 1];
        if (j1 - j0 >= min_row_deg) {
            if (lane == 0) total += (unsigned long long)(j1 - j0);
            continue;
        }
        for (int64_t jb = j0; jb < j1; jb += 128) {
            int c[4], full[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int64_t j = jb + 32 * u + lane;
                c[u] = j < j1 ? __ldg(cols + j) : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) full[u] = c[u] >= 0 && __ldg(col_deg + c[u]) >= min_col_deg;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                total += full[u];
                const int cell = c[u] >= 0 && !full[u] ? c[u] / DENSE_CELL_COLS : -1;
                const int before = __shfl_up_sync(0xffffffffu, cell, 1);
                const unsigned head = __ballot_sync(0xffffffffu, lane == 0 || cell != before);
                if (((head >> lane) & 1u) && cell >= 0) {
                    const unsigned above = lane == 31 ? 0u : head >> (lane + 1);
                    atomicAdd(&cell_count[cell], above ? __ffs(above) : 32 - lane);
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_cell_cols; i += blockDim.x)
        if (cell_count[i] >= min_count) total += cell_count[i];
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    if (lane == 0 && total) atomicAdd(bound, total);
}

struct CellGeometry {
    unsigned long long grid;  // keys per class: n_row_panels * n_col_blocks of the regular grid
    int64_t ncb;              // column blocks of the matrix
    int64_t nvcb;             // column blocks over the dense columns
};

template <class Key>
__global__ void cell_key_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, int64_t nnz,
                                const int32_t *__restrict__ row_vid, const int32_t *__restrict__ col_vid,
                                CellGeometry geo, Key *keys, int32_t *idx)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t r = rows[i], c = cols[i];
        const int32_t vr = row_vid[r], vc = col_vid[c];
        unsigned long long key;
        if (vr >= 0) key = (unsigned long long)(vr / DENSE_CELL_ROWS) * geo.ncb + (c / DENSE_CELL_COLS);
        else if (vc >= 0) key = geo.grid + (unsigned long long)(r / DENSE_CELL_ROWS) * geo.nvcb + (vc / DENSE_CELL_COLS);
        else key = 2 * geo.grid + (unsigned long long)(r / DENSE_CELL_ROWS) * geo.ncb + (c / DENSE_CELL_COLS);
        keys[i] = (Key)key;
        idx[i] = (int32_t)i;
    }
}
template <class Key>
struct KeyHead {
    const Key *keys;
    __device__ __forceinline__ int operator()(int j) const { return (j == 0 || keys[j] != keys[j - 1]) ? 1 : 0; }
};
template <class Key>
struct KeyHeadPred {
    const Key *keys;
    __device__ __forceinline__ bool operator()(int j) const { return j == 0 || keys[j] != keys[j - 1]; }
};
// per non-empty cell: dense or not, and how many nonzeros it contributes to the dense arrays
__global__ void classify_cells_kernel(const int32_t *__restrict__ cell_start, int n_cells, int min_count,
                                      int32_t *dense_flag, int64_t *dense_cnt)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n_cells; i += gridDim.x * blockDim.x) {
        if (i == n_cells) { dense_flag[i] = 0; dense_cnt[i] = 0; continue; }
        const int c = cell_start[i + 1] - cell_start[i];
        const int d = c >= min_count ? 1 : 0;
        dense_flag[i] = d;
        dense_cnt[i] = d ? c : 0;
    }
}
template <class Key>
__global__ void fill_dense_kernel(const Key *__restrict__ keys_s, const int32_t *__restrict__ idx_s,
                                  const int32_t *__restrict__ cellid /* inclusive head scan */,
                                  const int32_t *__restrict__ cell_start, const int32_t *__restrict__ dense_flag,
                                  const int32_t *__restrict__ dense_slot, const int64_t *__restrict__ dense_off,
                                  const int32_t *__restrict__ rows, const int32_t *__restrict__ cols,
                                  const int32_t *__restrict__ row_vid, const int32_t *__restrict__ col_vid, int64_t nnz,
                                  CellGeometry geo, DenseCell *cells, int32_t *idx_d, uint16_t *rc_d,
                                  unsigned char *is_dense)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        const int ci = cellid[j] - 1;
        if (!dense_flag[ci]) continue;
        const unsigned long long key = keys_s[j];
        const int cls = (int)(key / geo.grid);
        const unsigned long long rem = key % geo.grid;
        const unsigned long long nb = (cls == 1) ? (unsigned long long)geo.nvcb : (unsigned long long)geo.ncb;
        const int32_t row0 = (int32_t)(rem / nb) * DENSE_CELL_ROWS;  // virtual for class 0
        const int32_t col0 = (int32_t)(rem % nb) * DENSE_CELL_COLS;  // virtual for class 1
        const int32_t start = cell_start[ci];
        const int64_t pos = dense_off[ci] + (j - start);
        const int32_t orig = idx_s[j];
        const int32_t r = rows[orig], c = cols[orig];
        const int32_t rl = (cls == 0 ? row_vid[r] : r) - row0;
        const int32_t cl = (cls == 1 ? col_vid[c] : c) - col0;
        idx_d[pos] = orig;
        rc_d[pos] = (uint16_t)((rl << 8) | cl);
        is_dense[orig] = 1;
        if (j == start) {
            DenseCell dcell;
            dcell.row0 = row0;
            dcell.col0 = col0;
            dcell.slot = dense_off[ci];  // of its nonzeros in the lists, until the forms are known
            dcell.count = cell_start[ci + 1] - start;
            dcell.cls = cls;
            cells[dense_slot[ci]] = dcell;
        }
    }
}
// Row masks and run positions of every dense cell (one CTA per cell, grid-stride), and whether the cell qualifies for
// the row-mask form: inside every row the list entries (input order) have ascending columns, and either their input indices are
// consecutive but for one gap at most or index and column go up together (any number of columns may be in other cells then).  row_mask arrives zeroed.
__global__ void cell_row_masks_kernel(DenseCell *cells, int64_t n_cells, const int32_t *__restrict__ idx,
                                      const uint16_t *__restrict__ rc, unsigned long long *row_mask, int2 *row_base,
                                      uint32_t *row_span, unsigned long long *n_mask_cells)
{
    __shared__ int unordered, gapped, forms;
    __shared__ int gaps[DENSE_CELL_ROWS], first[DENSE_CELL_ROWS], split[DENSE_CELL_ROWS], second[DENSE_CELL_ROWS];
    for (int64_t cell = blockIdx.x; cell < n_cells; cell += gridDim.x) {
        if (threadIdx.x == 0) {
            unordered = gapped = 0;
            forms = CELL_RUNS;
        }
        for (int r = threadIdx.x; r < DENSE_CELL_ROWS; r += blockDim.x) {
            gaps[r] = first[r] = second[r] = 0;
            split[r] = DENSE_CELL_COLS;
        }
        __syncthreads();
        const DenseCell dc = cells[cell];
        const int32_t *ci = idx + dc.slot;
        const uint16_t *cr = rc + dc.slot;
        unsigned long long *mk = row_mask + cell * DENSE_CELL_ROWS;
        for (int t = threadIdx.x; t < dc.count; t += blockDim.x) {
            const unsigned code = cr[t];
            const int r = code >> 8, c = code & 255u;
            atomicOr(mk + r, 1ull << c);
            const unsigned prev = t > 0 ? cr[t - 1] : 0u;
            if (t == 0 || (prev >> 8) != (unsigned)r) {
                first[r] = ci[t];
            } else {
                if ((int)(prev & 255u) >= c) unordered = 1;
                if (ci[t] - ci[t - 1] != c - (int)(prev & 255u)) forms = 0;
                if (ci[t] != ci[t - 1] + 1) {
                    if (atomicAdd(&gaps[r], 1) > 0) gapped = 1;
                    split[r] = c;
                    second[r] = ci[t];
                }
            }
        }
        __threadfence_block();
        __syncthreads();
        for (int r = threadIdx.x; r < DENSE_CELL_ROWS; r += blockDim.x) {
            const unsigned long long m = atomicOr(mk + r, 0ull);
            const int s = split[r];
            const int before = s < DENSE_CELL_COLS ? __popcll(m & ((1ull << s) - 1ull)) : 0;
            row_base[cell * DENSE_CELL_ROWS + r] = make_int2(first[r], second[r] - before);
            const int c0 = m ? __ffsll(m) - 1 : 0;
            row_span[cell * DENSE_CELL_ROWS + r] = (uint32_t)c0 | (uint32_t)s << 16;
        }
        __syncthreads();
        if (threadIdx.x == 0 && !unordered && (forms || !gapped)) {
            cells[cell].cls = dc.cls | CELL_MASKED | forms;
            atomicAdd(n_mask_cells, 1ull);
        }
        __syncthreads();
    }
}

// Tables of the cells that are not in row-mask form (one CTA per cell, grid-stride); DenseCell::slot becomes the number of the
// table.  table arrives filled with -1.  Of several nonzeros of one row and column the first is entered, the others go to
// the remainder.  words[0]: tables, words[1]: nonzeros that went; both arrive 0.
__global__ void cell_tables_kernel(DenseCell *cells, int64_t n_cells, const int32_t *__restrict__ idx, const uint16_t *__restrict__ rc,
                                   int32_t *table, unsigned char *is_dense, unsigned long long *words)
{
    __shared__ unsigned long long slot;
    for (int64_t cell = blockIdx.x; cell < n_cells; cell += gridDim.x) {
        const DenseCell dc = cells[cell];
        if (dc.cls & CELL_MASKED) continue;  // the same for the whole block
        if (threadIdx.x == 0) slot = atomicAdd(words, 1ull);
        __syncthreads();
        unsigned *t = reinterpret_cast<unsigned *>(table) + slot * (DENSE_CELL_ROWS * DENSE_CELL_COLS);
        auto entry = [&](int i) {
            const unsigned code = rc[dc.slot + i];
            return t + (code >> 8) * DENSE_CELL_COLS + (code & 255u);
        };
        for (int i = threadIdx.x; i < dc.count; i += blockDim.x) atomicMin(entry(i), (unsigned)idx[dc.slot + i]);
        __threadfence_block();
        __syncthreads();
        unsigned long long gone = 0;
        for (int i = threadIdx.x; i < dc.count; i += blockDim.x) {
            const unsigned mine = (unsigned)idx[dc.slot + i];
            if (atomicMin(entry(i), 0xffffffffu) != mine) {
                is_dense[mine] = 0;
                ++gone;
            }
        }
        if (gone) atomicAdd(words + 1, gone);
        if (threadIdx.x == 0) cells[cell].slot = (int64_t)slot;
        __syncthreads();
    }
}

// Cells are in the order of (class, row0, col0): a unit begins at every second cell of the same rows.
struct UnitHead {
    const DenseCell *cells;
    __device__ __forceinline__ bool operator()(int c) const
    {
        const int cls = cells[c].cls & 0xff, row0 = cells[c].row0;
        int lo = 0, hi = c;  // first cell of these rows
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2, k = cells[mid].cls & 0xff;
            if (k < cls || (k == cls && cells[mid].row0 < row0)) lo = mid + 1;
            else hi = mid;
        }
        return ((c - lo) & 1) == 0;
    }
};
__global__ void unit_fill_kernel(const DenseCell *__restrict__ cells, const int32_t *__restrict__ heads, int n_cells, int n_units, DenseUnit *units)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < n_units; u += gridDim.x * blockDim.x) {
        const int c = heads[u], n = (u + 1 < n_units ? heads[u + 1] : n_cells) - c;
        DenseUnit d = {};
        d.n = n;
        d.row0 = cells[c].row0;
        for (int k = 0; k < n; ++k) {
            d.number[k] = cells[c + k].cls & CELL_MASKED ? c + k : (int32_t)cells[c + k].slot;
            d.col0[k] = cells[c + k].col0;
            d.cls[k] = cells[c + k].cls;
        }
        units[u] = d;
    }
}

struct NotDense {
    const unsigned char *is_dense;
    __device__ __forceinline__ bool operator()(int j) const { return is_dense[j] == 0; }
};

}  // namespace

void DensePlan::release()
{
    pool_free(cells); pool_free(units); pool_free(table); pool_free(rows_s); pool_free(cols_s); pool_free(perm_s);
    pool_free(dense_rows); pool_free(dense_cols); pool_free(row_mask); pool_free(row_base); pool_free(row_span);
    cells = nullptr; units = nullptr; table = nullptr; rows_s = cols_s = perm_s = nullptr;
    dense_rows = dense_cols = nullptr;
    row_mask = nullptr; row_base = nullptr; row_span = nullptr;
    n_cells = n_dense_nnz = n_sparse = n_dense_rows = n_dense_cols = n_units = n_table_cells = 0;
}

// Key: of a cell; 32 bits wherever they are enough (the sort moves two thirds of the bytes).
template <class Key>
static cudaError_t build_dense_cells_k(const int32_t *d_rows, const int32_t *d_cols, const int64_t *d_row_ptr, int64_t nnz,
                                       int64_t M, int64_t N, float min_density, float min_share, DensePlan *out,
                                       cudaStream_t stream)
{
    out->release();
    if (nnz == 0) return cudaSuccess;
    const int n = (int)nnz;
    const int min_count = (int)(min_density * DENSE_CELL_ROWS * DENSE_CELL_COLS);
    thrust::counting_iterator<int> counting(0);
    Scratch tmp;
    size_t tb = 0;

    // 0. dense rows and columns -> virtual ids and compacted lists
    Scratch lines;  // col_deg[N] | row_flag[M+1] | row_rank[M+1] | col_flag[N+1] | col_rank[N+1] | row_vid[M] | col_vid[N]
    const size_t m1 = (size_t)M + 1, n1 = (size_t)N + 1;
    CK(lines.reserve(sizeof(int32_t) * ((size_t)N + 2 * m1 + 2 * n1 + (size_t)M + (size_t)N)));
    int32_t *col_deg = (int32_t *)lines.ptr, *row_flag = col_deg + N, *row_rank = row_flag + m1;
    int32_t *col_flag = row_rank + m1, *col_rank = col_flag + n1, *row_vid = col_rank + n1, *col_vid = row_vid + M;
    CK(cudaMemsetAsync(col_deg, 0, sizeof(int32_t) * (size_t)N, stream));
    col_degree_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_cols, nnz, col_deg);
    const int64_t min_row_deg = std::max<int64_t>(N / 4, 4 * DENSE_CELL_COLS);
    const int64_t min_col_deg = std::max<int64_t>(M / 4, 4 * DENSE_CELL_ROWS);
    // most matrices that get here have no dense cells: find out before the sort
    const int64_t n_cell_cols = (N + DENSE_CELL_COLS - 1) / DENSE_CELL_COLS;
    if (n_cell_cols * 4 <= (200 << 10)) {
        static SmemOptinCache optin;
        const size_t smem = (size_t)n_cell_cols * 4;
        if (smem > (48 << 10)) CK(optin_dynamic_smem(dense_bound_kernel, smem, optin));
        Scratch bound;
        CK(bound.reserve(sizeof(unsigned long long)));
        CK(cudaMemsetAsync(bound.ptr, 0, sizeof(unsigned long long), stream));
        dense_bound_kernel<<<(unsigned)((M + DENSE_CELL_ROWS - 1) / DENSE_CELL_ROWS), 1024, smem, stream>>>(
            d_cols, d_row_ptr, col_deg, M, (int)n_cell_cols, min_row_deg, min_col_deg, min_count,
            (unsigned long long *)bound.ptr);
        CK(cudaGetLastError());
        unsigned long long most = 0;
        CK(cudaMemcpyAsync(&most, bound.ptr, sizeof(most), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        if ((double)most < (double)min_share * (double)nnz) return cudaSuccess;
    }
    dense_line_flags_kernel<<<grid_for(std::max(M, N) + 1), TPB, 0, stream>>>(d_row_ptr, M, min_row_deg, col_deg, N,
                                                                           min_col_deg, row_flag, col_flag);
    CK(cudaGetLastError());
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, row_flag, row_rank, (int)m1, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, row_flag, row_rank, (int)m1, stream));
    tb = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, col_flag, col_rank, (int)n1, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, col_flag, col_rank, (int)n1, stream));
    int n_dr = 0, n_dcol = 0;
    CK(cudaMemcpyAsync(&n_dr, row_rank + M, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaMemcpyAsync(&n_dcol, col_rank + N, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    CK(pool_alloc(&out->dense_rows, (size_t)(n_dr > 0 ? n_dr : 1)));
    CK(pool_alloc(&out->dense_cols, (size_t)(n_dcol > 0 ? n_dcol : 1)));
    dense_line_ids_kernel<<<grid_for(M), TPB, 0, stream>>>(row_flag, row_rank, M, row_vid, out->dense_rows);
    dense_line_ids_kernel<<<grid_for(N), TPB, 0, stream>>>(col_flag, col_rank, N, col_vid, out->dense_cols);
    CK(cudaGetLastError());
    out->n_dense_rows = n_dr;
    out->n_dense_cols = n_dcol;

    CellGeometry geo;
    geo.ncb = (N + DENSE_CELL_COLS - 1) / DENSE_CELL_COLS;
    geo.nvcb = std::max<int64_t>(1, (n_dcol + DENSE_CELL_COLS - 1) / DENSE_CELL_COLS);
    geo.grid = (unsigned long long)((M + DENSE_CELL_ROWS - 1) / DENSE_CELL_ROWS) * (unsigned long long)geo.ncb;

    // 1. nonzeros sorted by cell (stable: row-major inside a cell)
    Scratch keys;  // keys_in | keys_out | idx_in | idx_sorted | cellid (i32)
    CK(keys.reserve((size_t)nnz * (2 * sizeof(Key) + 4 + 4 + 4)));
    Key *k_in = (Key *)keys.ptr, *k_s = k_in + nnz;
    int32_t *i_in = (int32_t *)(k_s + nnz), *i_s = i_in + nnz, *cellid = i_s + nnz;
    cell_key_kernel<<<grid_for(nnz), TPB, 0, stream>>>(d_rows, d_cols, nnz, row_vid, col_vid, geo, k_in, i_in);
    CK(cudaGetLastError());
    int bits = 1;
    while (bits < (int)sizeof(Key) * 8 && (1ull << bits) <= 3 * geo.grid) ++bits;
    tb = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k_in, k_s, i_in, i_s, n, 0, bits, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, k_in, k_s, i_in, i_s, n, 0, bits, stream));

    // 2. non-empty cells: starts and the cell id of every sorted position
    auto heads = thrust::make_transform_iterator(counting, KeyHead<Key>{k_s});
    tb = 0;
    CK(cub::DeviceScan::InclusiveSum(nullptr, tb, heads, cellid, n, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceScan::InclusiveSum(tmp.ptr, tb, heads, cellid, n, stream));
    int n_cells = 0;
    CK(cudaMemcpyAsync(&n_cells, cellid + (nnz - 1), sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    Scratch cellbuf;  // dense_cnt i64[n+1] | dense_off i64[n+1] | cell_start i32[n+1] | dense_flag i32[n+1] | dense_slot i32[n+1] | n_sel
    const size_t nc1 = (size_t)n_cells + 1;
    CK(cellbuf.reserve(nc1 * (4 * 3 + 8 * 2) + 64));
    int64_t *dense_cnt = (int64_t *)cellbuf.ptr, *dense_off = dense_cnt + nc1;
    int32_t *cell_start = (int32_t *)(dense_off + nc1), *dense_flag = cell_start + nc1, *dense_slot = dense_flag + nc1;
    int *d_n_sel = (int *)(dense_slot + nc1);
    tb = 0;
    CK(cub::DeviceSelect::If(nullptr, tb, counting, cell_start, d_n_sel, n, KeyHeadPred<Key>{k_s}, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceSelect::If(tmp.ptr, tb, counting, cell_start, d_n_sel, n, KeyHeadPred<Key>{k_s}, stream));
    CK(cudaMemcpyAsync(cell_start + n_cells, &n, sizeof(int), cudaMemcpyHostToDevice, stream));

    // 3. classify, offsets of the dense cells' nonzeros and slots of the dense cells
    classify_cells_kernel<<<grid_for(nc1), TPB, 0, stream>>>(cell_start, n_cells, min_count, dense_flag, dense_cnt);
    CK(cudaGetLastError());
    tb = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, dense_cnt, dense_off, (int)nc1, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, dense_cnt, dense_off, (int)nc1, stream));
    tb = 0;
    CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, dense_flag, dense_slot, (int)nc1, stream));
    CK(tmp.reserve(tb));
    CK(cub::DeviceScan::ExclusiveSum(tmp.ptr, tb, dense_flag, dense_slot, (int)nc1, stream));
    int64_t n_dense_nnz = 0;
    int n_dense_cells = 0;
    CK(cudaMemcpyAsync(&n_dense_nnz, dense_off + n_cells, sizeof(int64_t), cudaMemcpyDeviceToHost, stream));
    CK(cudaMemcpyAsync(&n_dense_cells, dense_slot + n_cells, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    if (n_dense_cells == 0 || (double)n_dense_nnz < (double)min_share * (double)nnz) {  // not worth a split
        out->release();
        return cudaSuccess;
    }

    // 4. the dense arrays and the remainder
    auto body = [&]() -> cudaError_t {
        CK(pool_alloc(&out->cells, (size_t)n_dense_cells));
        Scratch lists;  // idx: input index of every dense-cell nonzero, grouped by cell, row-major inside; rc: (row - row0) << 8 | (col - col0)
        CK(lists.reserve((size_t)n_dense_nnz * 6));
        int32_t *idx = (int32_t *)lists.ptr;
        uint16_t *rc = (uint16_t *)(idx + n_dense_nnz);
        Scratch flags;
        CK(flags.reserve((size_t)nnz));
        CK(cudaMemsetAsync(flags.ptr, 0, (size_t)nnz, stream));
        fill_dense_kernel<<<grid_for(nnz), TPB, 0, stream>>>(k_s, i_s, cellid, cell_start, dense_flag, dense_slot, dense_off,
                                                            d_rows, d_cols, row_vid, col_vid, nnz, geo, out->cells,
                                                            idx, rc, (unsigned char *)flags.ptr);
        CK(cudaGetLastError());
        // row-mask form of the cells that allow it
        {
            const size_t lines_n = (size_t)n_dense_cells * DENSE_CELL_ROWS;
            CK(pool_alloc(&out->row_mask, lines_n));
            CK(pool_alloc(&out->row_base, lines_n));
            CK(pool_alloc(&out->row_span, lines_n));
            CK(cudaMemsetAsync(out->row_mask, 0, sizeof(unsigned long long) * lines_n, stream));
            Scratch cnt;
            CK(cnt.reserve(sizeof(unsigned long long)));
            CK(cudaMemsetAsync(cnt.ptr, 0, sizeof(unsigned long long), stream));
            cell_row_masks_kernel<<<grid_for((int64_t)n_dense_cells * TPB), TPB, 0, stream>>>(
                out->cells, n_dense_cells, idx, rc, out->row_mask, out->row_base,
                out->row_span, (unsigned long long *)cnt.ptr);
            CK(cudaGetLastError());
            unsigned long long n_mask = 0;
            CK(cudaMemcpyAsync(&n_mask, cnt.ptr, sizeof(n_mask), cudaMemcpyDeviceToHost, stream));
            CK(cudaStreamSynchronize(stream));
            out->n_table_cells = n_dense_cells - (int64_t)n_mask;
        }
        if (out->n_table_cells > 0) {
            const size_t entries = (size_t)out->n_table_cells * DENSE_CELL_ROWS * DENSE_CELL_COLS;
            CK(pool_alloc(&out->table, entries));
            CK(cudaMemsetAsync(out->table, 0xff, sizeof(int32_t) * entries, stream));
            Scratch words;
            CK(words.reserve(2 * sizeof(unsigned long long)));
            CK(cudaMemsetAsync(words.ptr, 0, 2 * sizeof(unsigned long long), stream));
            cell_tables_kernel<<<grid_for((int64_t)n_dense_cells * TPB), TPB, 0, stream>>>(out->cells, n_dense_cells, idx, rc, out->table,
                                                                                          (unsigned char *)flags.ptr, (unsigned long long *)words.ptr);
            CK(cudaGetLastError());
            unsigned long long gone = 0;
            CK(cudaMemcpyAsync(&gone, (unsigned long long *)words.ptr + 1, sizeof(gone), cudaMemcpyDeviceToHost, stream));
            CK(cudaStreamSynchronize(stream));
            n_dense_nnz -= (int64_t)gone;
        }
        // units of one or two cells
        {
            Scratch heads;
            CK(heads.reserve(sizeof(int32_t) * (size_t)n_dense_cells));
            tb = 0;
            CK(cub::DeviceSelect::If(nullptr, tb, counting, (int32_t *)heads.ptr, d_n_sel, n_dense_cells, UnitHead{out->cells}, stream));
            CK(tmp.reserve(tb));
            CK(cub::DeviceSelect::If(tmp.ptr, tb, counting, (int32_t *)heads.ptr, d_n_sel, n_dense_cells, UnitHead{out->cells}, stream));
            int n_units = 0;
            CK(cudaMemcpyAsync(&n_units, d_n_sel, sizeof(int), cudaMemcpyDeviceToHost, stream));
            CK(cudaStreamSynchronize(stream));
            CK(pool_alloc(&out->units, (size_t)n_units));
            unit_fill_kernel<<<grid_for(n_units), TPB, 0, stream>>>(out->cells, (const int32_t *)heads.ptr, n_dense_cells, n_units, out->units);
            CK(cudaGetLastError());
            out->n_units = n_units;
        }
        const int64_t n_sparse = nnz - n_dense_nnz;
        if (n_sparse > 0) {
            CK(pool_alloc(&out->perm_s, (size_t)n_sparse));
            CK(pool_alloc(&out->rows_s, (size_t)n_sparse));
            CK(pool_alloc(&out->cols_s, (size_t)n_sparse));
            tb = 0;
            CK(cub::DeviceSelect::If(nullptr, tb, counting, out->perm_s, d_n_sel, n, NotDense{(unsigned char *)flags.ptr}, stream));
            CK(tmp.reserve(tb));
            CK(cub::DeviceSelect::If(tmp.ptr, tb, counting, out->perm_s, d_n_sel, n, NotDense{(unsigned char *)flags.ptr}, stream));
            gather2_kernel<<<grid_for(n_sparse), TPB, 0, stream>>>(out->perm_s, d_rows, d_cols, n_sparse, out->rows_s, out->cols_s);
            CK(cudaGetLastError());
        }
        out->n_cells = n_dense_cells;
        out->n_dense_nnz = n_dense_nnz;
        out->n_sparse = n_sparse;
        return cudaStreamSynchronize(stream);
    };
    cudaError_t e = body();
    if (e != cudaSuccess) out->release();
    return e;
}

cudaError_t build_dense_cells(const int32_t *d_rows, const int32_t *d_cols, const int64_t *d_row_ptr, int64_t nnz,
                              int64_t M, int64_t N, float min_density, float min_share, DensePlan *out,
                              cudaStream_t stream)
{
    const double grid = (double)((M + DENSE_CELL_ROWS - 1) / DENSE_CELL_ROWS) * (double)((N + DENSE_CELL_COLS - 1) / DENSE_CELL_COLS);
    auto build = 3.0 * grid < 4.0e9 ? build_dense_cells_k<uint32_t> : build_dense_cells_k<unsigned long long>;
    return build(d_rows, d_cols, d_row_ptr, nnz, M, N, min_density, min_share, out, stream);
}

// ---------------------------------------------------------------------------
// Reference-layout tiling tables (test hook)
// ---------------------------------------------------------------------------
namespace {

// Head of a (column tile, row) segment in tiled order.
__global__ void seg_flag_kernel(const int32_t *__restrict__ rows_t, const int32_t *__restrict__ cols_t, int64_t nnz,
                                int col_tile, int32_t *flag)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x)
        flag[j] = (j == 0 || rows_t[j] != rows_t[j - 1] || cols_t[j] / col_tile != cols_t[j - 1] / col_tile) ? 1 : 0;
}

// tile_begin[t] = first tiled index whose tile id is >= t, for t in [0, n_slots).
__global__ void tile_begin_kernel(const int32_t *__restrict__ cols_t, int64_t nnz, int col_tile, int n_slots,
                                  int32_t *tile_begin)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_slots; t += gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = nnz;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (cols_t[mid] / col_tile < t) lo = mid + 1; else hi = mid;
        }
        tile_begin[t] = (int32_t)lo;
    }
}

// Per nonzero: tile-local active-row index; per segment: active_row entry and
// block-table entries; per tile: number of active rows.
__global__ void tiling_tables_kernel(const int32_t *__restrict__ rows_t, const int32_t *__restrict__ cols_t,
                                     const int32_t *__restrict__ flag, const int32_t *__restrict__ segid,
                                     const int32_t *__restrict__ tile_begin, int64_t nnz, int64_t M, int col_tile,
                                     int panel_rows, int64_t max_blk, int32_t *t_rows, int32_t *active_row,
                                     int32_t *block_table, int32_t *n_actv_row)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x) {
        const int T = cols_t[j] / col_tile;
        const int32_t tb = tile_begin[T], te = tile_begin[T + 1];
        const int32_t a = segid[j] - segid[tb];  // inclusive scan: the tile's first segment has local index 0
        if (t_rows) t_rows[j] = a;
        if (flag[j] && active_row) active_row[(int64_t)T * M + a] = rows_t[j];
        const bool seg_tail = (j + 1 == nnz) || flag[j + 1];
        if (seg_tail) {
            const bool last_in_tile = (j + 1 == te);
            if (block_table) {
                if ((a + 1) % panel_rows == 0) block_table[(int64_t)T * max_blk + (a + 1) / panel_rows - 1] = (int32_t)(j + 1);
                else if (last_in_tile) block_table[(int64_t)T * max_blk + (a + 1) / panel_rows] = (int32_t)(j + 1);
            }
            if (last_in_tile && n_actv_row) n_actv_row[T] = a + 1;
        }
    }
}

// The reference writes slot 0 of the NEXT tile's block table at the start of
// every tile with the current tile's start index (util.h:289-292).
__global__ void block_table_prewrite_kernel(const int32_t *__restrict__ tile_begin, int n_loop, int64_t max_blk,
                                            int32_t *block_table)
{
    for (int T = blockIdx.x * blockDim.x + threadIdx.x; T < n_loop; T += gridDim.x * blockDim.x)
        block_table[(int64_t)(T + 1) * max_blk] = (T == 0) ? 0 : tile_begin[T];
}

}  // namespace

cudaError_t export_reference_tiling(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t M, int64_t N,
                                    int panel_rows, int col_tile, const TilingTables &out, cudaStream_t stream)
{
    const int64_t ntile_c = N / col_tile + 1;
    const int64_t n_loop = (N + col_tile - 1) / col_tile;  // tiles the reference loop visits
    const int64_t max_blk = M / panel_rows + 1;
    const size_t n = (size_t)(nnz > 0 ? nnz : 1);

    Scratch idx;  // perm | rows_t | cols_t | flag | segid | local row ids
    CK(idx.reserve(sizeof(int32_t) * 6 * n));
    int32_t *perm = (int32_t *)idx.ptr, *rows_t = perm + n, *cols_t = rows_t + n, *flag = cols_t + n, *segid = flag + n;
    int32_t *lrow = segid + n;
    CK(build_tiled_order(d_rows, d_cols, nnz, N, col_tile, perm, rows_t, cols_t, stream));

    Scratch tabs;  // tile_begin[ntile_c+2] | n_actv[ntile_c] | block_table[(ntile_c+1)*max_blk]
    const size_t tb_n = (size_t)ntile_c + 2, bt_n = (size_t)((ntile_c + 1) * max_blk);
    CK(tabs.reserve(sizeof(int32_t) * (tb_n + (size_t)ntile_c + bt_n)));
    int32_t *tile_begin = (int32_t *)tabs.ptr, *n_actv = tile_begin + tb_n, *block_table = n_actv + ntile_c;
    CK(cudaMemsetAsync(tabs.ptr, 0, tabs.bytes, stream));
    Scratch act;
    int32_t *active = nullptr;
    if (out.active_row) {
        CK(act.reserve(sizeof(int32_t) * (size_t)(M * ntile_c > 0 ? M * ntile_c : 1)));
        CK(cudaMemsetAsync(act.ptr, 0, act.bytes, stream));
        active = (int32_t *)act.ptr;
    }

    tile_begin_kernel<<<grid_for(ntile_c + 1), TPB, 0, stream>>>(cols_t, nnz, col_tile, (int)(ntile_c + 1), tile_begin);
    CK(cudaGetLastError());
    if (nnz > 0) {
        seg_flag_kernel<<<grid_for(nnz), TPB, 0, stream>>>(rows_t, cols_t, nnz, col_tile, flag);
        CK(cudaGetLastError());
        size_t tmp_bytes = 0;
        CK(cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, flag, segid, (int)nnz, stream));
        Scratch tmp;
        CK(tmp.reserve(tmp_bytes));
        CK(cub::DeviceScan::InclusiveSum(tmp.ptr, tmp_bytes, flag, segid, (int)nnz, stream));
        CK(cudaStreamSynchronize(stream));
    }
    block_table_prewrite_kernel<<<grid_for(n_loop), TPB, 0, stream>>>(tile_begin, (int)n_loop, max_blk, block_table);
    CK(cudaGetLastError());
    if (nnz > 0) {
        tiling_tables_kernel<<<grid_for(nnz), TPB, 0, stream>>>(rows_t, cols_t, flag, segid, tile_begin, nnz, M,
                                                               col_tile, panel_rows, max_blk, lrow,
                                                               active, block_table, n_actv);
        CK(cudaGetLastError());
    }
    // copy out.  lastIdx_tile[t] = tile_begin[t] for t <= n_loop; the slot past the
    // loop (present when N is a multiple of col_tile) stays zero.
    auto d2h = [&](void *dst, const void *src, size_t bytes) {
        return dst ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream) : cudaSuccess;
    };
    if (nnz > 0) {
        CK(d2h(out.tiled_ind, perm, sizeof(int32_t) * nnz));
        CK(d2h(out.t_cols, cols_t, sizeof(int32_t) * nnz));
    }
    CK(cudaStreamSynchronize(stream));
    if (out.lastIdx_tile) {
        CK(cudaMemcpyAsync(out.lastIdx_tile, tile_begin, sizeof(int32_t) * (size_t)(n_loop + 1), cudaMemcpyDeviceToHost, stream));
        for (int64_t t = n_loop + 1; t <= ntile_c; ++t) out.lastIdx_tile[t] = 0;
    }
    CK(d2h(out.lastIdx_block_tile, block_table, sizeof(int32_t) * bt_n));
    CK(d2h(out.n_actv_row, n_actv, sizeof(int32_t) * (size_t)ntile_c));
    if (active) CK(d2h(out.active_row, active, sizeof(int32_t) * (size_t)(M * ntile_c)));
    if (nnz > 0) CK(d2h(out.t_rows, lrow, sizeof(int32_t) * nnz));
    CK(cudaStreamSynchronize(stream));
    if (out.max_active_row) {
        int32_t mx = 0;
        // small table: reduce on the host from the copied counts
        int32_t *tmp_host = out.n_actv_row;
        std::vector<int32_t> local;
        if (!tmp_host) {
            local.resize((size_t)ntile_c);
            CK(cudaMemcpy(local.data(), n_actv, sizeof(int32_t) * (size_t)ntile_c, cudaMemcpyDeviceToHost));
            tmp_host = local.data();
        }
        for (int64_t t = 0; t < ntile_c; ++t) mx = tmp_host[t] > mx ? tmp_host[t] : mx;
        *out.max_active_row = mx;
    }
    return cudaSuccess;
}

}  // namespace sddmm
