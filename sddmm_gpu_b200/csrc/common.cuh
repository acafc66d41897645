// Shared declarations of the sm_100a SDDMM engine (internal; the public surface
// is include/sddmm_b200.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <string>
#include <vector>

#include "sddmm_b200.h"

namespace sddmm {

// One unit of work of the row-panel kernel: a run of consecutive nonzeros (in the
// plan's processing order) whose rows all lie in [row_begin, row_begin + n_rows),
// n_rows <= the plan's panel height, so that the W rows they touch fit one
// shared-memory panel.  Built on the device by the binning pass.
struct WorkItem {
    int64_t nnz_begin;   // first nonzero (processing order)
    int64_t list_begin;  // offset of the item's distinct rows in the plan's item-row list
    int32_t nnz_count;
    int32_t row_begin;   // smallest row of the item
    int32_t n_rows;      // number of distinct rows (entries of the item-row list)
    int32_t reserved;
};

// A dense cell of S: rows [row0, row0 + DENSE_CELL_ROWS) x columns [col0, col0 +
// DENSE_CELL_COLS) (clipped).  cls 0: row0 indexes the list of compacted full rows;
// cls 1: col0 indexes the list of compacted full columns; cls 2: both are
// plain matrix coordinates.
constexpr int DENSE_CELL_ROWS = 128;
constexpr int DENSE_CELL_COLS = 64;
// Forms of a cell in DenseCell::cls, above the class: CELL_MASKED = the row-mask form (see DensePlan); CELL_RUNS = of those, a
// cell in which the input position of every row's nonzeros is their column plus a number of the row (columns may be missing: those
// that are in another cell); neither = the table form, the cell's input positions are table number `slot` of the plan.
constexpr int CELL_MASKED = 0x100, CELL_RUNS = 0x200;
struct DenseCell {
    int64_t slot;
    int32_t row0, col0;
    int32_t count;
    int32_t cls;
};
// One or two cells of the same rows: a product of the tcgen05 kernel.  number: of the cell or, in table form, of its table.
struct DenseUnit {
    int32_t number[2], n;
    int32_t row0, col0[2], cls[2];
};
struct DensePlan;

// The opt-in to more than 48 KB of dynamic shared memory (cudaFuncSetAttribute) is a
// property of a kernel ON ONE DEVICE: a process that drives several GPUs must make it
// on each of them.  One cache per kernel instantiation remembers the largest size
// already granted, per device ordinal; devices beyond the table are never cached.
struct SmemOptinCache {
    static constexpr int MAX_DEVICES = 64;
    std::atomic<size_t> granted[MAX_DEVICES];
    SmemOptinCache() { for (auto &g : granted) g.store(0, std::memory_order_relaxed); }
    bool needs(int device, size_t bytes) const
    {
        return device < 0 || device >= MAX_DEVICES || bytes > granted[device].load(std::memory_order_acquire);
    }
    void record(int device, size_t bytes)
    {
        if (device >= 0 && device < MAX_DEVICES) granted[device].store(bytes, std::memory_order_release);
    }
};

// Makes the opt-in for `kern` on the current device unless `cache` says it holds.
template <class Kern>
inline cudaError_t optin_dynamic_smem(Kern kern, size_t bytes, SmemOptinCache &cache)
{
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (!cache.needs(device, bytes)) return cudaSuccess;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cache.record(device, bytes);
    return e;
}

// Device status word written by kernels whose bounded waits give up.
enum DeviceStatus : int { DEV_OK = 0, DEV_MBARRIER_TIMEOUT = 1 };

struct PanelConfig {
    int panel_rows;      // rows of W per staged panel
    int item_nnz;        // nonzero budget of one work item
    int threads;         // CTA size
    int ctas_per_sm;     // resident CTAs per SM the launch is sized for
    size_t smem_bytes;   // dynamic shared memory per CTA
};

// Chooses panel height / item budget / CTA shape for a given K and hint.
PanelConfig choose_panel_config(int K, int panel_rows_hint, int sm_count, size_t smem_optin);

// Gather kernel (sddmm_gather.cu): any K % 4 == 0, no plan data needed; the default path.  perm as in launch_panel.
// clock: two device words that receive the kernel's start and end (clock_begin / clock_end), or null.
// beside (with perm only): may run beside the kernel before it in the stream, once that has signalled it; it ends no earlier.
// passes: the columns of W and H that a launch multiplies (without perm; with it there is one).  Every pass but the first adds to P.
struct GatherPasses {
    int n, floats;           // launches, columns of each (the last one may have fewer)
    bool few_lanes = false;  // the shape with fewer lanes for a nonzero, where there are two
    bool large_h = false;    // most rows of H come from DRAM
    bool awaited = false;    // by the host, as soon as it has been launched, with P in the GPU's memory
};
// One pass over whole rows of an H of N rows.
GatherPasses gather_whole(int64_t nnz, int64_t N, int K);
// What is best for an H of N rows; one pass where S values and P share memory.  tiled: the nonzeros are in the order of column tiles.
GatherPasses gather_passes(int64_t nnz, int64_t N, int K, bool tiled, const float *sval, const float *P);
cudaError_t launch_gather(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                          const float *W, const float *H, float *P, int64_t nnz, int K, GatherPasses passes, int sm_count,
                          unsigned long long *clock, cudaStream_t stream, bool beside = false);
// The same over operands stored in bfloat16 (rows of 2K bytes): K = 256, 512 or 1024.
bool gather_bf16_supports(int K);
GatherPasses gather_passes_bf16(int64_t nnz, int64_t N, int K, const float *sval, const float *P);
cudaError_t launch_gather_bf16(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval, const void *W,
                               const void *H, float *P, int64_t nnz, int64_t N, int K, int sm_count, unsigned long long *clock, cudaStream_t stream);

// Row-panel kernel: persistent CTAs walk the work items; the W rows an item
// touches (item_rows lists them) are staged into shared memory with bulk
// asynchronous copies (TMA, double-buffered on mbarriers) by a producer warp,
// H rows are gathered with software-pipelined 128-bit loads.
// perm == nullptr: P[j] = result of processing-order nonzero j (sval indexed the
// same way).  perm != nullptr: result of j goes to P[perm[j]], scaled by sval[perm[j]].
cudaError_t launch_panel(const WorkItem *items, int64_t n_items, const int32_t *item_rows,
                         const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                         const float *W, const float *H, float *P, int K,
                         const PanelConfig &cfg, int sm_count, int *dev_status,
                         cudaStream_t stream);

// dst[r*K + t] = src[t*n + r]: a K-major operand (K x n) into the row-major layout (n x K) the kernels read.
cudaError_t launch_transpose_operand(const float *src_kmajor, float *dst_rowmajor, int64_t n, int K, cudaStream_t stream);

// Rows [begin, end) of a row-major array in mapped, page-locked host memory that are to be copied to the same rows of a
// device array: those marked in col_used, those with a nonzero in row_ptr, or all of them (both null).  16-byte aligned.
struct UploadRows {
    const char *src = nullptr;
    char *dst = nullptr;
    const unsigned char *col_used = nullptr;
    const int64_t *row_ptr = nullptr;
    int64_t begin = 0, end = 0;
    int row_bytes = 16;
};
// Two such ranges and s_count floats (both addresses 16-byte aligned) in one launch; the GPU reads the host memory.
cudaError_t launch_upload_operands(const UploadRows &a, const UploadRows &b, const float *s_src, float *s_dst, int64_t s_count,
                                   int n_ctas, cudaStream_t stream);

// Copies the listed rows (K floats each) of a row-major array in mapped, page-locked
// host memory to the same rows of a device array; the GPU reads the host memory.
cudaError_t launch_upload_rows(const float *mapped_host, float *dev, const int32_t *d_row_list, int64_t n_rows, int K,
                               int n_ctas, cudaStream_t stream);

// Ring kernel: H rows gathered by bulk asynchronous copies (TMA) into per-warp
// shared-memory rings, work handed out dynamically through *work_counter (one
// device word, zeroed by the launcher).  K = 256, 512 or 1024.
bool ring_supports(int K);
// K that SDDMM_FLAG_KERNEL_RING takes.
inline bool rows_path_supports(int K) { return K == 32 || K == 64 || K == 128 || K == 256 || K == 512 || K == 1024; }
// Whether the ring kernel is the faster one for an H of N rows (see sddmm_ring.cu).
bool ring_preferred(int64_t N, int K);
bool ring_few(int64_t nnz, int row_bytes);  // ... also where the nonzeros are in input order
// cols_hinted: bit 31 of every column index marks a hub column (see build_hub_column_hints).
cudaError_t launch_ring(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                        const float *W, const float *H, float *P, int64_t nnz, int K, bool cols_hinted, int sm_count,
                        unsigned long long *work_counter, int *dev_status, cudaStream_t stream);

// The same TMA rings over operands stored in bfloat16 (rows of 2K bytes; products and sums in fp32):
// K = 256, 512, 1024 or 2048.  Opt-in, outside the fp32 tolerance contract.
bool ring_bf16_supports(int K);
cudaError_t launch_ring_bf16(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                             const void *W_bf16, const void *H_bf16, float *P, int64_t nnz, int K, bool cols_hinted, int sm_count,
                             unsigned long long *work_counter, int *dev_status, cudaStream_t stream);

// Dense-cell kernel: every dense cell is computed as the 128 x 64 block
// W[rows] * H[cols]^T -- fp32 FMAs, or (tensor) 3xTF32 on the tensor cores -- then
// the cell's nonzeros pick their entries: P[i] = block[r][c] (* sval[i]) for the nonzero at input position i.
cudaError_t launch_dense_cells(const DensePlan &d, const float *sval, const float *W, const float *H, float *P,
                               int64_t M, int64_t N, int K, bool tensor, int sm_count, cudaStream_t stream);

// The same dense cells on tcgen05: MMAs issued by one thread from shared-memory descriptors, accumulator in
// tensor memory (3xTF32).  dev_status receives DEV_MBARRIER_TIMEOUT if a bounded wait gives up.
cudaError_t launch_dense_cells_tc(const DensePlan &d, const float *sval, const float *W, const float *H, float *P, int64_t M, int64_t N,
                                  int K, int sm_count, int *dev_status, cudaStream_t stream);

// SpMM (W null) / fused SDDMM->SpMM (spmm.cu): device arrays, input order.  scratch: spmm_scratch_floats() floats for
// partial rows, the first spmm_counter_floats() of them zeroed once (every call leaves them zero); clock as in launch_gather.  K a multiple of 4, at most 1024 (spmm_supports).
struct SpmmCall {
    const int32_t *rows, *cols;
    const int64_t *row_ptr;
    const float *val;  // P values (SpMM) or S values (fused); null: ones
    const float *W, *H;
    float *P_out;      // fused: receives P, or null
    float *Y, *scratch;
    int64_t M, N, nnz;
    int K;
    unsigned long long *clock;
};
bool spmm_supports(int K);
size_t spmm_counter_floats(int64_t nnz, int64_t N, int K, int sm_count);
size_t spmm_scratch_floats(int64_t nnz, int64_t N, int K, int sm_count);
int spmm_passes(int64_t nnz, int64_t N, int K);  // launches of an SpMM
cudaError_t launch_spmm(const SpmmCall &call, int sm_count, int64_t *n_launches, cudaStream_t stream);

// float64 recomputation of every stride-th nonzero on the device (see check.cu).
struct CheckResult {
    unsigned long long n_checked;
    unsigned long long n_bad;      // sampled nonzeros with |P - ref| > tol * max(|ref|, A), or not finite
    double max_scaled_err;         // max |P - ref| / max(|ref|, A)
};
cudaError_t launch_check_result(const int32_t *rows, const int32_t *cols, const float *sval, const float *W, const float *H,
                                const float *P, int64_t nnz, int K, int64_t stride, double tol, CheckResult *d_out,
                                int sm_count, cudaStream_t stream);

// Self-test of the bounded-wait path: one warp waits (with a short poll limit) on
// an mbarrier that nothing ever arrives on, gives up, records DEV_MBARRIER_TIMEOUT
// in *dev_status and returns normally.  Nothing faults, traps or hangs.
cudaError_t launch_wait_timeout_probe(int *dev_status, cudaStream_t stream);

}  // namespace sddmm
