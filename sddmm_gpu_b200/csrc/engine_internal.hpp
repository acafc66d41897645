// Internal layout of the engine's handle and plan (shared by engine.cu and the
// multi-GPU layer); the public surface is include/sddmm_b200.h.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "binning.cuh"
#include "common.cuh"
#include "pool.hpp"
#include "sddmm_b200.h"

using namespace sddmm;

// Host-operand pipeline: S is cut into at most this many chunks of consecutive nonzeros.
#define SDDMM_PIPE_MAX_CHUNKS 16

#define SDDMM_EVENT_PAIRS 8
#define SDDMM_WORK_COUNTERS 1024

struct sddmm_handle_s {
    int device = 0;
    int sm_count = 0;
    size_t smem_optin = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    // guards free_clocks and the owners of events, which a plan that another thread destroys leaves
    std::mutex owners;
    // event pairs around the kernels of synchronous calls that no kernel clock times, taken in turn; a plan's time is
    // read from its pair when it is asked for, or before another plan takes the pair
    cudaEvent_t ev_begin[SDDMM_EVENT_PAIRS] = {}, ev_end[SDDMM_EVENT_PAIRS] = {};
    sddmm_plan_s *ev_owner[SDDMM_EVENT_PAIRS] = {};
    int next_pair = 0;
    int *h_status = nullptr;  // status word of bounded waits, in mapped host memory
    int *d_status = nullptr;  // its device address
    // dynamic work distribution of the ring kernel: a counter for each launch, taken in turn, since launches on other streams may overlap
    unsigned long long *d_work_counters = nullptr;
    unsigned next_work_counter = 0;
    unsigned long long *work_counter() { return d_work_counters + next_work_counter++ % SDDMM_WORK_COUNTERS; }
    // kernel clocks (two words each) of plans whose last synchronous call was a single gather launch
    unsigned long long *d_clocks = nullptr;
    unsigned long long *d_plan_words = nullptr;                          // of scan_coo
    volatile unsigned long long *h_words = nullptr;                      // mapped: what plan-time kernels answer
    unsigned long long *d_words = nullptr;                               // its device address
    cudaEvent_t ev_plan[2] = {};
    DevicePool pool;  // memory given back by plans and calls
    std::vector<int> free_clocks;
    std::string last_error;
    // dense cells: 0 = fp32 FMA, 1 = 3xTF32 on mma.sync, 2 = 3xTF32 on tcgen05 / tensor memory (SDDMM_DENSE_TENSOR)
    int dense_mode = 2;
    // pipelined execution with host operands: compute and download streams, one
    // "uploaded" and one "computed" event per chunk (created on first use)
    cudaStream_t pipe_compute = nullptr, pipe_download = nullptr;
    cudaEvent_t pipe_uploaded[SDDMM_PIPE_MAX_CHUNKS] = {};
    cudaEvent_t pipe_started[SDDMM_PIPE_MAX_CHUNKS] = {}, pipe_computed[SDDMM_PIPE_MAX_CHUNKS] = {};  // timing events
    cudaEvent_t pipe_joined = nullptr;
    sddmm_plan_s *pipe_owner = nullptr;  // whose last call's times the chunk events hold
    bool pipeline = true;  // SDDMM_PIPELINE=0 keeps upload, kernel and download strictly one after the other
    // pipelined calls whose host operands are page-locked and mapped upload only the rows of
    // W and H that a nonzero touches, read by the GPU (SDDMM_SPARSE_UPLOAD=0: whole arrays by cudaMemcpy)
    bool sparse_upload = true;
    int upload_ctas = 0;  // CTAs of the upload kernel (SDDMM_UPLOAD_CTAS; default half the SMs)
    int64_t n_launches = 0;  // kernels launched through this handle by sddmm_execute / sddmm_upload_rows
};

struct sddmm_plan_s {
    sddmm_handle_s *h = nullptr;
    int64_t M = 0, N = 0, nnz = 0;
    int K = 0;
    bool sorted = true;   // by row; false only behind SDDMM_PLAN_SKIP_VALIDATION, and then nothing may look at the row pointer
    int col_tile = 0;     // == N (clamped) when there is a single column tile
    int n_col_tiles = 1;
    PanelConfig cfg{};
    // pattern, input order
    int32_t *d_rows = nullptr, *d_cols = nullptr;
    bool owns_rows = true, owns_cols = true;
    // pattern, tiled order (only when n_col_tiles > 1)
    int32_t *d_rows_t = nullptr, *d_cols_t = nullptr, *d_perm = nullptr;
    int64_t *d_row_ptr = nullptr;
    WorkItem *d_items = nullptr;     // row-panel kernel; built when it is first asked for (ensure_items)
    int64_t n_items = -1;
    int32_t *d_item_rows = nullptr;  // distinct rows of every item, concatenated
    int32_t *d_cols_hint = nullptr;  // processing-order columns with hub marks (ring kernel), or null (ensure_hints)
    int64_t hub_budget = 0;          // bytes of H rows to keep in L2 (0 = no marks)
    bool hints_built = false;
    // dense cells + row-sorted remainder (single-tile plans of locally dense matrices)
    DensePlan dense;
    int64_t n_hub_cols = 0;
    int64_t n_item_rows = 0;
    int64_t n_nonempty_rows = 0, n_nonempty_cols = -1;
    // staging for host operands (allocated on first use)
    float *d_W = nullptr, *d_H = nullptr, *d_S = nullptr, *d_P = nullptr;
    float *d_Wt = nullptr, *d_Ht = nullptr;  // device copies of K-major host operands, before their transposition
    int64_t device_bytes = 0;
    float plan_ms = 0.f, last_ms = -1.f;
    // work was enqueued that nothing has waited for yet; asynchronous calls: on which stream, on several
    bool pending = false, async_pending = false, async_mixed = false;
    cudaStream_t async_stream = nullptr;
    int clock = -1;              // index of this plan's kernel clock in the handle's array
    enum { MS_KNOWN, MS_IN_CLOCK, MS_IN_EVENTS, MS_IN_PIPE } ms_state = MS_KNOWN;  // where the last call's kernel time is
    int ev_pair = -1;
    // chunks of the host-operand pipeline (0 = not pipelined): nonzeros
    // [pipe_nnz[i], pipe_nnz[i+1]); filled by ensure_pipe
    int n_pipe = 0, pipe_step = 1;  // chunks; chunks that the last call took together
    bool pipe_ready = false;
    int64_t pipe_nnz[SDDMM_PIPE_MAX_CHUNKS + 1] = {};
    // rows of W chunk i uploads: [pipe_w_begin[i], pipe_w_end[i]) (empty when an earlier chunk brought them)
    int64_t pipe_w_begin[SDDMM_PIPE_MAX_CHUNKS] = {}, pipe_w_end[SDDMM_PIPE_MAX_CHUNKS] = {};
    bool setup_unwaited = false;  // the row pointer or the marks were enqueued by a call that nothing has waited for
    unsigned char *d_col_used = nullptr;  // marks of the columns that hold a nonzero (row upload of H)
    int32_t *d_used_rows = nullptr, *d_used_cols = nullptr;  // ascending ids of the rows / columns holding a nonzero
    int64_t n_used_rows = 0, n_used_cols = 0;
    int64_t last_h2d_bytes = 0, last_d2h_bytes = 0;  // moved by the last sddmm_execute
    bool last_h2d_used_cols = false;                 // and the rows of H of the columns that hold a nonzero (counted on request)
    const char *last_kernel = "none";                // kernels the last sddmm_execute launched
    float *d_spmm_scratch = nullptr;  // partial rows of SpMM / fused SDDMM->SpMM, allocated on first use
    // An asynchronous call that uses the scratch and that nothing has waited for: its stream, and once a plan's calls have been
    // seen on more than one stream (spmm_event_kept) the event at its end.
    bool spmm_running = false, spmm_event_kept = false;
    cudaStream_t spmm_stream = nullptr;
    cudaEvent_t spmm_done = nullptr;
};


namespace sddmm {
constexpr int N_KERNEL_CLOCKS = 1024;

// Whether launch_rows takes the ring kernel: it is the faster one for this plan, or forced.  permuted: perm is given.
bool rows_on_ring(const sddmm_plan_s *p, bool force_ring, bool permuted);
// SDDMM over nonzeros in the plan's processing order, [first, first + count): the ring kernel (rows_on_ring) or the gather
// kernel in as many passes as are best (beside: see launch_gather; awaited: see GatherPasses).  Launches beyond the first are counted here.
cudaError_t launch_rows(sddmm_plan_s *p, const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval,
                        const float *W, const float *H, float *P, int64_t first, int64_t count, bool force_ring,
                        unsigned long long *clock, cudaStream_t stream, bool beside = false, bool awaited = false);
}  // namespace sddmm
