// GPU binning pass: everything the reference prepares on the host before its
// launch loop (make_CSR, TiledMatrix, rewrite_matrix_1D -- HiPC18/src/util.h:52-65,
// 131-153, 267-343), done on the device from the row-sorted COO.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "common.cuh"
#include "pool.hpp"

namespace sddmm {

// Device scratch whose lifetime is one binning call.
struct Scratch {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaError_t reserve(size_t n);
    void release();
    ~Scratch() { release(); }
};

// First look at the indices (see plan_scan_kernel): out_mapped[0] / [1] = first unsorted / out-of-range nonzero or
// ULLONG_MAX, [2] = rows with at least one nonzero, [3] = the kernel's time in ns.  words: PLAN_WORDS device words that
// init_plan_words has set up once.
constexpr int PLAN_WORDS = 5;
cudaError_t init_plan_words(unsigned long long *words);
cudaError_t scan_coo(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t M, int64_t N, unsigned long long *words,
                     unsigned long long *out_mapped, cudaStream_t stream);

// row_ptr[r] = first nonzero of row r (M + 1 entries, empty rows repeat).
cudaError_t build_row_ptr(const int32_t *d_rows, int64_t nnz, int64_t M, int64_t *d_row_ptr, cudaStream_t stream);

// d_used[c] = 1 for the columns that hold a nonzero, 0 for the others.
cudaError_t mark_used_cols(const int32_t *d_cols, int64_t nnz, int64_t N, unsigned char *d_used, cudaStream_t stream);

// A few entries of a device array (at.v = positions) to mapped host memory.
constexpr int PICK_MAX = 64;
struct PickAt {
    int64_t v[PICK_MAX];
};
cudaError_t pick_values(const int32_t *d_array, const PickAt &at, int n, unsigned long long *out_mapped, cudaStream_t stream);

// Number of distinct columns (marks a byte per column, then counts).
cudaError_t count_distinct_cols(const int32_t *d_cols, int64_t nnz, int64_t N, int64_t *host_out,
                                cudaStream_t stream);

// Stable partition of the nonzeros by column tile (tile = col / col_tile):
// d_perm[j] = input index of the j-th nonzero in tiled order (the reference's
// tiled_ind, util.h:301), d_rows_t/d_cols_t the permuted indices.
cudaError_t build_tiled_order(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t N,
                              int col_tile, int32_t *d_perm, int32_t *d_rows_t, int32_t *d_cols_t,
                              cudaStream_t stream);

// Work items over the processing-order arrays: maximal runs of nonzeros that
// share a column tile and a row panel (row / panel_rows), each cut into pieces of
// at most item_nnz nonzeros, plus the list of the distinct rows of every item
// (what the producer warp stages).  Allocates *d_items and *d_item_rows
// (cudaMalloc) and sets *n_items / *n_item_rows.
cudaError_t build_work_items(const int32_t *d_rows_p, const int32_t *d_cols_p, int64_t nnz,
                             int panel_rows, int col_tile, int item_nnz, WorkItem **d_items,
                             int64_t *n_items, int32_t **d_item_rows, int64_t *n_item_rows,
                             cudaStream_t stream);

// Ascending list of the rows of S that hold at least one nonzero (from the row
// pointer) or of the columns that do (from the column indices): the rows of W / H
// that an SDDMM actually reads.  Allocates *d_list (cudaMalloc) and sets *n_list.
cudaError_t build_used_row_list(const int64_t *d_row_ptr, int64_t M, int32_t **d_list, int64_t *n_list,
                                cudaStream_t stream);
cudaError_t build_used_col_list(const int32_t *d_cols, int64_t nnz, int64_t N, int32_t **d_list, int64_t *n_list,
                                cudaStream_t stream);

// Sort COO triples on the device, in place: by (a, b) keeping the input order of
// equal pairs (stable), or -- tie_by_value -- by (a, b, value), the order
// std::sort gives whole (a, b, value) tuples.  d_a / d_b are the major / minor
// index arrays (rows / cols, or cols / rows for a transposing sort).
cudaError_t sort_coo(int32_t *d_a, int32_t *d_b, float *d_v, int64_t nnz, bool tie_by_value, cudaStream_t stream);

// Hub-column hints for the ring kernel: d_cols_hinted[j] = d_cols_p[j] with bit 31
// set when the column is among the most popular ones whose rows of H together fit
// budget_bytes (chosen by exact column degree, most popular first).
cudaError_t build_hub_column_hints(const int32_t *d_cols_p, int64_t nnz, int64_t N, int64_t row_bytes,
                                   int64_t budget_bytes, int32_t *d_cols_hinted, int64_t *n_hub_cols,
                                   int *degree_threshold, cudaStream_t stream);

// Dense-cell classification.  S is cut into cells of DENSE_CELL_ROWS x
// DENSE_CELL_COLS -- over compacted (nearly) full rows, then compacted (nearly)
// full columns, then the regular grid; a cell holding at least min_density of its
// positions is "dense" and is computed as a small dense product by the dense-cell
// kernel, the nonzeros of all other cells form a row-sorted remainder that goes
// through the gather kernels with a permutation.  Nothing is built (n_cells == 0)
// when the dense cells would hold less than min_share of the nonzeros.
struct DensePlan {
    DenseCell *cells = nullptr;   // one descriptor per dense cell
    int64_t n_cells = 0;
    // Cells of the same rows in twos (consecutive ones, from the first cell of those rows on; the last one may be alone).  Also where each could
    // have an SM to itself (masks of K = 128, 77 to 145 cells, in twos / one by one, us: 1,211 tokens 16.3 / 16.3, 2,000 18.4 / 22.1, 3,000 15.3 / 17.5).
    DenseUnit *units = nullptr;
    int64_t n_units = 0;
    // Row-mask form of a cell (DenseCell::cls bit 8 set): per cell row a 64-bit column mask and the input positions of
    // its nonzeros as at most two runs: the nonzero in column c sits at popc(mask below c) past row_base.x, or past
    // row_base.y from column row_span >> 16 on (64: one run; the lowest byte of row_span: first column).  Valid for cells in which the nonzeros of every row have
    // ascending columns and at most one gap in their input positions (cells of compacted columns of a (row, col)-sorted input: the gap is the
    // band between them), or input positions that go up with the columns (CELL_RUNS, which goes by that alone: cells of the
    // regular grid; each column missing is one that went to the compacted full columns).  All other cells are in table form: the input position of every entry of the cell, -1 where S
    // holds nothing.  (A second nonzero of the same row and column is not in its cell then but in the remainder.)  A table is 32 KB, read twice, where
    // lists of 6 bytes a nonzero were read once.  Rows with their columns in random order, lists and one cell to a product / this, us: masks, K = 64,
    // 5,000 tokens 31 / 36, 20,000 113 / 125, 28,546 without global tokens 110 / 113, 65,536 435 / 485;  cells 0.3 and 0.6 full, 4,096 x 4,096, K = 64 71 / 67, 130 / 111,
    // K = 128 98 / 72, 138 / 117;  0.3 full, 16,384 x 16,384 1145 / 1340, K = 128 1536 / 1420.
    unsigned long long *row_mask = nullptr;  // [n_cells][DENSE_CELL_ROWS]
    int2 *row_base = nullptr;                // [n_cells][DENSE_CELL_ROWS]
    uint32_t *row_span = nullptr;            // [n_cells][DENSE_CELL_ROWS]
    int32_t *table = nullptr;                // [n_table_cells][DENSE_CELL_ROWS][DENSE_CELL_COLS]
    int64_t n_table_cells = 0;
    int64_t n_dense_nnz = 0;
    int32_t *rows_s = nullptr, *cols_s = nullptr, *perm_s = nullptr;  // remainder: indices and input positions
    int64_t n_sparse = 0;
    int32_t *dense_rows = nullptr, *dense_cols = nullptr;  // ids of the compacted full rows / columns
    int64_t n_dense_rows = 0, n_dense_cols = 0;
    void release();
};
// a cell is dense if it is a quarter full; cells are used if they hold half of S
constexpr float DENSE_MIN_FILL = 0.25f, DENSE_MIN_SHARE = 0.5f;
cudaError_t build_dense_cells(const int32_t *d_rows, const int32_t *d_cols, const int64_t *d_row_ptr, int64_t nnz,
                              int64_t M, int64_t N, float min_density, float min_share, DensePlan *out,
                              cudaStream_t stream);

// Reference-layout tiling tables (test hook); see sddmm_plan_export_tiling.
struct TilingTables {
    int32_t *t_rows, *t_cols, *tiled_ind, *lastIdx_tile, *lastIdx_block_tile, *active_row, *n_actv_row;
    int32_t *max_active_row;
};
cudaError_t export_reference_tiling(const int32_t *d_rows, const int32_t *d_cols, int64_t nnz, int64_t M,
                                    int64_t N, int panel_rows, int col_tile, const TilingTables &host_out,
                                    cudaStream_t stream);

}  // namespace sddmm
