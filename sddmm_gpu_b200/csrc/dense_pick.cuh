// The "pick" phase of the dense-cell kernels: the finished 128 x 64 block of a cell sits in shared
// memory (row-major, `stride` floats per row) and the cell's nonzeros take their entries, scale them
// by S and store them to P at their input positions.  NT threads (a multiple of 32), tid in [0, NT).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace sddmm {

template <int NT = 256>  // divides a quarter of the cell's entries
__device__ __forceinline__ void pick_block(const float *Ct, int stride, const DenseCell &dc, bool masked, bool runs, int64_t cell,
                                           int tid, const int32_t *__restrict__ table,
                                           const unsigned long long *__restrict__ row_mask,
                                           const int2 *__restrict__ row_base, const uint32_t *__restrict__ row_span, const float *__restrict__ sval,
                                           float *__restrict__ P)
{
    if (masked) {
        // Row r of the cell holds the columns of mask[r]; in column order its nonzeros are one or two runs of
        // consecutive input positions: the one in column c sits at popc(mask[r] below bit c) past base[r].x, or past
        // base[r].y from column span[r] >> 16 on; or (runs) as far past base[r].x as it is past the row's first column, span[r] & 255.  A warp takes four rows at a time, lane l the columns l and l + 32: the S
        // loads and the P stores of a row are a few contiguous runs.
        const unsigned long long *cm = row_mask + cell * DENSE_CELL_ROWS;
        const int2 *cb = row_base + cell * DENSE_CELL_ROWS;
        const uint32_t *cs = row_span + cell * DENSE_CELL_ROWS;
        const int lane = tid & 31, warp = tid >> 5;
        const unsigned below = (1u << lane) - 1u;
        for (int r0 = warp * 4; r0 < DENSE_CELL_ROWS; r0 += NT / 8) {
            unsigned lo[4], hi[4];
            int2 base[4];
            int split[4], c0[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const unsigned long long m = __ldg(cm + r0 + u);
                lo[u] = (unsigned)m;
                hi[u] = (unsigned)(m >> 32);
                base[u] = __ldg(cb + r0 + u);
                const uint32_t span = __ldg(cs + r0 + u);
                split[u] = (int)(span >> 16);
                c0[u] = (int)(span & 255u);
            }
            float s_lo[4], s_hi[4];
            int32_t p_lo[4], p_hi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                p_lo[u] = (lane < split[u] ? base[u].x : base[u].y) + __popc(lo[u] & below);
                p_hi[u] = (lane + 32 < split[u] ? base[u].x : base[u].y) + __popc(lo[u]) + __popc(hi[u] & below);
                if (runs) {
                    p_lo[u] = base[u].x + lane - c0[u];
                    p_hi[u] = p_lo[u] + 32;
                }
                s_lo[u] = s_hi[u] = 1.f;
                if (sval) {
                    if ((lo[u] >> lane) & 1u) s_lo[u] = __ldcs(sval + p_lo[u]);
                    if ((hi[u] >> lane) & 1u) s_hi[u] = __ldcs(sval + p_hi[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float *crow = Ct + (r0 + u) * stride;
                if ((lo[u] >> lane) & 1u) __stcs(P + p_lo[u], crow[lane] * s_lo[u]);
                if ((hi[u] >> lane) & 1u) __stcs(P + p_hi[u], crow[lane + 32] * s_hi[u]);
            }
        }
    } else {
        // table form: the input position of every entry
        const int32_t *t = table + dc.slot * (DENSE_CELL_ROWS * DENSE_CELL_COLS);
        for (int i = tid; i < DENSE_CELL_ROWS * DENSE_CELL_COLS; i += 4 * NT) {  // four independent entries per thread and trip
            int32_t o[4];
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = __ldg(t + i + u * NT);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = i + u * NT;
                v[u] = Ct[e / DENSE_CELL_COLS * stride + e % DENSE_CELL_COLS];
                if (sval && o[u] >= 0) v[u] *= __ldg(sval + o[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o[u] >= 0) P[o[u]] = v[u];
        }
    }
}

}  // namespace sddmm
