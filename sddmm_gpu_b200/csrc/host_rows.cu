// Row upload from mapped host memory: the GPU reads the listed rows of a
// row-major host array over PCIe and writes them to the same rows of a device
// array.  An SDDMM reads only the rows of W and H that a nonzero touches; on
// graph matrices close to half of the rows are untouched, and a plain
// cudaMemcpy of the whole array moves them all the same (the reference does,
// HiPC18/src/sddmm.cu:71-73).  The host array must be page-locked and mapped into
// the device's address space (every cudaHostAlloc / cudaHostRegister allocation
// is, under unified addressing); the caller checks that before launching.
//
// Few, small CTAs on purpose: the kernel is bound by the PCIe link, not by the
// SMs, and it shares the SMs with the SDDMM kernels of earlier chunks.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace sddmm {

namespace {

constexpr int UP_TPB = 256;
constexpr int UP_ROWS = 4;  // rows a warp moves together: 4 x 16 bytes in flight per lane

__global__ void __launch_bounds__(UP_TPB)
upload_rows_kernel(const char *__restrict__ src, char *__restrict__ dst, const int32_t *__restrict__ list,
                   int64_t n_rows, int row_bytes)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * UP_TPB + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * UP_TPB) >> 5;
    const int pieces = row_bytes >> 4;  // 16-byte pieces per row (row_bytes = 4K, K a multiple of 4)
    for (int64_t q = warp * UP_ROWS; q < n_rows; q += n_warps * UP_ROWS) {
        int64_t off[UP_ROWS];
#pragma unroll
        for (int j = 0; j < UP_ROWS; ++j)
            off[j] = q + j < n_rows ? (int64_t)__ldg(list + q + j) * row_bytes : -1;
        for (int c = lane; c < pieces; c += 32) {
            uint4 v[UP_ROWS];
#pragma unroll
            for (int j = 0; j < UP_ROWS; ++j)
                if (off[j] >= 0) v[j] = __ldcs(reinterpret_cast<const uint4 *>(src + off[j]) + c);
#pragma unroll
            for (int j = 0; j < UP_ROWS; ++j)
                if (off[j] >= 0) __stcs(reinterpret_cast<uint4 *>(dst + off[j]) + c, v[j]);
        }
    }
}

// One launch of the host-operand path: the used rows of W and of H in their ranges and a range of S values, read from
// mapped host memory.  A warp takes 16 rows at a time, lists the used ones and moves their 16-byte pieces, eight per lane
// in flight; S moves in tiles of 2048 values.  No list of rows has to exist: a mark per column and the row pointer do, so
// the first call of a plan pays two small kernels instead of two compactions and their waits.  Bound by the link: 45 to 50
// GB/s of 256- to 512-byte rows (56 GB/s for whole arrays).  Measured against a copy per array, R-MAT patterns (us a call):
// 19 K nonzeros K = 32 77 -> 37; 411 K, K = 64 430 -> 289; 1.5 M, K = 128 2336 -> 1640; 11.2 M, K = 68 8880 -> 6050.
constexpr int UP_S_TILE = 2048;
constexpr int UP_DEPTH = 8;  // 16-byte loads in flight per lane
constexpr int UP_TILE = 16;  // rows of a warp at a time: 8 to 32 measure alike, 2 is 5 % slower

__device__ __forceinline__ void upload_row_tile(const UploadRows &u, int64_t tile, int lane, unsigned char *list)
{
    const int64_t r0 = u.begin + tile * UP_TILE, r = r0 + lane;
    bool used = lane < UP_TILE && r < u.end;
    if (used && u.col_used) used = u.col_used[r] != 0;
    if (used && u.row_ptr) used = u.row_ptr[r + 1] > u.row_ptr[r];
    const unsigned mask = __ballot_sync(0xffffffffu, used);
    if (used) list[__popc(mask & ((1u << lane) - 1u))] = (unsigned char)lane;
    __syncwarp();
    const unsigned pieces = (unsigned)u.row_bytes >> 4, total = (unsigned)__popc(mask) * pieces;
    for (unsigned i0 = lane; i0 < total; i0 += 32 * UP_DEPTH) {
        uint4 v[UP_DEPTH];
        size_t off[UP_DEPTH];
#pragma unroll
        for (int k = 0; k < UP_DEPTH; ++k) {
            const unsigned i = i0 + 32 * k;
            if (i < total) {
                const unsigned q = i / pieces;
                off[k] = (size_t)(r0 + list[q]) * (unsigned)u.row_bytes + (size_t)(i - q * pieces) * 16;
                v[k] = __ldcs(reinterpret_cast<const uint4 *>(u.src + off[k]));
            }
        }
#pragma unroll
        for (int k = 0; k < UP_DEPTH; ++k)
            if (i0 + 32 * k < total) *reinterpret_cast<uint4 *>(u.dst + off[k]) = v[k];
    }
    __syncwarp();
}

__global__ void __launch_bounds__(UP_TPB)
upload_operands_kernel(UploadRows a, UploadRows b, const float *__restrict__ s_src, float *__restrict__ s_dst, int64_t s_count)
{
    __shared__ unsigned char lists[UP_TPB / 32][UP_TILE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t ta = (a.end - a.begin + UP_TILE - 1) / UP_TILE, tb = (b.end - b.begin + UP_TILE - 1) / UP_TILE, ts = (s_count + UP_S_TILE - 1) / UP_S_TILE;
    for (int64_t t = (int64_t)blockIdx.x * (UP_TPB / 32) + warp; t < ta + tb + ts; t += (int64_t)gridDim.x * (UP_TPB / 32)) {
        if (t < ta) {
            upload_row_tile(a, t, lane, lists[warp]);
        } else if (t < ta + tb) {
            upload_row_tile(b, t - ta, lane, lists[warp]);
        } else {
            const int64_t j0 = (t - ta - tb) * UP_S_TILE, n = s_count - j0 < UP_S_TILE ? s_count - j0 : UP_S_TILE;
            const int n4 = (int)(n / 4);
            for (int i = lane; i < n4; i += 32)
                reinterpret_cast<float4 *>(s_dst + j0)[i] = __ldcs(reinterpret_cast<const float4 *>(s_src + j0) + i);
            if (lane < (int)(n - 4 * n4)) s_dst[j0 + 4 * n4 + lane] = __ldcs(s_src + j0 + 4 * n4 + lane);
        }
    }
}

// 32 x 32 tiles through shared memory: coalesced reads along n, coalesced writes along K.
__global__ void __launch_bounds__(256)
transpose_operand_kernel(const float *__restrict__ src, float *__restrict__ dst, int64_t n, int K)
{
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
    const int64_t n_tiles_n = (n + 31) / 32;
    const int64_t n_tiles = n_tiles_n * ((K + 31) / 32);
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int64_t r0 = (t % n_tiles_n) * 32;
        const int k0 = (int)(t / n_tiles_n) * 32;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const int k = k0 + ty + j;
            const int64_t r = r0 + tx;
            tile[ty + j][tx] = (k < K && r < n) ? src[(int64_t)k * n + r] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const int64_t r = r0 + ty + j;
            const int k = k0 + tx;
            if (r < n && k < K) dst[r * K + k] = tile[tx][ty + j];
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_transpose_operand(const float *src_kmajor, float *dst_rowmajor, int64_t n, int K, cudaStream_t stream)
{
    if (n == 0 || K == 0) return cudaSuccess;
    const int64_t n_tiles = ((n + 31) / 32) * ((K + 31) / 32);
    const unsigned grid = (unsigned)(n_tiles < 148 * 16 ? n_tiles : 148 * 16);
    transpose_operand_kernel<<<grid, 256, 0, stream>>>(src_kmajor, dst_rowmajor, n, K);
    return cudaGetLastError();
}

cudaError_t launch_upload_operands(const UploadRows &a, const UploadRows &b, const float *s_src, float *s_dst, int64_t s_count,
                                   int n_ctas, cudaStream_t stream)
{
    const int64_t tiles = (a.end - a.begin + UP_TILE - 1) / UP_TILE + (b.end - b.begin + UP_TILE - 1) / UP_TILE +
                          (s_count + UP_S_TILE - 1) / UP_S_TILE;
    if (tiles <= 0) return cudaSuccess;
    const int64_t blocks = (tiles + UP_TPB / 32 - 1) / (UP_TPB / 32);
    upload_operands_kernel<<<(unsigned)(blocks < n_ctas ? blocks : n_ctas), UP_TPB, 0, stream>>>(a, b, s_src, s_dst, s_count);
    return cudaGetLastError();
}

cudaError_t launch_upload_rows(const float *mapped_host, float *dev, const int32_t *d_row_list, int64_t n_rows, int K,
                               int n_ctas, cudaStream_t stream)
{
    if (n_rows == 0) return cudaSuccess;
    upload_rows_kernel<<<(unsigned)n_ctas, UP_TPB, 0, stream>>>(reinterpret_cast<const char *>(mapped_host),
                                                               reinterpret_cast<char *>(dev), d_row_list, n_rows, K * 4);
    return cudaGetLastError();
}

}  // namespace sddmm
