// Launch arithmetic of the gather kernel, the same code on the host and on the device.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SDDMM_HD __host__ __device__ __forceinline__
#else
#define SDDMM_HD inline
#endif

namespace sddmm {

constexpr unsigned GATHER_TPB = 256;
// Nonzeros of one launch: the kernels count them in 32 bits.  (The kernel clock times one launch, so longer calls are timed by
// events.)
constexpr int64_t GATHER_SLICE = 1ll << 30;

// Number of a warp within its launch.  Not (block * threads per block + thread) / 32: a launch with a warp per nonzero has 2^32
// threads at 2^27 nonzeros.
SDDMM_HD unsigned gather_warp(unsigned block, unsigned threads_per_block, unsigned thread)
{
    return block * (threads_per_block / 32) + thread / 32;
}
// Blocks of a launch with a warp per nonzero.
SDDMM_HD unsigned gather_long_blocks(unsigned nnz)
{
    return (unsigned)(((uint64_t)nnz + GATHER_TPB / 32 - 1) / (GATHER_TPB / 32));
}

// First of the blocks that can be the last to run, of a grid of which `resident` blocks run at a time.
SDDMM_HD unsigned last_wave(unsigned blocks, unsigned resident) { return blocks > resident ? blocks - resident : 0; }

}  // namespace sddmm
