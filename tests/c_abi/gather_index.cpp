// Launch arithmetic of the gather kernel (csrc/gather_index.hpp) where 32-bit thread numbers would wrap: with a warp per nonzero a
// launch has 32 nnz threads.
#include <cstdio>
#include <initializer_list>

#include "gather_index.hpp"

using namespace sddmm;

int main()
{
    int failures = 0;
    const unsigned sizes[] = {1u, 8u, 9u, (1u << 27) - 1, 1u << 27, (1u << 27) + 1, (1u << 30) - 1, 1u << 30};
    for (unsigned nnz : sizes) {
        const unsigned blocks = gather_long_blocks(nnz);
        // every warp of a block has the nonzero after the warp before it, at the first and last blocks and around 2^32 threads
        unsigned long long bad = 0;
        const unsigned probes[] = {0, (1u << 24) - 1, 1u << 24, (1u << 24) + 1, blocks - 1};
        for (unsigned b : probes) {
            if (b >= blocks) continue;
            for (unsigned w = 0; w < GATHER_TPB / 32; ++w)
                for (unsigned lane : {0u, 31u})
                    bad += gather_warp(b, GATHER_TPB, w * 32 + lane) != (unsigned long long)b * (GATHER_TPB / 32) + w;
        }
        const bool covered = (unsigned long long)blocks * (GATHER_TPB / 32) >= nnz && (unsigned long long)(blocks - 1) * (GATHER_TPB / 32) < nnz;
        printf("%s: %u nonzeros, %u blocks, %llu wrong\n", bad == 0 && covered ? "ok" : "FAILED", nnz, blocks, bad);
        failures += bad != 0 || !covered;
    }
    return failures;
}
