// Gather kernel: the SDDMM of any K that is a multiple of 4, with or without a plan.
//
// The 32 lanes of a warp are sets of L lanes; a set takes a run of consecutive nonzeros and works on one nonzero at a
// time: lane l of the set holds the 16-byte pieces l, l + L, ... (F of them) of the W row and of the H row, so one
// load instruction of a set covers L * 16 consecutive bytes of one row.  H rows are loaded straight into registers, B
// nonzeros ahead of their use; the W row stays in registers until the row of S changes.  Rows, columns and S values of
// a step (8 nonzeros per set) are loaded one step ahead, one nonzero per lane, and spread by shuffles (STAGED: columns through shared memory); the 8 partial
// sums of a lane are reduced by one transposed butterfly, after which lane l stores nonzero l of the set.
//
// What bounds it.  Every nonzero brings one row of H from L2 (or L1, or DRAM) to its SM: 4K bytes, 16.7 TB/s at most
// over all SMs (a bare copy loop).  Latency is hidden by warps, not by a pipeline inside the warp: few registers per
// thread and many resident warps (24 to 48 per SM, __launch_bounds__ below) move more bytes than deeper batches with
// fewer warps (K = 128, 16.1 M nonzeros of an R-MAT matrix: 0.53 ms at 40 warps with one nonzero in flight per set,
// 0.59 ms at 24 warps with two, 0.64 ms at 16 warps with four).  Next to no shared memory (32 or 64 bytes a warp for
// the columns of a step, K = 324 to 384, 644 to 768 and 900 to 1024): the rest is L1, which serves the
// hub columns of a power-law matrix, and nothing is issued beyond the load, the packed FMAs (two per instruction) and
// 1/8 of a butterfly -- 9 warp instructions per nonzero at K = 128 where the shared-memory ring needed 34.  Grids are
// not persistent: a warp's share is 8, 16 or 32 nonzeros per set (4 where sets of four lanes are many), the hardware's block scheduler
// evens out the rest, and there is no work counter to clear before the launch.
//
// Measured against the shared-memory ring and panel kernels (R-MAT, 16.1 M nonzeros, 1 M x 1 M, and 4.1 M nonzeros,
// 300 K x 250 K; us before -> after):  K = 32: 250 -> 185, K = 64: 480 -> 296, K = 128: 832 -> 540, K = 256: 1250 ->
// 1146;  K = 100: 590 -> 135, K = 192: 752 -> 187, K = 300: 1233 -> 283, K = 512: 599 -> 522, K = 768: 2775 -> 820.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "device_utils.cuh"
#include "gather_index.hpp"

namespace sddmm {

using namespace dev;

namespace {

constexpr int GA_TPB = GATHER_TPB;
// Launched beside the kernel before it in the stream (the remainder of a matrix with dense cells): the persistent block of the dense-cell
// kernel leaves an SM 7,900 registers, room for two warps of any shape here (32 to 128 threads measure alike).  65,536-token mask, 0.3 M of
// 44 M nonzeros left over, K = 64: 180 us after the cells, 168 beside them; 12,777 tokens 37 -> 29.6.
constexpr int GA_TPB_BESIDE = 64;
constexpr int FEW_EACH = 2;  // nonzeros of a set (sddmm_gather_few_kernel)

// L lanes per nonzero, F 16-byte pieces per lane, B nonzeros of a set in flight, RB nonzeros per reduction, CTAS
// resident blocks per SM asked of the compiler.  EXACT: the L * F pieces are the row (no predicate on the last one).
// PF: the W rows of the next step are prefetched into L1.  BF16: W and H hold bfloat16 (a piece is 8 values).  STAGED: the columns of a step come from shared memory, two
// loads for 8, in place of a shuffle each: where a nonzero is six pieces of a lane or more (one in flight) that is faster, else slower (us, shuffles / this: K = 1024 0.75 M nonzeros,
// documents x words 163 / 141, 0.2 M 59.6 / 53.2, 0.6 M 159 / 151;  K = 768 106 / 101, 46.3 / 44.3, 112 / 109;  K = 384 62.0 / 59.8, 1.6 M 148 / 146;  but K = 896, 1.6 M 320 / 344,
// K = 256, 16.1 M 1080 / 1177, K = 128 520 / 642).
template <int L_, int F_, int B_, int RB_, bool EXACT_, bool PF_, int CTAS_, bool BF16_ = false, bool STAGED_ = false>
struct GatherShape {
    static constexpr bool STAGED = STAGED_;
    static constexpr int L = L_, F = F_, B = B_, RB = RB_, CTAS = CTAS_;
    static constexpr bool EXACT = EXACT_, PF = PF_, BF16 = BF16_;
    static constexpr int NB = L < 8 ? L : 8;  // nonzeros of a set per step
    static constexpr int G = 32 / L;          // sets of a warp
    static_assert(NB % RB == 0 && RB % B == 0 && RB <= L, "step geometry");
};

// A lane's share of the W row.
template <class S>
struct WShare {
    u64x2 v[S::F];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int f = 0; f < S::F; ++f) v[f] = u64x2{0, 0};
    }
    __device__ __forceinline__ void load(const char *wp, bool last_ok)
    {
#pragma unroll
        for (int f = 0; f < S::F; ++f)
            if (f < S::F - 1 || last_ok) v[f] = ldg_u64x2(wp + f * S::L * 16);
    }
    __device__ __forceinline__ float dot(const u64x2 (&h)[S::F]) const
    {
        if constexpr (S::BF16) {
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
            for (int f = 0; f < S::F; ++f) {
                fma_bf16x2((unsigned)v[f].a, (unsigned)h[f].a, s0, s1);
                fma_bf16x2((unsigned)(v[f].a >> 32), (unsigned)(h[f].a >> 32), s2, s3);
                fma_bf16x2((unsigned)v[f].b, (unsigned)h[f].b, s0, s1);
                fma_bf16x2((unsigned)(v[f].b >> 32), (unsigned)(h[f].b >> 32), s2, s3);
            }
            return (s0 + s1) + (s2 + s3);
        } else {
            unsigned long long a0 = 0, a1 = 0;  // two fp32 sums each
#pragma unroll
            for (int f = 0; f < S::F; ++f) {
                a0 = ffma2(v[f].a, h[f].a, a0);
                a1 = ffma2(v[f].b, h[f].b, a1);
            }
            return fold2(a0) + fold2(a1);
        }
    }
};

// What is multiplied and what becomes of a dot product: whole rows, the product stored (STORE) or stored through perm, the result of nonzero
// j to P[perm[j]], scaled by sval[perm[j]] (PERM); or one pass over some columns of rows that are `pitch` bytes apart (PASS): stored by
// the first pass, added to P by the later ones (`add`) -- by a reduction that nothing waits for, or, in the last pass (`finish`), read, added and scaled.
// red.global.add.f32 makes zeros of subnormal numbers, P's own among them.  Beside a part of 2^-100 and more that is less than its rounding; a smaller part is
// read, added and stored (every entry has one writer), a part that is zero is not added.  (All parts that way: graph of 97 M nonzeros, K = 256 8.6 -> 9.05 ms.)
enum GatherMode { STORE, PERM, PASS };

// pieces: 16-byte pieces of a row that are multiplied.  run_len: nonzeros of a set, a multiple of S::NB.
template <class S, GatherMode MODE>
__global__ void __launch_bounds__(GA_TPB, S::CTAS)
sddmm_gather_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, const int32_t *__restrict__ perm,
                    const float *__restrict__ sval, const char *__restrict__ W, const char *__restrict__ H,
                    float *__restrict__ P, unsigned nnz, int pieces, unsigned pitch, bool add, bool finish, unsigned run_len, unsigned long long *clock, unsigned meet_from)
{
    clock_begin(clock);
    constexpr bool HAS_PERM = MODE == PERM;
    const unsigned row_bytes = MODE == PASS ? pitch : (unsigned)pieces * 16u;  // from one row to the next
    constexpr int L = S::L, F = S::F, B = S::B, RB = S::RB, NB = S::NB, G = S::G;
    const int lane = threadIdx.x & 31, lig = lane & (L - 1), set = lane / L;
    const unsigned warp0 = gather_warp(blockIdx.x, blockDim.x, threadIdx.x) * (G * run_len);  // first nonzero of this warp
    if (warp0 >= nnz) return;
    const char *H_lane = H + lig * 16, *W_lane = W + lig * 16;
    const bool last_ok = S::EXACT || lig + (F - 1) * L < pieces;
    unsigned setmask = 0;  // lane 0 of every set
#pragma unroll
    for (int g = 0; g < G; ++g) setmask |= 1u << (g * L);

    __shared__ __align__(16) int step_cols[S::STAGED ? GA_TPB / 32 : 1][S::STAGED ? G * NB : 1];
    int *const my_cols = step_cols[S::STAGED ? threadIdx.x >> 5 : 0] + (S::STAGED ? set * NB : 0);
    WShare<S> w;
    w.clear();
    const int il = lig & (NB - 1);  // lanes >= NB of a set mirror a nonzero
    unsigned j = warp0 + set * run_len + il;
    auto at = [&](unsigned x) { return x < nnz ? x : nnz - 1; };  // past the end the last nonzero is read again, never stored
    int r, c, dst = 0;
    float s = 1.f;
    {
        const unsigned a = at(j);
        r = __ldg(rows + a);
        c = __ldg(cols + a);
        if (HAS_PERM) dst = __ldg(perm + a);
        else if (sval) s = __ldg(sval + a);
    }
    int cur = -1;  // row of the set's nonzero before this step
#pragma unroll 1
    for (unsigned step = run_len / NB; step > 0; --step) {
        int rn = 0, cn = 0, dn = 0;
        float sn = 1.f;
        if (step > 1) {
            const unsigned a = at(j + NB);
            rn = __ldg(rows + a);
            cn = __ldg(cols + a);
            if (HAS_PERM) dn = __ldg(perm + a);
            else if (sval) sn = __ldg(sval + a);
        }
        int before = __shfl_up_sync(FULL, r, 1, L);
        if (lig == 0) before = cur;
        const unsigned changed = __ballot_sync(FULL, r != before && lig < NB);
        cur = __shfl_sync(FULL, r, NB - 1, L);
        if (S::PF && step > 1) {
            int b2 = __shfl_up_sync(FULL, rn, 1, L);
            if (lig == 0) b2 = cur;
            if (rn != b2 && lig < NB) {
                const char *wp = W + (size_t)(unsigned)rn * row_bytes;
                for (unsigned o = 0; o < (unsigned)pieces * 16u; o += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(wp + o));
            }
        }
        if (HAS_PERM && sval) s = __ldg(sval + dst);
        float sum = 0.f;
        // (volatile: it is to be under way while the rows of H are, not waited for at the end of the step)
        if (MODE == PASS && add && finish && lig < NB) asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(sum) : "l"(P + at(j)));
        float res = 0.f;
        int cs[NB];
        if constexpr (S::STAGED) {
            static_assert(NB == 8, "two loads of four");
            __syncwarp();
            if (lig < NB) my_cols[lig] = c;
            __syncwarp();
#pragma unroll
            for (int x = 0; x < NB; x += 4) {
                const int4 t = *reinterpret_cast<const int4 *>(my_cols + x);
                cs[x] = t.x;
                cs[x + 1] = t.y;
                cs[x + 2] = t.z;
                cs[x + 3] = t.w;
            }
        }
#pragma unroll
        for (int h0 = 0; h0 < NB; h0 += RB) {
            float acc[RB];
#pragma unroll
            for (int b = 0; b < RB; b += B) {
                u64x2 h[B][F];
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const unsigned cj = S::STAGED ? (unsigned)cs[h0 + b + i] : (unsigned)__shfl_sync(FULL, c, h0 + b + i, L);
                    const char *hp = H_lane + (size_t)cj * row_bytes;
#pragma unroll
                    for (int f = 0; f < F; ++f)
                        h[i][f] = (f < F - 1 || last_ok) ? ldg_u64x2(hp + f * L * 16) : u64x2{0, 0};
                }
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const int x = h0 + b + i;
                    if (changed & (setmask << x)) {  // uniform over the warp: nonzero x of some set opens a row
                        const unsigned rj = (unsigned)__shfl_sync(FULL, r, x, L);
                        if ((changed >> (set * L + x)) & 1u) w.load(W_lane + (size_t)rj * row_bytes, last_ok);
                    }
                    acc[b + i] = w.dot(h[i]);
                }
            }
            reduce_transposed<L, RB>(acc, lig);
            // the sum of nonzero h0 + q of the set is in its lanes q (L / RB) and following
            const float t = RB == L ? acc[0] : __shfl_sync(FULL, acc[0], (lig & (RB - 1)) * (L / RB), L);
            if (RB == NB || il / RB == h0 / RB) res = t;
        }
        if (lig < NB && j < nnz) {
            if (MODE == PASS && add && !finish) {
                // (all of it predicated: with a branch around the rare addition 97 M nonzeros took 8.74 ms in place of 8.52)
                const unsigned small = fabsf(res) < 0x1p-100f;
                asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(P + j), "f"(res), "r"(small) : "memory");
                asm volatile("{\n\t.reg .pred p;\n\t.reg .f32 t;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.global.f32 t, [%0];\n\t@p add.rn.f32 t, t, %1;\n\t@p st.global.f32 [%0], t;\n\t}" ::"l"(P + j),
                             "f"(res), "r"((unsigned)(small && res != 0.f)) : "memory");
            } else {
                P[HAS_PERM ? (unsigned)dst : j] = (MODE == PASS ? sum + res : res) * s;
            }
        }
        j += NB;
        r = rn;
        c = cn;
        s = sn;
        dst = dn;
    }
    // (launched beside the kernel before it: that one is done when this one is)
    if (HAS_PERM && blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    clock_end(clock, meet_from);
}

// Few nonzeros, two for each set: rows of W and of H are asked for together, where the kernel above waits for an H row after the other and for the W row of every row of S
// that a step opens.  (All four rows of a set at once at F = 1; from F = 2 on the compiler keeps 32 to 40 registers and the second nonzero's rows follow the first's.)  The sums are
// the same, bit for bit: the same pieces to the same lanes, reduced in the same order.  What bounds it: three latencies, indices, rows, the wait
// for the call.  Synchronous calls, us, above / this: uniform, 16,777 nonzeros, K = 32 14.2 / 13.3, K = 64 14.5 / 13.6, K = 128 14.4 / 14.1;  4,000, K = 32, 128, 512 14.2 / 13.1, 14.0 /
// 13.6, 14.3 / 14.1;  40,000, K = 64 14.5 / 14.0;  R-MAT, 70,000, K = 32 14.7 / 14.2.  One or four for each set: 13.3, 13.7 and 13.6, 14.1 in the first two.
template <int L, int F, bool EXACT>
__global__ void __launch_bounds__(GA_TPB)
sddmm_gather_few_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, const float *__restrict__ sval,
                        const char *__restrict__ W, const char *__restrict__ H, float *__restrict__ P, unsigned nnz, int pieces,
                        unsigned long long *clock, unsigned meet_from)
{
    clock_begin(clock);
    using S = GatherShape<L, F, 1, 1, EXACT, false, 1>;
    constexpr int G = S::G, U = FEW_EACH;
    const int lane = threadIdx.x & 31, lig = lane & (L - 1), set = lane / L;
    const unsigned first = gather_warp(blockIdx.x, GA_TPB, threadIdx.x) * (G * U);  // nonzero u of a set: first + u G + set
    if (first >= nnz) return;
    const unsigned row_bytes = (unsigned)pieces * 16u;
    const char *H_lane = H + lig * 16, *W_lane = W + lig * 16;
    const bool last_ok = S::EXACT || lig + (F - 1) * L < pieces;
    unsigned r[U], c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const unsigned j = first + u * G + set, a = j < nnz ? j : nnz - 1;
        r[u] = (unsigned)__ldg(rows + a);
        c[u] = (unsigned)__ldg(cols + a);
    }
    // what this lane stores, if anything
    const unsigned mine = first + lig / (L / U) * G + set;
    const bool stores = lig % (L / U) == 0 && mine < nnz;
    float s = 1.f;
    if (stores && sval) s = __ldg(sval + mine);
    u64x2 h[U][F];
    WShare<S> w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const char *hp = H_lane + (size_t)c[u] * row_bytes;
#pragma unroll
        for (int f = 0; f < F; ++f) h[u][f] = f < F - 1 || last_ok ? ldg_u64x2(hp + f * L * 16) : u64x2{0, 0};
        w[u].clear();
        w[u].load(W_lane + (size_t)r[u] * row_bytes, last_ok);
    }
    float acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = w[u].dot(h[u]);
    reduce_transposed<L, U>(acc, lig);
    if (stores) P[mine] = acc[0] * s;
    clock_end(clock, meet_from);
}

// Rows of more than 256 pieces (K > 1024): a warp per nonzero, both rows in passes of 32 pieces.  The W row is read again for
// every nonzero, from L1: 9 TB/s of H rows on 1.9 M nonzeros of an R-MAT matrix, beside as much of W.
// Against the row-panel kernel, which stages W in shared memory (us, panel / this): R-MAT, 0.23 M nonzeros, K = 1028 460 / 100,
// 2048 490 / 192, 4096 879 / 366;  4.1 M nonzeros 5167 / 2017, 5985 / 4143, 11010 / 8561;  documents x words, 0.75 M nonzeros 731 /
// 311, 1009 / 577, 1372 / 1064.
template <bool HAS_PERM>
__global__ void __launch_bounds__(GA_TPB)
sddmm_gather_long_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, const int32_t *__restrict__ perm,
                         const float *__restrict__ sval, const char *__restrict__ W, const char *__restrict__ H,
                         float *__restrict__ P, unsigned nnz, int pieces, unsigned long long *clock, unsigned meet_from)
{
    clock_begin(clock);
    constexpr int U = 4;
    const int lane = threadIdx.x & 31;
    const unsigned j = gather_warp(blockIdx.x, GA_TPB, threadIdx.x);
    if (j >= nnz) return;
    const char *wp = W + (size_t)(unsigned)__ldg(rows + j) * pieces * 16 + lane * 16;
    const char *hp = H + (size_t)(unsigned)__ldg(cols + j) * pieces * 16 + lane * 16;
    unsigned long long a0 = 0, a1 = 0;
    for (int q = lane; q < pieces; q += 32 * U) {
        u64x2 h[U], w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = q + 32 * u < pieces;
            h[u] = in ? ldg_u64x2(hp + 512 * u) : u64x2{0, 0};
            w[u] = in ? ldg_u64x2(wp + 512 * u) : u64x2{0, 0};
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            a0 = ffma2(w[u].a, h[u].a, a0);
            a1 = ffma2(w[u].b, h[u].b, a1);
        }
        hp += 512 * U;
        wp += 512 * U;
    }
    float a = fold2(a0) + fold2(a1);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) a += __shfl_xor_sync(FULL, a, off);
    if (lane == 0) {
        const unsigned dst = HAS_PERM ? (unsigned)__ldg(perm + j) : j;
        if (sval) a *= __ldg(sval + dst);
        P[dst] = a;
    }
    clock_end(clock, meet_from);
}

struct GatherCall {
    const int32_t *rows, *cols, *perm;
    const float *sval;
    const char *W, *H;
    float *P;
    unsigned nnz;
    int pieces;
    bool pass;         // one of several passes (perm null)
    unsigned pitch;
    bool add, finish;
    int sm_count;
    unsigned long long *clock;
    bool beside;
    cudaStream_t stream;
    bool few_lanes = false, large_h = false, awaited = false;
};

template <class S>
cudaError_t launch_few(const GatherCall &c)
{
    const unsigned per_block = GA_TPB / S::L * FEW_EACH, blocks = (c.nnz + per_block - 1) / per_block;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(GA_TPB);
    cfg.stream = c.stream;
    return cudaLaunchKernelEx(&cfg, sddmm_gather_few_kernel<S::L, S::F, S::EXACT>, c.rows, c.cols, c.sval, c.W, c.H, c.P, c.nnz, c.pieces, c.clock,
                              last_wave(blocks, (unsigned)c.sm_count * (2048 / GA_TPB)));
}

template <class S, GatherMode MODE>
cudaError_t launch_mode(const GatherCall &c)
{
    // only the last piece of a lane is predicated: the ones before it have to lie inside the row
    if (c.pieces > S::L * S::F || c.pieces <= S::L * (S::F - 1)) return cudaErrorInvalidValue;
    // Up to 10 MB of H rows a call is a few latencies long, which count where it is waited for.  (Above it W rows that are read again for every nonzero cost more: synchronous calls
    // of 80,000 nonzeros, uniform, K = 64 15.3 / 15.0, K = 128 16.3 / 16.9;  40,000, K = 128 14.8 / 15.1, K = 256 16.0 / 16.7;  150,000, R-MAT, K = 32 15.2 / 15.3.  Asynchronous calls one
    // after the other take what the host needs to launch them, and that is more with the shorter kernel: 16,777 nonzeros, K = 32, 64 5.0 / 5.5, of 2.9 / 1.7, 3.0 / 1.9 on the GPU.)
    // (the shape of eight lanes and four pieces is taken from a million nonzeros on, and no call with bfloat16 operands asks)
    if constexpr (MODE == STORE && S::F <= 4 && !(S::L == 8 && S::F == 4) && !S::BF16)
        if (c.awaited && (uint64_t)c.nnz * (unsigned)c.pieces * 16u <= 10000000) return launch_few<S>(c);
    // A set's run.  A long one spreads what a run costs at its ends and keeps the W row over more nonzeros; the last wave of blocks, which
    // may be nearly empty, lasts as long as a run.  So by the nonzeros that there are for a resident set (us at runs of 8 / 16 / 32):
    // below 40: K = 32, 1.0 M nonzeros 18.6 / 21.1 / 27.3;  K = 64, 0.4 M 12.4 / 14.4 / 14.4, 0.7 M 19.6 / 20.7 / 24.0;  K = 128, 0.24 M 12.4 / 14.4 /
    // 14.2, 0.4 M, planned, called and closed 49.6 / 50.1 / 55.3;  K = 256, 0.18 M 18.0 / 17.5 / 19.2;  K = 512, 0.12 M 24.2 / 24.4 / 28.0;
    // from there on: K = 64, 1.6 M 51.8 / 48.5 / 51.8, 4.0 M 88.3 / 77.9 / 79.0;  K = 128, 1.0 M 43.1 / 41.0 / 44.4, 2.0 M 74.0 / 67.6 / 69.9;
    // K = 300, 1.0 M 79.9 / 76.0 / 84.9;  K = 256, 0.7 M 53.6 / 49.9 / 51.7, documents x words, 0.75 M 56.7 / 50.0 / 47.8;
    // two sets to a warp, from 256 on: K = 192, 2.5 M 122 / 109.5 / 108.6;  K = 300, 2.5 M 179 / 177 / 168;  K = 100, 4.1 M 149 / 130 / 125.
    const unsigned resident = (unsigned)c.sm_count * S::CTAS * (GA_TPB / 32) * S::G, share = c.nnz / resident;  // sets; nonzeros for each
    // a nonzero to a warp, 40 to 95 nonzeros for each (runs of 16 / 32): K = 256, 0.4 M 24.5 / 25.4, K = 512, 0.2 M 26.8 / 29.9, 0.22 M 24.8 / 28.7;  from there on: K = 256, 0.75 M 39.2 / 38.0,
    // K = 512, 0.6 M 74.0 / 72.2.
    unsigned run = share < 40 ? 8 : (S::L == 32 && (S::F > 4 || share >= 96)) || (S::L == 16 && share >= 256) ? 32 : 16;
    if (share < 8) run = S::NB;
    const unsigned tpb = c.beside ? GA_TPB_BESIDE : GA_TPB, per_block = run * S::G * (tpb / 32);
    const unsigned blocks = (unsigned)(((uint64_t)c.nnz + per_block - 1) / per_block);
    const unsigned meet_from = last_wave(blocks, (unsigned)c.sm_count * S::CTAS);
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(tpb);
    cfg.stream = c.stream;
    cfg.attrs = &attr;
    cfg.numAttrs = c.beside ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, sddmm_gather_kernel<S, MODE>, c.rows, c.cols, c.perm, c.sval, c.W, c.H, c.P, c.nnz, c.pieces, c.pitch, c.add,
                              c.finish, run, c.clock, meet_from);
}

template <class S>
cudaError_t launch_shape(const GatherCall &c)
{
    return c.perm ? launch_mode<S, PERM>(c) : c.pass ? launch_mode<S, PASS>(c) : launch_mode<S, STORE>(c);
}

// The shape for `pieces` pieces of a row: L * (F - 1) < pieces <= L * F, L small enough that a set's lanes
// are busy and large enough that F pieces of W and B * F of H stay in few registers.  Every line is the best of a sweep
// over (L, B, RB, prefetch, resident blocks) at a K of its range on the matrices named at the top of this file.
cudaError_t launch_pieces(const GatherCall &c)
{
    const int q = c.pieces;
#define GA_GO(L, F, B, RB, EXACT, PF, CTAS) return launch_shape<GatherShape<L, F, B, RB, EXACT, PF, CTAS>>(c)
    if (q <= 4) GA_GO(4, 1, 4, 4, false, false, 6);
    // Up to 16 pieces all eight sums of a step are reduced together, eight shuffles for 8 instead of ten; with 48 registers more blocks are resident.  us, four at
    // a time / this: K = 64 16.1 M nonzeros 285.7 / 279.9, 6.0 M 107.1 / 102.3, 1.5 M, columns alike 30.7 / 28.7, 0.2 M 9.0 / 8.2;  K = 56 6.0 M 110.1 / 103.8;  K = 32 6.0 M 72.4 /
    // 70.4, 1.6 M 22.4 / 20.9, documents x words, 0.7 M 12.0 / 10.5.  Passes, and rows of 52 to 64 columns of an H that is mostly read from DRAM, keep
    // four at a time (97 M nonzeros, 4.2 M rows of H: K = 256 7729 / 8641, K = 64 1805 / 1845; 1 M rows: above).
    if (q < 8) GA_GO(8, 1, 4, 8, false, false, 6);
    if (q == 8) GA_GO(8, 1, 4, 8, true, false, 6);
    if (q <= 12) GA_GO(4, 3, 2, 4, false, true, 4);
    // Where two or three waves of blocks are all, their number counts and a block's own time: four rows at a time on four resident blocks where that takes no more waves than two on five (a tenth
    // of a wave more is lost in the ends of the one before).  Same bits; us, two / four, and where the host waits: K = 64, uniform, 0.15 M nonzeros 6.2 / 6.6 (16.2 / 16.4), 0.175 M 6.4 / 8.2
    // (16.5 / 18.1), 0.26 M 10.3 / 10.3 (19.5 / 19.1), 0.3 M 10.3 / 10.3 (19.7 / 19.4), 0.35 M 10.3 / 12.3 (20.2 / 21.8), 0.45 M 12.9 / 12.3 (23.0 / 22.7);  K = 52, R-MAT, 0.205 M 8.2 / 9.7 (17.8 / 18.7).
    auto waves = [&](unsigned per_block, unsigned ctas, unsigned slack) {
        const unsigned blocks = c.nnz / per_block + 1, wave = (unsigned)c.sm_count * ctas;
        return (blocks - (blocks > slack ? slack : 0) + wave - 1) / wave;
    };
    const unsigned at_four = waves(256, 4, 0);
    if (q > 12 && q <= 16 && !c.pass && at_four > 1 && at_four <= 3 && at_four == waves(256, 5, (unsigned)c.sm_count / 2)) GA_GO(8, 2, 4, 8, false, false, 4);
    if (q < 16 && (c.pass || c.large_h)) GA_GO(8, 2, 4, 4, false, true, 4);
    if (q < 16) GA_GO(8, 2, 2, 8, false, true, 5);
    if (q == 16 && (c.pass || c.large_h)) GA_GO(8, 2, 4, 4, true, true, 4);
    if (q == 16) GA_GO(8, 2, 2, 8, true, false, 5);
    if (q <= 24) GA_GO(8, 3, 2, 8, false, true, 4);
    // Here sixteen lanes take two pieces each, 25 to 31 of the 32, or eight lanes four.  Eight lanes need fewer shuffles, but a wave of them is more nonzeros, and fewer warps: for
    // many nonzeros of an H that L1 holds little of (gather_passes).  K = 100, us, sixteen / eight: 6.0 M nonzeros 175.6 / 168.0, 4.1 M 126.6 / 121.5, 1.6 M 53.7 / 51.7, 1.5 M, columns
    // alike 51.4 / 47.4;  but 0.2 M 11.5 / 14.3, documents x words 0.75 M, 4,000 words 1.8 M 27.0 / 28.7, 59.9 / 61.7, and
    // 97 M of an H of 1.7 GB 3690 / 3863.
    if (q < 32 && c.few_lanes) GA_GO(8, 4, 1, 8, false, true, 4);
    if (q < 32) GA_GO(16, 2, 2, 8, false, true, 5);
    if (q == 32) GA_GO(16, 2, 2, 8, true, false, 5);
    if (q <= 48) GA_GO(16, 3, 2, 8, false, true, 4);
    if (q < 64) GA_GO(16, 4, 1, 8, false, true, 4);
    if (q == 64) GA_GO(32, 2, 2, 8, true, false, 5);
    if (q <= 80) GA_GO(16, 5, 1, 8, false, true, 4);
#define GA_STAGED(L, F, B, RB, EXACT, PF, CTAS) return launch_shape<GatherShape<L, F, B, RB, EXACT, PF, CTAS, false, true>>(c)
    if (q <= 96) GA_STAGED(16, 6, 1, 8, false, false, 4);
    if (q < 128) GA_GO(32, 4, 2, 8, false, true, 3);
    // (two at a time on three blocks / this, us: 0.75 M nonzeros, documents x words 69.9 / 65.8, 0.6 M 75.6 / 72.2, 1.6 M 182.4 / 179.9, 0.2 M 27.0 / 26.8, 32 K, uniform 10.3 / 8.2, 60 K 14.3 / 13.0;
    // two at a time where that takes no more waves, from the second on: 50 K 11.1 / 12.3, 78 K 15.3 / 16.4, documents x words, 50 K 8.5 / 10.3)
    const unsigned at_one = waves(64, 4, 0);
    if (q == 128 && at_one > 1 && at_one <= 3 && at_one == waves(64, 3, 0)) GA_GO(32, 4, 2, 8, true, true, 3);
    if (q == 128) GA_GO(32, 4, 1, 8, true, false, 4);
    if (q <= 160) GA_GO(32, 5, 1, 8, false, false, 4);
    if (q == 192) GA_STAGED(32, 6, 1, 8, true, false, 4);  // (0.75 M nonzeros 104.6 / 100.9)
    if (q <= 192) GA_STAGED(32, 6, 1, 8, false, false, 4);
    if (q <= 224) GA_GO(32, 7, 1, 8, false, false, 3);
    if (q <= 256) GA_STAGED(32, 8, 1, 8, false, false, 3);
#undef GA_STAGED
#undef GA_GO
    return cudaErrorInvalidValue;
}

}  // namespace

// (where the lines lie: launch_pieces)
GatherPasses gather_whole(int64_t nnz, int64_t N, int K)
{
    const int64_t h_bytes = N * K * 4;
    return {1, K, nnz >= 1000000 && h_bytes >= 8000000 && h_bytes < 300000000, h_bytes >= 500000000};
}

// Long rows in passes over their columns.  A pass multiplies `floats` columns of every row; its part of H is so much smaller that more
// of the gathers hit L2, and it runs on one of the shapes that take few registers.  Against that a pass costs the indices again and a
// sum in P that is written and read: 16 bytes a nonzero.  Sustained us, one pass -> passes of 64 / 96 / 192 (R-MAT unless said):
//   K = 256: 4.2 M rows of H, 97 M nonzeros 9330 (the ring kernel) -> 8340 / - / -, another GPU 8922 (one pass of this kernel) -> 8552 /
//   8669 / 8877; 50 M nonzeros 4740 -> 4676 / 4687 / 4757; 25 M 2421 -> 2514 / 2448 / 2502; 3 M rows, 36 M 3078 -> 3168 / 3111 / 3127;
//   1.5 M rows, 18 M 1409 -> 1532 / 1438 / 1454; K = 300, 1.5 M rows 1803 -> 2163 / 2016 / 1904
//   K = 384: 20 K rows 44 -> 74 / 63 / 47; 300 K 515 -> 587 / 506 / 494; 1.5 M 2578 -> 2224 / 2112 / 2114; 4.2 M 16233 -> 13008 / 12806 / 13466
//   K = 512: 300 K rows 607 -> 773 / 666 / 635; 700 K 1245 -> 1381 / 1253 / 1214; 1.5 M 3052 -> 3053 / 2894 / 2830
//   K = 768: 100 K rows, 1.2 M nonzeros 255 -> 392 / 295 / 255; 200 K, uniform, 2 M 972 -> 712 / 646 / 770; 150 K, uniform, 0.3 M 197 -> 228
//   / 190 / 217; 700 K, 8.4 M 2356 -> 2081 / 1836 / 1822; 1.5 M, 18 M 5688 -> 4545 / 4267 / 4212
//   few nonzeros, H of 1.6 and of 3.2 GB, one pass -> passes of 192 (K = 512 and 1024: see ring_few), all columns alike; R-MAT:
//   K = 384: 0.25 M 90 -> 91, 90 -> 92, 60 -> 63, 70 -> 71; 0.5 M 156 -> 153, 158 -> 156, 105 -> 105, 125 -> 124; 1 M 271 -> 253, 277 -> 262, 182 -> 172, 213 -> 202
//   K = 768: 0.25 M 167 -> 179, 169 -> 183, 107 -> 113, 126 -> 125; 0.5 M 296 -> 293, 300 -> 307, 187 -> 180, 223 -> 211; 1 M 522 -> 474, 531 -> 507, 327 -> 292, 387 -> 343
//   K = 1028: 20 K rows, 0.24 M 105 -> 205 / 143 / 134; 100 K, 1.2 M 548 -> 551 / 426 / 384; 1 M, 12 M 6685 -> 4807 / 4261 / 4189
// Where rows are no multiple of 128 bytes, neighbouring passes touch the same lines: a pass of 192 then costs a sixth more, and a last one
// of a few columns as much as a third of that (12 nonzeros a row; one pass -> 192, all columns alike, R-MAT).  It still pays up to 384 columns, and
// from 640 on, where one pass runs on few warps:
//   K = 324, H of 1.3 GB 2890 -> 2861, 1564 -> 1378;  3 GB 6826 -> 6879, 4172 -> 3598;   K = 392 2543 -> 2920, 1406 -> 1333;  6023 -> 7054, 3604 -> 3449
//   K = 452 2541 -> 2785, 1358 -> 1293;  6020 -> 6836, 3542 -> 3345;   K = 584 2490 -> 2755, 1273 -> 1237;  5904 -> 6799, 3417 -> 3225
//   K = 644 2705 -> 2674, 1453 -> 1237;  6384 -> 6683, 3908 -> 3122;   K = 780 2490 -> 2659, 1343 -> 1216;  5891 -> 6715, 3501 -> 3087;  0.6 GB 1092 -> 1008, 540 -> 536
//   K = 900 2707 -> 2523, 1546 -> 1188;  6366 -> 6463, 4013 -> 2995;   K = 1060 2677 -> 2451, 1930 -> 1168;  6394 -> 6364, 4817 -> 2919
// and with rows that are: K = 352 2662 -> 2425, 1445 -> 1221;  6265 -> 5880, 3785 -> 3085;   K = 416 2420 -> 2474, 1341 -> 1196;  5738 -> 5979, 3474 -> 3074
//   K = 512 2380 -> 2305, 1223 -> 1129;  5642 -> 5673, 3254 -> 2885;   K = 640 2382 -> 2261, 1162 -> 1098;  5647 -> 5624, 3334 -> 2793
// 193 to 320 columns, 16 nonzeros a row, one pass -> 64: K = 256, 4.3 GB 10612 -> 10663, 6403 -> 5979;  8.2 GB 20431 -> 21017, 12972 -> 12923;  16 GB 40877 -> 43462,
//   28282 -> 27961;   K = 320, 4.5 GB 11657 -> 11535, 6863 -> 6515;   K = 224, 4.1 GB 10898 -> 11299, 6617 -> 6412;   K = 196 12237 -> 16677, 7471 -> 8135;
//   K = 260 12684 -> 17282, 7300 -> 8052;   K = 300 14697 -> 19795, 8501 -> 9396
// In the order of column tiles a tile's rows of H stay in L2 as they are: K = 256, 67 M nonzeros, tiles of 65,536 columns, R-MAT 5470 -> 6932.  Longer rows gain
// all the same (their rows of W are read again for every tile): K = 512, 18 M, tiles of 32,768, one pass -> 192 10656 -> 8919, 3129 -> 3082.
GatherPasses gather_passes(int64_t nnz, int64_t N, int K, bool tiled, const float *sval, const float *P)
{
    const int64_t h_bytes = N * K * 4;
    const GatherPasses whole = gather_whole(nnz, N, K);
    if (sval && sval < P + nnz && P < sval + nnz) return whole;  // the first pass would overwrite S values that the last one needs
    int floats = K;
    if (K > 320) {
        const bool lines = K % 32 == 0;
        const bool pays = lines || K <= 384 || K > 1024 || (K > 640 && (K % 192 >= 32 || h_bytes < 1000000000));
        // (the shapes for 512 and 640 floats are the ones that hold their own longest)
        if (pays && nnz >= (h_bytes >= 1500000000 ? 500000 : 1000000) && h_bytes >= (K > 480 && K <= 640 ? 1000000000 : 400000000))
            floats = lines && N > 2000000 ? 96 : 192;
    } else if (K > 192 && K % 64 == 0 && !tiled && h_bytes >= 4000000000 && h_bytes < 8000000000 && nnz >= 16 * N) {
        floats = 64;
    }
    return floats < K ? GatherPasses{(K + floats - 1) / floats, floats} : whole;
}

cudaError_t launch_gather(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval, const float *W,
                          const float *H, float *P, int64_t nnz, int K, GatherPasses passes, int sm_count, unsigned long long *clock,
                          cudaStream_t stream, bool beside)
{
    if (perm) passes = {1, K, passes.few_lanes, passes.large_h};
    for (int pass = 0; pass < passes.n; ++pass) {
        const int k0 = pass * passes.floats, width = K - k0 < passes.floats ? K - k0 : passes.floats;
        for (int64_t j0 = 0; j0 < nnz; j0 += GATHER_SLICE) {
            GatherCall c;
            c.nnz = (unsigned)(nnz - j0 < GATHER_SLICE ? nnz - j0 : GATHER_SLICE);
            c.rows = rows + j0;
            c.cols = cols + j0;
            c.perm = perm ? perm + j0 : nullptr;
            c.sval = sval && !perm ? sval + j0 : sval;
            if (pass < passes.n - 1) c.sval = nullptr;  // the sum is scaled
            c.W = reinterpret_cast<const char *>(W + k0);
            c.H = reinterpret_cast<const char *>(H + k0);
            c.P = perm ? P : P + j0;
            c.pieces = width / 4;
            c.pass = passes.n > 1;
            c.pitch = (unsigned)K * 4u;
            c.add = pass > 0;
            c.finish = pass == passes.n - 1;
            c.sm_count = sm_count;
            c.clock = clock;
            c.beside = beside && j0 == 0;
            c.stream = stream;
            c.few_lanes = passes.few_lanes;
            c.large_h = passes.large_h;
            c.awaited = passes.awaited;
            cudaError_t e;
            if (c.pieces <= 256) {
                e = launch_pieces(c);
            } else {
                const unsigned blocks = gather_long_blocks(c.nnz), meet_from = last_wave(blocks, (unsigned)sm_count * 8);
                if (perm) sddmm_gather_long_kernel<true><<<blocks, GA_TPB, 0, stream>>>(c.rows, c.cols, c.perm, c.sval, c.W, c.H, c.P, c.nnz, c.pieces, clock, meet_from);
                else sddmm_gather_long_kernel<false><<<blocks, GA_TPB, 0, stream>>>(c.rows, c.cols, c.perm, c.sval, c.W, c.H, c.P, c.nnz, c.pieces, clock, meet_from);
                e = cudaGetLastError();
            }
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

// bfloat16 rows of 2K bytes.  16.1 M nonzeros, 1 M x 1 M, K = 256: 677 us widening to fp32 first, 569 us with the
// mixed-precision FMA (fewer registers: five resident blocks instead of four); K = 512: 1378 -> 1190.
bool gather_bf16_supports(int K) { return K == 256 || K == 512 || K == 1024; }

// Passes of 256 values, sustained us, the ring kernel / one pass / these: K = 1024, 0.3 M rows of H - / 544 / 583, 0.7 M 1394 / 1406 / 1405, 1 M 2775 / 2747 /
// 2600, 1.5 M 4320 / 4466 / 4119;  K = 512, 1.5 M 2036 / 2047 / 2038, 4.2 M 9298 / 9264 / 8920;  K = 256, 4.2 M 4864 / 4218 / -.
// From a million nonzeros and one for each row of H on; K = 1024 below a million on the rings (ring_few).  All columns alike, R-MAT: K = 512, H of 4.3 GB, 0.3 M nonzeros 68 / 66 / 78,
// 60 / 55 / 66; 1 M 179 / 177 / 188, 161 / 164 / 162; 3 M 490 / 488 / 483, 412 / 422 / 393;  K = 1024, 2.1 GB, 0.02 M 18.5 / 16.4 / 41; 0.3 M 128 / 136 / 154,
// 88 / 101 / 110; 1 M 345 / 337 / 349, 239 / 243 / 253; 3 M 934 / 896 / 872, 628 / 611 / 598;  4.3 GB, 1 M 351 / 342 / 368, 274 / 294 / 285; 3 M 953 / 913 / 934,
// 706 / 718 / 683.
GatherPasses gather_passes_bf16(int64_t nnz, int64_t N, int K, const float *sval, const float *P)
{
    const GatherPasses whole = {1, K};
    if (sval && sval < P + nnz && P < sval + nnz) return whole;
    return nnz >= 1000000 && nnz >= N && N * K * 2 >= (K >= 1024 ? 1900000000 : 4000000000) && K > 256 ? GatherPasses{K / 256, 256} : whole;
}

cudaError_t launch_gather_bf16(const int32_t *rows, const int32_t *cols, const int32_t *perm, const float *sval, const void *W,
                               const void *H, float *P, int64_t nnz, int64_t N, int K, int sm_count, unsigned long long *clock, cudaStream_t stream)
{
    if (nnz == 0) return cudaSuccess;
    if (nnz > INT32_MAX) return cudaErrorInvalidValue;  // plans hold fewer
    GatherPasses p = gather_passes_bf16(nnz, N, K, sval, P);
    if (perm) p = {1, K};
    for (int pass = 0; pass < p.n; ++pass) {
        GatherCall c = {rows, cols, perm, pass < p.n - 1 ? nullptr : sval, static_cast<const char *>(W) + 2 * pass * p.floats,
                        static_cast<const char *>(H) + 2 * pass * p.floats, P, (unsigned)nnz, p.floats / 8, p.n > 1, (unsigned)K * 2u, pass > 0,
                        pass == p.n - 1, sm_count, clock, false, stream};
        cudaError_t e = cudaErrorInvalidValue;
        if (p.floats == 256) e = launch_shape<GatherShape<16, 2, 2, 8, true, false, 5, true>>(c);
        else if (p.floats == 512) e = launch_shape<GatherShape<16, 4, 1, 8, true, true, 4, true>>(c);
        else if (p.floats == 1024) e = launch_shape<GatherShape<32, 4, 2, 8, true, true, 3, true>>(c);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace sddmm
