// The step after SDDMM in its callers: Y = P * H with P on the sparsity pattern of S
// (SpMM), and the fused form Y = (S o (W H^T)) * H that never writes P to memory.
//
// The reference stops at SDDMM; its README motivates SDDMM as "a core component in
// reformulations of many machine learning algorithms" (README.md:1), where the
// sampled product is at once multiplied back into a dense factor.  These kernels
// have therefore no counterpart to be pinned to: the parity tests use a CPU loop of
// the same definition (oracle/sddmm_oracle.c, oracle_spmm*).
//
//     Y[r, :] = sum over the nonzeros i of row r of  p_i * H[col_i, :]
//     p_i     = Pval[i]                                    (SpMM; 1 when Pval is NULL)
//             = (sum_t W[r, t] H[col_i, t]) * Sval[i]      (fused; Sval NULL = 1)
//
// Shape.  The lane sets of the gather kernel (sddmm_gather.cu): a set of L lanes takes a RUN of consecutive nonzeros, one
// at a time, lane l holding the 16-byte pieces l, l + L, ... of the H row, of the Y row being summed and (fused) of the
// W row; B nonzeros of H are in flight per set.  When the row of S changes the set stores the finished row of Y and
// starts the next one.  Runs are equal shares of the nonzeros whatever the rows look like, so a power-law matrix
// loads every warp alike, and nothing is built per plan.
//
// A row that crosses a run boundary is in parts: what the run in which it ends has of it (its head) and what the runs before that one have (their tails).  The runs of a
// block follow one another, so a block adds up its own parts: tails go to shared memory, heads to Y for the time being, and behind a barrier the run in which a row ends
// adds the tails before it, in order.  (Y of the fused form may be W: each row of W is used up before its row of Y is stored.  Heads go to scratch then, ON_W, since other runs may
// still read the row of W.  Heads in scratch for all calls: 1 to 10 % slower, K = 32 10 %, K = 256 3 %, since what picks the address sits in the loop.)  Only the row that a block begins with and the one that goes on behind it concern other blocks.  Their parts
// go to scratch -- 2 b: block b's part of a row that ends in it, 2 b + 1: of one that goes on -- and the block that arrives last at a row (a counter per row) adds them
// up in order: no atomics on Y, the result does not depend on scheduling, and there is no second launch (a fix-up kernel took a third of a call with ten thousand
// nonzeros).  Parts are added in groups of 16 or 8 blocks, each by its last block, and the groups by the last of those, so that a row of hundreds of blocks does not end in one long
// chain.  With a fence, a counter and two reads of the row pointer at both ends of every run, a run's ends took some 8 us, what 40 nonzeros at K = 64 take (us, then / now:
// SpMM, 0.2 M nonzeros, K = 64, 128 14.4 / 12.3, 17.0 / 14.4;  1.2 M, K = 64, 128 31.0 / 26.6, 47 / 41;  6.0 M, K = 64 114 / 100;  fused, 30 K nonzeros, K = 64 12.2 / 9.2;
// 0.2 M, K = 128 24.5 / 20.5;  1.2 M, K = 128 75 / 62;  1.5 M, columns alike, K = 32 39 / 29).  Rows of S without nonzeros are zeroed by blocks of their own at the end of the grid.
//
// What bounds it: the gathers, as in SDDMM (4K bytes of H per nonzero from L2, some 65 to 70 bytes a clock and SM at most; used twice in the fused form), hidden
// by resident warps: SpMM takes 59 bytes a clock at K = 64, 70 at K = 256 (6.0 M nonzeros).  The fused form also computes: a block of B nonzeros is reduced, spread
// and added with nothing of its warp in flight (6.0 M nonzeros, K = 256: 1,180 clocks of 2,220 wait for memory), and more warps or more rows in flight do not fit the
// registers.  Measured and not kept: rows of H through a ring of shared memory by 16-byte or bulk copies (the ring takes what L1 gave: 16.1 M, K = 256, 1407 with a ring of 64 KB a block while L1 had 32 KB, 2180
// with 9 KB; bulk copies 1617 - 2490), H rows of the next block in registers (two nonzeros a block, 1571).
// At K = 64 the gather kernel alone runs at 14.2 TB/s of gathered bytes.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "device_utils.cuh"
#include "gather_index.hpp"

namespace sddmm {

using namespace dev;

namespace {

constexpr int SP_TPB = 256;
constexpr int SP_NB = 8;         // nonzeros of a set per index step (4 when a set is 4 lanes)
constexpr int SP_MAX_RUN = 1024;

constexpr int TAILS = 8;         // tails of a block's runs that are added before they go to the row

// L lanes per nonzero, F pieces per lane, B nonzeros of a set in flight, CTAS resident blocks asked of the compiler.  PF: the
// W rows of the next step are prefetched into L1.  JOINT: the B dot products are reduced together and a block of B that opens
// no row is summed without the tests for it.  Taken where a nonzero has a whole warp or a set few pieces, while with several sets in a warp
// most blocks open a row in one of them (K = 128 871 -> 965).  STAGED (a warp for a nonzero): rows, columns and S values of 32 nonzeros in shared memory, see the
// kernel.  LIMIT: a shape that rounds as much as this one may (run_length).  FAR: tails in scratch instead of shared memory, which is L1 that four blocks of SpMM with a warp for a nonzero miss (6.0 M nonzeros, K = 256: 348 / 330 us, 338
// with no shared memory and the run ends of before; K = 512 722 / 726).
template <int L_, int F_, int B_, bool EXACT_, int CTAS_, bool FUSED_ = false, bool PF_ = false, bool JOINT_ = true, bool STAGED_ = false, bool FAR_ = false, class LIMIT_ = void>
struct SpmmShape {
    using LIMIT = LIMIT_;
    static constexpr int L = L_, F = F_, B = B_, CTAS = CTAS_;
    static constexpr bool EXACT = EXACT_, FUSED = FUSED_, PF = PF_, JOINT = JOINT_, STAGED = STAGED_, FAR = FAR_;
    static constexpr int NB = L < SP_NB ? L : SP_NB, G = 32 / L;
    static constexpr int SETS = SP_TPB / 32 * G;         // of a block
    static constexpr int TAIL_BYTES = FAR ? 0 : SP_TPB * F * 16;  // a row for each of them
    static_assert(NB % B == 0, "step geometry");
    static_assert(!FAR || !FUSED, "a set has one row in scratch");
    static constexpr int SLOTS = FUSED || FAR ? SETS : 0;  // rows of a block's sets in scratch: heads of the fused form (ON_W), tails of FAR
    static_assert(!STAGED || (FUSED && JOINT && L == 32 && B > 1), "staged: a warp for a nonzero");
};

// STAGED: what a warp knows of the 32 nonzeros at hand.
struct Staged {
    int32_t row[32], col[32];
    float val[32], p[32];  // p: the weights
};
template <int B> struct Vec;
template <> struct Vec<2> { using I = int2; using V = float2; };
template <> struct Vec<4> { using I = int4; using V = float4; };
template <int B, class T>
__device__ __forceinline__ void lds_vec(T (&out)[B], const T *p)
{
    using X = typename std::conditional<std::is_same<T, float>::value, typename Vec<B>::V, typename Vec<B>::I>::type;
    const X v = *reinterpret_cast<const X *>(p);
    out[0] = v.x, out[1] = v.y;
    if constexpr (B == 4) out[2] = v.z, out[3] = v.w;
}

__device__ __forceinline__ void stg_u64x2(char *p, u64x2 v)
{
    asm volatile("st.global.cs.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v.a), "l"(v.b) : "memory");
}
__device__ __forceinline__ u64x2 lds_u64x2(uint32_t p)
{
    u64x2 r;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "r"(p) : "memory");
    return r;
}
__device__ __forceinline__ u64x2 ldcg_u64x2(const char *p)  // from L2: written by another SM during this launch
{
    u64x2 r;
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ unsigned long long pair_of(float x)
{
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b)
{
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b)
{
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

template <class S, bool ON_W>
__global__ void __launch_bounds__(SP_TPB, S::CTAS)
spmm_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ cols, const float *__restrict__ val,
            const char *__restrict__ W, const char *__restrict__ H, float *__restrict__ P_out, char *__restrict__ Y,
            char *scratch, unsigned *arrived, const int64_t *__restrict__ row_ptr, unsigned nnz, int64_t M, int pieces, unsigned pitch,
            unsigned run_len, unsigned gather_blocks, unsigned long long *clock, unsigned meet_from)
{
    constexpr int L = S::L, F = S::F, B = S::B, NB = S::NB, G = S::G, T = S::SETS;
    constexpr bool FUSED = S::FUSED;
    constexpr unsigned GROUP = T == 8 && (F == 5 || F == 6) ? 8 : 16;  // parts that one block adds, at most eight times one after the other where a block is few sets
    extern __shared__ __align__(16) char tails[];  // what the sets have of rows that go on behind their runs, a piece for each lane
    __shared__ int first_row[T];
    __shared__ unsigned openers[2];  // the sets whose tail is the beginning of its row, a bit each
    __shared__ __align__(16) Staged staged[S::STAGED ? SP_TPB / 32 : 1];
    // From one row to the next.  (The fused form multiplies whole rows and holds one value less: with a second one it spills, 1707 -> 1801 us
    // at K = 256, 16.1 M nonzeros.)
    const unsigned row_bytes = !FUSED ? pitch : (unsigned)pieces * 16u;
    clock_begin(clock);
    const int lane = threadIdx.x & 31;
    if (blockIdx.x >= gather_blocks) {
        // 32 rows of S per warp: those without nonzeros are written as zeros
        const int64_t r0 = ((int64_t)(blockIdx.x - gather_blocks) * (SP_TPB / 32) + (threadIdx.x >> 5)) * 32;
        const int64_t r = r0 + lane;
        unsigned empty = __ballot_sync(FULL, r < M && row_ptr[r] == row_ptr[r + 1]);
        while (empty) {
            char *out = Y + (size_t)(r0 + __ffs(empty) - 1) * row_bytes;
            empty &= empty - 1;
            for (int q = lane; q < pieces; q += 32) stg_u64x2(out + q * 16, u64x2{0, 0});
        }
        if (clock && threadIdx.x == 0) clock_note(clock);
        return;
    }
    const int lig = lane & (L - 1), set = lane / L;
    const unsigned warp = (blockIdx.x * SP_TPB + threadIdx.x) >> 5;
    const unsigned run = warp * G + set;
    if (threadIdx.x < 2) openers[threadIdx.x] = 0;
    __syncthreads();
    if (warp * G * run_len >= nnz) return;
    const unsigned j0 = run * run_len;
    const char *H_lane = H + lig * 16, *W_lane = W + lig * 16;
    const bool last_ok = S::EXACT || lig + (F - 1) * L < pieces;
    unsigned setmask = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) setmask |= 1u << (g * L);

    u64x2 y[F], w[F];
#pragma unroll
    for (int f = 0; f < F; ++f) y[f] = w[f] = u64x2{0, 0};
    auto load_w = [&](unsigned r) {
        const char *wp = W_lane + (size_t)r * row_bytes;
#pragma unroll
        for (int f = 0; f < F; ++f)
            if (f < F - 1 || last_ok) w[f] = ldg_u64x2(wp + f * L * 16);
    };
    auto flush = [&](char *out) {
        out += lig * 16;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            if (f < F - 1 || last_ok) stg_u64x2(out + f * L * 16, y[f]);
            y[f] = u64x2{0, 0};
        }
    };
    auto at = [&](unsigned x) { return x < nnz ? x : nnz - 1; };
    // Past the end of the matrix a run sees the last nonzero again and again.  Its H row is replaced by zeros there, but a weight
    // that is not finite would make NaN of them.  So the weight is zero as well; or, where several weights are reduced together
    // (PAD), the first of those nonzeros opens a row of its own: the last row is stored before it, and what comes
    // after is not stored.  (Each where it costs nothing measurable.  fused, 16.1 M nonzeros, K = 256, us: without either 1646,
    // zero weights 1683, a row of its own 1638; 6.0 M, K = 512: 1088 / 1095 / 1142; SpMM, 6.0 M, K = 128: 224 / 224 / 229.)
    constexpr bool PAD = FUSED && S::JOINT;
    // A row for each set, behind the blocks' parts.  (The block is read again each time: an address that waits in registers all through the loop makes shapes spill.)
    auto slot_of = [&](int q) {
        unsigned block;
        asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block));
        return scratch + (size_t)(2 * gather_blocks + block * T + q) * row_bytes;
    };
    int cur = __ldg(rows + at(j0));                                // row being summed: that of the nonzero before this step
    auto began_before = [&](int row) { return j0 > 0 && __ldg(rows + at(j0 - 1)) == row; };  // it began in an earlier run
    bool head = began_before(cur);                                 // and nothing of it has been stored yet
    const bool enters = head;
    const int my_set = (threadIdx.x >> 5) * G + set;
    if (lig == 0) first_row[my_set] = cur;
    if (FUSED) load_w((unsigned)cur);
    auto store_row = [&] {  // the finished row; the head of one that began before this run for now
        char *out = Y + (size_t)(unsigned)cur * row_bytes;
        if (ON_W && head) out = slot_of(my_set);
        flush(out);
        head = false;
    };
    auto next_row = [&](int to) {
        store_row();
        cur = to;
    };
    auto add = [&](float weight, const u64x2 (&h)[F]) {
        const unsigned long long pp = pair_of(weight);
#pragma unroll
        for (int f = 0; f < F; ++f) {
            y[f].a = ffma2(pp, h[f].a, y[f].a);
            y[f].b = ffma2(pp, h[f].b, y[f].b);
        }
    };
    // B nonzeros of one row are summed before they are added to it: a long row's chain of roundings is a B-th as long, which is what
    // lets runs be as long as they are (SpMM, 6.0 M nonzeros, K = 64, against 64 bits: runs of 80 one by one 1.4e-7 to 1.6e-7, runs of 320
    // 2.6e-7, in blocks of four 1.4e-7).
    auto add_block = [&](const float (&p)[B], const u64x2 (&h)[B][F]) {
#pragma unroll
        for (int f = 0; f < F; ++f) {
            unsigned long long pp = pair_of(p[0]), ta = mul2(pp, h[0][f].a), tb = mul2(pp, h[0][f].b);
#pragma unroll
            for (int i = 1; i < B; ++i) {
                pp = pair_of(p[i]);
                ta = ffma2(pp, h[i][f].a, ta);
                tb = ffma2(pp, h[i][f].b, tb);
            }
            y[f].a = add2(y[f].a, ta);
            y[f].b = add2(y[f].b, tb);
        }
    };
    // Two sums from three pieces on: one sum of six terms and more loses more to rounding (operands of both signs, rms: K = 384 8.19e-8 / 8.03e-8, K = 512 8.62e-8 / 8.29e-8,
    // K = 768 9.39e-8 / 8.76e-8).
    auto dot = [&](const u64x2 (&h)[F]) {
        unsigned long long a = 0, b = 0;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            a = ffma2(w[f].a, h[f].a, a);
            if constexpr (F > 2) b = ffma2(w[f].b, h[f].b, b);
            else a = ffma2(w[f].b, h[f].b, a);
        }
        return F > 2 ? fold2(a) + fold2(b) : fold2(a);
    };
    if constexpr (S::STAGED) {
        // Rows, columns and S values of 32 nonzeros lie in shared memory, from where a block of B takes its columns and its weights by one
        // load each that all lanes share.  With a shuffle for each they take as much of the load/store pipe as half of the loads of H, and registers that make the loop
        // spill.  us, so / this: 16.1 M nonzeros, K = 256 1598 / 1455 (sustained 1776 / 1571);  6.0 M, K = 200, 256, 384, 512 528 / 456, 528 / 475, 800 / 732, 990 / 915;
        // 0.2 M, K = 256, 512 28.9 / 26.7, 48 / 45;  1.2 M, K = 768 344 / 297;  but K = 640, 1024 259 / 264, 395 / 404.
        Staged &st = staged[threadIdx.x >> 5];
        int rn, cn;
        float sn = 1.f;
        auto fetch = [&](unsigned done) {  // the nonzeros from `done` of the run on
            const unsigned a = at(j0 + done + lane);
            rn = __ldg(rows + a);
            cn = __ldg(cols + a);
            if (val) sn = __ldg(val + a);
        };
        fetch(0);
#pragma unroll 1
        for (unsigned done = 0; done < run_len; done += 32) {
            st.row[lane] = rn;
            st.col[lane] = cn;
            st.val[lane] = sn;
            int before = __shfl_up_sync(FULL, rn, 1);
            if (lane == 0) before = cur;
            const unsigned changed = __ballot_sync(FULL, rn != before || j0 + done + lane == nnz);  // (the padding opens a row)
            __syncwarp();
            if (S::PF && lane >= B && (changed >> lane) & 1u) {
                // the W rows that these nonzeros open, into L1
                const char *wp = W + (size_t)(unsigned)rn * row_bytes;
                for (unsigned o = 0; o < row_bytes; o += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(wp + o));
            }
            if (done + 32 < run_len) fetch(done + 32);
            const int n = min(run_len - done, 32u);
#pragma unroll 1
            for (int b = 0; b < n; b += B) {
                int c[B];
                lds_vec<B>(c, &st.col[b]);
                u64x2 h[B][F];
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const char *hp = H_lane + (size_t)(unsigned)c[i] * row_bytes;
#pragma unroll
                    for (int f = 0; f < F; ++f) h[i][f] = f < F - 1 || last_ok ? ldg_u64x2(hp + f * L * 16) : u64x2{0, 0};
                }
                const unsigned here = (changed >> b) & ((1u << B) - 1u);
                float acc[B], p[B];
                if (here == 0) {
#pragma unroll
                    for (int i = 0; i < B; ++i) acc[i] = dot(h[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < B; ++i) {
                        if (here >> i & 1u) load_w((unsigned)st.row[b + i]);
                        acc[i] = dot(h[i]);
                    }
                }
                reduce_transposed<L, B>(acc, lig);
                const int mine = b + lane / (L / B);
                const float scaled = acc[0] * st.val[mine];
                if (lane % (L / B) == 0) st.p[mine] = scaled;
                __syncwarp();
                lds_vec<B>(p, &st.p[b]);
                if (here == 0) {
                    add_block(p, h);
                } else {
#pragma unroll
                    for (int i = 0; i < B; ++i) {
                        if (here >> i & 1u) next_row(st.row[b + i]);
                        add(p[i], h[i]);
                    }
                }
            }
            __syncwarp();
            if (P_out) {
                if (lane < n && j0 + done + lane < nnz) P_out[j0 + done + lane] = st.p[lane];
                __syncwarp();
            }
        }
    } else {
        const int il = lig & (NB - 1);
        unsigned j = j0 + il;
        int r, c;
        float s = 1.f;
        {
            const unsigned a = at(j);
            r = __ldg(rows + a);
            c = __ldg(cols + a);
            if (val) s = __ldg(val + a);
        }
#pragma unroll 1
        for (unsigned step = run_len / NB; step > 0; --step) {
            int rn = 0, cn = 0;
            float sn = 1.f;
            if (step > 1) {
                const unsigned a = at(j + NB);
                rn = __ldg(rows + a);
                cn = __ldg(cols + a);
                if (val) sn = __ldg(val + a);
            }
            int before = __shfl_up_sync(FULL, r, 1, L);
            if (lig == 0) before = cur;
            const unsigned changed = __ballot_sync(FULL, (r != before || (PAD && j == nnz && (G == 1 || j0 < nnz))) && lig < NB);
            const bool full = __all_sync(FULL, j < nnz);
            if (!FUSED && !full && j >= nnz) s = 0.f;
            if (FUSED && S::PF && step > 1) {
                // the W rows that the next step opens, into L1
                int b2 = __shfl_up_sync(FULL, rn, 1, L);
                const int last = __shfl_sync(FULL, r, NB - 1, L);
                if (lig == 0) b2 = last;
                if (rn != b2 && lig < NB) {
                    const char *wp = W + (size_t)(unsigned)rn * row_bytes;
                    for (unsigned o = 0; o < row_bytes; o += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(wp + o));
                }
            }
            float p_mine = 0.f;
            auto load_h = [&](int b, u64x2 (&h)[B][F]) {
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const unsigned cj = (unsigned)__shfl_sync(FULL, c, b + i, L);
                    const char *hp = H_lane + (size_t)cj * row_bytes;
                    if (full) {
#pragma unroll
                        for (int f = 0; f < F; ++f) h[i][f] = f < F - 1 || last_ok ? ldg_u64x2(hp + f * L * 16) : u64x2{0, 0};
                    } else {  // the end of the matrix
                        const bool ok = j - il + b + i < nnz;
#pragma unroll
                        for (int f = 0; f < F; ++f) h[i][f] = ok && (f < F - 1 || last_ok) ? ldg_u64x2(hp + f * L * 16) : u64x2{0, 0};
                    }
                }
            };
#pragma unroll
            for (int b = 0; b < NB; b += B) {
                u64x2 h[B][F];
                load_h(b, h);
                float p[B];  // the nonzeros' weights, the same in all lanes of the set
                const unsigned here = changed >> b;
                auto opens = [&](int i) { return (here & (setmask << i)) != 0; };  // uniform over the warp: some set goes on to another row
                auto mine = [&](int i) { return ((here >> (set * L + i)) & 1u) != 0; };
                // most blocks of B stay within their rows: one test for the block instead of two for each nonzero
                const bool stays = (here & (setmask * ((1u << B) - 1u))) == 0;
                if (FUSED && S::JOINT) {
                    // all B products first, so that their reductions overlap: one transposed butterfly leaves product i with the
                    // i-th B-th of the set's lanes, where it is scaled; then B broadcasts
                    float acc[B];
                    if (stays) {
#pragma unroll
                        for (int i = 0; i < B; ++i) acc[i] = dot(h[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < B; ++i) {
                            if (opens(i)) {
                                const int rj = __shfl_sync(FULL, r, b + i, L);
                                if (mine(i)) load_w((unsigned)rj);
                            }
                            acc[i] = dot(h[i]);
                        }
                    }
                    reduce_transposed<L, B>(acc, lig);
                    const float scaled = acc[0] * __shfl_sync(FULL, s, b + lig / (L / B), L);
#pragma unroll
                    for (int i = 0; i < B; ++i) p[i] = __shfl_sync(FULL, scaled, i * (L / B), L);
                    if (stays) {
                        add_block(p, h);
                    } else {
#pragma unroll
                        for (int i = 0; i < B; ++i) {
                            if (opens(i)) {
                                const int rj = __shfl_sync(FULL, r, b + i, L);
                                if (mine(i)) next_row(rj);
                            }
                            add(p[i], h[i]);
                        }
                    }
                    if (P_out) {
#pragma unroll
                        for (int i = 0; i < B; ++i)
                            if (il == b + i) p_mine = p[i];
                    }
                } else {
                    if (!FUSED) {
#pragma unroll
                        for (int i = 0; i < B; ++i) p[i] = __shfl_sync(FULL, s, b + i, L);
                        if (B > 1 && stays) {
                            add_block(p, h);
                            continue;
                        }
                    }
                    auto weight = [&](int i) {  // fused: of nonzero i of the block
                        const int x = b + i;
                        unsigned long long a0 = 0, a1 = 0;
#pragma unroll
                        for (int f = 0; f < F; ++f) {
                            a0 = ffma2(w[f].a, h[i][f].a, a0);
                            a1 = ffma2(w[f].b, h[i][f].b, a1);
                        }
                        float a = fold2(a0) + fold2(a1);
#pragma unroll
                        for (int off = L / 2; off >= 1; off >>= 1) a += __shfl_xor_sync(FULL, a, off);
                        p[i] = a * __shfl_sync(FULL, s, x, L);
                        if (!full && j - il + x >= nnz) p[i] = 0.f;
                        if (il == x) p_mine = p[i];
                    };
                    if (FUSED && B > 1 && stays) {
#pragma unroll
                        for (int i = 0; i < B; ++i) weight(i);
                        add_block(p, h);
                        continue;
                    }
#pragma unroll
                    for (int i = 0; i < B; ++i) {
                        const int x = b + i;
                        if (opens(i)) {
                            const int rj = __shfl_sync(FULL, r, x, L);
                            if (mine(i)) {
                                next_row(rj);
                                if (FUSED) load_w((unsigned)rj);
                            }
                        }
                        if (FUSED) weight(i);
                        add(p[i], h[i]);
                    }
                }
            }
            if (FUSED && P_out && lig < NB && j < nnz) P_out[j] = p_mine;
            j += NB;
            r = rn;
            c = cn;
            s = sn;
        }
    }
    auto tail_of = [&](int q) { return smem_u32(tails) + q / G * (F * 512) + (q % G * L + lig) * 16; };
    bool goes_on = false;
    if (G == 1 || j0 < nnz) {
        const unsigned end = j0 + run_len;
        goes_on = end < nnz && __ldg(rows + end) == cur;
        if (goes_on) {
            if constexpr (S::FAR) {
                flush(slot_of(my_set));
            } else {
#pragma unroll
                for (int f = 0; f < F; ++f)
                    asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(tail_of(my_set) + f * 512), "l"(y[f].a), "l"(y[f].b) : "memory");
            }
            if (!head && lig == 0) atomicOr(&openers[my_set / 32], 1u << (my_set & 31));
        } else if (!PAD || end <= nnz) {  // (else it was stored when the padding opened)
            store_row();
        }
    }
    __syncthreads();
    // y += the tails of the sets before set `to` that belong to the row at hand, in their order; whether the row began in this block.  Eight are added before they go to the row: a
    // block of sets of eight lanes may have 31, of four 63, and one by one they lose more to rounding than the runs do.  (Relative rms error against 64 bits, one by one or in two sums / so:
    // documents x words, 0.75 M nonzeros, fused, K = 160 6.6e-8 / 5.3e-8, K = 48 5.7e-8 / 4.9e-8, SpMM, K = 48 5.5e-8 / 4.6e-8.  Two or four sums side by side hold more registers: fused, K = 48,
    // six matrices 5 to 12 % slower.)
    auto add_tails = [&](int to) {
        unsigned long long before = openers[0];
        if (T > 32) before |= (unsigned long long)openers[1] << 32;
        if (to < 64) before &= (1ull << to) - 1;
        const int from = before ? 63 - __clzll((long long)before) : 0;
        constexpr int AHEAD = FUSED ? 1 : 4;  // (the fused form has fewer registers to spare: K = 128 4 6 % slower)
        auto tail = [&](int q, int f) {
            return !S::FAR ? lds_u64x2(tail_of(q) + f * 512) : f < F - 1 || last_ok ? ldcg_u64x2(slot_of(q) + (f * L + lig) * 16) : u64x2{0, 0};
        };
#pragma unroll 1
        for (int q0 = from; q0 < to; q0 += TAILS) {
            u64x2 sum[F];
#pragma unroll
            for (int f = 0; f < F; ++f) sum[f] = tail(q0, f);
            const int q1 = min(q0 + TAILS, to);
#pragma unroll AHEAD
            for (int q = q0 + 1; q < q1; ++q) {
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const u64x2 v = tail(q, f);
                    sum[f].a = add2(sum[f].a, v.a);
                    sum[f].b = add2(sum[f].b, v.b);
                }
            }
#pragma unroll
            for (int f = 0; f < F; ++f) {
                y[f].a = add2(y[f].a, sum[f].a);
                y[f].b = add2(y[f].b, sum[f].b);
            }
        }
        return before != 0;
    };
    // The row in y is one of several blocks': its part goes to scratch -- part 2 b of block b: the row ends there, 2 b + 1: it goes on -- and the block that
    // arrives last adds the parts up.
    const unsigned lanes = L == 32 ? FULL : ((1u << (L & 31)) - 1u) << (set * L);
    auto hand_over = [&](size_t row) {
        auto arrive = [&](unsigned *count) {  // how many came before; everything this set stored is visible first
            __threadfence();
            __syncwarp(lanes);
            unsigned before = 0;
            if (lig == 0) before = atomicAdd(count, 1u);
            return __shfl_sync(lanes, before, set * L);
        };
        const unsigned per_block = T * run_len, me = blockIdx.x;
        const unsigned first = (unsigned)row_ptr[row] / per_block, last = (unsigned)(row_ptr[row + 1] - 1) / per_block;
        auto part = [&](unsigned q) { return scratch + (size_t)(2 * q + (q < last ? 1 : 0)) * row_bytes + lig * 16; };
        auto add_up = [&](unsigned q0, unsigned q1, unsigned step) {  // y = parts q0, q0 + step, ... <= q1
            constexpr int U = F <= 2 ? 4 : F <= 4 || F > 6 ? 2 : 1;  // (two of five or six pieces spill)
#pragma unroll
            for (int f = 0; f < F; ++f) y[f] = u64x2{0, 0};
#pragma unroll 1
            for (unsigned q = q0; q <= q1; q += U * step) {
                u64x2 v[U][F];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int f = 0; f < F; ++f)
                        v[u][f] = q + u * step <= q1 && (f < F - 1 || last_ok) ? ldcg_u64x2(part(q + u * step) + f * L * 16) : u64x2{0, 0};
#pragma unroll
                for (int u = U / 2; u >= 1; u /= 2)
#pragma unroll
                    for (int x = 0; x < u; ++x)
#pragma unroll
                        for (int f = 0; f < F; ++f) {
                            v[x][f].a = add2(v[x][f].a, v[x + u][f].a);
                            v[x][f].b = add2(v[x][f].b, v[x + u][f].b);
                        }
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    y[f].a = add2(y[f].a, v[0][f].a);
                    y[f].b = add2(y[f].b, v[0][f].b);
                }
            }
        };
        flush(part(me) - lig * 16);
        const unsigned g0 = first + (me - first) / GROUP * GROUP, g1 = min(g0 + GROUP - 1, last);
        // (a group that is the row's last block only needs no counter, and has none: the next row may begin in that block)
        if (g1 > g0) {
            if (arrive(&arrived[2 * g0]) != g1 - g0) return;
            if (lig == 0) arrived[2 * g0] = 0;  // for the next call
            __threadfence();
        }
        add_up(g0, g1, 1);
        if (g0 != first || g1 != last) {
            flush(part(g0) - lig * 16);
            if (arrive(&arrived[2 * first + 1]) != (last - first) / GROUP) return;
            if (lig == 0) arrived[2 * first + 1] = 0;
            __threadfence();
            add_up(first, last, GROUP);
        }
        flush(Y + row * row_bytes);
        if (clock && lig == 0) clock_note(clock);  // (a row of many blocks: this may outlast every block that starts later)
    };
    if (enters && !head) {  // a row that began before this run has ended in it
        const size_t row = (size_t)(unsigned)first_row[my_set];
        const char *const mine = (ON_W ? slot_of(my_set) : Y + row * row_bytes) + lig * 16;
#pragma unroll
        for (int f = 0; f < F; ++f)
            y[f] = f < F - 1 || last_ok ? ldcg_u64x2(mine + f * L * 16) : u64x2{0, 0};
        if (add_tails(my_set)) flush(Y + row * row_bytes);
        else hand_over(row);
    }
    if (goes_on && my_set == T - 1) {
#pragma unroll
        for (int f = 0; f < F; ++f) y[f] = u64x2{0, 0};
        (void)add_tails(T);
        hand_over((size_t)(unsigned)cur);
    }
    clock_end(clock, meet_from);
}

// Runs are cut so that they fill whole waves of resident sets: a wave lasts as long as its runs, and a last one that is nearly empty as
// long as a full one (SpMM, K = 64, 6.0 M nonzeros, us: 2.0 waves 117, 2.5 waves 127, 2.8 waves 121, 4.0 waves 124).  How many: each
// run pays for its two ends, so few; but rows of a power-law matrix make some
// runs slower than others, the fused form more than SpMM, and long runs spread a wave over more rows of H than L2 holds.  us at
// 1 / 2 / 3 / 4 / 6 / 8 waves (s: nonzeros for a resident set):
//   SpMM, K = 64: s = 14 12.6 / 12.4 / 12.5 / 12.5 / 12.5 / 12.5 (runs of 24 at least);  80, columns alike 28.8 / 31.6 / 35.4 / 37.2 / 37.2 / 37.3;  317 100 / 99.5 / 101 / 102 / 107 / 112
//   K = 256: 127 40.9 / 43.9 / 46.1 / 50.4 / 54.5 / 54.6;  K = 100: 577 137 / 135 / 136 / 138 / 143 / 148, 845 183 / 181 / 181 / 183 / 186 / 192;  K = 200: 1267 295 / 295 / 297 / 299 / 302 / 308
//   fused, sets of eight lanes, K = 64: s = 14 14.4 / 17.2 / 17.2 / 17.2 / 17.2 / 17.2;  80, columns alike 41.7 / 43.8 / 49.0 / 50.5 / 52.8 / 52.8;  317 194 / 179 / 174 / 172 / 168 / 169
//   K = 128: 72 75 / 74 / 74 / 74 / 79 / 79;  317 303 / 279 / 276 / 273 / 271 / 270
//   fused, a warp for a nonzero, K = 256: s = 58 26.7 / 26.9 / 28.7 / 30.6 / 30.6 / 39.6;  330 133 / 116 / 113 / 110 / 110 / 111;  423, columns alike 138 / 145 / 150 / 158 / 165 / 168;
//   1690 528 / 530 / 514 / 517 / 475 / 473;  4531 at 12 / 16 1492 / 1478
// (SpMM: what asks for more than two are roundings.)
template <class S>
unsigned run_length(int64_t nnz, int sm_count)
{
    const int64_t wave = (int64_t)sm_count * S::CTAS * (SP_TPB / 32) * S::G, s = nnz / wave + 1;
    int64_t waves;
    if (S::B == 1) {
        // One nonzero at a time: a row that fills a run has as many roundings one after the other as the run is long.  32 nonzeros and up to a
        // third of a set's share, 80 and up to a sixth, 160 and up to a twelfth.
        waves = s <= 32 ? 1 : s <= 64 ? 2 : s <= 240 ? 3 : s <= 480 ? (s + 79) / 80 : std::min<int64_t>(12, std::max<int64_t>(6, (s + 159) / 160));
    } else {
        // B at a time (add_block): a B-th of the roundings.  At most as many as where one at a time is added, and 80 up to 1,920 nonzeros.
        // (Relative error of sums of positive terms, rms of all entries, one at a time / the waves of the table alone / with this limit: 8 M nonzeros, rows of
        // 700, K = 192 8.4e-8 / 1.4e-7 / 7.1e-8, K = 200 9.7e-8 / 2.0e-7 / 9.1e-8;  28 M, K = 64 9.8e-8 / 1.5e-7 / 8.6e-8;  and of one at a time, 0.28 M, rows of 80,
        // K = 576 5.5e-8 / 1.4e-7 / 6.2e-8.  It costs up to 5 % of the time: K = 192, 4 M 216 -> 220 us, K = 384 446 -> 460, K = 512, 3 M 439 -> 460; K = 40 79 -> 88.)
        const int64_t chain = s < 240 ? std::max<int64_t>(24, s / 3) : std::max<int64_t>(80, s / 24);
        waves = S::FUSED && S::L == 32 ? (s <= 120 ? 1 : s <= 330 ? 2 : s > 1500 ? (s + 299) / 300 : (s + 169) / 170)
              : S::FUSED ? (s <= 120 ? 1 : s <= 240 ? 2 : std::max<int64_t>(std::min<int64_t>(12, (s + 79) / 80), (s + 299) / 300))
                         : s <= 340 ? 1 : std::max<int64_t>(2, (s + 759) / 760);
        waves = std::max(waves, (s + S::B * chain - 1) / (S::B * chain));
    }
    // Fewer, longer runs where they would be very short (us at runs of 8 / 16 / 24, SpMM: s = 3, K = 128 10.5 / 11.0 / 11.9, K = 512 12.0 / 10.3 / 12.0;  s = 6, K = 192 14.8 / 14.3 / 15.3,
    // K = 512 15.8 / 14.3 / 12.3;  s = 8, K = 128 13.8 / 12.3 / 14.3, K = 192 16.0 / 14.4 / 16.4;  s = 10, K = 256 15.5 / 12.5 / 12.3, K = 512 18.4 / 15.0 / 16.4;  s = 14, K = 64 20.6 / 16.4 / 16.5,
    // K = 300 19.0 / 16.8 / 15.1, K = 512 22.5 / 19.0 / 16.4;  fused: s = 6, K = 64 14.2 / 14.7 / 16.4, K = 256 12.4 / 13.6 / 16.4, K = 512 20.5 / 19.5 / 22.3;  s = 14, K = 64 22.6 / 18.4 / 20.5,
    // K = 512 31.0 / 24.5 / 25.9).
    int64_t least = S::NB, most = SP_MAX_RUN;
    if (!S::FUSED && s > 4) least = (s > 12 ? 3 : 2) * S::NB;
    if (S::FUSED && S::F >= 4 && s > 5) least = 2 * S::NB;
    // The share s of a set, and with it the table, depends on how many sets are resident and on how many nonzeros they take at a time.  A shape with another of either than the one that the
    // roundings were measured with (LIMIT) has runs no longer than that one's.  A run of n nonzeros adds n / B times to a row's sum, one after the other, and a long row loses a third of
    // that to rounding, in squares and for the run's part of it: n^2 / B counts.  More waves then, not runs that end in the middle of one (fused, K = 256, 0.2 M nonzeros on three
    // resident blocks, runs of 48 32.4 us, of 32 28.2).  Rows of 700 positive terms, squares of the relative error in 2^-48 / 3, by the table alone / so: fused, K = 256, 6.5 M nonzeros
    // 4.7 / 3.2, K = 512, 2.0 M 4.1 / 2.9, SpMM, K = 200, 1.4 M 6.0 / 3.1.
    if constexpr (!std::is_void<typename S::LIMIT>::value)
        most = std::max<int64_t>(S::NB, (int64_t)(run_length<typename S::LIMIT>(nnz, sm_count) * std::sqrt((double)S::B / S::LIMIT::B) + S::NB / 2) / S::NB * S::NB);
    least = std::min(least, most);
    auto cut = [&] { return std::max(least, (nnz / (waves * wave) + S::NB) / S::NB * S::NB); };  // rounded up: one run less than a wave, not one more
    while (cut() > most && cut() > S::NB) ++waves;
    return (unsigned)std::min(cut(), most);
}

template <class S>
cudaError_t launch_shape(const SpmmCall &a, int k0, int width, int sm_count, int64_t *n_launches, cudaStream_t stream)
{
    const int pieces = width / 4;
    if (pieces > S::L * S::F || pieces <= S::L * (S::F - 1)) return cudaErrorInvalidValue;
    const unsigned run = run_length<S>(a.nnz, sm_count), per_block = S::SETS * run;
    const unsigned gather_blocks = (unsigned)((a.nnz + per_block - 1) / per_block);
    const unsigned zero_blocks = (unsigned)((a.M + SP_TPB - 1) / SP_TPB);
    // scratch: two counters per block, zero between calls, then the parts, then a row for each set (SLOTS)
    unsigned *const arrived = reinterpret_cast<unsigned *>(a.scratch);
    char *const parts = reinterpret_cast<char *>(a.scratch + spmm_counter_floats(a.nnz, a.N, a.K, sm_count));
    constexpr int smem = S::TAIL_BYTES;
    static_assert(smem + sizeof(Staged) * (SP_TPB / 32) + 512 <= 48 * 1024, "without opt-in");
    auto launch = [&](auto kernel) {
        kernel<<<gather_blocks + zero_blocks, SP_TPB, smem, stream>>>(
            a.rows, a.cols, a.val, reinterpret_cast<const char *>(a.W), reinterpret_cast<const char *>(a.H + k0), a.P_out,
            reinterpret_cast<char *>(a.Y + k0), parts, arrived, a.row_ptr, (unsigned)a.nnz, a.M, pieces, (unsigned)a.K * 4u, run, gather_blocks, a.clock, last_wave(gather_blocks, (unsigned)sm_count * S::CTAS));
    };
    if (S::FUSED && a.Y < a.W + a.M * a.K && a.W < a.Y + a.M * a.K) launch(spmm_kernel<S, S::FUSED>);
    else launch(spmm_kernel<S, false>);
    ++*n_launches;
    return cudaGetLastError();
}

// Calls f with the shape for K (L * (F - 1) < K / 4 <= L * F).  The fused form holds the W row as well and wants fewer
// nonzeros in flight; every line is the best of a sweep over (L, B, prefetch, joint reduction, resident blocks).  The fused ones against the LIMIT lines that they took the place of, us,
// 6.0 M / 1.2 M nonzeros: K = 32 161 / 37, this 130 / 32;  K = 160 411 / 98, this 330 / 78;  K = 320 780 / 168, this 628 / 131;  K = 256 531 / 127, this 474 / 114;  K = 512 996 / 212, this
// 941 / 206.  SpMM, K = 200, three blocks / this: 6.0 M 357 / 301, 1.35 M 83 / 77, 1.5 M, columns alike 103 / 86.  Not taken, since short rows lose more to rounding: fused, K = 96, one at a time
// (239 / 57 -> 218 / 50, but rows of 100, 30 M nonzeros, squares of the relative error in 2^-48 / 3 7.6 -> 11.0), K = 32, four at a time (130 / 32 -> 120 / 31; rows of 15, 1.5 M
// 5.39e-8 -> 5.48e-8).
template <class Fn>
auto with_shape(int K, bool fused, int64_t nnz, Fn f)
{
    const int q = K / 4;
    if (fused) {
        if (q <= 4) return f(SpmmShape<4, 1, 2, false, 4, true, true, false>());
        if (q < 8) return f(SpmmShape<8, 1, 2, false, 5, true, true, true, false, false, SpmmShape<8, 1, 2, false, 4, true>>());
        if (q == 8) return f(SpmmShape<8, 1, 2, true, 5, true, true, true, false, false, SpmmShape<8, 1, 2, false, 4, true>>());
        if (q <= 12) return f(SpmmShape<4, 3, 2, false, 4, true, true, false>());
        if (q < 16) return f(SpmmShape<8, 2, 2, false, 4, true, true, false>());
        if (q == 16) return f(SpmmShape<8, 2, 2, true, 4, true, true, false>());
        if (q <= 24) return f(SpmmShape<8, 3, 2, false, 3, true, true, false>());
        if (q < 32) return f(SpmmShape<8, 4, 1, false, 3, true, true, false>());
        if (q == 32) return f(SpmmShape<8, 4, 1, true, 4, true, false, false>());
        if (q <= 40) return f(SpmmShape<8, 5, 1, false, 3, true, true, false, false, false, SpmmShape<16, 3, 1, false, 4, true>>());
        if (q <= 48) return f(SpmmShape<16, 3, 1, false, 4, true, true, false>());
        if (q <= 64) return f(SpmmShape<32, 2, 4, false, 3, true, true, true, true, false, SpmmShape<32, 2, 4, false, 4, true>>());
        if (q <= 80) return f(SpmmShape<16, 5, 1, false, 3, true, true, false, false, false, SpmmShape<32, 3, 1, false, 4, true>>());
        if (q <= 96) return f(SpmmShape<32, 3, 2, false, 3, true, true, true, true, false, SpmmShape<32, 3, 1, false, 4, true>>());
        if (q <= 128) return f(SpmmShape<32, 4, 2, false, 3, true, false, true, true, false, SpmmShape<32, 4, 1, false, 4, true>>());
        if (q <= 160) return f(SpmmShape<32, 5, 1, false, 3, true, false, false>());
        if (q <= 192) return f(SpmmShape<32, 6, 2, false, 2, true, false, true, true, false, SpmmShape<32, 6, 1, false, 2, true>>());
        if (q <= 224) return f(SpmmShape<32, 7, 1, false, 2, true, false, false>());
        return f(SpmmShape<32, 8, 1, false, 2, true, false, false>());
    }
    if (q <= 4) return f(SpmmShape<4, 1, 4, false, 4>());
    if (q <= 8) return f(SpmmShape<8, 1, 4, false, 4>());
    if (q <= 12) return f(SpmmShape<4, 3, 2, false, 4>());
    if (q < 16) return f(SpmmShape<8, 2, 4, false, 3>());
    if (q == 16) return f(SpmmShape<8, 2, 4, true, 4>());
    if (q <= 24) return f(SpmmShape<8, 3, 2, false, 4>());
    if (q < 32) return f(SpmmShape<16, 2, 4, false, 3>());
    if (q == 32) return f(SpmmShape<16, 2, 4, true, 4>());
    if (q <= 48) return f(SpmmShape<16, 3, 2, false, 4>());
    // (few nonzeros, tails in shared memory; us, this / the lines below: K = 200, a block fewer, 0.26 M 24.6 / 26.5, documents x words, 0.75 M 43.6 / 45.3, but 1.2 M 73 / 68;  K = 256, three blocks / four /
    // four and tails in scratch: 60 K 10.4 / 12.3 / -, 79 K 12.4 / 14.4 / 14.4, 70 K 12.3 / 12.3 / 14.4, 0.1 M 18.2 / 14.0 / -, 0.2 M 21 / 20.3 / 20.6, 0.28 M 30.5 / 25.1 / 24.7)
    if (q > 48 && q < 64 && nnz < 1000000) return f(SpmmShape<32, 2, 4, false, 3>());
    if (q == 64 && nnz < 85000) return f(SpmmShape<32, 2, 4, true, 3, false, false, true, false, false, SpmmShape<32, 2, 4, true, 4>>());
    if (q == 64 && nnz < 300000) return f(SpmmShape<32, 2, 4, true, 4>());
    if (q < 64) return f(SpmmShape<32, 2, 4, false, 4, false, false, true, false, true, SpmmShape<32, 2, 4, false, 3>>());
    if (q == 64) return f(SpmmShape<32, 2, 4, true, 4, false, false, true, false, true>());
    if (q <= 96) return f(SpmmShape<32, 3, 2, false, 3>());
    if (q <= 128) return f(SpmmShape<32, 4, 2, false, 3>());
    if (q <= 160) return f(SpmmShape<32, 5, 1, false, 3>());
    if (q <= 192) return f(SpmmShape<32, 6, 1, false, 3>());
    if (q <= 224) return f(SpmmShape<32, 7, 1, false, 2>());
    return f(SpmmShape<32, 8, 1, false, 2>());
}

}  // namespace

// SpMM of long rows with a large H in passes of 192 columns (of H and of Y; the fused form needs whole rows).  More gathers of a pass hit L2,
// and the shapes for more columns hold so many registers that few warps are resident.  Sustained us, one pass / these: K = 384, 0.3 M rows
// of H 573 / 570, 0.7 M 1166 / 1062, 1 M 2163 / 1975; K = 512, 0.3 M 734 / 782, 0.7 M 1449 / 1453, 1 M 2806 / 2678, 1.5 M 4516 / 4181; K = 256, 1.5 M 2096 / 2138.
// Rows of whole 128-byte lines, and no narrow last pass: neighbouring passes touch the same lines otherwise (one pass / these, all columns alike, R-MAT: K = 352,
// 1.8 GB of H 3451 / 3447, 2110 / 2025;  K = 324 3715 / 4062, 2312 / 2353;  K = 388 3608 / 4350, 2168 / 2427;  K = 416 3378 / 3586, 1961 / 2012;  K = 544 3505 / 3372,
// 2146 / 1896;  K = 608 3453 / 3468, 2058 / 1932;  K = 644 3563 / 3931, 2130 / 2123;  K = 704 3389 / 3291, 2029 / 1799;  K = 772 3596 / 4001, 2203 / 2132).  Above 768
// columns, where a row whole runs on very few warps, also other rows of an H that is not too large (K = 900, 1.0 GB 1940 / 1891, 1111 / 1089; 1.8 GB 3545 / 3733, 2178 / 1993;
// K = 1020 1907 / 1806, 1075 / 1043; 3488 / 3656, 2139 / 1973).
static int pass_floats(int64_t nnz, int64_t N, int K)
{
    const int64_t h_bytes = N * K * 4;
    const bool pays = K % 32 == 0 ? K % 192 == 0 || K % 192 >= 64 || K > 512 : K > 768 && h_bytes < 1500000000;
    return K > 320 && pays && nnz >= 1000000 && h_bytes >= (K > 480 && K <= 512 ? 1700000000 : 900000000) ? 192 : K;
}

int spmm_passes(int64_t nnz, int64_t N, int K)
{
    const int w = pass_floats(nnz, N, K);
    return (K + w - 1) / w;
}

bool spmm_supports(int K) { return K > 0 && K % 4 == 0 && K <= 1024; }

// The largest f(shape, blocks of runs) of either form and of every pass.
template <class Fn>
static size_t largest(int64_t nnz, int64_t N, int K, int sm_count, Fn f)
{
    auto of = [&](int width, bool fused) {
        return with_shape(width, fused, nnz, [&](auto s) {
            const size_t per_block = (size_t)decltype(s)::SETS * run_length<decltype(s)>(nnz, sm_count);
            return f(s, ((size_t)nnz + per_block - 1) / per_block);
        });
    };
    size_t n = std::max(of(K, false), of(K, true));
    const int w = pass_floats(nnz, N, K);
    if (w < K) n = std::max(n, of(w, false));
    if (K % w) n = std::max(n, of(K % w, false));
    return n;
}
size_t spmm_counter_floats(int64_t nnz, int64_t N, int K, int sm_count)
{
    return (2 * largest(nnz, N, K, sm_count, [](auto, size_t blocks) { return blocks; }) + 31) / 32 * 32;
}
size_t spmm_scratch_floats(int64_t nnz, int64_t N, int K, int sm_count)
{
    return spmm_counter_floats(nnz, N, K, sm_count) + largest(nnz, N, K, sm_count, [](auto s, size_t blocks) { return blocks * (2 + decltype(s)::SLOTS); }) * (size_t)K;
}

cudaError_t launch_spmm(const SpmmCall &a, int sm_count, int64_t *n_launches, cudaStream_t stream)
{
    if (a.M == 0) return cudaSuccess;
    const int w = a.W ? a.K : pass_floats(a.nnz, a.N, a.K);
    for (int k0 = 0; k0 < a.K; k0 += w) {
        const int width = std::min(w, a.K - k0);
        const cudaError_t e = with_shape(width, a.W != nullptr, a.nnz, [&](auto s) { return launch_shape<decltype(s)>(a, k0, width, sm_count, n_launches, stream); });
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace sddmm
