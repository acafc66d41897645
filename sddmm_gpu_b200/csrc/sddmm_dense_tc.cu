// Dense-cell kernel on the 5th-generation tensor cores (tcgen05, accumulator in
// tensor memory), warp-specialised.
//
// Same job as sddmm_dense_kernel, two cells of the same rows at a time (DenseUnit): their 2 x 64 columns are the M = 128 side of
// the product and the 128 rows the N side, D = H[cols] * W[rows]^T, so that a lane of tensor memory is a COLUMN of S and a
// tensor-memory column a row of S.  A warp that reads 32 lanes then holds 32 neighbouring columns of a row in
// its lanes: S values and P entries of a row are contiguous over the lanes, and the block goes from tensor memory to P without a
// pass through shared memory.  The product is issued by ONE thread as tcgen05.mma instructions (M = 128, N = 128, K = 8 per
// instruction, kind::tf32) that read both operands from shared memory through matrix descriptors and accumulate into 128 columns
// of tensor memory (TMEM).  fp32-level accuracy comes from 3xTF32 as in the mma.sync
// variant: every operand is written to shared memory twice, as its TF32 head (x
// with the 13 low mantissa bits cleared) and its tail (x - head, exact), and
// every k-step issues head*tail + tail*head + head*head.  (The head tile is the
// raw fp32 data: the tensor core reads only the TF32 bits of an element.)
//
// One persistent CTA per SM, three roles that overlap through mbarriers:
//   warps 0-7   producers: copy H / W rows of a K chunk (32 k) into the head tiles of one
//               of three head stages with cp.async, two chunks ahead, and compute the tail tiles from them into one of
//               two tail stages;
//   warp  8     one thread issues the MMAs of a chunk when its stages are full and
//               commits them to the chunk's "done" barrier; after a unit's last
//               chunk it commits to the accumulator's "full" barrier;
//   warps 9-24  epilogue: a warp reads 32 rows x 32 columns of the finished block (tcgen05.ld, eight rows at a time), multiplies them by the
//               S values, which it has loaded one unit ahead, and stores them to P.  The warps of a group of four meet only where
//               they wait for the product.
//
// Shared-memory operand layout (K-major, 128-byte swizzle): a tile of 128 rows x 32 k is 128 lines of
// 128 bytes, one per row, in groups of eight rows (1024 bytes, the descriptor's stride-dimension
// offset); inside a group the 16-byte piece c of row r sits at piece c ^ (r % 8) of the row's line --
// the layout a tile copy with the 128-byte swizzle would produce, and the one the tensor core reads
// without bank conflicts.  One instruction consumes 32 bytes of every row, so k-step s starts 32 s
// bytes into the tile.  Producer thread f writes bytes [16 f, 16 f + 16) of a tile, i.e. piece f % 8
// of row f / 8, which holds the four k from 4 ((f % 8) ^ (f / 8 % 8)) on: the eight lanes of a row
// read its 128 contiguous bytes in global memory and fill one 128-byte line of shared memory.
//
// What bounds it: the epilogue's S loads and P stores (512 of each for a unit and SM, through a load/store path that the producers
// share): 65,536-token mask with 80 global tokens, K = 64: 130 us, 104 without them, 352 MB of S and P in all (54 us at the copy rate).
// A cell at a time (N = 64, rows on the lanes, every block parked in shared memory between tensor memory and P) it took 164 us: the one
// issuing thread needed 3,700 clocks for the 24 MMAs of a cell, parking and picking four passes over shared memory and three
// barriers of 512 threads.  Now / then, us: K = 128 174 / 239, K = 64 without global tokens, 28,546 tokens, 41 / 49.  What decides is the
// register budget of the epilogue (72 at 25 warps): the same code with 72 bytes of spills took 145 us, with 556 bytes 297.
//
// Every wait is bounded (mbarrier polls with a limit; on expiry the role sets the
// device status word and leaves its loop, the others run into their own limits),
// the only CTA-wide barriers are at the start and the end, and the TMEM columns
// are released on every path.
#include <cuda_runtime.h>
#include <stdint.h>

#include "binning.cuh"
#include "common.cuh"
#include "device_utils.cuh"

namespace sddmm {

using namespace dev;

namespace {

constexpr int DR = DENSE_CELL_ROWS;          // 128 = N of the MMA = TMEM columns per accumulator
constexpr int DC = DENSE_CELL_COLS;          // 64; two cells are M of the MMA = TMEM lanes
constexpr int TM = 2 * DC;
constexpr int KC = 32;                       // K chunk of one operand stage
constexpr int HEADS = 3, TAILS = 2;          // stages of head and of tail tiles
constexpr int TILE_BYTES = 128 * KC * 4;     // 16 KB, of either operand
constexpr int STAGE_BYTES = 2 * TILE_BYTES;  // H tile, then W tile
static_assert(DR == 128 && TM == 128, "one tile size for both operands");
// Epilogue: group g of four warps has rows 32 g .. + 32 of the unit, a warp the 32 tensor-memory lanes that its number mod 4 names (it
// can read no others).
constexpr int EPI_GROUPS = DR / 32, EPI_WARPS = EPI_GROUPS * 4;
constexpr int BATCH = 8, N_BATCH = 32 / BATCH;  // rows read from tensor memory together
// 32 rows of S as a warp picks them, for its 32 columns.  run (every row at input position x + column): x and the columns held.
// masked: the position of the first column held, the columns held, the position it would have from behind the gap, the first column there.
union EpiRows {
    int2 run[32];
    int4 masked[32];
};
constexpr int N_PRODUCERS = 256;
constexpr int MMA_WARP = N_PRODUCERS / 32, EPI_WARP0 = MMA_WARP + 1;
constexpr int TC_THREADS = N_PRODUCERS + 32 + EPI_WARPS * 32;  // 800
constexpr int TC_SMEM_BYTES = (HEADS + TAILS) * STAGE_BYTES + EPI_WARPS * 2 * (int)sizeof(EpiRows);  // 180,224 bytes
// Accumulators: all of tensor memory (no second CTA fits an SM anyway).
constexpr unsigned N_ACC = 4;
constexpr uint32_t TMEM_COLS = N_ACC * DR;  // 512
constexpr uint32_t LBO = 16, SBO = 8 * KC * 4;  // leading offset unused by swizzled K-major tiles; 8 rows of 128 bytes

// Shared-memory matrix descriptor: start address, leading / stride byte offsets (all >> 4), version 1,
// layout type 2 = 128-byte swizzle (bits 61-63).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor of kind::tf32: D = fp32 (bits 4-5 = 1), A = B = TF32 (bits 7-9, 10-12 = 2), both
// K-major (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(DR >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

__device__ __forceinline__ void mma_tf32_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(IDESC), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Eight tensor-memory columns of this warp's 32 lanes; complete behind tcgen05.wait::ld.
__device__ __forceinline__ void tmem_ld(uint32_t (&v)[8], uint32_t taddr)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

// tail = x - head(x) of four consecutive k of one row (head = x with the 13 low mantissa bits cleared), exact
__device__ __forceinline__ void tail_store(const float4 v, unsigned char *dst)
{
    float4 lo;
    lo.x = v.x - __uint_as_float(__float_as_uint(v.x) & 0xffffe000u);
    lo.y = v.y - __uint_as_float(__float_as_uint(v.y) & 0xffffe000u);
    lo.z = v.z - __uint_as_float(__float_as_uint(v.z) & 0xffffe000u);
    lo.w = v.w - __uint_as_float(__float_as_uint(v.w) & 0xffffe000u);
    *reinterpret_cast<float4 *>(dst) = lo;
}
// 16-byte asynchronous copy global -> shared; src_bytes = 0 fills the 16 bytes with zeros
__device__ __forceinline__ void cp_async16_zfill(void *dst_smem, const void *src, int src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src), "r"(src_bytes) : "memory");
}

// S value and P entry of a lane, if `held`: predicated, not branched around (a branch each made it 25 instructions for a row of a warp), and
// not kept in L1, which is small beside the operand stages (65,536-token mask, K = 64, us: stores 184 -> 165, loads 156 -> 152).
__device__ __forceinline__ void load_if(float &v, const float *p, unsigned held)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.global.nc.L1::no_allocate.f32 %0, [%1];\n\t}" : "+f"(v) : "l"(p), "r"(held));
}
__device__ __forceinline__ void store_if(float *p, float v, unsigned held)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.L1::no_allocate.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"(held) : "memory");
}

// barrier.cta.red.and over the 128 threads of an epilogue group (named barrier 1 + group): one answer for all of them
__device__ __forceinline__ bool group_all(int group, bool mine)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)mine), "r"(1 + group)
        : "memory");
    return r != 0;
}

// A warp waits for a barrier phase: lane 0 polls (32 lanes polling one word cost 32 accesses of the shared-memory
// pipe per poll), the others take its answer; __syncwarp orders the warp's memory accesses behind the wait.  The polling
// loop is a call: inlined at five places it took instruction cache and registers from the roles (with the vote in place
// of a shuffle, 65,536-token mask: K = 64 168.5 -> 166, K = 128 245 -> 239.5 us).
__device__ __noinline__ bool wait_polling(uint64_t *bar, unsigned parity) { return mbar_wait_bounded(bar, parity); }
__device__ __forceinline__ bool wait_bar(uint64_t *bar, unsigned parity)
{
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = mbar_try_wait(bar, parity) || wait_polling(bar, parity);
    ok = __all_sync(FULL, ok);
    __syncwarp();
    return ok;
}

__global__ void __launch_bounds__(TC_THREADS, 1)
sddmm_dense_tc_kernel(const DenseUnit *__restrict__ units, int64_t n_units,
                      const int32_t *__restrict__ table, const unsigned long long *__restrict__ row_mask,
                      const int2 *__restrict__ row_base, const uint32_t *__restrict__ row_span, const int32_t *__restrict__ dense_rows, int64_t n_dense_rows,
                      const int32_t *__restrict__ dense_cols, int64_t n_dense_cols, const float *__restrict__ sval,
                      const float *__restrict__ W, const float *__restrict__ H, float *__restrict__ P, int64_t M,
                      int64_t N, int K, int *dev_status)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *const tails = smem + HEADS * STAGE_BYTES;
    EpiRows *const epi_rows = reinterpret_cast<EpiRows *>(smem + (HEADS + TAILS) * STAGE_BYTES);
    __shared__ uint64_t full_bar[HEADS], done_bar[HEADS], acc_full[N_ACC], acc_empty[N_ACC];
    __shared__ uint32_t tmem_holder;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int s = 0; s < HEADS; ++s) {
            mbar_init(&full_bar[s], N_PRODUCERS / 32);  // one arrival per producer warp, after all its lanes' stores
            mbar_init(&done_bar[s], 1);                 // one tcgen05.commit
        }
        for (unsigned b = 0; b < N_ACC; ++b) {
            mbar_init(&acc_full[b], 1);                 // one tcgen05.commit
            mbar_init(&acc_empty[b], EPI_WARPS);        // one arrival per epilogue warp, after its last tcgen05.ld
        }
        mbar_fence_init();
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "n"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;
    // every block runs: the gather kernel of the remaining nonzeros may start beside this one
    if (tid == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n_chunks = (K + KC - 1) / KC;
    bool ok = true;
    // The units of this CTA: every gridDim.x-th of the list.
    const int my_units = (int64_t)blockIdx.x < n_units ? (int)((n_units - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
    auto unit_of = [&](int i) -> const DenseUnit & { return units[(int64_t)i * gridDim.x + blockIdx.x]; };

    if (warp < MMA_WARP) {
        // ---------------- producers ----------------
        // The head tile of an operand is the raw fp32 data (the tensor core reads only the TF32 bits of an
        // element), so it is brought in by 16-byte cp.async copies, two chunks ahead and without holding a
        // register; the tail tile (x minus its TF32 head, exact) is computed from the head tile in shared memory.
        // Thread f owns bytes [16 f, 16 f + 16) of every tile, so it only ever reads what it copied itself.
        const unsigned total = (unsigned)my_units * (unsigned)n_chunks;
        // the k group of this thread's pieces, f = tid + 256 i: piece f % 8 of row f / 8 holds group (f % 8) ^ (f / 8 % 8)
        const int kq = ((tid & 7) ^ ((tid >> 3) & 7)) * 4;
        // issue cursor: unit, chunk and this thread's operand rows of that unit (`there`: a bit each, else zeros).  Looking them up is
        // two dependent loads for compacted lines, so it runs ahead: the descriptor two units, the rows one.
        int iunit = 0, ichunk = 0;
        unsigned gi = 0, there = 0;
        DenseUnit ahead = {};
        int hrow[4], wrow[4], hnext[4], wnext[4];
        auto load_unit = [&](int i) { if (i < my_units) ahead = unit_of(i); };
        auto load_rows = [&]() {
            const int cls = ahead.cls[0] & 0xff;  // of both cells
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned r = (tid >> 3) + 32 * i;
                const unsigned row = (unsigned)ahead.row0 + r, col = (unsigned)ahead.col0[i / 2] + r % DC;
                wnext[i] = cls == 0 ? (row < n_dense_rows ? __ldg(dense_rows + row) : -1) : row < M ? (int)row : -1;  // 0: compacted full rows
                hnext[i] = cls == 1 ? (col < n_dense_cols ? __ldg(dense_cols + col) : -1) : col < N ? (int)col : -1;  // 1: compacted full columns
                if (i / 2 >= ahead.n) hnext[i] = -1;
            }
        };
        if (my_units > 0) {
            load_unit(0);
            load_rows();
            load_unit(1);
        }
        // Waits for the MMAs of chunk gi - 3, whose head stage chunk gi takes, and copies chunk gi (nothing past the end; an empty
        // group keeps the count uniform).  False on a timed-out wait.
        auto issue = [&]() -> bool {
            const unsigned s = gi % HEADS;
            if (gi >= HEADS && !wait_bar(&done_bar[s], (gi / HEADS - 1u) & 1u)) return false;
            if (gi < total) {
                if (ichunk == 0) {
                    there = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        there |= (unsigned)(hnext[i] >= 0) << i | (unsigned)(wnext[i] >= 0) << (4 + i);
                        hrow[i] = hnext[i] >= 0 ? hnext[i] : 0;
                        wrow[i] = wnext[i] >= 0 ? wnext[i] : 0;
                    }
                    load_rows();
                    load_unit(iunit + 2);
                }
                unsigned char *st = smem + s * STAGE_BYTES + tid * 16;
                const int k = ichunk * KC + kq;
                const unsigned in = k < K ? there : 0u;  // rows outside the matrix and k beyond K arrive as zeros
                const float *h = H + (k < K ? k : 0), *w = W + (k < K ? k : 0);
#pragma unroll
                for (int i = 0; i < 4; ++i) cp_async16_zfill(st + i * N_PRODUCERS * 16, h + (int64_t)hrow[i] * K, in >> i & 1u ? 16 : 0);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    cp_async16_zfill(st + TILE_BYTES + i * N_PRODUCERS * 16, w + (int64_t)wrow[i] * K, in >> (4 + i) & 1u ? 16 : 0);
                if (++ichunk == n_chunks) {
                    ichunk = 0;
                    ++iunit;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            ++gi;
            return true;
        };
        ok = issue() && issue();
        for (unsigned g = 0; g < total && ok; ++g) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // this thread's copies of chunk g have landed
            // the tail stage was last read by the MMAs of chunk g - 2: issue() has waited for those
            const unsigned char *head = smem + (g % HEADS) * STAGE_BYTES + tid * 16;
            unsigned char *tail = tails + (g % TAILS) * STAGE_BYTES + tid * 16;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                tail_store(*reinterpret_cast<const float4 *>(head + i * N_PRODUCERS * 16), tail + i * N_PRODUCERS * 16);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // my copies and stores -> visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[g % HEADS]);
            // only now the copies of chunk g + 2: they need the stage of chunk g - 1, whose MMAs ran meanwhile
            ok = issue();
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else if (warp == MMA_WARP) {
        // ---------------- MMA issue: the whole warp walks the loop, lane 0 issues ----------------
        unsigned g = 0;
        const uint64_t head0 = smem_desc(smem_u32(smem), LBO, SBO), tail0 = smem_desc(smem_u32(tails), LBO, SBO);
        for (int i = 0; i < my_units && ok; ++i) {
            const unsigned b = (unsigned)i % N_ACC;
            // the epilogue has read this accumulator
            if (!wait_bar(&acc_empty[b], ((unsigned)i / N_ACC & 1u) ^ 1u)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem + b * DR;
            for (int c = 0; c < n_chunks; ++c) {
                const unsigned s = g % HEADS;
                if (!wait_bar(&full_bar[s], (g / HEADS) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t head = head0 + s * (STAGE_BYTES >> 4), tail = tail0 + g % TAILS * (STAGE_BYTES >> 4);
                if (lane == 0) {
#pragma unroll
                    for (int ks = 0; ks < KC / 8; ++ks) {
                        const uint64_t o = ks * 2, w = TILE_BYTES >> 4;  // eight k = 32 bytes of every row per instruction; the W tile
                        mma_tf32_ss(d, head + o, tail + w + o, (c > 0 || ks > 0) ? 1u : 0u);  // a unit's very first MMA overwrites
                        mma_tf32_ss(d, tail + o, head + w + o, 1u);
                        mma_tf32_ss(d, head + o, head + w + o, 1u);
                    }
                    mma_commit(&done_bar[s]);  // arrives when the MMAs issued so far have finished reading the stages
                    if (c == n_chunks - 1) mma_commit(&acc_full[b]);
                }
                __syncwarp();
                ++g;
            }
        }
    } else {
        // ---------------- epilogue ----------------
        // Warp (group, quarter) reads rows 32 * group .. + 32 of the unit for the 32 columns of its quarter: half of the columns of
        // cell quarter / 2.
        const int ew = warp - EPI_WARP0, group = ew >> 2, quarter = warp & 3;
        const int sub = quarter >> 1, half = quarter & 1;
        EpiRows *const slots = epi_rows + ew * 2;
        const unsigned lane_bit = 1u << lane, below = lane_bit - 1u;
        // This warp's 32 rows of a unit pass through: descriptor, three units ahead -> the rows' geometry in registers (lane l: row l),
        // two ahead -> in shared memory -> S values, one ahead -> picked.  Nothing waits for a load it has just issued.
        int d_number = 0, d_n = 0, d_cls = 0;  // descriptor
        auto fetch_unit = [&](int i) {
            d_n = 0;
            if (i < my_units) {
                const DenseUnit &u = unit_of(i);
                d_number = __ldg(&u.number[sub]);
                d_n = __ldg(&u.n);
                d_cls = __ldg(&u.cls[sub]);
            }
        };
        // number (in table form, of the table) and form of this warp's cell of the unit in one word
        enum { TABLE, MASKED, RUNS, NONE };
        auto cell_of_unit = [&]() -> int {
            return sub >= d_n ? (int)NONE : d_number << 2 | (d_cls & CELL_RUNS ? RUNS : d_cls & CELL_MASKED ? MASKED : TABLE);
        };
        uint2 mask;
        int2 base;
        uint32_t span;
        auto fetch_rows = [&](int c) {
            mask = make_uint2(0u, 0u);
            if ((c & 3) == RUNS || (c & 3) == MASKED) {
                const int64_t line = (int64_t)(c >> 2) * DR + group * 32 + lane;
                mask = __ldg(reinterpret_cast<const uint2 *>(row_mask) + line);
                base = __ldg(row_base + line);
                span = __ldg(row_span + line);
            } else if ((c & 3) == TABLE) {
                // the lines of these rows into L2, a line for each lane: load_s would wait for them one batch after the other
                asm volatile("prefetch.global.L2 [%0];" ::"l"(table + ((int64_t)(c >> 2) * DR + group * 32 + lane) * DC + 32 * half));
            }
        };
        auto stage = [&](int c, EpiRows *slot) {
            const int before = half ? __popc(mask.x) : 0, first = (int)(span & 255u) - 32 * half;
            const int held = (int)(half ? mask.y : mask.x);
            __syncwarp();  // the rows that were in this slot have been picked
            if ((c & 3) == MASKED) slot->masked[lane] = make_int4(base.x + before, held, base.y + before, (int)(span >> 16) - 32 * half);
            else slot->run[lane] = make_int2(base.x - first, held);
            __syncwarp();
        };
        // input position of this lane's column in row u of the slot, if it is held
        auto masked_at = [&](const EpiRows *slot, int u) {
            const int4 r = slot->masked[u];
            return (unsigned)r.y & lane_bit ? (lane < r.w ? r.x : r.z) + __popc((unsigned)r.y & below) : -1;
        };
        auto table_at = [&](int c) { return table + ((int64_t)(c >> 2) * DR + group * 32) * DC + 32 * half + lane; };
        auto load_s = [&](int c, const EpiRows *slot, int t, float (&s)[BATCH]) {
            if (!sval) return;
            if ((c & 3) >= RUNS) {
                const float *const S_lane = sval + lane;
#pragma unroll
                for (int u = 0; u < BATCH; u += 2) {
                    const int4 r = *reinterpret_cast<const int4 *>(&slot->run[t * BATCH + u]);
                    load_if(s[u], S_lane + r.x, (unsigned)r.y & lane_bit);
                    load_if(s[u + 1], S_lane + r.z, (unsigned)r.w & lane_bit);
                }
            } else if ((c & 3) == MASKED) {
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int j = masked_at(slot, t * BATCH + u);
                    load_if(s[u], sval + j, j >= 0);
                }
            } else {
                const int32_t *tab = table_at(c);
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int j = __ldg(tab + (t * BATCH + u) * DC);
                    load_if(s[u], sval + j, j >= 0);
                }
            }
        };
        auto pick = [&](int c, const EpiRows *slot, int t, const uint32_t (&v)[BATCH], const float (&s)[BATCH]) {
            if ((c & 3) >= RUNS) {
                float *const P_lane = P + lane;
#pragma unroll
                for (int u = 0; u < BATCH; u += 2) {
                    const int4 r = *reinterpret_cast<const int4 *>(&slot->run[t * BATCH + u]);
                    store_if(P_lane + r.x, __uint_as_float(v[u]) * s[u], (unsigned)r.y & lane_bit);
                    store_if(P_lane + r.z, __uint_as_float(v[u + 1]) * s[u + 1], (unsigned)r.w & lane_bit);
                }
            } else if ((c & 3) == MASKED) {
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int j = masked_at(slot, t * BATCH + u);
                    store_if(P + j, __uint_as_float(v[u]) * s[u], j >= 0);
                }
            } else {
                const int32_t *tab = table_at(c);
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int j = __ldg(tab + (t * BATCH + u) * DC);
                    store_if(P + j, __uint_as_float(v[u]) * s[u], j >= 0);
                }
            }
        };
        float s[N_BATCH][BATCH];
#pragma unroll
        for (int t = 0; t < N_BATCH; ++t)
#pragma unroll
            for (int u = 0; u < BATCH; ++u) s[t][u] = 1.f;
        fetch_unit(0);
        int cell = cell_of_unit();
        fetch_rows(cell);
        fetch_unit(1);
        stage(cell, slots);
        int next = cell_of_unit();
        fetch_rows(next);
        fetch_unit(2);
#pragma unroll
        for (int t = 0; t < N_BATCH; ++t) load_s(cell, slots, t, s[t]);
#pragma unroll 1
        for (int i = 0; i < my_units; ++i) {
            EpiRows *const slot = slots + (i & 1), *const other = slots + (~i & 1);
            stage(next, other);
            const int then = cell_of_unit();
            fetch_rows(then);
            fetch_unit(i + 3);
            // One warp of the group polls, the barrier holds the others: polls take shared-memory bandwidth from the tensor core
            const unsigned b = (unsigned)i % N_ACC;
            ok = group_all(group, quarter != 0 || wait_bar(&acc_full[b], ((unsigned)i / N_ACC) & 1u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t block = tmem + ((uint32_t)(quarter * 32) << 16) + b * DR + group * 32;
#pragma unroll
            for (int t = 0; t < N_BATCH; ++t) {
                uint32_t v[BATCH];
                tmem_ld(v, block + t * BATCH);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (t == N_BATCH - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[b]);  // the accumulator may be overwritten
                }
                pick(cell, slot, t, v, s[t]);
                load_s(next, other, t, s[t]);
            }
            cell = next;
            next = then;
        }
    }
    if (!ok && lane == 0) report_timeout(dev_status);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
}

}  // namespace

cudaError_t launch_dense_cells_tc(const DensePlan &d, const float *sval, const float *W, const float *H, float *P, int64_t M, int64_t N,
                                  int K, int sm_count, int *dev_status, cudaStream_t stream)
{
    if (d.n_cells == 0) return cudaSuccess;
    int64_t blocks = sm_count;  // one persistent CTA per SM
    if (blocks > d.n_units) blocks = d.n_units;
    static SmemOptinCache optin;  // per device
    {
        cudaError_t e = optin_dynamic_smem(sddmm_dense_tc_kernel, TC_SMEM_BYTES, optin);
        if (e != cudaSuccess) return e;
    }
    sddmm_dense_tc_kernel<<<(unsigned)blocks, TC_THREADS, TC_SMEM_BYTES, stream>>>(
        d.units, d.n_units, d.table, d.row_mask, d.row_base, d.row_span, d.dense_rows, d.n_dense_rows, d.dense_cols, d.n_dense_cols,
        sval, W, H, P, M, N, K, dev_status);
    return cudaGetLastError();
}

}  // namespace sddmm
