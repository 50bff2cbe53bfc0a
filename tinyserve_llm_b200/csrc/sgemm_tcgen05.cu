// float32 matrix product y[M, N] = x[M, K] . W[N, K]^T on the fifth-generation tensor cores, to float32's own accuracy.
//
// Every operand enters as the sum of two TF32 numbers, v = hi + lo (hi is v to the nearest of 11 significant bits, lo the rest,
// of which the tensor cores drop the last bit: 2^-23 of v), and W x = W_hi x_hi + W_hi x_lo + W_lo x_hi in tcgen05.mma kind::tf32
// with float32 accumulators; the small terms go first.  The tensor cores cut what an accumulator cannot hold, so they add up 32
// terms of k only: a block's sum leaves tensor memory and is added to the running sum in registers by an ordinary rounded
// addition (every second block's: 3 to 7 % faster, twice the error).  Measured against 64-bit products: 1.9e-7 (2,048 terms) and 1.8e-7 (8,192), where the multiply-add chain of sgemm.cu is
// 8.0e-7 and 1.6e-6 off; 1.3e-7 against 1.5e-7 at 64 terms.  An element that comes out infinite or NaN (infinite inputs, for
// which hi + lo does not stand, or an overflow) is worked out again by that chain, so such elements are what plain arithmetic gives.
//
// A row's result does not depend on what else is in the batch: the blocks of k, the segments k is cut into and the order
// they are added up in follow from N and K alone, and the rows' tile (the MMA's N side) does not enter an element's sum.
//
// Two CTAs a tile (`cta_group::2`): 256 rows of W, 128 in each CTA (the MMA's lanes), against BX rows of x, half in each CTA; the first CTA's
// thread issues the MMAs for both.  x is split into two matrices by a kernel ahead.  Per CTA: warp 0 issues TMA loads into a ring of raw
// tiles of W, warp 2 those of x's two tiles, warp 1 the MMAs, warps 4..11 split W (two teams, a block each): a thread puts its row into
// tensor memory as hi and lo (the MMA's A operand, so that neither passes through shared memory again); the warps from 12 on add the blocks'
// sums up.
// mbarriers: `raw_full` / `raw_empty` TMA <-> split, `ready` / `free` split and TMA of x <-> MMA, `sum_full` / `sum_empty` MMA <-> adders; `ready`
// and `sum_empty` are the first CTA's, on which both CTAs' warps arrive, `free` and `sum_full` are signalled in both.
// Split warps that wrote x's tiles would have to release each block's at cluster scope for MMAs the other CTA issues: 33 -> 50 us in the first
// row below at 1 row, 45 -> 57 at 100 (released by warps of their own 42 and 53).  Up to 16 rows the first CTA holds all of them, splits them itself, with
// no such order, and the second one's half is zeros (LOCAL): a kernel less, 2.5 us.
// K is cut into segments, enough of them that the tiles of W times the segments fill the SMs.  Where there are rows of x enough
// to fill them anyway a pair takes the segments one after another and adds each one's sum to y; else each segment is a pair's
// work, its sums go to scratch, and a second kernel adds them up in the same order.
// Measured on a B200, products with cold weights one after another, us: sgemm.cu, this product with one CTA a tile and the MMAs issued by
// one lane, and now:
//   rows of x             1                8               100              300             512             1,024
//   16,384 x 2,048   192 / 53 / 34   192 / 53 / 35    306 / 63 / 48     - / 170 / 127   - / 222 / 174    - / 405 / 331
//   2,048 x 8,192                    677 / 29 / 21    636 / 36 / 31     -  / 89 / 70    - / 118 / 96     - / 275 / 186
//   3,072 x 2,048                                                     241 /  86 / 37     - / 115 / 48
// A block of k took 0.75 to 0.93 us whatever BX was: 12 MMAs issued by one lane are 58 cycles each at the least (elect_one), and x's
// tile, loaded and split whole by every CTA, moved more bytes through shared memory than W's.  Now 0.48 (BX 32), 0.57 (64) and 0.68 us
// (128), of which the MMAs at the tensor cores' rate are 0.1, 0.22 and 0.41; W's stream alone takes 30 us in the first row.  What is left
// is the adders' reading of tensor memory (7 us in the first row at 128 rows), the split (3) and a pair in seven without a tile there.
//
// Every wait on an mbarrier gives up after about two seconds and records where in an error word the host reads.
#include "tcgen05.cuh"

namespace {

constexpr int BW = 128, BK = 32;                     // rows of W a CTA, half of a tile; k a block: 128 bytes, one swizzled row
constexpr int X_WARP = 2, SPLIT_WARPS = 4, SPLITS_FROM = 4, ADDERS_FROM = SPLITS_FROM + 2 * SPLIT_WARPS;    // two teams of split warps
__host__ __device__ constexpr int share_of(int bx) { return bx >= 64 ? 4 : 2; }           // adder warps a quarter of the lanes
__host__ __device__ constexpr int threads_of(int bx) { return 32 * (ADDERS_FROM + 4 * share_of(bx)); }
constexpr int W_BYTES = BW * BK * 4;
constexpr int PAIRS_OF_SMS = 74;
constexpr long long MAX_SCRATCH = 64ll << 20;        // floats: more than that and the segments are taken in turn
constexpr int MIN_SEGMENT = 8;                       // blocks of k a segment has at least (256 terms)

struct SgemmParams {
    float* y;                                        // output, or the segments' sums [segments][M][N]
    const float* x;
    const float* w;
    int M, N, K;
    long long ldx, ldw, ldy, segment_stride;
    int blocks, per_segment, in_turn;                // blocks of k in all, and a segment; 1: a CTA takes all segments in turn
    int items;                                       // tiles, times segments unless in turn: a pair's
    int* error;
};

// A from tensor memory (the 128 lanes of either CTA the rows, a column a number of K), B from both CTAs' shared memory
__device__ __forceinline__ void umma_tf32(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]),
          "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}

// v to the nearest number of 11 significant bits.  The rest, v - hi, has at most 12, of which the tensor cores drop the last; past
// the largest number hi is infinite and the rest NaN, and for a NaN the rest is one, so the sum never hides either.
__device__ __forceinline__ float to_tf32(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); }

__device__ __forceinline__ void split_four(float4 v, float4& hi, float4& lo) {
    hi = make_float4(to_tf32(v.x), to_tf32(v.y), to_tf32(v.z), to_tf32(v.w));
    lo = make_float4(v.x - hi.x, v.y - hi.y, v.z - hi.z, v.w - hi.w);
}

struct Item { int n0, m0, segment, first, count; };    // a pair's piece of work: a tile and the blocks of k it takes
__device__ __forceinline__ Item item_of(const SgemmParams& p, int item, int bx) {
    const int n_tiles = (p.N + 2 * BW - 1) / (2 * BW), m_tiles = (p.M + bx - 1) / bx;
    Item it;
    it.n0 = item % n_tiles * 2 * BW;
    it.m0 = item / n_tiles % m_tiles * bx;
    it.segment = item / n_tiles / m_tiles;
    it.first = it.segment * p.per_segment;
    it.count = p.in_turn ? p.blocks : min(p.per_segment, p.blocks - it.first);
    return it;
}

// A persistent CTA an SM: the four kinds of warps walk over the same items, each counting blocks (g) over all of them, so that
// the loads and MMAs of an item run under the sums of the one before.
// LOCAL: x's rows (raw, map_hi) fill at most the first CTA's half of the tile, which splits them itself; the second one's half is zeros.
template <int BX, int RING, int PAIRS, int SUMS, bool LOCAL>
__global__ void __launch_bounds__(threads_of(BX), 1)
sgemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                     SgemmParams p) {
    // RING of W (LOCAL: and x); PAIRS of [x hi | x lo], this CTA's half of the rows
    constexpr int X_BYTES = BX / 2 * BK * 4, RAW_BYTES = W_BYTES + (LOCAL ? X_BYTES : 0);
    constexpr int A_COLS = SUMS * BX, TMEM_USED = A_COLS + PAIRS * 2 * BK;            // PAIRS of [W hi | W lo]
    constexpr int TMEM_COLS = TMEM_USED <= 256 ? 256 : 512;
    static_assert(TMEM_USED <= 512, "tensor memory has 512 columns");
    // a slot's barrier is waited on by one team only: the other could come to it a round early, where the parity it waits
    // for stands for the round before the first
    static_assert(RING % 2 == 0 && PAIRS % 2 == 0, "a ring slot and a pair of operand tiles belong to one team");
    static_assert(W_BYTES % 1024 == 0 && X_BYTES % 1024 == 0, "tiles lie on the swizzle's boundaries");
    constexpr int OWN = BX / share_of(BX);           // columns of an adder
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t raw_full_bar[RING], raw_empty_bar[RING], ready_bar[PAIRS], free_bar[PAIRS], sum_full_bar[SUMS], sum_empty_bar[SUMS];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int failed;
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* x_tiles = ring + RING * RAW_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)pair_rank(), pair = blockIdx.x / 2, pairs = gridDim.x / 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < RING; ++s) {
            mbar_init(&raw_full_bar[s], 1);
            mbar_init(&raw_empty_bar[s], SPLIT_WARPS);
        }
        for (int b = 0; b < PAIRS; ++b) {
            mbar_init(&ready_bar[b], 2 * SPLIT_WARPS + (LOCAL ? 0 : 1));          // both CTAs' split warps, and x's bytes
            mbar_init(&free_bar[b], 1);
        }
        for (int b = 0; b < SUMS; ++b) {
            mbar_init(&sum_full_bar[b], 1);
            mbar_init(&sum_empty_bar[b], 2 * 4 * share_of(BX));
        }
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot;
    if (LOCAL && rank) {
        for (int e = threadIdx.x; e < PAIRS * 2 * X_BYTES / 16; e += threads_of(BX)) reinterpret_cast<float4*>(x_tiles)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    pair_sync();                                     // both CTAs' barriers exist, and the zeros
    chain_wait();
    chain_release();

    // The adders' sums want more registers than an even share: the launch's 896 x 72 as 128 x 40 + 256 x 56 + 512 x 88.
    constexpr bool SHARES = threads_of(BX) == 896;
    if (warp < SPLITS_FROM) {
        if (SHARES) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            int g = 0;
            for (int at = pair; at < p.items && !failed; at += pairs) {
                const Item it = item_of(p, at, BX);
                for (int i = 0; i < it.count; ++i, ++g) {
                    const int s = g % RING;
                    if (!mbar_wait(&raw_empty_bar[s], ((g / RING) & 1) ^ 1, p.error, 21)) { failed = 1; break; }
                    mbar_expect_tx(&raw_full_bar[s], LOCAL && rank == 0 ? RAW_BYTES : W_BYTES);
                    tma_load_2d(ring + s * RAW_BYTES, &map_w, &raw_full_bar[s], (it.first + i) * BK, it.n0 + rank * BW);
                    if (LOCAL && rank == 0) tma_load_2d(ring + s * RAW_BYTES + W_BYTES, &map_hi, &raw_full_bar[s], (it.first + i) * BK, it.m0);
                }
            }
        } else if (!LOCAL && warp == X_WARP && lane == 0) {
            int g = 0;
            for (int at = pair; at < p.items && !failed; at += pairs) {
                const Item it = item_of(p, at, BX);
                for (int i = 0; i < it.count; ++i, ++g) {
                    const int a = g % PAIRS;
                    if (!mbar_wait(&free_bar[a], ((g / PAIRS) & 1) ^ 1, p.error, 27)) { failed = 1; break; }
                    const uint32_t ready = in_first_cta(&ready_bar[a]);
                    if (rank == 0) mbar_expect_tx(&ready_bar[a], 4 * X_BYTES);        // of both CTAs
                    unsigned char* tile = x_tiles + a * 2 * X_BYTES;
                    tma_load_2d_pair(tile, &map_hi, ready, (it.first + i) * BK, it.m0 + rank * (BX / 2));
                    tma_load_2d_pair(tile + X_BYTES, &map_lo, ready, (it.first + i) * BK, it.m0 + rank * (BX / 2));
                }
            }
        } else if (warp == 1 && rank == 0) {
            // float32 accumulator, TF32 operands, B K-major, 256 x BX over both CTAs; the warp as one, so that operands stay in uniform registers
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BX >> 3) << 17) | ((uint32_t)(2 * BW >> 4) << 24);
            const uint32_t leader = elect_one();
            int g = 0;
            bool ok = true;                          // the same in all lanes
            for (int at = pair; at < p.items && ok; at += pairs) {
                const Item it = item_of(p, at, BX);
                for (int i = 0; i < it.count; ++i, ++g) {
                    const int a = g % PAIRS, b = g % SUMS;
                    ok = mbar_wait(&sum_empty_bar[b], ((g / SUMS) & 1) ^ 1, p.error, 24) &&
                         mbar_wait(&ready_bar[a], (g / PAIRS) & 1, p.error, 23) && !failed;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { failed = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t w_hi = tmem_base + A_COLS + a * 2 * BK, w_lo = w_hi + BK, d = tmem_base + b * BX;
                    const uint64_t x_hi = smem_desc(x_tiles + a * 2 * X_BYTES), x_lo = smem_desc(x_tiles + a * 2 * X_BYTES + X_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 8; ++k) umma_tf32(leader, d, w_hi + 8 * k, x_lo + 2 * k, idesc, k != 0);   // 8 numbers of K: 8 columns, 32 bytes
#pragma unroll
                    for (int k = 0; k < BK / 8; ++k) umma_tf32(leader, d, w_lo + 8 * k, x_hi + 2 * k, idesc, 1);
#pragma unroll
                    for (int k = 0; k < BK / 8; ++k) umma_tf32(leader, d, w_hi + 8 * k, x_hi + 2 * k, idesc, 1);
                    if (leader) {
                        umma_commit_pair(&free_bar[a]);
                        umma_commit_pair(&sum_full_bar[b]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < ADDERS_FROM) {
        if (SHARES) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // blocks in turn between the teams: a block's split is a chain of waits, loads and stores, and two run side by side
        const int team = (warp - SPLITS_FROM) / SPLIT_WARPS, quarter = warp & 3, row = quarter * 32 + lane;   // a warp reaches the quarter of the lanes its number gives
        const uint32_t lane_addr = tmem_base + A_COLS + ((uint32_t)(quarter * 32) << 16);
        int total = 0;
        for (int at = pair; at < p.items; at += pairs) total += item_of(p, at, BX).count;
        for (int g = team; g < total; g += 2) {
            const int s = g % RING, a = g % PAIRS;
            bool ok = mbar_wait(&raw_full_bar[s], (g / RING) & 1, p.error, 22) && !failed;
            ok = ok && mbar_wait(&free_bar[a], ((g / PAIRS) & 1) ^ 1, p.error, 26);
            if (!__all_sync(0xffffffffu, ok)) { failed = 1; break; }                  // what follows wants the whole warp
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned char* w_row = ring + s * RAW_BYTES + row * 128;            // 16-byte piece c lies at c ^ (row % 8)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float hi[16], lo[16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(w_row + (((4 * half + c) ^ (row & 7)) << 4));
                    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        hi[4 * c + j] = to_tf32(e[j]);
                        lo[4 * c + j] = e[j] - hi[4 * c + j];
                    }
                }
                tmem_st16(lane_addr + a * 2 * BK + 16 * half, hi);
                tmem_st16(lane_addr + a * 2 * BK + BK + 16 * half, lo);
            }
            if (LOCAL && rank == 0) {
                const float4* raw = reinterpret_cast<const float4*>(ring + s * RAW_BYTES + W_BYTES);
                float4* x_hi = reinterpret_cast<float4*>(x_tiles + a * 2 * X_BYTES);
                for (int e = quarter * 32 + lane; e < X_BYTES / 16; e += 32 * SPLIT_WARPS)
                    split_four(raw[e], x_hi[e], x_hi[X_BYTES / 16 + e]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");          // the MMAs read x through the async proxy
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if (rank == 0) mbar_arrive(&ready_bar[a]);
                else mbar_arrive_remote(in_first_cta(&ready_bar[a]));
                mbar_arrive(&raw_empty_bar[s]);
            }
        }
    } else {
        if (SHARES) asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
        const int quarter = warp & 3, side = (warp - ADDERS_FROM) >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + side * OWN;
        float sum[OWN];
#pragma unroll
        for (int j = 0; j < OWN; ++j) sum[j] = 0.f;
        int sums = 0;
        bool ok = true;                              // the same in all lanes
        for (int at = pair; at < p.items && ok; at += pairs) {
            const Item it = item_of(p, at, BX);
            const int n = it.n0 + rank * BW + quarter * 32 + lane, m_first = it.m0 + side * OWN;
            for (int from = 0; from < it.count && ok; from += p.per_segment) {        // a segment
                const int blocks = min(p.per_segment, it.count - from);
                for (int i = 0; i < blocks; ++i, ++sums) {
                    const int b = sums % SUMS;
                    ok = __all_sync(0xffffffffu, mbar_wait(&sum_full_bar[b], (sums / SUMS) & 1, p.error, 25) && !failed);
                    if (!ok) { failed = 1; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t v[OWN];
#pragma unroll
                    for (int j = 0; j < OWN; j += 8) tmem_ld8(lane_addr + b * BX + j, v + j);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");  // read: the accumulator goes back before the additions
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(in_first_cta(&sum_empty_bar[b]));
#pragma unroll
                    for (int j = 0; j < OWN; ++j) sum[j] += __uint_as_float(v[j]);
                }
                if (!ok) break;
                float* y = p.y + it.segment * p.segment_stride + (long long)m_first * p.ldy + n;
                const int k0 = (it.first + from) * BK, k1 = min(p.K, k0 + blocks * BK);
                const int rows = n < p.N ? p.M - m_first : 0;
                uint32_t odd = 0;
                if (from) {                          // the segments before this one: a few loads under way together
                    const float* at_y = y;
#pragma unroll
                    for (int j0 = 0; j0 < OWN; j0 += 8) {
                        float before[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j, at_y += p.ldy) before[j] = j0 + j < rows ? *at_y : 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (!isfinite(sum[j0 + j])) odd |= 1u << (j0 + j);
                            sum[j0 + j] += before[j];
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < OWN; ++j)
                        if (!isfinite(sum[j])) odd |= 1u << j;
                }
                if (rows < OWN) odd &= rows > 0 ? (1u << rows) - 1 : 0;      // hi + lo does not stand for infinite or the largest numbers
                float* to_y = y;
#pragma unroll
                for (int j = 0; j < OWN; ++j, to_y += p.ldy) {
                    if (j < rows && !(odd >> j & 1)) *to_y = sum[j];
                    sum[j] = 0.f;
                }
                // Those again by multiply-adds.  A row of x with a NaN, which padding may be, gives NaN everywhere: one look tells.
                for (int j = 0; j < OWN && __any_sync(0xffffffffu, odd >> j); ++j) {
                    const bool mine = odd >> j & 1;
                    if (!__any_sync(0xffffffffu, mine)) continue;
                    const float* x = p.x + (m_first + j) * p.ldx;
                    float v = 0.f;
                    bool nan = false;
                    for (int k = k0 + lane; k < k1; k += 32) nan |= x[k] != x[k];
                    if (__any_sync(0xffffffffu, nan)) v = __uint_as_float(0x7fffffffu);
                    else if (mine)
                        for (int k = k0; k < k1; ++k) v = fmaf(x[k], p.w[n * p.ldw + k], v);
                    if (mine) y[j * p.ldy] = from ? y[j * p.ldy] + v : v;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_sync();                                     // neither CTA leaves while the other's MMAs or arrivals may reach it
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// y[m, n] = the segments' sums in order; four neighbours a thread where rows allow
template <int V>
__global__ void __launch_bounds__(256) add_segments_kernel(const float* __restrict__ parts, float* __restrict__ y, int segments,
                                                           long long segment_stride, int M, int N, long long ldy) {
    chain_wait();
    chain_release();
    const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= (long long)M * N) return;
    float sum[V];
#pragma unroll
    for (int j = 0; j < V; ++j) sum[j] = parts[e + j];
#pragma unroll 4
    for (int s = 1; s < segments; ++s) {
        float next[V];
        if (V == 4) *reinterpret_cast<float4*>(next) = *reinterpret_cast<const float4*>(parts + s * segment_stride + e);
        else next[0] = parts[s * segment_stride + e];
#pragma unroll
        for (int j = 0; j < V; ++j) sum[j] += next[j];
    }
    float* out = y + e / N * ldy + e % N;
    if (V == 4) *reinterpret_cast<float4*>(out) = *reinterpret_cast<float4*>(sum);
    else out[0] = sum[0];
}

// How K is cut, from N and K alone: enough segments that the tiles of W fill the SMs once, none shorter than MIN_SEGMENT blocks.
void cut(int N, int K, int* blocks, int* per_segment, int* segments) {
    *blocks = (K + BK - 1) / BK;
    const int tiles = (N + 2 * BW - 1) / (2 * BW);
    int s = PAIRS_OF_SMS / tiles;
    if (s > *blocks / MIN_SEGMENT) s = *blocks / MIN_SEGMENT;
    if (s < 1) s = 1;
    *per_segment = (*blocks + s - 1) / s;
    *segments = (*blocks + *per_segment - 1) / *per_segment;
}

// x as two TF32 numbers an element, in matrices of their own [M][K].  Its error: to_tf32.  Bound by its launch: 100 to 512 rows of 2,048 take 3.5
// to 4 us by themselves, 2.5 in a chain.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, long long ldx, float* __restrict__ hi,
                                                         float* __restrict__ lo, int M, int K) {
    chain_wait();
    chain_release();
    const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= (long long)M * K) return;
    split_four(*reinterpret_cast<const float4*>(x + e / K * ldx + e % K), *reinterpret_cast<float4*>(hi + e), *reinterpret_cast<float4*>(lo + e));
}

// hi, lo: x's pieces in rows of K, or null: LOCAL
template <int BX, int RING, int PAIRS, int SUMS, bool LOCAL>
int launch(SgemmParams p, const float* hi, const float* lo, int segments, cudaStream_t stream) {
    CUtensorMap map_w, map_hi, map_lo;
    if (make_tile_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p.w, p.N, p.K, p.ldw, BW, "sgemm_tcgen05")) return 1;
    if (make_tile_map(&map_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, LOCAL ? p.x : hi, p.M, p.K, LOCAL ? p.ldx : p.K, BX / 2, "sgemm_tcgen05")) return 1;
    if (LOCAL) map_lo = map_hi;                          // not read
    else if (make_tile_map(&map_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, lo, p.M, p.K, p.K, BX / 2, "sgemm_tcgen05")) return 1;
    constexpr size_t smem = (size_t)RING * (W_BYTES + (LOCAL ? BX / 2 * BK * 4 : 0)) + PAIRS * BX * BK * 4 + 1024;
    static_assert(smem <= 226 * 1024, "shared memory of an SM");
    auto kernel = sgemm_tcgen05_kernel<BX, RING, PAIRS, SUMS, LOCAL>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    p.items = ((p.N + 2 * BW - 1) / (2 * BW)) * ((p.M + BX - 1) / BX) * (p.in_turn ? 1 : segments);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (p.items < PAIRS_OF_SMS ? p.items : PAIRS_OF_SMS));
    cfg.blockDim = dim3(threads_of(BX));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ts_chaining_enabled() ? 2 : 1;
    TS_CHAINED_CHECK("sgemm_tcgen05", cudaLaunchKernelEx(&cfg, kernel, map_w, map_hi, map_lo, p));
    return 0;
}

// Rows of x a CTA, and whether it takes the segments in turn.  Neither enters an element's sum.
struct Shape { int bx, in_turn; };
Shape choose(int M, int N, int blocks, int per_segment, int segments) {
    static const struct { int bx; double ns; } kinds[3] = {{32, 480}, {64, 570}, {128, 680}};   // of a block of k, as measured
    Shape best{128, segments > 1};
    double least = 1e30;
    for (const auto& kind : kinds)
        for (int in_turn = 0; in_turn < (segments > 1 ? 2 : 1); ++in_turn) {
            if (segments > 1 && !in_turn && (long long)segments * M * N > MAX_SCRATCH) continue;
            const long long items = (long long)((N + 2 * BW - 1) / (2 * BW)) * ((M + kind.bx - 1) / kind.bx) * (in_turn ? 1 : segments);
            // in turn, each segment but the first waits for the sums before it to come back from memory
            double ns = (double)((items + PAIRS_OF_SMS - 1) / PAIRS_OF_SMS) *
                        (500.0 + (in_turn ? blocks : per_segment) * kind.ns + (in_turn ? (segments - 1) * 3000.0 : 0.0));
            if (segments > 1 && !in_turn) ns += 2500.0 + (double)segments * M * N * 8.0 / 5000.0;     // the second kernel
            if (ns < least) {
                least = ns;
                best = Shape{kind.bx, in_turn};
            }
        }
    return best;
}

}  // namespace

// Terms from which on a sum of split products is no further from 64 bits than the multiply-add chain.  Below, what the split drops counts
// for more than the chain's roundings (relative error, chain and here: 4 terms 4.0e-8 / 9.3e-8, 16 7.4e-8 / 1.0e-7, 32 1.03e-7 / 1.30e-7,
// 48 1.25e-7 both, 64 1.43e-7 / 1.34e-7, 2,048 8.1e-7 / 1.5e-7).
constexpr int MIN_TERMS = 64;

// 1 if the sum is long enough and TMA takes the sizes and addresses: 16-byte aligned bases and rows.
bool sgemm_tcgen05_supported(const float* x, const float* w, int K, long long ldx, long long ldw) {
    return K >= MIN_TERMS && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0;
}

// Rows of x that the first CTA of a pair splits itself: half of the narrowest tile.
constexpr int LOCAL_ROWS = 16;

// Rows of x that are split at a time: their pieces stay within MAX_SCRATCH (no fewer than a tile of rows).
static int rows_at_once(int M, int K) {
    const long long rows = MAX_SCRATCH / 2 / K / 128 * 128;
    return rows >= M ? M : rows < 128 ? (M < 128 ? M : 128) : (int)rows;
}

// Floats of scratch a product of these sizes needs: x's pieces, and the segments' sums where they are apart.
long long sgemm_tcgen05_scratch_floats(int M, int N, int K) {
    int blocks, per, segments;
    cut(N, K, &blocks, &per, &segments);
    const int rows = rows_at_once(M, K);
    long long sums = 0;
    for (const int m : {rows, M % rows}) {
        const long long need = (long long)segments * m * N;
        if (m > 0 && segments > 1 && !choose(m, N, blocks, per, segments).in_turn && need > sums) sums = need;
    }
    return (M <= LOCAL_ROWS ? 0 : 2ll * rows * K) + sums;
}

static int run_rows(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, float* scratch,
                    float* sums, int* error, cudaStream_t stream) {
    int blocks, per, segments;
    cut(N, K, &blocks, &per, &segments);
    const Shape shape = choose(M, N, blocks, per, segments);
    const bool parts = segments > 1 && !shape.in_turn;
    const bool local = M <= LOCAL_ROWS;
    float *hi = local ? nullptr : scratch, *lo = local ? nullptr : scratch + (long long)M * K;
    if (!local) {
        const long long pieces = (long long)M * K / 4;
        TS_CHAINED_CHECK("sgemm_tcgen05 (split)", launch_chained(split_rows_kernel, dim3((unsigned)((pieces + 255) / 256)), dim3(256), 0,
                                                                 stream, x, ldx, hi, lo, M, K));
    }
    SgemmParams p{parts ? sums : y, x, w, M, N, K, ldx, ldw, parts ? N : ldy, parts ? (long long)M * N : 0, blocks, per,
                  shape.in_turn, 0, error};
    const int failed = local ? launch<32, 10, 4, 4, true>(p, hi, lo, segments, stream)
                     : shape.bx == 32 ? launch<32, 10, 6, 4, false>(p, hi, lo, segments, stream)
                     : shape.bx == 64 ? launch<64, 10, 4, 4, false>(p, hi, lo, segments, stream) : launch<128, 10, 4, 2, false>(p, hi, lo, segments, stream);
    if (failed || !parts) return failed;
    const bool vec = N % 4 == 0 && ldy % 4 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)sums % 16 == 0;
    const long long items = (long long)M * N / (vec ? 4 : 1);
    auto kernel = vec ? add_segments_kernel<4> : add_segments_kernel<1>;
    TS_CHAINED_CHECK("sgemm_tcgen05 (segments)",
                     launch_chained(kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, stream, (const float*)sums, y,
                                    segments, (long long)M * N, M, N, ldy));
    return 0;
}

int sgemm_tcgen05(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                  float* scratch, int* error, cudaStream_t stream) {
    const int rows = rows_at_once(M, K);
    float* sums = scratch + (M <= LOCAL_ROWS ? 0 : 2ll * rows * K);
    for (int m = 0; m < M; m += rows)
        if (run_rows(x + m * ldx, w, y + m * ldy, M - m < rows ? M - m : rows, N, K, ldx, ldw, ldy, scratch, sums, error, stream)) return 1;
    return 0;
}
