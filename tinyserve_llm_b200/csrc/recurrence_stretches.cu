// The plain recurrence (gated linear attention, retention) over bfloat16 prompt portions, sixteen tokens at a time (the tile's algebra:
// recurrence_tiles.cu), its read-outs side by side.
//
//   o_t = sum_i q_(t,i) d_(t,i) S_0[i] + sum_{j<=t} P[t][j] v_j,   S_B = d_B S_0 + sum_j (k_j a_(j+1) ... a_B) v_j^T
//
// What a tile adds to the state does not depend on the state, so the chain through a portion is one multiply-add a tile.  Three kernels:
//   prepare   per tile and head the "pack", in the order of the fragments below: queries with the decays up to them, P, the decays over
//             the tile, keys with the decays behind them, values;
//   states    walks the tiles and keeps the state before every stretch of STRETCH tiles, and the one behind the portion; a CTA owns a
//             head, 32 rows and 64 columns of the state (of eight such CTAs a head each reads a quarter of the keys and half the values);
//   read-out  all stretches side by side, each from the state kept for it; a CTA owns a head and 32 columns.  Inside a stretch it moves the
//             state on by the same operations as the states kernel, so every state is the number one walk over the whole portion would
//             have there: where a prompt was cut at multiples of sixteen tokens does not show.
//
// Arithmetic.  Values are bfloat16 numbers.  Keys and P enter as three bfloat16 pieces each, x = b0 + b1 + b2, which hold all 24 bits; their
// products with values are exact, the large ones (b0) of a tile's sixteen tokens summed by one MMA that begins at zero, the small ones by two
// more, and both sums are added by ordinary float32 additions.  Queries and the state they meet are split into two TF32 numbers as in
// recurrence_tiles.cu, every eight channels' large parts in an MMA of their own.  Relative error of outputs / states against 64 bits, gated
// linear attention over 2,048 tokens: see there.
//
// A value that is infinite or NaN is left out of the product with P (0 times it would be NaN) and added to the rows from its own on.
//
// Measured on a B200, 2,048 tokens, 8 heads of 128 x 256, us: preparation 31 -> 32 (it now lays out values and pieces too), one walk that did
// all 141 (one warp a scheduler in a chain of products) -> states 25, read-outs 39.  The states are bound by a step's own chain of shared
// memory reads, MMAs and a barrier (with two steps less in flight 32, with copies a thread computes addresses for 41); the read-outs by
// instructions: 48 % of issue slots, 317 a warp and tile of 32 columns where the walk had 677 for 16.
#include "recurrence_tiles.cuh"

namespace {

constexpr int STRETCH = 8;                               // tiles: 128 tokens
constexpr int WALK_COLS = 64, WALK_WARPS = 16, WALK_TILES = 4, WALK_STAGES = 4;   // of a CTA of the states kernel; tiles a step, steps in flight
constexpr int READ_COLS = 32, READ_WARPS = 4;            // of a CTA of the read-out
constexpr int RP = READ_COLS + 8;                        // pitch of the partial sums: a warp's fragments fall into different banks

// Fragments of mma.sync, lane = 4 r + c (r 0..7, c 0..3).  m16n8k8 (TF32): A (r, c), (r + 8, c), (r, c + 4), (r + 8, c + 4); B (c, r),
// (c + 4, r).  m16n8k16 (bfloat16 pairs): A (r, 2c..), (r + 8, 2c..), (r, 2c + 8..), (r + 8, 2c + 8..); B (2c.., r), (2c + 8.., r).
// C of both: (r, 2c), (r, 2c + 1), (r + 8, 2c), (r + 8, 2c + 1).
// The state is held as C fragments of S^T (16 columns x 8 rows of S).  As B fragments of S for the queries they hold rows 2c and
// 2c + 1 where the product counts k = c and c + 4: the queries' fragments take their channels in the same order.
//
// A pack, for ROWS rows, in words of four bytes:
//   queries [ROWS / 8][lane][4] float32 | P [3 pieces][lane][4] | by 32 rows: keys [4][3 pieces][lane][2], decays [32] float32 |
//   values [blocks of 16 columns][lane][4], columns up to a multiple of 64
constexpr int ROW_BLOCK = 32, KEY_WORDS = 24 * ROW_BLOCK, ROW_WORDS = KEY_WORDS + ROW_BLOCK;      // of 32 rows
__host__ __device__ constexpr int p_at(int rows) { return 16 * rows; }
__host__ __device__ constexpr int rows_at(int rows) { return p_at(rows) + 384; }
__host__ __device__ constexpr int values_at(int rows) { return rows_at(rows) + rows / ROW_BLOCK * ROW_WORDS; }
__host__ __device__ constexpr int pack_words(int rows, int blocks) { return values_at(rows) + 128 * blocks; }

__device__ __forceinline__ uint32_t pair_of(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float low_of(uint32_t x) { return __uint_as_float(x << 16); }
__device__ __forceinline__ float high_of(uint32_t x) { return __uint_as_float(x & 0xffff0000u); }
// Two numbers as three pairs of bfloat16 pieces.
__device__ __forceinline__ void pieces_of(float x0, float x1, uint32_t (&piece)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        piece[i] = pair_of(x0, x1);
        x0 -= low_of(piece[i]);
        x1 -= high_of(piece[i]);
    }
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16_fresh(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void load_values(uint32_t (&v)[4], const float* block, int lane) {
    const uint4 x = *reinterpret_cast<const uint4*>(block + 4 * lane);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
// Eight rows of sixteen columns of the state after a tile; v the values of those columns, k the keys' pieces of those rows, d the decays
// of rows 2c and 2c + 1.
__device__ __forceinline__ void advance(float (&S)[4], const uint32_t (&v)[4], const uint2 (&k)[3], float2 d) {
    float big[4], small[4];
    mma_bf16_fresh(small, v, k[2].x, k[2].y);
    mma_bf16(small, v, k[1].x, k[1].y);
    mma_bf16_fresh(big, v, k[0].x, k[0].y);
    S[0] = fmaf(d.x, S[0], big[0] + small[0]);
    S[1] = fmaf(d.y, S[1], big[1] + small[1]);
    S[2] = fmaf(d.x, S[2], big[2] + small[2]);
    S[3] = fmaf(d.y, S[3], big[3] + small[3]);
}

struct StretchArgs {
    float* pack;
    const __nv_bfloat16* v; long long v_stride;          // elements between tokens; a head's values start at h * vdim
    const int* cu_q; const int* slots; const int* prefill_seqs;
    float* state; long long slot_stride;                 // floats between slots; a slot holds [heads, dim, vdim]
    float* kept;                                         // states before stretches: [stretches][heads][blocks][G][lane][4]
    float* out;                                          // [tokens, heads * vdim] float32
    int heads, dim, vdim;
    int blocks;                                          // blocks of 16 columns in a pack and in `kept`
};

// Where the state before a stretch lies: numbered as tiles are, in stretches.
__device__ __forceinline__ float4* kept_state(const StretchArgs& p, int rows, int seq, int begin, int stretch, int h, int block) {
    const long long at = ((begin / (B * STRETCH) + seq + stretch) * (long long)p.heads + h) * p.blocks + block;
    return reinterpret_cast<float4*>(p.kept + at * rows * 16);
}

// grid (tiles, heads, portions), 128 threads
template <int ROWS>
__global__ void __launch_bounds__(128, ROWS == 128 ? 7 : 1) stretch_prepare_kernel(PlainArgs p, StretchArgs s) {
    extern __shared__ float smem[];
    __shared__ float scores[B][B + 1];
    const int seq = p.prefill_seqs[blockIdx.z], tile = blockIdx.x, h = blockIdx.y;
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || tile * B >= n) return;
    const int t0 = begin + tile * B, m = min(B, n - tile * B);
    const PlainTile<ROWS> x(smem);
    load_plain<__nv_bfloat16, ROWS>(p, x, h, t0, m);
    float* pack = s.pack + (tile_slot(seq, begin, tile) * p.heads + h) * pack_words(ROWS, s.blocks);
    for (int col = threadIdx.x; col < 16 * s.blocks; col += 128) {       // zeros past the portion's tokens and the head's columns
        const __nv_bfloat16* v = s.v + (long long)t0 * s.v_stride + (long long)h * s.vdim + min(col, s.vdim - 1);
        __nv_bfloat16 e[B];
#pragma unroll
        for (int t = 0; t < B; ++t) e[t] = v[min(t, m - 1) * s.v_stride];
        uint32_t* to = reinterpret_cast<uint32_t*>(pack + values_at(ROWS) + (col / 16 * 32 + 4 * (col % 8)) * 4 + (col >> 3 & 1));
#pragma unroll
        for (int c = 0; c < 8; ++c) {                    // tokens 2c, 2c + 1: lane c % 4 of the column's four, its second pair from c = 4 on
            const uint32_t lo = __bfloat16_as_ushort(e[2 * c]), hi = __bfloat16_as_ushort(e[2 * c + 1]);
            to[c % 4 * 4 + c / 4 * 2] = col < s.vdim ? (2 * c < m ? lo : 0u) | (2 * c + 1 < m ? hi << 16 : 0u) : 0u;
        }
    }
    __syncthreads();
    plain_scores<ROWS>(x, p.dim, [&](int t, int j, float y) { scores[t][j] = y; });
    for (int i = threadIdx.x; i < ROWS; i += 128) {
        const int g = i / 8, c = i % 8 / 2, odd = i & 1;
        float* rows = pack + rows_at(ROWS) + i / ROW_BLOCK * ROW_WORDS;
        float q[B], k[B];
        rows[KEY_WORDS + i % ROW_BLOCK] = plain_sides<ROWS>(x, i, [&](int t, float y) { q[t] = y; }, [&](int t, float y) { k[t] = y; });
#pragma unroll
        for (int r = 0; r < 8; ++r)
            *reinterpret_cast<float2*>(pack + (g * 32 + 4 * r + c) * 4 + 2 * odd) = make_float2(q[r], q[r + 8]);
        uint32_t piece[8][3];                            // lane 4 (i % 8) + c holds tokens 2c, 2c + 1 and 2c + 8, 2c + 9
#pragma unroll
        for (int e = 0; e < 8; ++e) pieces_of(k[2 * (e >> 1) + 8 * (e & 1)], k[2 * (e >> 1) + 8 * (e & 1) + 1], piece[e]);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            uint4* to = reinterpret_cast<uint4*>(rows + ((i % ROW_BLOCK / 8 * 3 + b) * 32 + 4 * (i % 8)) * 2);
            to[0] = make_uint4(piece[0][b], piece[1][b], piece[2][b], piece[3][b]);
            to[1] = make_uint4(piece[4][b], piece[5][b], piece[6][b], piece[7][b]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int r = threadIdx.x >> 2, c = threadIdx.x & 3;
        uint32_t piece[4][3];
#pragma unroll
        for (int e = 0; e < 4; ++e) pieces_of(scores[r + 8 * (e & 1)][2 * c + 8 * (e >> 1)], scores[r + 8 * (e & 1)][2 * c + 8 * (e >> 1) + 1], piece[e]);
#pragma unroll
        for (int b = 0; b < 3; ++b)
            *reinterpret_cast<uint4*>(pack + p_at(ROWS) + (b * 32 + threadIdx.x) * 4) = make_uint4(piece[0][b], piece[1][b], piece[2][b], piece[3][b]);
    }
}

constexpr int WALK_TILE = ROW_WORDS + 8 * WALK_COLS;       // words of a tile: keys and decays of 32 rows, values of 64 columns

// grid (row blocks x column blocks, heads, portions).  Warp w: rows 8 (w % 4) .. + 7 and columns 16 (w / 4) .. + 15 of the CTA's.
template <int ROWS>
__global__ void __launch_bounds__(WALK_WARPS * 32) stretch_states_kernel(StretchArgs p) {
    constexpr int THREADS = WALK_WARPS * 32, ROW_BLOCKS = ROWS / ROW_BLOCK, STAGE = WALK_TILES * WALK_TILE;
    extern __shared__ __align__(16) float smem[];
    chain_wait();
    const int row0 = blockIdx.x % ROW_BLOCKS * ROW_BLOCK, j0 = blockIdx.x / ROW_BLOCKS * WALK_COLS, h = blockIdx.y, seq = p.prefill_seqs[blockIdx.z];
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin, slot = p.slots[seq];
    if (n <= 1 || slot < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const int group = warp & 3, col = warp / 4 * 16;
    float* st = p.state + (long long)slot * p.slot_stride + (long long)h * p.dim * p.vdim;
    auto element = [&](int e, int& i, int& j) {
        i = row0 + 8 * group + 2 * c + (e & 1);
        j = j0 + col + r + 8 * (e >> 1);
        return i < p.dim && j < p.vdim;
    };
    float S[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        int i, j;
        S[e] = element(e, i, j) ? st[(long long)i * p.vdim + j] : 0.f;
    }
    const int tiles = (n + B - 1) / B;
    // what this thread copies of every tile: 16 bytes of the rows' part of the pack, or of the columns'
    static_assert(WALK_TILE / 4 <= THREADS, "a thread a piece");
    const long long pack_step = (long long)p.heads * pack_words(ROWS, p.blocks);
    const float* from = p.pack + tile_slot(seq, begin, 0) * pack_step + (long long)h * pack_words(ROWS, p.blocks) + 4 * tid +
                        (4 * tid < ROW_WORDS ? rows_at(ROWS) + row0 / ROW_BLOCK * ROW_WORDS : values_at(ROWS) + 8 * j0 - ROW_WORDS);
    auto issue = [&](int tile0) {
        float* stage = smem + tile0 / WALK_TILES % WALK_STAGES * STAGE + 4 * tid;
        if (4 * tid < WALK_TILE) {
#pragma unroll
            for (int k = 0; k < WALK_TILES; ++k) {
                if (tile0 + k < tiles) cp16(stage + k * WALK_TILE, from);
                from += pack_step;
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    constexpr int AHEAD = (WALK_STAGES - 1) * WALK_TILES;        // a step takes a fifth of a trip to L2
#pragma unroll
    for (int k = 0; k < AHEAD; k += WALK_TILES) issue(k);
    for (int tile0 = 0; tile0 < tiles; tile0 += WALK_TILES) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(WALK_STAGES - 2) : "memory");
        __syncthreads();                                 // these tiles are in, and the stage of those before has been read
        issue(tile0 + AHEAD);                            // (past the last tile: an empty group)
        static_assert(STRETCH % WALK_TILES == 0, "a stretch begins with a step");
        if (tile0 % STRETCH == 0)
            kept_state(p, ROWS, seq, begin, tile0 / STRETCH, h, (j0 + col) / 16)[(row0 / 8 + group) * 32 + lane] = make_float4(S[0], S[1], S[2], S[3]);
        const float* stage = smem + tile0 / WALK_TILES % WALK_STAGES * STAGE;
        auto step = [&](int k) {
            const float* tile = stage + k * WALK_TILE;
            uint2 key[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) key[b] = *reinterpret_cast<const uint2*>(tile + ((group * 3 + b) * 32 + lane) * 2);
            const float2 d = *reinterpret_cast<const float2*>(tile + KEY_WORDS + 8 * group + 2 * c);
            uint32_t v[4];
            load_values(v, tile + ROW_WORDS + 8 * col, lane);
            advance(S, v, key, d);
        };
        if (tile0 + WALK_TILES <= tiles) {
#pragma unroll
            for (int k = 0; k < WALK_TILES; ++k) step(k);
        } else {
            for (int k = 0; k < tiles - tile0; ++k) step(k);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        int i, j;
        if (element(e, i, j)) st[(long long)i * p.vdim + j] = S[e];
    }
}

__device__ __forceinline__ bool not_finite(uint32_t x, uint32_t exponent) { return (x & exponent) == exponent; }
constexpr uint32_t LOW_EXPONENT = 0x7f80u, HIGH_EXPONENT = 0x7f800000u;

// What values that are not finite (as a B fragment: tokens 2c, 2c + 1 and 2c + 8, 2c + 9 of column r) add to tokens at or after them, by P's
// pieces: a C fragment.  Out of line: it is hardly ever called.
__device__ __noinline__ float4 add_odd_values(const uint32_t* pieces, uint32_t b0, uint32_t b1, int r, int c) {
    float y[4] = {};
    for (int j = 0; j < B; ++j)
        for (int side = 0; side < 2; ++side) {
            const uint32_t x0 = __shfl_sync(0xffffffffu, b0, 4 * (2 * c + side) + (j & 7) / 2), x1 = __shfl_sync(0xffffffffu, b1, 4 * (2 * c + side) + (j & 7) / 2);
            const uint32_t x = j < 8 ? x0 : x1;
            const float v = j & 1 ? high_of(x) : low_of(x);
            if (isfinite(v)) continue;
            for (int half = 0; half < 2; ++half) {
                if (j > r + 8 * half) continue;
                float s = 0.f;
                for (int b = 2; b >= 0; --b) {
                    const uint32_t w = pieces[(b * 32 + 4 * r + (j & 7) / 2) * 4 + half + 2 * (j >> 3)];
                    s += j & 1 ? high_of(w) : low_of(w);
                }
                y[2 * half + side] = fmaf(s, v, y[2 * half + side]);
            }
        }
    return make_float4(y[0], y[1], y[2], y[3]);
}

// grid (stretches x column blocks, heads, portions).  Warp w holds rows 8 NT w .. of the state, and makes the outputs of columns 8 w .. + 7.
template <int NT>
__global__ void __launch_bounds__(READ_WARPS * 32) stretch_read_kernel(StretchArgs p) {
    constexpr int ROWS = READ_WARPS * 8 * NT, THREADS = READ_WARPS * 32, SHARED = values_at(ROWS), STAGE = SHARED + 8 * READ_COLS;
    static_assert(READ_COLS == 8 * READ_WARPS, "a warp makes eight columns of the output");
    extern __shared__ __align__(16) float smem[];
    float* red = smem + 2 * STAGE;                       // [READ_WARPS][16][RP]
    chain_wait();
    const int col_blocks = (p.vdim + READ_COLS - 1) / READ_COLS;
    const int j0 = blockIdx.x % col_blocks * READ_COLS, stretch = blockIdx.x / col_blocks, h = blockIdx.y, seq = p.prefill_seqs[blockIdx.z];
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || p.slots[seq] < 0) return;
    const int tile0 = stretch * STRETCH, tiles = min((n + B - 1) / B, tile0 + STRETCH);
    if (tile0 >= tiles) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const long long first = tile_slot(seq, begin, 0);
    auto issue = [&](int tile) {
        float* stage = smem + (tile & 1) * STAGE;
        const float* pack = p.pack + ((first + tile) * p.heads + h) * pack_words(ROWS, p.blocks);
#pragma unroll
        for (int e = 0; e < SHARED / 4; e += THREADS)
            if (e + tid < SHARED / 4) cp16(stage + 4 * (e + tid), pack + 4 * (e + tid));
        if (tid < 2 * READ_COLS) cp16(stage + SHARED + 4 * tid, pack + values_at(ROWS) + 8 * j0 + 4 * tid);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(tile0);
    float S[NT][2][4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const float4* from = kept_state(p, ROWS, seq, begin, stretch, h, j0 / 16 + half);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const float4 x = from[(warp * NT + nt) * 32 + lane];
            S[nt][half][0] = x.x, S[nt][half][1] = x.y, S[nt][half][2] = x.z, S[nt][half][3] = x.w;
        }
    }
    for (int tile = tile0; tile < tiles; ++tile) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();                                 // the tile is in; the other stage and the sums have been read
        if (tile + 1 < tiles) issue(tile + 1);
        const float* pack = smem + (tile & 1) * STAGE;
        {   // the queries against this warp's rows of S
            float big[4][4] = {}, small[4][4] = {};
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const float4 q = *reinterpret_cast<const float4*>(pack + ((warp * NT + nt) * 32 + lane) * 4);
                const SplitA a = split_a(q.x, q.y, q.z, q.w);
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int side = 0; side < 2; ++side)
                        mma_split<true>(big[2 * half + side], small[2 * half + side], a, split_tf32(S[nt][half][2 * side]), split_tf32(S[nt][half][2 * side + 1]));
            }
#pragma unroll
            for (int nj = 0; nj < 4; ++nj)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<float2*>(red + (warp * B + r + 8 * half) * RP + 8 * nj + 2 * c) =
                        make_float2(big[nj][2 * half] + small[nj][2 * half], big[nj][2 * half + 1] + small[nj][2 * half + 1]);
        }
        uint32_t v[2][4];                                // values of columns 0..15 and 16..31
#pragma unroll
        for (int half = 0; half < 2; ++half) load_values(v[half], pack + SHARED + 128 * half, lane);
        if (tile + 1 < tiles) {                          // the state after the tile
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int group = warp * NT + nt;
                const float* rows = pack + rows_at(ROWS) + group / 4 * ROW_WORDS;
                uint2 key[3];
#pragma unroll
                for (int b = 0; b < 3; ++b) key[b] = *reinterpret_cast<const uint2*>(rows + ((group % 4 * 3 + b) * 32 + lane) * 2);
                const float2 d = *reinterpret_cast<const float2*>(rows + KEY_WORDS + group % 4 * 8 + 2 * c);
#pragma unroll
                for (int half = 0; half < 2; ++half) advance(S[nt][half], v[half], key, d);
            }
        }
        __syncthreads();                                 // the partial sums are in
        {
            uint32_t b0 = 0, b1 = 0;                     // the values of this warp's columns as a B fragment
#pragma unroll
            for (int w = 0; w < READ_WARPS; ++w)
                if (w == warp) b0 = v[w / 2][w & 1], b1 = v[w / 2][2 + (w & 1)];
            float4 late = make_float4(0.f, 0.f, 0.f, 0.f);
            const bool odd = not_finite(b0, LOW_EXPONENT) || not_finite(b0, HIGH_EXPONENT) || not_finite(b1, LOW_EXPONENT) || not_finite(b1, HIGH_EXPONENT);
            if (__any_sync(0xffffffffu, odd)) {
                late = add_odd_values(reinterpret_cast<const uint32_t*>(pack + p_at(ROWS)), b0, b1, r, c);
                if (not_finite(b0, LOW_EXPONENT)) b0 &= 0xffff0000u;
                if (not_finite(b0, HIGH_EXPONENT)) b0 &= 0xffffu;
                if (not_finite(b1, LOW_EXPONENT)) b1 &= 0xffff0000u;
                if (not_finite(b1, HIGH_EXPONENT)) b1 &= 0xffffu;
            }
            uint32_t a[3][4];
#pragma unroll
            for (int b = 0; b < 3; ++b) load_values(a[b], pack + p_at(ROWS) + 128 * b, lane);
            float big[4], small[4];
            mma_bf16_fresh(small, a[2], b0, b1);
            mma_bf16(small, a[1], b0, b1);
            mma_bf16_fresh(big, a[0], b0, b1);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float q0 = 0.f, q1 = 0.f;
#pragma unroll
                for (int w = 0; w < READ_WARPS; ++w) {
                    const float2 q = *reinterpret_cast<const float2*>(red + (w * B + r + 8 * half) * RP + 8 * warp + 2 * c);
                    q0 += q.x;
                    q1 += q.y;
                }
                const float y0 = q0 + (big[2 * half] + small[2 * half] + (half ? late.z : late.x));
                const float y1 = q1 + (big[2 * half + 1] + small[2 * half + 1] + (half ? late.w : late.y));
                const int t = tile * B + r + 8 * half, j = j0 + 8 * warp + 2 * c;
                if (t < n) {
                    float* dst = p.out + ((long long)(begin + t) * p.heads + h) * p.vdim + j;
                    if (j < p.vdim) dst[0] = y0;
                    if (j + 1 < p.vdim) dst[1] = y1;
                }
            }
        }
    }
}

int blocks_of(int vdim) { return (vdim + WALK_COLS - 1) / WALK_COLS * (WALK_COLS / 16); }
long long packs_floats(int num_tokens, int num_seqs, int heads, int dim, int vdim) {
    return ((long long)num_tokens / B + num_seqs + 1) * heads * pack_words(padded_rows(dim), blocks_of(vdim));
}
long long kept_floats(int num_tokens, int num_seqs, int heads, int dim, int vdim) {
    return ((long long)num_tokens / (B * STRETCH) + num_seqs + 1) * heads * blocks_of(vdim) * padded_rows(dim) * 16;
}

template <int ROWS>
int launch(const PlainArgs& a, const StretchArgs& p, int portions, int max_q_len, cudaStream_t stream) {
    const int tiles = (max_q_len + B - 1) / B;
    const size_t prepare_smem = PlainTile<ROWS>::BYTES;
    auto prepare = stretch_prepare_kernel<ROWS>;
    cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prepare_smem);
    prepare<<<dim3(tiles, p.heads, portions), 128, prepare_smem, stream>>>(a, p);
    TS_LAUNCH_CHECK("plain_tiles (prepare)");
    const size_t walk_smem = sizeof(float) * WALK_STAGES * WALK_TILES * WALK_TILE;
    auto walk = stretch_states_kernel<ROWS>;
    cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem);
    const dim3 walk_grid(ROWS / ROW_BLOCK * ((p.vdim + WALK_COLS - 1) / WALK_COLS), p.heads, portions);
    TS_CHAINED_CHECK("plain_tiles (states)", launch_chained(walk, walk_grid, dim3(WALK_WARPS * 32), walk_smem, stream, p));
    const size_t read_smem = sizeof(float) * (2 * (values_at(ROWS) + 8 * READ_COLS) + READ_WARPS * B * RP);
    auto read = stretch_read_kernel<ROWS / (8 * READ_WARPS)>;
    cudaFuncSetAttribute(read, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)read_smem);
    const long long blocks = (long long)((p.vdim + READ_COLS - 1) / READ_COLS) * ((tiles + STRETCH - 1) / STRETCH);
    TS_REQUIRE(blocks < 0x7fffffffll, "plain_tiles: grid too large");
    TS_CHAINED_CHECK("plain_tiles (read-out)", launch_chained(read, dim3((unsigned)blocks, p.heads, portions), dim3(READ_WARPS * 32), read_smem, stream, p));
    return 0;
}

}  // namespace

long long plain_stretches_floats(int num_tokens, int num_seqs, int heads, int dim, int vdim) {
    return packs_floats(num_tokens, num_seqs, heads, dim, vdim) + kept_floats(num_tokens, num_seqs, heads, dim, vdim);
}

int plain_stretches(const PlainArgs& a, const __nv_bfloat16* v, long long v_stride, const int* slots, int portions, int max_q_len, float* state,
                    long long slot_stride, int num_tokens, int num_seqs, float* out, int vdim, cudaStream_t stream) {
    float* kept = a.pack + packs_floats(num_tokens, num_seqs, a.heads, a.dim, vdim);
    const StretchArgs p{a.pack, v, v_stride, a.cu_q, slots, a.prefill_seqs, state, slot_stride, kept, out, a.heads, a.dim, vdim, blocks_of(vdim)};
    const int rows = padded_rows(a.dim);
    return rows == 64 ? launch<64>(a, p, portions, max_q_len, stream) : rows == 128 ? launch<128>(a, p, portions, max_q_len, stream)
                                                                                    : launch<256>(a, p, portions, max_q_len, stream);
}
