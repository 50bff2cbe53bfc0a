// Paged causal grouped-query softmax attention in float32 for prompt portions and single tokens: tiles of query rows against tiles
// of 64 keys, both products with multiply-adds in float32.  (attention_generic.cu walks over the keys once per token and head.)
//
// A CTA owns one kv head and a run of tokens of one request; its rows are (token, head of the group), so a key tile is read
// once for all heads of the group.  16 x 8 threads (BQ 32) or 16 x 4 (BQ 16: steps of single tokens), each with four rows and
// four keys of the scores, then the same four rows and HD / 16 channels of the output.  Keys and values come by cp.async, the next
// tile's keys under this tile's softmax and second product, the next values under the next scores.
//
// The order of every sum depends on the query's position only: key tiles count from key 0, a score is a chain over the
// channels, a row's weights and its output are chains over the keys of a tile, masked keys add exact zeros.  BQ does not enter.
//
// What bounds it: the multiply-adds and the 16-byte reads that feed them (8 for 64 of them), with two to four warps a scheduler to
// hide both; a step of a few rows the serial walk over its key tiles.  Measured on a B200, 32:8 heads of 64, us, before (one warp a
// token and head, every key row read from L2 by each) and now: 512 tokens 598 / 61; 600 tokens 819 / 76; 4 portions of up to 150
// behind up to 400 467 / 54; 64 tokens behind 4,000 1,114 / 290; 8 single tokens behind 2,000 163 / 157; one behind 400 42 / 38.
// Taken are heads of 64 and 128 channels in groups of two and more.  Both sides over other sizes: heads of 16 and 32 have forms of
// their own in the generic kernel (8 single tokens behind 2,000, 32:8 heads of 32: 108 / 157), heads between would be padded (32:8 of 80:
// 171 / 260; of 112, 32:4: 209 / 255), and a group of one leaves fifteen of a single token's sixteen rows empty (64 single
// tokens behind 500, 16:16 heads of 128: 163 / 261; 32 behind 150, 32:32 of 64: 32 / 43).  With groups of two nothing was slower
// (16:8 heads of 64, 8 single tokens behind 2,000: 157 / 149, 512 tokens 323 / 47; of 128 426 / 252 and 654 / 81).
// The bounds by `hd` cut nothing off, but with HD in their place the compiler unrolls the loads of a tile ahead of everything else: 8
// single tokens behind 2,000 take 171 us (16:8 of 64) and 288 (24:8 of 128) instead of 149 and 248.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BK = 64, TX = 16, PP = BK + 4;         // keys a tile; threads across; pitch of the weights

__device__ __forceinline__ void cp16(float* smem, const float* gmem, bool ok) {
    const int bytes = ok ? 16 : 0;                   // 0: zeros are written
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

struct Args {
    const float* q; long long q_stride;
    float* out;
    const float* k_pool; const float* v_pool;
    KVGeometry geo;
    const int* block_table; int table_width;
    const int* positions; const int* cu_q;
    int num_tokens, num_seqs, steps, nh, nkv, window;  // steps: the largest power of two up to num_seqs
    int hd;                                          // HD, which the kernel takes as a number it does not know (see below)
    float scale;
};

// Padding rows behind the last request: zeros, so that nothing that reads them meets NaNs of someone else's memory.  Out of line: in line
// it takes registers from the loop over the keys (24:8 heads of 128, 8 single tokens behind 2,000: 247 -> 257 us).
__device__ __noinline__ void clear_padding(float* out, const int* end, int num_tokens, int first, int stride, long long row, int width) {
    for (int t = *end + first; t < num_tokens; t += stride)
        for (int d = threadIdx.x; d < width; d += blockDim.x) out[t * row + d] = 0.f;
}

template <int HD, int BQ>
__global__ void __launch_bounds__(BQ * 4) paged_attention_f32_kernel(Args p) {
    constexpr int THREADS = BQ * 4, PITCH = HD + 4, NC = HD / 64;                     // NC: runs of four channels a thread
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                // [BQ][PITCH]
    float* ks = qs + BQ * PITCH;                     // [BK][PITCH]
    float* vs = ks + BK * PITCH;
    float* ps = vs + BK * PITCH;                     // [BQ][PP]
    __shared__ int first_key[BQ], last_key[BQ];
    __shared__ long long key_at[2][BK];
    const int kvh = blockIdx.x, group = p.nh / p.nkv, per_tile = BQ / group;
    // request s's tiles begin at cu_q[s] / per_tile + s, which leaves room for its last, partly filled one; the tiles with the
    // most keys before them go first
    const int tile_at = gridDim.y - 1 - blockIdx.y;
    clear_padding(p.out + (long long)kvh * group * HD, p.cu_q + p.num_seqs, p.num_tokens, tile_at, gridDim.y, p.nh * HD, group * HD);
    int seq = 0;
    for (int step = p.steps; step > 0; step >>= 1)
        if (seq + step < p.num_seqs && p.cu_q[seq + step] / per_tile + seq + step <= tile_at) seq += step;
    const int begin = p.cu_q[seq], t0 = begin + (tile_at - begin / per_tile - seq) * per_tile;
    const int tokens = min(per_tile, p.cu_q[seq + 1] - t0), rows = tokens * group;
    if (tokens <= 0) return;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;

    for (int e = tid; e < BQ * (HD / 4); e += THREADS) {
        const int r = e / (HD / 4), d = e % (HD / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows && d < p.hd)
            v = *reinterpret_cast<const float4*>(p.q + (t0 + r / group) * p.q_stride + (long long)(kvh * group + r % group) * p.hd + d);
        *reinterpret_cast<float4*>(qs + r * PITCH + d) = make_float4(v.x * p.scale, v.y * p.scale, v.z * p.scale, v.w * p.scale);
    }
    for (int r = tid; r < BQ; r += THREADS) {
        const int pos = r < rows ? p.positions[t0 + r / group] : -1;
        last_key[r] = pos;
        first_key[r] = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    }
    __syncthreads();
    const int from = first_key[0] / BK, to = last_key[rows - 1] / BK;                 // positions rise along a run
    const int* table = p.block_table + (long long)seq * p.table_width;
    const int keys_end = last_key[rows - 1] + 1;
    const long long head_off = p.geo.entry_offset + (long long)kvh * p.geo.page_tokens * p.hd;
    // Where a tile's keys lie, looked up a tile ahead; -1: a page given back or a bad table, and the key is not seen.
    auto locate = [&](int tile) {
        for (int r = tid; r < BK; r += THREADS) {
            const int j = tile * BK + r, page = j < keys_end ? table[j / p.geo.page_tokens] : -1;
            key_at[tile & 1][r] = page >= 0 && page < p.geo.num_pages
                                      ? (long long)page * p.geo.page_stride + head_off + (long long)(j % p.geo.page_tokens) * p.hd : -1;
        }
    };
    auto load = [&](float* dst, const float* pool, int tile) {
        for (int e = tid; e < BK * (HD / 4); e += THREADS) {
            const int r = e / (HD / 4), d = e % (HD / 4) * 4;
            const long long at = key_at[tile & 1][r];
            const bool ok = at >= 0 && d < p.hd;
            cp16(dst + r * PITCH + d, ok ? pool + at + d : pool, ok);
        }
        commit();
    };
    float o[4][NC * 4], m[4], l[4];
    int lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
        lo[i] = first_key[ty * 4 + i];
        hi[i] = last_key[ty * 4 + i];
#pragma unroll
        for (int c = 0; c < NC * 4; ++c) o[i][c] = 0.f;
    }
    const bool live = (ty & ~1) * 4 < rows;          // a warp holds two of the sixteen rows of threads: one without rows only loads
    locate(from);
    __syncthreads();
    load(ks, p.k_pool, from);
    load(vs, p.v_pool, from);
    for (int tile = from; tile <= to; ++tile) {
        wait_group<1>();
        __syncthreads();                             // the tile's keys are in
        if (tile < to) locate(tile + 1);
        float s[4][4];
        if (live) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty * 4 + i) * PITCH + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + TX * j) * PITCH + d);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                        s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                        s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                        s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                    }
            }
        }
        __syncthreads();                             // the keys have been read
        if (tile < to) load(ks, p.k_pool, tile + 1);
        else commit();                               // an empty group: the count of groups stays
        if (live) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = tile * BK + tx + TX * j;
                const bool there = key_at[tile & 1][tx + TX * j] >= 0;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (!there || key < lo[i] || key > hi[i]) s[i][j] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float top = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
                for (int x = TX / 2; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
                const float next = fmaxf(m[i], top);
                const float base = next == -INFINITY ? 0.f : next;                    // nothing seen yet: every weight is 0
                const float shrink = next == m[i] ? 1.f : expf(m[i] - base);
                m[i] = next;
                l[i] *= shrink;
#pragma unroll
                for (int c = 0; c < NC * 4; ++c) o[i][c] *= shrink;
#pragma unroll
                for (int j = 0; j < 4; ++j) ps[(ty * 4 + i) * PP + tx + TX * j] = s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - base);
            }
        }
        wait_group<1>();
        __syncthreads();                             // the tile's values and weights are in
        // a tile with keys that some row does not see: those are stepped over, whatever lies in their values
        auto add_values = [&](auto edge) {
#pragma unroll 2
            for (int j = 0; j < BK; j += 4) {
                float w[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(ps + (ty * 4 + i) * PP + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const int key = tile * BK + j + jj;
                    float4 v[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) v[c] = *reinterpret_cast<const float4*>(vs + (j + jj) * PITCH + 64 * c + tx * 4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (edge.value && (key < lo[i] || key > hi[i])) continue;
                        l[i] += w[i][jj];
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            o[i][4 * c] = fmaf(w[i][jj], v[c].x, o[i][4 * c]);
                            o[i][4 * c + 1] = fmaf(w[i][jj], v[c].y, o[i][4 * c + 1]);
                            o[i][4 * c + 2] = fmaf(w[i][jj], v[c].z, o[i][4 * c + 2]);
                            o[i][4 * c + 3] = fmaf(w[i][jj], v[c].w, o[i][4 * c + 3]);
                        }
                    }
                }
            }
        };
        if (live) {
            if (tile * BK + BK - 1 > last_key[0] || tile * BK < first_key[rows - 1]) add_values(std::true_type{});
            else add_values(std::false_type{});
        }
        __syncthreads();                             // the values and weights have been read
        if (tile < to) load(vs, p.v_pool, tile + 1);
        else commit();
    }
    wait_group<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (r >= rows) continue;
        const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
        float* out = p.out + ((long long)(t0 + r / group) * p.nh + kvh * group + r % group) * p.hd;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = 64 * c + tx * 4;
            if (d < p.hd)
                *reinterpret_cast<float4*>(out + d) = make_float4(o[i][4 * c] * inv, o[i][4 * c + 1] * inv, o[i][4 * c + 2] * inv, o[i][4 * c + 3] * inv);
        }
    }
}

// Query rows a CTA: 16 where every request feeds one token, whose group's heads are all the rows there are.  Else 32, not 64: twice
// the CTAs to share out (512 tokens, 32:8 heads of 64: 84 against 102 us before the tiles went longest first).
int rows_of(int max_q_len) { return max_q_len <= 1 ? 16 : 32; }
long long tiles_of(int num_tokens, int num_seqs, int group, int rows) { return (long long)num_tokens / (rows / group) + num_seqs; }

template <int HD, int BQ>
int launch(const Args& p, int num_tokens, cudaStream_t stream) {
    constexpr size_t smem = sizeof(float) * ((BQ + 2 * BK) * (HD + 4) + BQ * PP);
    auto kernel = paged_attention_f32_kernel<HD, BQ>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<dim3(p.nkv, (unsigned)tiles_of(num_tokens, p.num_seqs, p.nh / p.nkv, BQ)), BQ * 4, smem, stream>>>(p);
    TS_LAUNCH_CHECK("paged_attention_f32");
    return 0;
}

}  // namespace

// Whether these sizes and addresses are taken: 16-byte rows, the sizes named above, a group's heads inside a tile, no more tiles
// than a grid holds (131,000 prompt tokens and more: so many have no steps of other sizes beside them).  Which
// of the two kernels takes a model's attention follows from its sizes alone, so a row's result stays independent of its step.
TS_API int ts_paged_attention_f32_takes(int nh, int nkv, int hd) { return (hd == 64 || hd == 128) && nh / nkv >= 2 && nh / nkv <= 16; }

bool paged_attention_f32_supported(const void* q, long long q_stride, const void* out, const void* k_pool, const void* v_pool,
                                   const KVGeometry& geo, int num_seqs, int num_tokens, int max_q_len, int nh, int nkv, int hd) {
    return ts_paged_attention_f32_takes(nh, nkv, hd) && nkv <= 65535 && q_stride % 4 == 0 && geo.page_stride % 4 == 0 && geo.entry_offset % 4 == 0 &&
           ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) % 16 == 0 &&
           tiles_of(num_tokens, num_seqs, nh / nkv, rows_of(max_q_len)) <= 65535;
}

int paged_attention_f32(const float* q, long long q_stride, float* out, const float* k_pool, const float* v_pool, KVGeometry geo,
                        const int* block_table, int table_width, const int* positions, const int* cu_q, int num_seqs,
                        int num_tokens, int max_q_len, int nh, int nkv, int hd, float scale, int window, cudaStream_t stream) {
    int steps = 1;
    while (2 * steps <= num_seqs) steps *= 2;
    const Args p{q, q_stride, out, k_pool, v_pool, geo, block_table, table_width, positions, cu_q, num_tokens, num_seqs, steps, nh, nkv, window, hd, scale};
    if (rows_of(max_q_len) == 16) return hd == 64 ? launch<64, 16>(p, num_tokens, stream) : launch<128, 16>(p, num_tokens, stream);
    return hd == 64 ? launch<64, 32>(p, num_tokens, stream) : launch<128, 32>(p, num_tokens, stream);
}
