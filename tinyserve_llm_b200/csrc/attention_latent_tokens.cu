// Attention over a cached latent for prompt portions: the computation of attention_latent_mma.cu (mma.sync m16n8k16 on bfloat16
// operands, the folded query's latent part and the probabilities each as the sum of two bfloat16 pieces, float32 softmax and
// sums), four consecutive tokens of a request a CTA instead of one: those whose positions are the same but for their last two bits, so
// that the order of a token's sums depends on its position only, wherever the portion was cut.  Requests that feed one token are left
// to the other kernel.
//
// The tokens' windows overlap in all but three keys at either end, so a tile of keys is read from L2 once for 4 x 16 rows (token,
// head) where it was read for 16.  Eight warps.  Scores: a warp takes one token's 16 heads and 16 of the tile's 32 keys.  Output: a
// warp takes all 64 rows and an eighth of the channels (128 registers a thread at 512 channels).  Two key tiles of 32 rows, the next
// one on its way by cp.async.  Keys that only some of the four tokens see (at most six) come as a tile of their own, whose weights
// meet the values by plain multiply-adds under a row's own mask; all other tiles hold keys that every token sees.
//
// Measured on a B200, 16 heads, latent of 512 + 64 channels, window 1,024, us, one token a CTA and now: 2,048 tokens 723 / 504, 1,000
// behind 2,000 cached ones 461 / 360, 514 242 / 181 (other sizes: ts_latent_attention_portions).  A tile takes 4.8 us, of which its MMAs are 2.2: two warps a
// scheduler wait on one another's products and reads.  Tried and no faster: scores and values in warps of their own a tile apart (539
// at 2,048 tokens), scores by quarters of the channels with half the ldmatrix (537).
#include "mma_tile.cuh"

namespace {

constexpr int TOKENS = 4, HEADS = 16, ROWS = TOKENS * HEADS, KEYS = 32, WARPS = 8, PAD = 8, EDGE = 8, PPITCH = KEYS + PAD;

struct LatentArgs {
    const float* q_lat; long long ql_token_stride, ql_head_stride;
    const __nv_bfloat16* q; long long q_stride;
    int q_head_width, q_rot_offset;
    const float* freq; float magnitude; const float* sink;
    const __nv_bfloat16* k_pool; KVGeometry geo;
    const int* block_table; int table_width;
    const int* positions; const int* seq_of_token; const int* cu_q;
    int num_seqs, steps;                             // steps: the largest power of two up to num_seqs
    __nv_bfloat16* out;
    int heads, rot; float scale; int window;
    int wide;                                        // 1: 16-byte loads of q_lat
};

__host__ __device__ constexpr size_t latent_tokens_smem(int rank, int rot) {
    return (size_t)(ROWS + 2 * KEYS) * (rank + rot + PAD) * 2 + (size_t)ROWS * (rank + PAD) * 2 + (size_t)2 * ROWS * PPITCH * 2 +
           (size_t)ROWS * EDGE * 4 + (size_t)3 * ROWS * 4 + (size_t)2 * KEYS * 8;
}

// NT: eights of output channels a warp (rank = 64 NT)
template <int NT>
__global__ void __launch_bounds__(WARPS * 32, 1) latent_attention_tokens_kernel(LatentArgs p) {
    constexpr int RANK = 64 * NT, LPITCH = RANK + PAD, THREADS = WARPS * 32;
    extern __shared__ __align__(16) unsigned char raw[];
    const int width = RANK + p.rot, pitch = width + PAD;
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(raw);            // [64][pitch]: the folded queries, rounded
    __nv_bfloat16* Ks = Qs + ROWS * pitch;                                // [2][32][pitch]
    __nv_bfloat16* Ql = Ks + 2 * KEYS * pitch;                            // [64][LPITCH]: what rounding left of their latent part
    __nv_bfloat16* Ps = Ql + ROWS * LPITCH;                               // [64][40]
    __nv_bfloat16* Pl = Ps + ROWS * PPITCH;
    long long* row_base = reinterpret_cast<long long*>(Pl + ROWS * PPITCH);      // [2][32] element offset of a key's row, -1: none
    float* Pe = reinterpret_cast<float*>(row_base + 2 * KEYS);            // [64][8]: weights of the edge keys, -1: not seen
    float* red = Pe + ROWS * EDGE;                                        // [2][64]
    float* corr_s = red + 2 * ROWS;                                       // [64]
    float2* turn = reinterpret_cast<float2*>(Ps);                         // [4][rot / 2] at first: cosines and sines (rot <= 256)

    // request s's tiles begin at cu_q[s] / 4 + 2 s, which leaves room for its first and last, partly filled ones; the last
    // ones, whose tokens see most, go first
    const int tile_at = gridDim.x - 1 - blockIdx.x;
    int seq = 0;
    for (int step = p.steps; step > 0; step >>= 1)
        if (seq + step < p.num_seqs && p.cu_q[seq + step] / TOKENS + 2 * (seq + step) <= tile_at) seq += step;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || p.seq_of_token[begin] < 0) return;     // a single token, or a request that is left out
    const int start = p.positions[begin], last = start + n - 1;
    // the run's positions, pos0 .. pos1, of which the portion may hold the middle or one end: first .. first + tokens - 1
    const int pos0 = (start / TOKENS + tile_at - begin / TOKENS - 2 * seq) * TOKENS, pos1 = pos0 + TOKENS - 1;
    const int first = max(pos0, start), t0 = begin + first - start, tokens = min(pos1, last) - first + 1;
    if (tokens <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h0 = blockIdx.y * HEADS;
    const int lo0 = p.window > 0 ? max(0, pos0 - p.window + 1) : 0, lo1 = p.window > 0 ? max(0, pos1 - p.window + 1) : 0;
    // keys all of the run see, and the others: below lo1 and above pos0 (a window shorter than the run: there is no key in between)
    const int body0 = min(lo1, pos0 + 1), body = pos0 + 1 - body0, edges = (body0 - lo0) + (pos1 - pos0);
    const int tiles = (body + KEYS - 1) / KEYS, first_tile = edges > 0 ? -1 : 0;
    auto edge_key = [&](int e) { return e < body0 - lo0 ? lo0 + e : pos0 + 1 + e - (body0 - lo0); };
    const int* table = p.block_table + (long long)seq * p.table_width;

    auto locate = [&](int tile) {                    // tile -1: the edge keys
        if (tid < KEYS) {
            const bool any = tile < 0 ? tid < edges : tile * KEYS + tid < body;
            const int j = tile < 0 ? edge_key(tid) : body0 + tile * KEYS + tid;
            long long base = -1;
            if (any && j <= last) {                  // a key behind the portion's end may lie past the table
                const int page = table[j / p.geo.page_tokens];
                if (page >= 0 && page < p.geo.num_pages)
                    base = (long long)page * p.geo.page_stride + p.geo.entry_offset + (long long)(j % p.geo.page_tokens) * width;
            }
            row_base[(tile & 1) * KEYS + tid] = base;
        }
    };
    const int chunks = width / 8;
    auto load = [&](int tile) {
        __nv_bfloat16* dst = Ks + (tile & 1) * KEYS * pitch;
#pragma unroll
        for (int i = 0; i < KEYS / WARPS; ++i) {
            const int r = warp * (KEYS / WARPS) + i;
            const long long base = row_base[(tile & 1) * KEYS + r];
            for (int c = lane; c < chunks; c += 32) cp_async16(dst + r * pitch + c * 8, p.k_pool + (base >= 0 ? base : 0) + c * 8, base >= 0);
        }
        cp_async_commit();
    };
    locate(first_tile);
    const int half = p.rot / 2;
    for (int e = tid; e < TOKENS * half; e += THREADS) {
        float sn, cs;
        sincosf((float)(first + e / half) * p.freq[e % half], &sn, &cs);
        turn[e] = make_float2(cs * p.magnitude, sn * p.magnitude);
    }
    __syncthreads();
    load(first_tile);

    // the folded queries, [W_uk^T q_flat | rotated q_rot], in bfloat16 pieces; many loads on their way at a time
    if (p.wide) {
#pragma unroll 8
        for (int e = tid; e < ROWS * (RANK / 4); e += THREADS) {
            const int r = e / (RANK / 4), d = e % (RANK / 4) * 4, tk = r / HEADS, h = h0 + r % HEADS;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tk < tokens && h < p.heads) x = *reinterpret_cast<const float4*>(p.q_lat + (t0 + tk) * p.ql_token_stride + h * p.ql_head_stride + d);
            const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
            *reinterpret_cast<uint2*>(Qs + r * pitch + d) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
            *reinterpret_cast<uint2*>(Ql + r * LPITCH + d) =
                make_uint2(pack_bf16(x.x - __low2float(a), x.y - __high2float(a)), pack_bf16(x.z - __low2float(b), x.w - __high2float(b)));
        }
    } else {
        for (int e = tid; e < ROWS * RANK; e += THREADS) {
            const int r = e / RANK, d = e % RANK, tk = r / HEADS, h = h0 + r % HEADS;
            const float x = tk < tokens && h < p.heads ? p.q_lat[(t0 + tk) * p.ql_token_stride + h * p.ql_head_stride + d] : 0.f;
            const __nv_bfloat16 hi = __float2bfloat16_rn(x);
            Qs[r * pitch + d] = hi;
            Ql[r * LPITCH + d] = __float2bfloat16_rn(x - __bfloat162float(hi));
        }
    }
#pragma unroll 8
    for (int e = tid; e < ROWS * half; e += THREADS) {
        const int r = e / half, i = e % half, tk = r / HEADS, h = h0 + r % HEADS;
        float u = 0.f, v = 0.f;
        if (tk < tokens && h < p.heads) {
            const __nv_bfloat16* qr = p.q + (long long)(t0 + tk) * p.q_stride + (long long)h * p.q_head_width + p.q_rot_offset;
            u = __bfloat162float(qr[i]);
            v = __bfloat162float(qr[i + half]);
        }
        const float2 t = turn[tk * half + i];
        Qs[r * pitch + RANK + i] = __float2bfloat16_rn(u * t.x - v * t.y);
        Qs[r * pitch + RANK + i + half] = __float2bfloat16_rn(v * t.x + u * t.y);
    }
    float o[TOKENS][NT][4];
#pragma unroll
    for (int mt = 0; mt < TOKENS; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[mt][nt][c] = 0.f;
    const int row = lane >> 2, quad = lane & 3;
    const int mine = warp >> 1, side = warp & 1;     // scores: the token and the half of the keys of this warp
    const bool scores = mine < tokens;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};        // rows `row` and `row + 8` of the token
    const int ch0 = warp * (RANK / WARPS);
    for (int tile = first_tile; tile < tiles; ++tile) {
        if (tile + 1 < tiles) locate(tile + 1);
        cp_async_wait<0>();
        __syncthreads();                             // this tile is in, the one before has been read, the next one's rows are known
        if (tile + 1 < tiles) load(tile + 1);
        const __nv_bfloat16* K = Ks + (tile & 1) * KEYS * pitch;
        const long long* base = row_base + (tile & 1) * KEYS;
        float s[2][4];
        if (scores) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
            const __nv_bfloat16* qa = Qs + (mine * HEADS + (lane & 15)) * pitch + (lane >> 4) * 8;
            const __nv_bfloat16* la = Ql + (mine * HEADS + (lane & 15)) * LPITCH + (lane >> 4) * 8;
            const __nv_bfloat16* kb = K + (side * 16 + ((lane >> 4) << 3) + (lane & 7)) * pitch + ((lane >> 3) & 1) * 8;
            float low[2][4] = {};                    // the small pieces' sums: a chain of their own
#pragma unroll 8
            for (int k0 = 0; k0 < RANK; k0 += 16) {
                uint32_t a[4], al[4], b[4];
                ldmatrix_x4(a, qa + k0);
                ldmatrix_x4(b, kb + k0);
                ldmatrix_x4(al, la + k0);
                mma_bf16(s[0], a, b[0], b[1]);
                mma_bf16(s[1], a, b[2], b[3]);
                mma_bf16(low[0], al, b[0], b[1]);
                mma_bf16(low[1], al, b[2], b[3]);
            }
            for (int k0 = RANK; k0 < width; k0 += 16) {
                uint32_t a[4], b[4];
                ldmatrix_x4(a, qa + k0);
                ldmatrix_x4(b, kb + k0);
                mma_bf16(s[0], a, b[0], b[1]);
                mma_bf16(s[1], a, b[2], b[3]);
            }
            // thread: rows `row` (c 0, 1) and `row + 8` (c 2, 3); keys 16 side + 8 i + 2 quad + {0, 1}
            const int pos = first + mine, lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
            float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int key = side * 16 + 8 * i + 2 * quad + (c & 1);
                    bool seen = base[key] >= 0;
                    if (tile < 0 && seen) {
                        const int j = edge_key(key);
                        seen = j >= lo && j <= pos;
                    }
                    s[i][c] = seen ? (s[i][c] + low[i][c]) * p.scale : -INFINITY;
                    top[c >> 1] = fmaxf(top[c >> 1], s[i][c]);
                }
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2) {
                top[r2] = fmaxf(top[r2], __shfl_xor_sync(0xffffffffu, top[r2], 1));
                top[r2] = fmaxf(top[r2], __shfl_xor_sync(0xffffffffu, top[r2], 2));
                if (quad == 0) red[side * ROWS + mine * HEADS + row + 8 * r2] = top[r2];
            }
        }
        __syncthreads();                             // both halves' maxima are in
        if (scores) {
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2) {
                const int r = mine * HEADS + row + 8 * r2;
                const float next = fmaxf(m_run[r2], fmaxf(red[r], red[ROWS + r]));
                const float corr = next == -INFINITY ? 1.f : expf(m_run[r2] - next);
                m_run[r2] = next;
                l_run[r2] *= corr;
                if (side == 0 && quad == 0) corr_s[r] = corr;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float w[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    w[c] = s[i][c] == -INFINITY ? 0.f : expf(s[i][c] - m_run[c >> 1]);
                    l_run[c >> 1] += w[c];
                }
                const int col = side * 16 + 8 * i + 2 * quad, r = mine * HEADS + row;
                if (tile < 0) {
                    if (col < EDGE)
#pragma unroll
                        for (int c = 0; c < 4; ++c) Pe[(r + 8 * (c >> 1)) * EDGE + col + (c & 1)] = s[i][c] == -INFINITY ? -1.f : w[c];
                } else {
                    const __nv_bfloat162 h01 = __floats2bfloat162_rn(w[0], w[1]), h23 = __floats2bfloat162_rn(w[2], w[3]);
                    *reinterpret_cast<__nv_bfloat162*>(Ps + r * PPITCH + col) = h01;
                    *reinterpret_cast<__nv_bfloat162*>(Ps + (r + 8) * PPITCH + col) = h23;
                    *reinterpret_cast<__nv_bfloat162*>(Pl + r * PPITCH + col) = __floats2bfloat162_rn(w[0] - __low2float(h01), w[1] - __high2float(h01));
                    *reinterpret_cast<__nv_bfloat162*>(Pl + (r + 8) * PPITCH + col) = __floats2bfloat162_rn(w[2] - __low2float(h23), w[3] - __high2float(h23));
                }
            }
        }
        __syncthreads();                             // the weights are in
        if (tile < 0) {
#pragma unroll
            for (int mt = 0; mt < TOKENS; ++mt) {
                if (mt >= tokens) break;
                for (int e = 0; e < edges; ++e) {
                    const float w0 = Pe[(mt * HEADS + row) * EDGE + e], w1 = Pe[(mt * HEADS + row + 8) * EDGE + e];
                    if (w0 < 0.f && w1 < 0.f) continue;
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(K + e * pitch + ch0 + nt * 8 + 2 * quad));
                        if (!(w0 < 0.f)) { o[mt][nt][0] = fmaf(w0, v.x, o[mt][nt][0]); o[mt][nt][1] = fmaf(w0, v.y, o[mt][nt][1]); }
                        if (!(w1 < 0.f)) { o[mt][nt][2] = fmaf(w1, v.x, o[mt][nt][2]); o[mt][nt][3] = fmaf(w1, v.y, o[mt][nt][3]); }
                    }
                }
            }
            continue;
        }
#pragma unroll
        for (int mt = 0; mt < TOKENS; ++mt) {
            if (mt >= tokens) break;
            const float c0 = corr_s[mt * HEADS + row], c1 = corr_s[mt * HEADS + row + 8];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                o[mt][nt][0] *= c0; o[mt][nt][1] *= c0;
                o[mt][nt][2] *= c1; o[mt][nt][3] *= c1;
            }
        }
#pragma unroll
        for (int kk = 0; kk < KEYS; kk += 16) {
            uint32_t b[NT / 2][4];
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2)
                ldmatrix_x4_trans(b[nt / 2], K + (kk + ((lane >> 3) & 1) * 8 + (lane & 7)) * pitch + ch0 + nt * 8 + (lane >> 4) * 8);
#pragma unroll
            for (int mt = 0; mt < TOKENS; ++mt) {
                if (mt >= tokens) break;
                uint32_t a[4], al[4];
                ldmatrix_x4(a, Ps + (mt * HEADS + (lane & 15)) * PPITCH + kk + (lane >> 4) * 8);
                ldmatrix_x4(al, Pl + (mt * HEADS + (lane & 15)) * PPITCH + kk + (lane >> 4) * 8);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_bf16(o[mt][nt], a, b[nt / 2][2 * (nt & 1)], b[nt / 2][2 * (nt & 1) + 1]);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_bf16(o[mt][nt], al, b[nt / 2][2 * (nt & 1)], b[nt / 2][2 * (nt & 1) + 1]);
            }
        }
    }
    // the rows' sums over a token's two warps, then the output
    __syncthreads();
    if (scores) {
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            l_run[r2] += __shfl_xor_sync(0xffffffffu, l_run[r2], 1);
            l_run[r2] += __shfl_xor_sync(0xffffffffu, l_run[r2], 2);
            if (quad == 0) red[side * ROWS + mine * HEADS + row + 8 * r2] = l_run[r2];
        }
    }
    __syncthreads();
    if (scores && side == 0 && quad == 0) {
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            const int r = mine * HEADS + row + 8 * r2, h = h0 + row + 8 * r2;
            const float l = red[r] + red[ROWS + r];
            float inv = l > 0.f ? 1.f / l : 0.f;
            if (p.sink && l > 0.f && h < p.heads) {  // exp(sink) joins the sum; above the maximum in the form that cannot overflow
                const float d = p.sink[h] - m_run[r2], e = expf(-fabsf(d));
                inv = d <= 0.f ? 1.f / (l + e) : e / (l * e + 1.f);
            }
            corr_s[r] = inv;
        }
    }
    __syncthreads();
#pragma unroll
    for (int mt = 0; mt < TOKENS; ++mt) {
        if (mt >= tokens) break;
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            const int h = h0 + row + 8 * r2;
            if (h >= p.heads) continue;
            const float inv = corr_s[mt * HEADS + row + 8 * r2];
            __nv_bfloat16* dst = p.out + ((long long)(t0 + mt) * p.heads + h) * RANK + ch0 + 2 * quad;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
                *reinterpret_cast<__nv_bfloat162*>(dst + nt * 8) = __floats2bfloat162_rn(o[mt][nt][2 * r2] * inv, o[mt][nt][2 * r2 + 1] * inv);
        }
    }
}

}  // namespace

// Latents of 384 or 512 channels whose tiles fit shared memory (the rotated part in steps of 16: ts_latent_mma_supported).
bool ts_latent_tokens_supported(int rank, int rot) {
    return (rank == 384 || rank == 512) && rot <= 256 && latent_tokens_smem(rank, rot) <= 227 * 1024;
}

int ts_latent_attention_tokens_launch(const float* q_lat, long long ql_t, long long ql_h, const void* q, long long q_stride,
                                      int q_head_width, int q_rot_offset, const float* freq, float magnitude, const float* sink,
                                      const void* k_pool, KVGeometry geo, const int* block_table, int table_width,
                                      const int* positions, const int* seq_of_token, const int* cu_q, int num_seqs, void* out,
                                      int num_tokens, int heads, int rank, int rot, float scale, int window, cudaStream_t stream) {
    int steps = 1;
    while (2 * steps <= num_seqs) steps *= 2;
    const int wide = ql_t % 4 == 0 && ql_h % 4 == 0 && (uintptr_t)q_lat % 16 == 0;
    const LatentArgs p{q_lat, ql_t, ql_h, (const __nv_bfloat16*)q, q_stride, q_head_width, q_rot_offset, freq, magnitude, sink,
                       (const __nv_bfloat16*)k_pool, geo, block_table, table_width, positions, seq_of_token, cu_q, num_seqs, steps, (__nv_bfloat16*)out,
                       heads, rot, scale, window, wide};
    const dim3 grid(num_tokens / TOKENS + 2 * num_seqs, (heads + HEADS - 1) / HEADS);
    const size_t smem = latent_tokens_smem(rank, rot);
#define TS_LATENT_TOKENS(NT)                                                                                                       \
    do {                                                                                                                           \
        cudaFuncSetAttribute(latent_attention_tokens_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);          \
        latent_attention_tokens_kernel<NT><<<grid, WARPS * 32, smem, stream>>>(p);                                                 \
    } while (0)
    if (rank == 384) TS_LATENT_TOKENS(6);
    else TS_LATENT_TOKENS(8);
#undef TS_LATENT_TOKENS
    TS_LAUNCH_CHECK("latent_attention (tokens)");
    return 0;
}
