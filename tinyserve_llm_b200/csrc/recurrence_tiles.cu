// The recurrences of linear_recurrence.cu over prompt portions, sixteen tokens at a time.
//
// What one token writes into the state the next one reads, so a scan token by token is a chain.  Inside a tile
// of B = 16 tokens the chain can be written out (S_0 the state before the tile, columns of S independent):
//
// Delta rule with one decay a head (a_t), step size b_t.  With c_t = a_1 ... a_t and G[t][j] = a_(j+1) ... a_t,
//   u_t = b_t (v_t - c_t S_0^T k_t - sum_{j<t} G[t][j] (k_j . k_t) u_j)
//   o_t = c_t S_0^T q_t + sum_{j<=t} G[t][j] (k_j . q_t) u_j,     S_B = c_B S_0 + sum_j G[B][j] k_j u_j^T
// The first line is a unit lower triangular system, U = M diag(b) (V - diag(c) R), R = S_0^T K, with
// M = (I + A)^-1, A[t][j] = b_t G[t][j] (k_j . k_t) for j < t (the entries of M stay below one in size: each is
// a product of the contractions a (I - b k k^T) between two unit vectors).
//
// Time mixing with decays per channel (a_(t,i)) and a bonus.  With d_(t,i) = a_(1,i) ... a_(t,i),
//   o_t = sum_i r_(t,i) d_(t-1,i) S_0[i] + sum_{j<t} P[t][j] v_j + bonus_t v_t,
//   P[t][j] = sum_i r_(t,i) k_(j,i) a_(j+1,i) ... a_(t-1,i),   S_B = d_B S_0 + sum_j (k_j a_(j+1) ... a_B) v_j^T
//
// Plain recurrence (gated linear attention, retention): the same with the token's own write in its read-out,
//   o_t = sum_i q_(t,i) d_(t,i) S_0[i] + sum_{j<=t} P[t][j] v_j,   P[t][j] = sum_i q_(t,i) k_(j,i) a_(j+1,i) ... a_(t,i)
//
// Delta rule with decays per channel: with G[t][j]_i = a_(j+1,i) ... a_(t,i),
//   u_t = b_t (v_t - (d_t k_t)^T S_0 - sum_{j<t} (sum_i k_(t,i) k_(j,i) G[t][j]_i) u_j),
//   o_t = (d_t q_t)^T S_0 + sum_{j<=t} (sum_i q_(t,i) k_(j,i) G[t][j]_i) u_j,   S_B = d_B S_0 + sum_j (G[B][j] k_j) u_j^T,
// the system of the first line solved as above; its k side has two sets of rows, those that read S_0 and those that update it.
//
// No decay is ever divided by another: products of decays are taken as they are needed.
//
// What the plain recurrence and the delta rule with decays per channel hold to (relative error of outputs / states against 64 bits, the
// walk token by token and here; the plain recurrence over bfloat16 values: recurrence_stretches.cu): gated linear attention over 2,048 tokens
// 1.73e-7 / 1.47e-7 and 1.20e-7 / 5.4e-8, constant decays 2.5e-7 / 2.4e-7 and 1.45e-7 / 1.04e-7, the delta rule over portions of 1,001, 667 and 333 tokens 3.0e-7 / 4.2e-7 and 1.9e-7 / 1.8e-7.
// Three things bring that: the products of decays from a tile's ends are taken in 64 bits and rounded once (sixteen roundings of one
// constant decay all err to one side, tile after tile: 6.2e-7 / 5.9e-7); a decay near one enters them with the bits past float32's that
// 1 + expm1 knows; no accumulator of the tensor cores, which cut what it cannot hold, takes more than one large part.  Sums inside a
// tile stay in float32 (in 64 bits they cost 20 us and gained nothing by then).
//
// A token's values, keys and decays reach its own and later tokens only, also where they are infinite or NaN: coefficients above the
// diagonal are zeros, and a value that has no split is left out of the product with them (0 times it would be NaN) and added to the
// rows from its own on.  A tile pays a vote for it.
//
// A first kernel works out, per tile and q/k head (time mixing: head), what all columns of the state share: the
// "pack" (16 rows for the q side, 16 or 32 for the k side, one with the channels' decays over the tile) and the coefficients
// (W = M diag(b); P W, so that O = diag(c) S_0^T Q + (P W) (V - diag(c) R) does not wait for U; c; G[B]).  The second
// kernel walks the tiles: a CTA owns one request, one head and 16 columns of the state and does three small
// products a tile on tensor cores,
//   [q side | k side] S_0   (each warp its own rows of S, the partial sums meet in shared memory in warp order)
//   U (two warps) and O (two warps) from the 16 x 16 coefficients
//   K^T U, by which the state moves on
// with the next tile's pack and coefficients on their way by cp.async.  The products are float32 to rounding: every
// factor is split into two TF32 numbers, x = hi + lo, and hi hi + hi lo + lo hi is summed in float32 (what is
// left out is 2^-22 of a term).  The state stays in registers, in the layout in which the third product
// leaves it (its transpose) and the first one takes it; the update is added to it by an ordinary fused
// multiply-add, so that what the tensor cores round is the update and not the state.
//
// A tile cut short by the portion's end is filled up with tokens that change nothing (k = 0, decay 1).  Requests that
// feed one token are left to the other scan.  Tiles count from the portion's first token, so where a prompt was cut
// moves sums inside rounding only.
#include "recurrence_tiles.cuh"

namespace {

constexpr int COLS = 16;           // value channels a CTA
constexpr int WARPS = 4, THREADS = WARPS * 32;   // of the scan
constexpr int CP = 20;             // pitch of a coefficient matrix: a warp's fragment loads fall into different banks
constexpr int COEF = 2 * B * CP + 2 * B;   // W [16][20], P W (time mixing: P) [16][20], c [16], g [16]
constexpr int RP = 24;             // pitch of the partial sums and of U: likewise
// A pack: 16 rows of the q side, `sets` times 16 of the k side, one with the channels' decays, each of `rows` floats and a pad
// that does the same for it.
__host__ __device__ constexpr int pack_pitch(int rows) { return rows + 8; }
__host__ __device__ constexpr int pack_floats(int rows, int sets) { return ((1 + sets) * B + 1) * pack_pitch(rows); }
enum { DELTA = 0, MIX = 1, CHANNEL = 2, PLAIN = 3 };   // delta rule, a decay a head; time mixing; delta rule, a decay a channel; plain
__host__ __device__ constexpr int sets_of(int mode) { return mode == CHANNEL ? 2 : 1; }

__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

struct PrepareArgs {
    const void* q; const void* k; long long qk_stride;   // delta: float32 after the convolution; mixing: r, k as projected
    const float* gates;                                  // delta: [tokens, 2 heads], logits of b, then of the decay; mixing: z [tokens, heads * dim]
    const float* bias;                                   // delta: dt_bias [heads]; mixing: w0 [heads * dim]
    const float* rate;                                   // delta: A_log [heads]; mixing: u [heads * dim]
    const int* cu_q; const int* prefill_seqs;
    float* pack; float* coef;
    int heads, kv_heads, dim, rows;                      // rows: dim rounded up to what the scan's threads hold
    float unit_eps, q_scale;
};

// grid (tiles, q/k heads, portions), 128 threads
__global__ void __launch_bounds__(128) delta_tile_prepare_kernel(PrepareArgs p) {
    extern __shared__ float smem[];
    const int seq = p.prefill_seqs[blockIdx.z], tile = blockIdx.x, g = blockIdx.y;
    if (seq < 0) return;                                 // a padding entry of the list
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || tile * B >= n) return;
    const int t0 = begin + tile * B, m = min(B, n - tile * B);
    const int pitch = p.rows + 1;
    float* qs = smem;                                    // [16][pitch]
    float* ks = qs + B * pitch;
    float* kk = ks + B * pitch;                          // [16][17]: k_t . k_j
    float* qk = kk + B * (B + 1);                        // q_t . k_j
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = warp; t < B; t += 4) {
        const float* qr = (const float*)p.q + (long long)(t0 + t) * p.qk_stride + (long long)g * p.dim;
        const float* kr = (const float*)p.k + (long long)(t0 + t) * p.qk_stride + (long long)g * p.dim;
        float sq = 0.f, sk = 0.f;
        for (int i = lane; i < p.rows; i += 32) {
            const bool ok = t < m && i < p.dim;
            const float qv = ok ? qr[i] : 0.f, kv = ok ? kr[i] : 0.f;
            qs[t * pitch + i] = qv;
            ks[t * pitch + i] = kv;
            sq += qv * qv;
            sk += kv * kv;
        }
        const float iq = p.q_scale / sqrtf(warp_sum(sq) + p.unit_eps), ik = 1.f / sqrtf(warp_sum(sk) + p.unit_eps);
        for (int i = lane; i < p.rows; i += 32) { qs[t * pitch + i] *= iq; ks[t * pitch + i] *= ik; }   // the lane's own elements
    }
    __syncthreads();
    const long long slot = tile_slot(seq, begin, tile);
    float* pack = p.pack + (slot * p.kv_heads + g) * pack_floats(p.rows, 1);
    for (int e = threadIdx.x; e < B * p.rows; e += 128) {
        const int t = e / p.rows, i = e % p.rows;
        pack[t * pack_pitch(p.rows) + i] = qs[t * pitch + i];
        pack[(B + t) * pack_pitch(p.rows) + i] = ks[t * pitch + i];
    }
    {   // the dot products: thread (t, pair of j)
        const int t = threadIdx.x >> 3, j = (threadIdx.x & 7) * 2;
        float k0 = 0.f, k1 = 0.f, q0 = 0.f, q1 = 0.f;
        for (int i = 0; i < p.dim; ++i) {
            const float kt = ks[t * pitch + i], qt = qs[t * pitch + i], a = ks[j * pitch + i], b = ks[(j + 1) * pitch + i];
            k0 = fmaf(kt, a, k0); k1 = fmaf(kt, b, k1);
            q0 = fmaf(qt, a, q0); q1 = fmaf(qt, b, q1);
        }
        kk[t * (B + 1) + j] = k0; kk[t * (B + 1) + j + 1] = k1;
        qk[t * (B + 1) + j] = q0; qk[t * (B + 1) + j + 1] = q1;
    }
    __syncthreads();
    // a warp a value head of the group; lane j holds column j (lanes 16..31 mirror lanes 0..15 and store nothing)
    const int group = p.heads / p.kv_heads, j = lane & (B - 1);
    for (int hh = warp; hh < group; hh += 4) {
        const int h = g * group + hh;
        float b = 0.f, a = 1.f;                          // a token past the portion's end changes nothing
        if (j < m) {
            const float* gr = p.gates + (long long)(t0 + j) * 2 * p.heads;
            b = 1.f / (1.f + expf(-gr[h]));
            a = expf(-expf(p.rate[h]) * softplus(gr[p.heads + h] + p.bias[h]));
        }
        float* out = p.coef + (slot * p.heads + h) * COEF;
        float M[B], P[B];
        float decay = 1.f, c = 1.f, c_own = 1.f;         // G[t][j] as t runs; c_t; c_j
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const float at = __shfl_sync(0xffffffffu, a, t), bt = __shfl_sync(0xffffffffu, b, t);
            c *= at;
            if (t == j) c_own = c;
            if (t > j) decay *= at;
            const float A = t > j ? bt * decay * kk[t * (B + 1) + j] : 0.f;
            P[t] = t >= j ? decay * qk[t * (B + 1) + j] : 0.f;
            float row = t == j ? 1.f : 0.f;              // M[t][j] = delta - sum_s A[t][s] M[s][j]
#pragma unroll
            for (int s = 0; s < t; ++s) row = fmaf(-__shfl_sync(0xffffffffu, A, s), M[s], row);
            M[t] = row;
        }
#pragma unroll
        for (int t = 0; t < B; ++t) {
            float pw = 0.f;
#pragma unroll
            for (int s = 0; s <= t; ++s) pw = fmaf(__shfl_sync(0xffffffffu, P[t], s), M[s] * b, pw);
            if (lane < B) {                              // 0 where t < j, whatever the later token's step size is
                out[t * CP + j] = t >= j ? M[t] * b : 0.f;
                out[B * CP + t * CP + j] = t >= j ? pw : 0.f;
            }
        }
        if (lane < B) {
            out[2 * B * CP + j] = c_own;
            out[2 * B * CP + B + j] = decay;
        }
    }
}

// grid (tiles, heads, portions), 128 threads: thread (j, channel group of 8) for the coefficients
template <typename T>
__global__ void __launch_bounds__(128) mix_tile_prepare_kernel(PrepareArgs p) {
    extern __shared__ float smem[];
    const int seq = p.prefill_seqs[blockIdx.z], tile = blockIdx.x, h = blockIdx.y;
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || tile * B >= n) return;
    const int t0 = begin + tile * B, m = min(B, n - tile * B);
    const int pitch = p.rows + 1;
    float* rs = smem;                                    // [16][pitch]
    float* ks = rs + B * pitch;
    float* as = ks + B * pitch;
    const long long slot = tile_slot(seq, begin, tile);
    float* pack = p.pack + (slot * p.heads + h) * pack_floats(p.rows, 1);
    const long long width = (long long)p.heads * p.dim, hc = (long long)h * p.dim;
    for (int e = threadIdx.x; e < B * p.rows; e += 128) {
        const int t = e / p.rows, i = e % p.rows;
        const bool ok = t < m && i < p.dim;
        float rv = 0.f, kv = 0.f, av = 1.f;
        if (ok) {
            rv = to_float<T>(((const T*)p.q)[(long long)(t0 + t) * p.qk_stride + hc + i]);
            kv = to_float<T>(((const T*)p.k)[(long long)(t0 + t) * p.qk_stride + hc + i]);
            av = expf(-expf(p.gates[(long long)(t0 + t) * width + hc + i] + p.bias[hc + i]));
        }
        rs[t * pitch + i] = rv;
        ks[t * pitch + i] = kv;
        as[t * pitch + i] = av;
    }
    __syncthreads();
    {   // P[t][j], t >= j: thread j = tid / 8 walks t with the running product of its channels
        const int j = threadIdx.x >> 3, part = threadIdx.x & 7;
        float sum[B];
#pragma unroll
        for (int t = 0; t < B; ++t) sum[t] = 0.f;
        for (int i = part; i < p.dim; i += 8) {
            float run = ks[j * pitch + i];
            const float own = run * rs[j * pitch + i] * p.rate[hc + i];                 // the bonus's share
#pragma unroll
            for (int t = 0; t < B; ++t) {
                if (t == j) sum[t] += own;
                if (t > j) {
                    sum[t] = fmaf(rs[t * pitch + i], run, sum[t]);
                    run *= as[t * pitch + i];
                }
            }
        }
        float* out = p.coef + (slot * p.heads + h) * COEF + B * CP;
#pragma unroll
        for (int t = 0; t < B; ++t) {
            float s = sum[t];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (part == 0) out[t * CP + j] = s;                                         // 0 where t < j
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < p.rows; i += 128) {    // a thread a channel: products from the left and from the right
        const int pp = pack_pitch(p.rows);
        float left = 1.f, right = 1.f;
        for (int t = 0; t < B; ++t) {
            pack[t * pp + i] = rs[t * pitch + i] * left;
            left *= as[t * pitch + i];
        }
        for (int t = B - 1; t >= 0; --t) {
            pack[(B + t) * pp + i] = ks[t * pitch + i] * right;
            right *= as[t * pitch + i];
        }
        pack[2 * B * pp + i] = left;
    }
}

// The plain recurrence's pack and P, float32.  grid (tiles, heads, portions), 128 threads.
template <int ROWS>
__global__ void __launch_bounds__(128) plain_tile_prepare_kernel(PlainArgs p) {
    extern __shared__ float smem[];
    const int seq = p.prefill_seqs[blockIdx.z], tile = blockIdx.x, h = blockIdx.y;
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || tile * B >= n) return;
    const PlainTile<ROWS> x(smem);
    load_plain<float, ROWS>(p, x, h, begin + tile * B, min(B, n - tile * B));
    __syncthreads();
    const long long slot = tile_slot(seq, begin, tile);
    float* out = p.coef + (slot * p.heads + h) * COEF + B * CP;
    plain_scores<ROWS>(x, p.dim, [&](int t, int j, float s) { out[t * CP + j] = s; });
    float* pack = p.pack + (slot * p.heads + h) * pack_floats(ROWS, 1);
    for (int i = threadIdx.x; i < ROWS; i += 128) {
        const int pp = pack_pitch(ROWS);
        pack[2 * B * pp + i] = plain_sides<ROWS>(x, i, [&](int t, float q) { pack[t * pp + i] = q; }, [&](int t, float k) { pack[(B + t) * pp + i] = k; });
    }
}

struct ChannelArgs {
    const float* q; const float* k; long long qk_stride;     // after the convolution
    const float* z;                                          // [tokens, heads * dim] decay logits
    const void* b; long long b_stride;                       // [tokens, heads] step sizes' logits
    const float* bias; const float* rate;                    // dt_bias [heads * dim], A_log [heads]
    const int* cu_q; const int* prefill_seqs;
    float* pack; float* coef;
    int heads, kv_heads, dim;
    float unit_eps, q_scale;
};

// The pack and the coefficients of the delta rule with decays per channel.  grid (tiles, value heads, portions), 128 threads.
// Bound by instructions (decays, running products) and by waits for its loads: all of a warp's four tokens' are under way together, seven
// CTAs share an SM.  Three portions of 1,001, 667 and 333 tokens, 8 heads of 128: 29 us (33 with a token's loads at a time and one channel a
// read of shared memory); the walk behind it 86, token by token 300.
template <typename T, int ROWS>
__global__ void __launch_bounds__(128, ROWS == 128 ? 7 : 1) channel_tile_prepare_kernel(ChannelArgs p) {
    extern __shared__ float smem[];
    const int seq = p.prefill_seqs[blockIdx.z], tile = blockIdx.x, h = blockIdx.y, g = h / (p.heads / p.kv_heads);
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin;
    if (n <= 1 || tile * B >= n) return;
    const int t0 = begin + tile * B, m = min(B, n - tile * B);
    constexpr int pitch = ROWS + 2;                      // even: two channels a read
    float* qs = smem;                                    // [16][pitch]
    float* ks = qs + B * pitch;
    float* as = ks + B * pitch;
    float* kk = as + B * pitch;                          // [16][17]: sum_i k_t k_j G[t][j]
    float* qk = kk + B * (B + 1);                        // sum_i q_t k_j G[t][j]
    __nv_bfloat16* rest = reinterpret_cast<__nv_bfloat16*>(qk + B * (B + 1));      // [16][pitch]: what the decays lack
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float rate = expf(p.rate[h]);
    constexpr int EACH = ROWS / 32, DEEP = ROWS > 128 ? 1 : 4;          // channels a lane; tokens whose loads are under way together
    for (int first = warp; first < B; first += 4 * DEEP) {
        float q[DEEP][EACH], k[DEEP][EACH], z[DEEP][EACH];
#pragma unroll
        for (int e = 0; e < DEEP; ++e) {
            const int t = first + 4 * e;
            const float* qr = p.q + (long long)(t0 + t) * p.qk_stride + (long long)g * p.dim;
            const float* kr = p.k + (long long)(t0 + t) * p.qk_stride + (long long)g * p.dim;
            const float* zr = p.z + ((long long)(t0 + t) * p.heads + h) * p.dim;
#pragma unroll
            for (int u = 0; u < EACH; ++u) {
                const int i = lane + 32 * u;
                const bool ok = t < m && i < p.dim;      // a token past the portion's end changes nothing
                q[e][u] = ok ? qr[i] : 0.f;
                k[e][u] = ok ? kr[i] : 0.f;
                z[e][u] = ok ? zr[i] : 0.f;
            }
        }
#pragma unroll
        for (int e = 0; e < DEEP; ++e) {
            const int t = first + 4 * e;
            float sq = 0.f, sk = 0.f;
#pragma unroll
            for (int u = 0; u < EACH; ++u) {
                const int i = lane + 32 * u;
                float more = 0.f;
                as[t * pitch + i] = t < m && i < p.dim ? decay_of(-rate * softplus(z[e][u] + p.bias[h * p.dim + i]), more) : 1.f;
                rest[t * pitch + i] = __float2bfloat16_rn(more);
                sq += q[e][u] * q[e][u];
                sk += k[e][u] * k[e][u];
            }
            const float iq = p.q_scale / sqrtf(warp_sum(sq) + p.unit_eps), ik = 1.f / sqrtf(warp_sum(sk) + p.unit_eps);
#pragma unroll
            for (int u = 0; u < EACH; ++u) {
                qs[t * pitch + lane + 32 * u] = q[e][u] * iq;
                ks[t * pitch + lane + 32 * u] = k[e][u] * ik;
            }
        }
    }
    __syncthreads();
    {   // t >= j: thread j = tid / 8 walks t with the running product of its channels
        const int j = threadIdx.x >> 3, part = threadIdx.x & 7;
        float sum_k[B], sum_q[B];
#pragma unroll
        for (int t = 0; t < B; ++t) sum_k[t] = sum_q[t] = 0.f;
        for (int i = 2 * part; i < p.dim; i += 16) {     // two channels (those past dim hold zeros)
            float2 run = *reinterpret_cast<const float2*>(ks + j * pitch + i);
#pragma unroll
            for (int t = 0; t < B; ++t) {
                if (t < warp * 4) continue;                                             // the warp's four j begin here
                if (t > j) {
                    const float2 a = *reinterpret_cast<const float2*>(as + t * pitch + i);
                    run.x *= a.x;
                    run.y *= a.y;
                }
                if (t >= j) {
                    const float2 kt = *reinterpret_cast<const float2*>(ks + t * pitch + i), qt = *reinterpret_cast<const float2*>(qs + t * pitch + i);
                    sum_k[t] = fmaf(kt.y, run.y, fmaf(kt.x, run.x, sum_k[t]));
                    sum_q[t] = fmaf(qt.y, run.y, fmaf(qt.x, run.x, sum_q[t]));
                }
            }
        }
#pragma unroll
        for (int t = 0; t < B; ++t) {
            float a = sum_k[t], b = sum_q[t];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
            }
            if (part == 0) {
                kk[t * (B + 1) + j] = a;
                qk[t * (B + 1) + j] = b;
            }
        }
    }
    __syncthreads();
    const long long slot = tile_slot(seq, begin, tile);
    float* pack = p.pack + (slot * p.heads + h) * pack_floats(ROWS, 2);
    for (int i = threadIdx.x; i < ROWS; i += 128) {    // a thread a channel: products from the left and from the right
        const int pp = pack_pitch(ROWS);
        double decay[B], left = 1.0, right = 1.0;
#pragma unroll
        for (int t = 0; t < B; ++t) {
            decay[t] = whole(as[t * pitch + i], rest[t * pitch + i]);
            left *= decay[t];
            pack[t * pp + i] = (float)((double)qs[t * pitch + i] * left);
            pack[(B + t) * pp + i] = (float)((double)ks[t * pitch + i] * left);
        }
#pragma unroll
        for (int t = B - 1; t >= 0; --t) {
            pack[(2 * B + t) * pp + i] = (float)((double)ks[t * pitch + i] * right);
            right *= decay[t];
        }
        pack[3 * B * pp + i] = (float)left;
    }
    if (warp) return;
    // lane j holds column j (lanes 16..31 mirror lanes 0..15 and store nothing)
    const int j = lane & (B - 1);
    const float b = j < m ? 1.f / (1.f + expf(-to_float<T>(((const T*)p.b)[(long long)(t0 + j) * p.b_stride + h]))) : 0.f;
    float* out = p.coef + (slot * p.heads + h) * COEF;
    float M[B];
#pragma unroll
    for (int t = 0; t < B; ++t) {
        const float bt = __shfl_sync(0xffffffffu, b, t);
        const float A = t > j ? bt * kk[t * (B + 1) + j] : 0.f;
        float row = t == j ? 1.f : 0.f;                  // M[t][j] = delta - sum_s A[t][s] M[s][j]
#pragma unroll
        for (int s = 0; s < t; ++s) row = fmaf(-__shfl_sync(0xffffffffu, A, s), M[s], row);
        M[t] = row;
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
        const float P = t >= j ? qk[t * (B + 1) + j] : 0.f;
        float pw = 0.f;
#pragma unroll
        for (int s = 0; s <= t; ++s) pw = fmaf(__shfl_sync(0xffffffffu, P, s), M[s] * b, pw);
        if (lane < B) {                                  // 0 where t < j, whatever the later token's step size is
            out[t * CP + j] = t >= j ? M[t] * b : 0.f;
            out[B * CP + t * CP + j] = t >= j ? pw : 0.f;
        }
    }
}

struct ScanArgs {
    const float* pack; const float* coef;
    const void* v; long long v_stride;                   // elements between tokens; a head's values start at h * vdim
    const int* cu_q; const int* slots; const int* prefill_seqs;
    float* state; long long slot_stride;                 // floats between slots; a slot holds [heads, dim, vdim]
    float* out;                                          // [tokens, heads * vdim] float32
    int heads, qk_group, dim, vdim;
    int* error; long long wait_cycles;                   // the delta rules' walk: where a wait that ran out says so, and when it does
};

// Numbers from here on have no split (their hi would be infinite).
constexpr float SPLITS = 3.4e38f;

// What the tokens without a split (as a B fragment: tokens c, c + 4, c + 8, c + 12 of column r) add to tokens at or after them, by the
// coefficients m [16][CP]: a C fragment.  Out of line: it is hardly ever called.
__device__ __noinline__ float4 add_odd_tokens(const float* m, float x0, float x4, float x8, float x12, int r, int c) {
    const float x[4] = {x0, x4, x8, x12};
    float y[4] = {};
#pragma unroll
    for (int j = 0; j < B; ++j)
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const float v = __shfl_sync(0xffffffffu, x[j >> 2], 4 * (2 * c + side) + (j & 3));
            if (fabsf(v) < SPLITS) continue;
#pragma unroll
            for (int half = 0; half < 2; ++half)
                if (j <= r + 8 * half) y[2 * half + side] = fmaf(m[(r + 8 * half) * CP + j], v, y[2 * half + side]);
        }
    return make_float4(y[0], y[1], y[2], y[3]);
}

// Coefficients m [16][CP] times x (as a B fragment: tokens c, c + 4, c + 8, c + 12 of column r): a C fragment.
template <bool FRESH>
__device__ __forceinline__ void times_coefficients(float (&y)[4], const float* m, const float (&x)[4], int r, int c) {
    float big[4], small[4];
    float kept[4];                                       // what is not finite stays out of the product, where 0 times it is NaN
    bool odd = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const bool ok = fabsf(x[k]) < SPLITS;
        kept[k] = ok ? x[k] : 0.f;
        odd |= !ok;
    }
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
        const float* a = m + r * CP + 8 * ks + c;
        const SplitA w = split_a(a[0], a[8 * CP], a[4], a[8 * CP + 4]);
        const Split x0 = split_tf32(kept[2 * ks]), x1 = split_tf32(kept[2 * ks + 1]);
        if (ks == 0) mma_split_first(big, small, w, x0, x1);
        else mma_split<FRESH>(big, small, w, x0, x1);
    }
    float4 late = make_float4(0.f, 0.f, 0.f, 0.f);       // and reaches its own and later tokens by itself
    if (__any_sync(0xffffffffu, odd)) late = add_odd_tokens(m, x[0], x[1], x[2], x[3], r, c);
    y[0] = big[0] + small[0] + late.x;
    y[1] = big[1] + small[1] + late.y;
    y[2] = big[2] + small[2] + late.z;
    y[3] = big[3] + small[3] + late.w;
}

// NT: eights of rows of the state a warp holds.  Fragments of mma.m16n8k8, lane = 4 r + c (r 0..7, c 0..3):
//   A (16 x 8): (r, c), (r + 8, c), (r, c + 4), (r + 8, c + 4);   B (8 x 8): (c, r), (c + 4, r);
//   C (16 x 8): (r, 2c), (r, 2c + 1), (r + 8, 2c), (r + 8, 2c + 1).
// The state is held as C fragments of S^T (16 columns x 8 rows of S).  Read as B fragments of S they hold rows 2c and
// 2c + 1 where the product counts k = c and c + 4: the A side takes its k in the same order.
template <typename T, int NT, int MODE>
__global__ void __launch_bounds__(THREADS) recurrence_tiles_kernel(ScanArgs p) {
    constexpr int WROWS = 8 * NT, ROWS = WARPS * WROWS;  // rows of a warp; rows of the state
    constexpr int PP = pack_pitch(ROWS);
    constexpr int PACK = pack_floats(ROWS, 1), STAGE = PACK + COEF;
    constexpr bool FRESH = MODE == PLAIN;                // (time mixing sums as it did before)
    static_assert(MODE == MIX || MODE == PLAIN && sizeof(T) == 4, "delta rules: below; plain bfloat16: recurrence_stretches.cu");
    extern __shared__ __align__(16) float smem[];
    float* red = smem + 2 * STAGE;                       // [WARPS][B][RP]
    float* G_s = red + WARPS * B * RP;                   // [B][RP]: the values
    const int seq = p.prefill_seqs[blockIdx.z], h = blockIdx.y, j0 = blockIdx.x * COLS;
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin, slot = p.slots[seq];
    if (n <= 1 || slot < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    float* st = p.state + (long long)slot * p.slot_stride + (long long)h * p.dim * p.vdim;

    auto element = [&](int nt, int e, int& i, int& j) {  // row and column of S of register e of tile nt
        i = warp * WROWS + 8 * nt + 2 * c + (e & 1);
        j = j0 + r + 8 * (e >> 1);
        return i < p.dim && j < p.vdim;
    };
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, j;
            S[nt][e] = element(nt, e, i, j) ? st[(long long)i * p.vdim + j] : 0.f;
        }
    const int tiles = (n + B - 1) / B;
    const long long first = tile_slot(seq, begin, 0);
    auto issue = [&](int tile) {
        float* stage = smem + (tile & 1) * STAGE;
        const float* pack = p.pack + ((first + tile) * p.heads + h) * (long long)PACK;
        const float* coef = p.coef + ((first + tile) * p.heads + h) * (long long)COEF;
#pragma unroll
        for (int e = 0; e < PACK / 4; e += THREADS)
            if (e + tid < PACK / 4) cp16(stage + 4 * (e + tid), pack + 4 * (e + tid));
#pragma unroll
        for (int e = 0; e < COEF / 4; e += THREADS)
            if (e + tid < COEF / 4) cp16(stage + PACK + 4 * (e + tid), coef + 4 * (e + tid));
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // Warps 0 and 1 hand the values on, warps 2 and 3 make O, for columns 8 (warp & 1) .. + 7 each.
    // Their values, as B fragments: tokens c, c + 4, c + 8, c + 12 of column r.
    const int nt_uo = warp & 1, col = 8 * nt_uo + r;
    const bool makes_o = warp >= 2;
    static_assert(WARPS == 4, "two warps hand the values on, two make O");
    const T* v = (const T*)p.v + (long long)(begin + c) * p.v_stride + (long long)h * p.vdim + j0 + col;
    T vnow[4], vnext[4];
    auto fetch_v = [&](int tile, T (&x)[4]) {            // as loaded: converting would wait for the load
#pragma unroll
        for (int k = 0; k < 4; ++k)
            x[k] = tile * B + c + 4 * k < n && j0 + col < p.vdim ? v[(long long)(tile * B + 4 * k) * p.v_stride] : from_float<T>(0.f);
    };
    issue(0);
    fetch_v(0, vnow);
#pragma unroll
    for (int k = 0; k < 4; ++k) vnext[k] = vnow[k];
    for (int tile = 0; tile < tiles; ++tile) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();                                 // the tile's inputs are in; the other stage, U and the sums have been read
        if (tile + 1 < tiles) {
            issue(tile + 1);
            fetch_v(tile + 1, vnext);
        }
        const float* pack = smem + (tile & 1) * STAGE;
        const float* coef = pack + PACK;
        if (!makes_o) {                                  // what the update takes is there from the start
#pragma unroll
            for (int k = 0; k < 4; ++k) G_s[(c + 4 * k) * RP + col] = to_float<T>(vnow[k]);
        }
        // product 1: the pack's rows against this warp's rows of S
        {
            float big[2][4] = {}, small[2][4] = {};
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                Split b[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) b[e] = split_tf32(S[nt][e]);
                const float* row = pack + r * PP + warp * WROWS + 8 * nt + 2 * c;
                const float2 lo = *reinterpret_cast<const float2*>(row), hi = *reinterpret_cast<const float2*>(row + 8 * PP);
                const SplitA a = split_a(lo.x, hi.x, lo.y, hi.y);
                mma_split<FRESH>(big[0], small[0], a, b[0], b[1]);
                mma_split<FRESH>(big[1], small[1], a, b[2], b[3]);
            }
#pragma unroll
            for (int nj = 0; nj < 2; ++nj)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<float2*>(red + (warp * B + r + 8 * half) * RP + 8 * nj + 2 * c) =
                        make_float2(big[nj][2 * half] + small[nj][2 * half], big[nj][2 * half + 1] + small[nj][2 * half + 1]);
        }
        __syncthreads();                                 // the partial sums are in
        if (makes_o) {
            float x[4];                                  // V at tokens c + 4 k of column `col`
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = to_float<T>(vnow[k]);
            float y[4];
            times_coefficients<FRESH>(y, coef + B * CP, x, r, c);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = r + 8 * half;
                float q0 = 0.f, q1 = 0.f;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) {
                    const float2 q = *reinterpret_cast<const float2*>(red + (w * B + t) * RP + 8 * nt_uo + 2 * c);
                    q0 += q.x;
                    q1 += q.y;
                }
                const int j = j0 + 8 * nt_uo + 2 * c;
                if (tile * B + t < n) {
                    float* dst = p.out + ((long long)(begin + tile * B + t) * p.heads + h) * p.vdim + j;
                    if (j < p.vdim) dst[0] = q0 + y[2 * half];
                    if (j + 1 < p.vdim) dst[1] = q1 + y[2 * half + 1];
                }
            }
        }
        // product 3, S^T <- decay S^T + G^T K, and the state after the tile
        {
            SplitA a[2];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const float* g = G_s + (8 * ks + c) * RP + r;
                a[ks] = split_a(g[0], g[8], g[4 * RP], g[4 * RP + 8]);
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float big[4] = {}, small[4] = {};
                const float* k = pack + (B + c) * PP + warp * WROWS + 8 * nt + r;
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const Split k0 = split_tf32(k[8 * ks * PP]), k1 = split_tf32(k[(8 * ks + 4) * PP]);
                    mma_split<FRESH>(big, small, a[ks], k0, k1);
                }
                const float2 d = *reinterpret_cast<const float2*>(pack + 2 * B * PP + warp * WROWS + 8 * nt + 2 * c);
                S[nt][0] = fmaf(d.x, S[nt][0], big[0] + small[0]);
                S[nt][1] = fmaf(d.y, S[nt][1], big[1] + small[1]);
                S[nt][2] = fmaf(d.x, S[nt][2], big[2] + small[2]);
                S[nt][3] = fmaf(d.y, S[nt][3], big[3] + small[3]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) vnow[k] = vnext[k];
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, j;
            if (element(nt, e, i, j)) st[(long long)i * p.vdim + j] = S[nt][e];
        }
}

// The delta rules' walk.  A CTA owns one request, one head and 16 columns.  Eight warps hold the state's rows.  A tile is a chain: k side
// against S_0, its sum over the warps, U, the update.  What it does not wait for is beside it: the q side's product runs while two warps
// without rows make U and two more (P W) (V - R), and those sum up and store the output under the update (all meet before the next tile).
// Packs and coefficients come by bulk copies, two tiles in shared memory.  Every wait for them gives up after about two seconds and says
// so in an error word; the CTA then stores nothing of that tile and the later ones, leaves the state as it was, waits once more, as long, for
// the copies on their way (the shared memory they write will be another CTA's) and returns.
// Bound by the chain.  Three portions of 1,001, 667 and 333 tokens, 8 heads of 128 x 128: 86 us, where four warps that did both sides
// before U, made U and O and copied the tiles themselves took 100.
constexpr int DELTA_WARPS = 8, HELPERS = 4, HOLDERS = DELTA_WARPS * 32, DELTA_THREADS = HOLDERS + HELPERS * 32;

template <int NT, int MODE>
__global__ void __launch_bounds__(DELTA_THREADS) delta_tiles_kernel(ScanArgs p) {
    constexpr int WROWS = 8 * NT, ROWS = DELTA_WARPS * WROWS;
    constexpr int PP = pack_pitch(ROWS);
    constexpr int SETS = sets_of(MODE), PACK = pack_floats(ROWS, SETS), STAGE = PACK + COEF, SUMS = DELTA_WARPS * B * RP;
    constexpr bool FRESH = MODE == CHANNEL;
    static_assert(MODE == DELTA || MODE == CHANNEL, "the delta rules");
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ int failed;
    float* red_k = smem + 2 * STAGE;                     // [DELTA_WARPS][B][RP], and of the q side
    float* red_q = red_k + SUMS;
    float* X_s = red_q + SUMS;                           // [B][RP]: V - R; (P W) of it
    float* O_s = X_s + B * RP;
    float* G_s = O_s + B * RP;                           // [2][B][RP]: G[B] U as two TF32 numbers
    const int seq = p.prefill_seqs[blockIdx.z], h = blockIdx.y, j0 = blockIdx.x * COLS;
    if (seq < 0) return;
    const int begin = p.cu_q[seq], n = p.cu_q[seq + 1] - begin, slot = p.slots[seq];
    if (n <= 1 || slot < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
    const bool holds = warp < DELTA_WARPS;
    const int qk_heads = p.heads / p.qk_group, qh = h / p.qk_group;
    float* st = p.state + (long long)slot * p.slot_stride + (long long)h * p.dim * p.vdim;
    auto element = [&](int nt, int e, int& i, int& j) {  // row and column of S of register e of tile nt
        i = warp * WROWS + 8 * nt + 2 * c + (e & 1);
        j = j0 + r + 8 * (e >> 1);
        return i < p.dim && j < p.vdim;
    };
    float S[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, j;
            S[nt][e] = holds && element(nt, e, i, j) ? st[(long long)i * p.vdim + j] : 0.f;
        }
    const int tiles = (n + B - 1) / B;
    const long long first = tile_slot(seq, begin, 0);
    auto issue = [&](int tile) {                         // one thread
        float* stage = smem + (tile & 1) * STAGE;
        mbar_expect_tx(&full[tile & 1], STAGE * 4);
        bulk_copy(stage, p.pack + ((first + tile) * qk_heads + qh) * (long long)PACK, PACK * 4, &full[tile & 1]);
        bulk_copy(stage + PACK, p.coef + ((first + tile) * p.heads + h) * (long long)COEF, COEF * 4, &full[tile & 1]);
    };
    static_assert(PACK % 4 == 0 && COEF % 4 == 0, "bulk copies go by 16 bytes");
    // the holders' threads a value of the tile: token tx, column cx; the helpers' two outputs: tokens tx and tx + 8
    const int tx = (holds ? tid : tid - HOLDERS) / COLS, cx = tid % COLS;
    static_assert(HOLDERS == B * COLS && HELPERS * 64 == B * COLS && HELPERS == 4, "a thread a value, or two; two helpers for U and two for O");
    const bool in_columns = j0 + cx < p.vdim;
    const float* v = (const float*)p.v + (long long)(begin + tx) * p.v_stride + (long long)h * p.vdim + j0 + cx;
    float* out = p.out + ((long long)(begin + tx) * p.heads + h) * p.vdim + j0 + cx;
    const long long v_step = B * p.v_stride, token_step = (long long)p.heads * p.vdim;
    auto fetch_v = [&](int tile) { return holds && in_columns && tile * B + tx < n ? v[tile * v_step] : 0.f; };
    if (tid == 0) {
        failed = 0;
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        issue(0);
    }
    float vnow = fetch_v(0);
    for (int tile = 0; tile < tiles; ++tile) {
        __syncthreads();                                 // the barriers exist; the other stage, U and the sums have been read
        if (tid == 0 && tile + 1 < tiles) issue(tile + 1);
        if (!mbar_wait(&full[tile & 1], tile >> 1 & 1, p.error, holds ? 31 : 32, p.wait_cycles)) failed = 1;
        float vnext = 0.f;
        if (tile + 1 < tiles) vnext = fetch_v(tile + 1);
        const float* pack = smem + (tile & 1) * STAGE;
        const float* coef = pack + PACK;
        Split s[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[nt][e] = split_tf32(S[nt][e]);
        auto against_state = [&](const float* rows, float* red) {    // 16 rows of the pack against this warp's rows of S
            float big[2][4], small[2][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const float* row = rows + r * PP + warp * WROWS + 8 * nt + 2 * c;
                const float2 lo = *reinterpret_cast<const float2*>(row), hi = *reinterpret_cast<const float2*>(row + 8 * PP);
                const SplitA a = split_a(lo.x, hi.x, lo.y, hi.y);
#pragma unroll
                for (int nj = 0; nj < 2; ++nj) {
                    if (nt == 0) mma_split_first(big[nj], small[nj], a, s[nt][2 * nj], s[nt][2 * nj + 1]);
                    else mma_split<FRESH>(big[nj], small[nj], a, s[nt][2 * nj], s[nt][2 * nj + 1]);
                }
            }
#pragma unroll
            for (int nj = 0; nj < 2; ++nj)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<float2*>(red + (warp * B + r + 8 * half) * RP + 8 * nj + 2 * c) =
                        make_float2(big[nj][2 * half] + small[nj][2 * half], big[nj][2 * half + 1] + small[nj][2 * half + 1]);
        };
        if (holds) against_state(pack + B * PP, red_k);
        __syncthreads();                                 // the k side's partial sums are in
        const int gone = failed;                         // the same in all threads; looked at where its load has long come back
        if (holds) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < DELTA_WARPS; ++w) sum += red_k[(w * B + tx) * RP + cx];
            X_s[tx * RP + cx] = MODE == DELTA ? fmaf(-coef[2 * B * CP + tx], sum, vnow) : vnow - sum;
        }
        __syncthreads();                                 // V - R is in
        if (holds) {
            against_state(pack, red_q);
        } else {
            const bool makes_u = warp < DELTA_WARPS + 2;
            const int col = 8 * (warp & 1);
            float x[4], y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) x[k] = X_s[(c + 4 * k) * RP + col + r];
            times_coefficients<FRESH>(y, coef + (makes_u ? 0 : B * CP), x, r, c);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = r + 8 * half;
                if (makes_u) {
                    const float g = MODE == DELTA ? coef[2 * B * CP + B + t] : 1.f;
                    const Split a = split_tf32(g * y[2 * half]), b = split_tf32(g * y[2 * half + 1]);
                    *reinterpret_cast<uint2*>(G_s + t * RP + col + 2 * c) = make_uint2(a.hi, b.hi);
                    *reinterpret_cast<uint2*>(G_s + (B + t) * RP + col + 2 * c) = make_uint2(a.lo, b.lo);
                } else {
                    *reinterpret_cast<float2*>(O_s + t * RP + col + 2 * c) = make_float2(y[2 * half], y[2 * half + 1]);
                }
            }
        }
        __syncthreads();                                 // what the update takes is in, and all of the output
        if (gone) {
            for (int t = tile; tid == 0 && t < tiles && t < tile + 2; ++t) mbar_wait(&full[t & 1], t >> 1 & 1, p.error, 31);
            return;
        }
        if (holds) {                                     // S^T <- decay S^T + G^T K: the state after the tile
            SplitA a[2];
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const uint32_t* g = reinterpret_cast<const uint32_t*>(G_s) + (8 * ks + c) * RP + r;
                a[ks] = SplitA{{g[0], g[8], g[4 * RP], g[4 * RP + 8]}, {g[B * RP], g[B * RP + 8], g[(B + 4) * RP], g[(B + 4) * RP + 8]}};
            }
            const float cB = MODE == DELTA ? coef[2 * B * CP + B - 1] : 1.f;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float big[4], small[4];
                const float* k = pack + (SETS * B + c) * PP + warp * WROWS + 8 * nt + r;
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const Split k0 = split_tf32(k[8 * ks * PP]), k1 = split_tf32(k[(8 * ks + 4) * PP]);
                    if (ks == 0) mma_split_first(big, small, a[0], k0, k1);
                    else mma_split<FRESH>(big, small, a[1], k0, k1);
                }
                float2 d = make_float2(cB, cB);
                if (MODE != DELTA) d = *reinterpret_cast<const float2*>(pack + (1 + SETS) * B * PP + warp * WROWS + 8 * nt + 2 * c);
                S[nt][0] = fmaf(d.x, S[nt][0], big[0] + small[0]);
                S[nt][1] = fmaf(d.y, S[nt][1], big[1] + small[1]);
                S[nt][2] = fmaf(d.x, S[nt][2], big[2] + small[2]);
                S[nt][3] = fmaf(d.y, S[nt][3], big[3] + small[3]);
            }
        } else {
#pragma unroll
            for (int t = tx; t < B; t += B / 2) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < DELTA_WARPS; ++w) sum += red_q[(w * B + t) * RP + cx];
                const float y = O_s[t * RP + cx];
                if (in_columns && tile * B + t < n) out[(tile * B + t - tx) * token_step] = MODE == DELTA ? fmaf(coef[2 * B * CP + t], sum, y) : y + sum;
            }
        }
        vnow = vnext;
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int i, j;
            if (holds && element(nt, e, i, j)) st[(long long)i * p.vdim + j] = S[nt][e];
        }
}

template <typename T, int MODE>
int launch_scan(const ScanArgs& p, int portions, cudaStream_t stream) {
    const dim3 grid((p.vdim + COLS - 1) / COLS, p.heads, portions);
#define TS_TILES(NT)                                                                                                 \
    do {                                                                                                             \
        constexpr int ROWS = WARPS * 8 * NT;                                                                         \
        if constexpr (MODE == DELTA || MODE == CHANNEL) {                                                            \
            static_assert(sizeof(T) == 4, "the delta rules' values are float32");                                    \
            const size_t smem = sizeof(float) * (2 * (pack_floats(ROWS, sets_of(MODE)) + COEF) + (2 * DELTA_WARPS + 4) * B * RP); \
            auto kernel = delta_tiles_kernel<NT * WARPS / DELTA_WARPS, MODE>;                                        \
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                    \
            kernel<<<grid, DELTA_THREADS, smem, stream>>>(p);                                                        \
        } else {                                                                                                     \
            const size_t smem = sizeof(float) * (2 * (pack_floats(ROWS, 1) + COEF) + (WARPS + 1) * B * RP);          \
            auto kernel = recurrence_tiles_kernel<T, NT, MODE>;                                                      \
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                    \
            kernel<<<grid, THREADS, smem, stream>>>(p);                                                              \
        }                                                                                                            \
    } while (0)
    const int rows = padded_rows(p.dim);
    if (rows == 64) TS_TILES(2);
    else if (rows == 128) TS_TILES(4);
    else TS_TILES(8);
#undef TS_TILES
    TS_LAUNCH_CHECK("recurrence_tiles");
    return 0;
}

}  // namespace

// Floats of the two buffers the tile kernels need: packs (`heads`: the q/k heads) and coefficients (`heads`: the value heads).
// `sets`: k-side sets of rows (2: delta rule with decays per channel).
TS_API long long ts_recurrence_tiles_pack_floats(int num_tokens, int num_seqs, int heads, int dim, int sets) {
    return ((long long)num_tokens / B + num_seqs + 1) * heads * pack_floats(padded_rows(dim), sets);
}
TS_API long long ts_recurrence_tiles_coef_floats(int num_tokens, int num_seqs, int heads) {
    return ((long long)num_tokens / B + num_seqs + 1) * heads * COEF;
}

// The delta rule with one decay a head over a step's prompt portions (`prefill_seqs`: the requests that feed more than
// one token, -1: none; `max_q_len` bounds their lengths).  q, k: float32 [tokens, kv_heads * dim] stretches after the
// convolution; gates [tokens, 2 heads]; v [tokens, heads * vdim] float32 stretch.  Rows of other requests are left alone.
TS_API int ts_delta_tiles(const float* q, const float* k, long long qk_stride, const float* gates, const float* dt_bias,
                          const float* a_log, const float* v, long long v_stride, const int* cu_q, const int* slots,
                          const int* prefill_seqs, int portions, int max_q_len, float* state, long long slot_stride,
                          float* pack, float* coef, float* out, int heads, int kv_heads, int dim, int vdim,
                          float unit_eps, float q_scale, int* error, long long wait_cycles, cudaStream_t stream) {
    TS_REQUIRE(error != nullptr, "delta_tiles: an error word is needed");
    TS_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && dim <= 256 && vdim > 0,
               "delta_tiles: %d heads over %d q/k heads of %d channels", heads, kv_heads, dim);
    TS_REQUIRE(slot_stride >= (long long)heads * dim * vdim, "delta_tiles: a state slot is too small");
    TS_REQUIRE(portions >= 0 && portions <= 65535 && heads <= 65535, "delta_tiles: grid too large");
    if (portions == 0 || max_q_len <= 1) return 0;
    PrepareArgs a{q, k, qk_stride, gates, dt_bias, a_log, cu_q, prefill_seqs, pack, coef, heads, kv_heads, dim, padded_rows(dim),
                  unit_eps, q_scale};
    const size_t smem = sizeof(float) * (2 * B * (a.rows + 1) + 2 * B * (B + 1));
    delta_tile_prepare_kernel<<<dim3((max_q_len + B - 1) / B, kv_heads, portions), 128, smem, stream>>>(a);
    TS_LAUNCH_CHECK("delta_tiles (prepare)");
    ScanArgs s{pack, coef, v, v_stride, cu_q, slots, prefill_seqs, state, slot_stride, out, heads, heads / kv_heads, dim, vdim, error, wait_cycles};
    return launch_scan<float, DELTA>(s, portions, stream);
}

// Time mixing over a step's prompt portions: r, k, v [tokens, heads * dim] of one dtype (r and k with one row stride),
// z float32 [tokens, heads * dim], w0 and u [heads * dim].
TS_API int ts_mix_tiles(const void* r, const void* k, long long rk_stride, const float* z, const float* w0, const float* u,
                        const void* v, long long v_stride, const int* cu_q, const int* slots, const int* prefill_seqs,
                        int portions, int max_q_len, float* state, long long slot_stride, float* pack, float* coef,
                        float* out, int heads, int dim, int dtype, cudaStream_t stream) {
    TS_REQUIRE(heads > 0 && dim > 0 && dim <= 256, "mix_tiles: %d heads of %d channels", heads, dim);
    TS_REQUIRE(slot_stride >= (long long)heads * dim * dim, "mix_tiles: a state slot is too small");
    TS_REQUIRE(portions >= 0 && portions <= 65535 && heads <= 65535, "mix_tiles: grid too large");
    if (portions == 0 || max_q_len <= 1) return 0;
    PrepareArgs a{r, k, rk_stride, z, w0, u, cu_q, prefill_seqs, pack, coef, heads, heads, dim, padded_rows(dim), 0.f, 1.f};
    const size_t smem = sizeof(float) * (3 * B * (a.rows + 1));
    const dim3 grid((max_q_len + B - 1) / B, heads, portions);
    ScanArgs s{pack, coef, v, v_stride, cu_q, slots, prefill_seqs, state, slot_stride, out, heads, 1, dim, dim, nullptr, 0};
    if (dtype == TS_F32) {
        cudaFuncSetAttribute(mix_tile_prepare_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        mix_tile_prepare_kernel<float><<<grid, 128, smem, stream>>>(a);
        TS_LAUNCH_CHECK("mix_tiles (prepare)");
        return launch_scan<float, MIX>(s, portions, stream);
    }
    if (dtype == TS_BF16) {
        cudaFuncSetAttribute(mix_tile_prepare_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        mix_tile_prepare_kernel<__nv_bfloat16><<<grid, 128, smem, stream>>>(a);
        TS_LAUNCH_CHECK("mix_tiles (prepare)");
        return launch_scan<__nv_bfloat16, MIX>(s, portions, stream);
    }
    return ts_fail("mix_tiles: unknown dtype code %d", dtype);
}

// Floats of the buffer of `ts_plain_tiles`.
TS_API long long ts_plain_tiles_floats(int num_tokens, int num_seqs, int heads, int dim, int vdim, int dtype) {
    if (dtype == TS_BF16) return plain_stretches_floats(num_tokens, num_seqs, heads, dim, vdim);
    return ts_recurrence_tiles_pack_floats(num_tokens, num_seqs, heads, dim, 1) + ts_recurrence_tiles_coef_floats(num_tokens, num_seqs, heads);
}

// The plain recurrence over a step's prompt portions: q, k, v as `ts_linear_recurrence` takes them; `buffer` has the floats of
// `ts_plain_tiles_floats`.  bfloat16 goes by stretches.
TS_API int ts_plain_tiles(const void* q, const void* k, const void* v, long long q_stride, long long k_stride, long long v_stride,
                          const float* z, long long z_stride, const float* bias, const float* head_decay, float inv_tau,
                          float q_scale, float k_scale, const float* freq, int rot_dims, const int* positions, const int* cu_q,
                          const int* slots, const int* prefill_seqs, int portions, int max_q_len, int num_tokens, int num_seqs,
                          float* state, long long slot_stride, float* buffer, float* out, int heads, int dim, int vdim, int dtype,
                          cudaStream_t stream) {
    TS_REQUIRE(heads > 0 && dim > 0 && dim <= 256 && vdim > 0, "plain_tiles: %d heads of %d channels", heads, dim);
    TS_REQUIRE(rot_dims >= 0 && rot_dims <= dim && rot_dims % 2 == 0, "plain_tiles: rotation over %d of %d channels", rot_dims, dim);
    TS_REQUIRE((z != nullptr) != (head_decay != nullptr), "plain_tiles: either decay logits or one decay per head");
    TS_REQUIRE(slot_stride >= (long long)heads * dim * vdim, "plain_tiles: a state slot is too small");
    TS_REQUIRE(portions >= 0 && portions <= 65535 && heads <= 65535, "plain_tiles: grid too large");
    TS_REQUIRE(dtype == TS_F32 || dtype == TS_BF16, "plain_tiles: unknown dtype code %d", dtype);
    if (portions == 0 || max_q_len <= 1) return 0;
    PlainArgs a{q, k, q_stride, k_stride, z, z_stride, bias, head_decay, inv_tau, q_scale, k_scale, freq, freq ? rot_dims : 0,
                positions, cu_q, prefill_seqs, buffer, nullptr, heads, dim};
    if (dtype == TS_BF16)
        return plain_stretches(a, (const __nv_bfloat16*)v, v_stride, slots, portions, max_q_len, state, slot_stride, num_tokens, num_seqs, out, vdim, stream);
    a.coef = buffer + ts_recurrence_tiles_pack_floats(num_tokens, num_seqs, heads, dim, 1);
    const int rows = padded_rows(dim);
    const size_t smem = rows == 64 ? PlainTile<64>::BYTES : rows == 128 ? PlainTile<128>::BYTES : PlainTile<256>::BYTES;   // 29 KB at 128 channels
    const dim3 grid((max_q_len + B - 1) / B, heads, portions);
    const ScanArgs s{a.pack, a.coef, v, v_stride, cu_q, slots, prefill_seqs, state, slot_stride, out, heads, 1, dim, vdim, nullptr, 0};
    auto kernel = rows == 64 ? plain_tile_prepare_kernel<64> : rows == 128 ? plain_tile_prepare_kernel<128> : plain_tile_prepare_kernel<256>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<grid, 128, smem, stream>>>(a);
    TS_LAUNCH_CHECK("plain_tiles (prepare)");
    return launch_scan<float, PLAIN>(s, portions, stream);
}

// The delta rule with decays per channel over a step's prompt portions: q, k float32 [tokens, kv_heads * dim] stretches after the
// convolution, v float32 [tokens, heads * vdim], z float32 [tokens, heads * dim], b [tokens, heads] logits of dtype `b_dtype`.
TS_API int ts_channel_tiles(const float* q, const float* k, long long qk_stride, const float* z, const void* b, long long b_stride,
                            int b_dtype, const float* dt_bias, const float* a_log, const float* v, long long v_stride,
                            const int* cu_q, const int* slots, const int* prefill_seqs, int portions, int max_q_len, float* state,
                            long long slot_stride, float* pack, float* coef, float* out, int heads, int kv_heads, int dim,
                            int vdim, float unit_eps, float q_scale, int* error, long long wait_cycles, cudaStream_t stream) {
    TS_REQUIRE(error != nullptr, "channel_tiles: an error word is needed");
    TS_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && dim <= 256 && vdim > 0,
               "channel_tiles: %d heads over %d q/k heads of %d channels", heads, kv_heads, dim);
    TS_REQUIRE(slot_stride >= (long long)heads * dim * vdim, "channel_tiles: a state slot is too small");
    TS_REQUIRE(portions >= 0 && portions <= 65535 && heads <= 65535, "channel_tiles: grid too large");
    if (portions == 0 || max_q_len <= 1) return 0;
    const ChannelArgs a{q, k, qk_stride, z, b, b_stride, dt_bias, a_log, cu_q, prefill_seqs, pack, coef, heads, kv_heads, dim,
                        unit_eps, q_scale};
    const int rows = padded_rows(dim);
    const size_t smem = sizeof(float) * (3 * B * (rows + 2) + 2 * B * (B + 1)) + 2 * B * (rows + 2);
    const dim3 grid((max_q_len + B - 1) / B, heads, portions);
    TS_REQUIRE(b_dtype == TS_F32 || b_dtype == TS_BF16, "channel_tiles: unknown dtype code %d", b_dtype);
#define TS_CHANNEL_PREPARE(T)                                                                                                  \
    do {                                                                                                                       \
        auto kernel = rows == 64 ? channel_tile_prepare_kernel<T, 64> : rows == 128 ? channel_tile_prepare_kernel<T, 128>      \
                                                                                    : channel_tile_prepare_kernel<T, 256>;     \
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                                  \
        kernel<<<grid, 128, smem, stream>>>(a);                                                                                \
    } while (0)
    if (b_dtype == TS_F32) TS_CHANNEL_PREPARE(float);
    else TS_CHANNEL_PREPARE(__nv_bfloat16);
#undef TS_CHANNEL_PREPARE
    TS_LAUNCH_CHECK("channel_tiles (prepare)");
    const ScanArgs s{pack, coef, v, v_stride, cu_q, slots, prefill_seqs, state, slot_stride, out, heads, 1, dim, vdim, error, wait_cycles};
    return launch_scan<float, CHANNEL>(s, portions, stream);
}
