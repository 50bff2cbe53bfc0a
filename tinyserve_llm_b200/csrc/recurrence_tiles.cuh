// What the recurrences over prompt portions sixteen tokens at a time share (recurrence_tiles.cu, recurrence_stretches.cu).
#pragma once

#include "tcgen05.cuh"

// The plain recurrence's inputs.
struct PlainArgs {
    const void* q; const void* k; long long q_stride, k_stride;
    const float* z; long long z_stride; const float* bias;   // decay logits a channel (a = sigmoid(z + bias)^inv_tau), or
    const float* head_decay;                                 // one decay a head
    float inv_tau, q_scale, k_scale;
    const float* freq; int rot_dims; const int* positions;   // rotation by halves over the first rot_dims channels
    const int* cu_q; const int* prefill_seqs;
    float* pack; float* coef;
    int heads, dim;
};

namespace {

constexpr int B = 16;              // tokens a tile

// Where a request's tiles lie among all tiles: request s's first at cu_q[s] / 16 + s.  Every request has room for its own
// (a portion of n tokens takes ceil(n / 16), and the next request's first lies at least that much further on).
__device__ __forceinline__ long long tile_slot(int seq, int begin, int tile) { return begin / B + seq + tile; }

// exp(x), x <= 0, as a float32 number and what that lacks: near one, where a portion multiplies many of them, 1 + expm1(x) is known to
// more bits than float32 holds.
__device__ __forceinline__ float decay_of(float x, float& rest) {
    const float a = expf(x);
    rest = 0.f;
    if (!(x > -0.6f)) return a;
    const float m = expm1f(x), near = 1.f + m;
    rest = m - (near - 1.f);
    return near;
}

__device__ __forceinline__ double whole(float a, __nv_bfloat16 rest) { return (double)a + (double)__bfloat162float(rest); }


// A tile's queries, keys and decays in shared memory (and what the decays lack), for the preparation's 128 threads.
template <int ROWS>
struct PlainTile {
    static constexpr int PITCH = ROWS + 2;               // even: two channels a load
    float *q, *k, *a;                                    // [16][PITCH]
    __nv_bfloat16* rest;
    static constexpr size_t BYTES = (3 * sizeof(float) + sizeof(__nv_bfloat16)) * B * PITCH;
    __device__ __forceinline__ PlainTile(float* smem)
        : q(smem), k(q + B * PITCH), a(k + B * PITCH), rest(reinterpret_cast<__nv_bfloat16*>(a + B * PITCH)) {}
};

// A thread a channel (ROWS 64: two threads), four tokens' loads under way together.
template <typename T, int ROWS>
__device__ __forceinline__ void load_plain(const PlainArgs& p, const PlainTile<ROWS>& x, int h, int t0, int m) {
    constexpr int pitch = PlainTile<ROWS>::PITCH, LANES = ROWS < 128 ? ROWS : 128, STEP = 128 / LANES, DEEP = 4;
    const int half = p.rot_dims / 2;
    for (int i = threadIdx.x % LANES; i < ROWS; i += LANES) {
        const int ic = min(i, p.dim - 1);                // loads stay inside; what is not there is selected away
        const bool turns = ic < p.rot_dims;
        const int f = ic < half ? ic : ic - half, other = turns ? (ic < half ? ic + half : ic - half) : ic;
        const float freq = turns ? p.freq[f] : 0.f, bias = p.z && p.bias ? p.bias[h * p.dim + ic] : 0.f, fixed = p.z ? 1.f : p.head_decay[h];
        for (int first = threadIdx.x / LANES; first < B; first += STEP * DEEP) {
            T q[DEEP], k[DEEP], qo[DEEP], ko[DEEP];
            float z[DEEP];
            int at[DEEP];
#pragma unroll
            for (int e = 0; e < DEEP; ++e) {
                const long long row = t0 + min(first + e * STEP, m - 1);
                const T *qr = (const T*)p.q + row * p.q_stride + (long long)h * p.dim, *kr = (const T*)p.k + row * p.k_stride + (long long)h * p.dim;
                q[e] = qr[ic];
                k[e] = kr[ic];
                if (p.rot_dims) {
                    qo[e] = qr[other];
                    ko[e] = kr[other];
                    at[e] = p.positions[row];
                }
                z[e] = p.z ? p.z[row * p.z_stride + (long long)h * p.dim + ic] : 0.f;
            }
#pragma unroll
            for (int e = 0; e < DEEP; ++e) {
                const int t = first + e * STEP;
                float qv = 0.f, kv = 0.f, av = 1.f, more = 0.f;      // a token past the portion's end changes nothing
                if (t < m && i < p.dim) {
                    qv = to_float<T>(q[e]);
                    kv = to_float<T>(k[e]);
                    if (turns) {
                        float sn, cs;
                        sincosf((float)at[e] * freq, &sn, &cs);
                        const float u = to_float<T>(qo[e]), w = to_float<T>(ko[e]);
                        qv = i < half ? qv * cs - u * sn : qv * cs + u * sn;
                        kv = i < half ? kv * cs - w * sn : kv * cs + w * sn;
                    }
                    qv *= p.q_scale;
                    kv *= p.k_scale;
                    av = fixed;
                    if (p.z) {
                        const float y = z[e] + bias;
                        av = decay_of((fminf(y, 0.f) - log1pf(expf(-fabsf(y)))) * p.inv_tau, more);
                    }
                }
                x.q[t * pitch + i] = qv;
                x.k[t * pitch + i] = kv;
                x.a[t * pitch + i] = av;
                x.rest[t * pitch + i] = __float2bfloat16_rn(more);
            }
        }
    }
}

// P[t][j] of the plain recurrence, 0 where t < j: thread j = tid / 8 walks t with the running products of two of its channels at a time
template <int ROWS, typename Store>
__device__ __forceinline__ void plain_scores(const PlainTile<ROWS>& x, int dim, Store store) {
    constexpr int pitch = PlainTile<ROWS>::PITCH;
    const int j = threadIdx.x >> 3, part = threadIdx.x & 7;
    float sum[B];
#pragma unroll
    for (int t = 0; t < B; ++t) sum[t] = 0.f;
    for (int i = 2 * part; i < dim; i += 16) {           // (channels past dim hold zeros)
        float2 run = *reinterpret_cast<const float2*>(x.k + j * pitch + i);
#pragma unroll
        for (int t = 0; t < B; ++t) {
            if (t < (int)(threadIdx.x >> 5) * 4) continue;                              // the warp's four j begin here
            if (t > j) {
                const float2 a = *reinterpret_cast<const float2*>(x.a + t * pitch + i);
                run.x *= a.x;
                run.y *= a.y;
            }
            if (t >= j) {
                const float2 q = *reinterpret_cast<const float2*>(x.q + t * pitch + i);
                sum[t] = fmaf(q.y, run.y, fmaf(q.x, run.x, sum[t]));
            }
        }
    }
#pragma unroll
    for (int t = 0; t < B; ++t) {
        float s = sum[t];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (part == 0) store(t, j, s);
    }
}

// Channel i's queries times the decays from the tile's beginning to their own, its keys times those behind theirs; the product of all.
template <int ROWS, typename StoreQ, typename StoreK>
__device__ __forceinline__ float plain_sides(const PlainTile<ROWS>& x, int i, StoreQ store_q, StoreK store_k) {
    constexpr int pitch = PlainTile<ROWS>::PITCH;
    double decay[B], left = 1.0, right = 1.0;
#pragma unroll
    for (int t = 0; t < B; ++t) {
        decay[t] = whole(x.a[t * pitch + i], x.rest[t * pitch + i]);
        left *= decay[t];
        store_q(t, (float)((double)x.q[t * pitch + i] * left));
    }
#pragma unroll
    for (int t = B - 1; t >= 0; --t) {
        store_k(t, (float)((double)x.k[t * pitch + i] * right));
        right *= decay[t];
    }
    return (float)left;
}

// `bytes` (a multiple of 16) from memory to shared memory by the copy engine, counted on `bar`: the threads' own 16-byte copies of a tile
// of 29 KB held up the shared-memory pipe for 400 ns of 1,570.
__device__ __forceinline__ void bulk_copy(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void cp16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// A float32 number as the sum of two TF32 numbers (11 significant bits each): hi is x to the nearest (half of its last
// place added before the low 13 bits go), lo what is left, of which the tensor cores read the leading bits: 2^-23 of x is lost.
struct Split { uint32_t hi, lo; };
__device__ __forceinline__ Split split_tf32(float x) {
    Split s;
    s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    s.lo = __float_as_uint(x - __uint_as_float(s.hi));
    return s;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
struct SplitA { uint32_t hi[4], lo[4]; };
__device__ __forceinline__ SplitA split_a(float a0, float a1, float a2, float a3) {
    const Split s0 = split_tf32(a0), s1 = split_tf32(a1), s2 = split_tf32(a2), s3 = split_tf32(a3);
    return SplitA{{s0.hi, s1.hi, s2.hi, s3.hi}, {s0.lo, s1.lo, s2.lo, s3.lo}};
}
__device__ __forceinline__ void mma_tf32_fresh(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// The first of several products of split factors that are added up: both sums begin with it.
__device__ __forceinline__ void mma_split_first(float (&big)[4], float (&small)[4], const SplitA& a, Split b0, Split b1) {
    mma_tf32_fresh(big, a.hi, b0.hi, b1.hi);
    mma_tf32_fresh(small, a.hi, b0.lo, b1.lo);
    mma_tf32(small, a.lo, b0.hi, b1.hi);
}
// The two large and the small parts of a product of split factors, each in an accumulator of its own (no long chain).  FRESH: every
// large part begins at zero and is added by an ordinary rounded addition, where the tensor cores cut what an accumulator cannot hold.
template <bool FRESH>
__device__ __forceinline__ void mma_split(float (&big)[4], float (&small)[4], const SplitA& a, Split b0, Split b1) {
    if (FRESH) {
        float part[4];
        mma_tf32_fresh(part, a.hi, b0.hi, b1.hi);
#pragma unroll
        for (int i = 0; i < 4; ++i) big[i] += part[i];
    } else {
        mma_tf32(big, a.hi, b0.hi, b1.hi);
    }
    mma_tf32(small, a.hi, b0.lo, b1.lo);
    mma_tf32(small, a.lo, b0.hi, b1.hi);
}

int padded_rows(int dim) { return dim <= 64 ? 64 : dim <= 128 ? 128 : 256; }

}  // namespace

// The plain recurrence over bfloat16 prompt portions (recurrence_stretches.cu), and the floats of its buffer.
int plain_stretches(const PlainArgs& a, const __nv_bfloat16* v, long long v_stride, const int* slots, int portions, int max_q_len, float* state,
                    long long slot_stride, int num_tokens, int num_seqs, float* out, int vdim, cudaStream_t stream);
long long plain_stretches_floats(int num_tokens, int num_seqs, int heads, int dim, int vdim);
