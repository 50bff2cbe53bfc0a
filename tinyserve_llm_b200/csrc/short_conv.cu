// Short causal convolution over time, one filter per channel, followed by silu:
//
//   y[t, c] = silu( sum_{j < taps} w[c, j] * x[t - (taps - 1 - j), c] )        zeros before the sequence's start
//
// The last taps - 1 inputs of a request are part of its state (float32, [taps - 1][channels] in the
// request's slot, oldest first), so a prompt may be cut anywhere and decoding is the same kernel: an
// input from before this step's first token is read from the slot.  A second kernel, launched behind
// the first, moves the slot on.  Sums are float32; the output is float32.
#include "common.cuh"

// grid: (channel blocks, groups of `group` tokens); a CTA's threads are neighbouring channels, each walks the group's
// tokens (8 in a step of many tokens, 1 in a small step, where the walk would only lengthen the step)

template <typename T>
__global__ void short_conv_silu_kernel(const T* __restrict__ x, long long x_stride, const float* __restrict__ w,
                                       const int* __restrict__ seq_of_token, const int* __restrict__ cu_q,
                                       const int* __restrict__ slots, const float* __restrict__ state, long long slot_stride,
                                       float* __restrict__ y, int num_tokens, int channels, int taps, int group) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int t_end = min(num_tokens, (int)(blockIdx.y + 1) * group);
    const float* wc = w + (long long)c * taps;
    for (int t = blockIdx.y * group; t < t_end; ++t) {
        const int seq = seq_of_token[t];
        if (seq < 0) { y[(long long)t * channels + c] = 0.f; continue; }      // a padding row
        const int slot = slots[seq];
        const int begin = cu_q[seq];
        const float* st = state + (long long)slot * slot_stride;
        float acc = 0.f;
        for (int j = 0; j < taps; ++j) {
            const int src = t - begin - (taps - 1 - j);    // token of this step, or (negative) one of the slot's
            float v;
            if (src >= 0) v = to_float<T>(x[(long long)(begin + src) * x_stride + c]);
            else v = slot >= 0 ? st[(long long)(taps - 1 + src) * channels + c] : 0.f;
            acc = fmaf(wc[j], v, acc);
        }
        y[(long long)t * channels + c] = acc / (1.f + expf(-acc));
    }
}

// The same for steps of many tokens and four taps: a thread walks CONV_RUN tokens of four neighbouring channels with the last three
// inputs in registers, all its loads asked for at the start.  The other kernel reads every input four times, two bytes a load, and looks
// the token's request up for each; 2,002 tokens of 2,048 channels, bfloat16: 28.9 us, and 12.3 here (4 by the bytes).
constexpr int CONV_RUN = 8, CONV_TAPS = 4;

template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&v)[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

template <typename T>
__global__ void __launch_bounds__(128)
short_conv_silu_runs_kernel(const T* __restrict__ x, long long x_stride, const float* __restrict__ w,
                            const int* __restrict__ seq_of_token, const int* __restrict__ cu_q, const int* __restrict__ slots,
                            const float* __restrict__ state, long long slot_stride, float* __restrict__ y, int num_tokens, int channels) {
    const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
    if (c >= channels) return;
    const int t0 = blockIdx.y * CONV_RUN, count = min(CONV_RUN, num_tokens - t0);
    float in[CONV_RUN][4], wc[4][CONV_TAPS], last[CONV_TAPS - 1][4];      // last: the inputs before the next token, oldest first
    int seqs[CONV_RUN];
#pragma unroll
    for (int i = 0; i < CONV_RUN; ++i) {
        seqs[i] = -1;
        if (i < count) {
            seqs[i] = seq_of_token[t0 + i];
            load4<T>(x + (long long)(t0 + i) * x_stride + c, in[i]);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) load4<float>(w + (long long)(c + e) * CONV_TAPS, wc[e]);
    int seq = -2;
#pragma unroll
    for (int i = 0; i < CONV_RUN; ++i) {
        if (i >= count) break;
        float out[4] = {0.f, 0.f, 0.f, 0.f};                              // a padding row
        if (seqs[i] >= 0) {
            if (seqs[i] != seq) {                                         // the run's first token, or another request's
                const int begin = cu_q[seqs[i]], slot = slots[seqs[i]];
#pragma unroll
                for (int j = 0; j < CONV_TAPS - 1; ++j) {
                    const int src = t0 + i - begin - (CONV_TAPS - 1 - j);  // token of this step, or (negative) one of the slot's
#pragma unroll
                    for (int e = 0; e < 4; ++e) last[j][e] = 0.f;
                    if (src >= 0) load4<T>(x + (long long)(begin + src) * x_stride + c, last[j]);
                    else if (slot >= 0) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) last[j][e] = state[(long long)slot * slot_stride + (long long)(CONV_TAPS - 1 + src) * channels + c + e];
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < CONV_TAPS - 1; ++j) acc = fmaf(wc[e][j], last[j][e], acc);
                acc = fmaf(wc[e][CONV_TAPS - 1], in[i][e], acc);
                out[e] = acc / (1.f + expf(-acc));
#pragma unroll
                for (int j = 0; j < CONV_TAPS - 2; ++j) last[j][e] = last[j + 1][e];
                last[CONV_TAPS - 2][e] = in[i][e];
            }
        }
        seq = seqs[i];
        *reinterpret_cast<float4*>(y + (long long)(t0 + i) * channels + c) = make_float4(out[0], out[1], out[2], out[3]);
    }
}

template <typename T>
static bool short_conv_runs(const void* x, long long x_stride, const float* w, const int* seq_of_token, const int* cu_q, const int* slots,
                            const float* state, long long slot_stride, float* y, int num_tokens, int channels, int taps, cudaStream_t stream) {
    // enough tokens that runs of eight still fill the SMs, and rows that start on the loads' boundaries
    if (taps != CONV_TAPS || num_tokens < 256 || channels % 4 || x_stride % 4 || (uintptr_t)x % (4 * sizeof(T)) || ((uintptr_t)w | (uintptr_t)y) % 16 ||
        (num_tokens + CONV_RUN - 1) / CONV_RUN > 65535)
        return false;
    const dim3 grid((channels / 4 + 127) / 128, (num_tokens + CONV_RUN - 1) / CONV_RUN);
    short_conv_silu_runs_kernel<T><<<grid, 128, 0, stream>>>((const T*)x, x_stride, w, seq_of_token, cu_q, slots, state, slot_stride, y,
                                                             num_tokens, channels);
    return true;
}

// state <- the last taps - 1 inputs after this step; one thread a (request, channel), oldest entry first, so an
// entry is read before it is overwritten
template <typename T>
__global__ void short_conv_advance_kernel(const T* __restrict__ x, long long x_stride, const int* __restrict__ cu_q,
                                          const int* __restrict__ slots, float* __restrict__ state, long long slot_stride,
                                          int num_seqs, int channels, int taps) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)num_seqs * channels) return;
    const int seq = (int)(idx / channels), c = (int)(idx % channels);
    const int slot = slots[seq];
    const int begin = cu_q[seq], n = cu_q[seq + 1] - begin;
    if (slot < 0 || n <= 0) return;
    float* st = state + (long long)slot * slot_stride;
    for (int i = 0; i < taps - 1; ++i) {
        const int src = n - (taps - 1) + i;
        st[(long long)i * channels + c] = src >= 0 ? to_float<T>(x[(long long)(begin + src) * x_stride + c])
                                                   : st[(long long)(i + n) * channels + c];
    }
}

TS_API int ts_short_conv_silu(const void* x, long long x_stride, const float* w, const int* seq_of_token, const int* cu_q,
                              const int* slots, int num_seqs, float* state, long long slot_stride, float* y, int num_tokens,
                              int channels, int taps, int dtype, cudaStream_t stream) {
    TS_REQUIRE(num_tokens >= 0 && channels > 0 && taps > 0, "short_conv: bad sizes");
    TS_REQUIRE(slot_stride >= (long long)(taps - 1) * channels, "short_conv: a state slot is too small");
    if (num_tokens == 0 || num_seqs == 0) return 0;
    const int group = num_tokens >= 512 ? 8 : 1;
    TS_REQUIRE(num_tokens <= 65535 * group, "short_conv: %d tokens a step are not supported", num_tokens);
    const dim3 blocks((channels + 255) / 256, (num_tokens + group - 1) / group);
    const unsigned blocks2 = (unsigned)(((long long)num_seqs * channels + 255) / 256);
    if (dtype == TS_F32) {
        if (!short_conv_runs<float>(x, x_stride, w, seq_of_token, cu_q, slots, state, slot_stride, y, num_tokens, channels, taps, stream))
            short_conv_silu_kernel<float><<<blocks, 256, 0, stream>>>((const float*)x, x_stride, w, seq_of_token, cu_q, slots,
                                                                  state, slot_stride, y, num_tokens, channels, taps, group);
        if (taps > 1)
            short_conv_advance_kernel<float><<<blocks2, 256, 0, stream>>>((const float*)x, x_stride, cu_q, slots, state,
                                                                          slot_stride, num_seqs, channels, taps);
    } else if (dtype == TS_BF16) {
        if (!short_conv_runs<__nv_bfloat16>(x, x_stride, w, seq_of_token, cu_q, slots, state, slot_stride, y, num_tokens, channels, taps, stream))
            short_conv_silu_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)x, x_stride, w, seq_of_token,
                                                                          cu_q, slots, state, slot_stride, y, num_tokens, channels, taps, group);
        if (taps > 1)
            short_conv_advance_kernel<__nv_bfloat16><<<blocks2, 256, 0, stream>>>((const __nv_bfloat16*)x, x_stride, cu_q, slots,
                                                                                  state, slot_stride, num_seqs, channels, taps);
    } else {
        return ts_fail("short_conv: unknown dtype code %d", dtype);
    }
    TS_LAUNCH_CHECK("short_conv");
    return 0;
}
