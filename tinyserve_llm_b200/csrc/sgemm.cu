// float32 matrix product C[M, N] = A[M, K] . B[N, K]^T: the engine's true 32-bit projection (no tensor-core mode that
// rounds its inputs).  A single product of 64 terms and more whose rows TMA takes runs in sgemm_tcgen05.cu, no further from 64
// bits; this file's kernel, FFMA with float32 accumulation, takes the others and batches of products.  Each output element
// sums over k in ascending order, so a row's result does not depend on what else is in the batch.
// Any M, N, K; rows of A and B are K-contiguous (the checkpoint's [out_features, in_features]).
// A batched form runs one such product per blockIdx.z.
#include "common.cuh"

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

__global__ void __launch_bounds__(256)
sgemm_nt_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C, int M, int N, int K,
                long long lda, long long ldb, long long ldc, long long batch_a, long long batch_b, long long batch_c) {
    A += blockIdx.z * batch_a;                            // one product per blockIdx.z (strides 0: a single product)
    B += blockIdx.z * batch_b;
    C += blockIdx.z * batch_c;
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int tr = (tid / 16) * TM, tc = (tid % 16) * TN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    const int lk = tid % BK, lr = tid / BK;               // each thread loads 4 rows at column lk
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < BM / 16; ++i) {
            const int r = lr + 16 * i;
            const int gr = row0 + r, gk = k0 + lk;
            As[lk][r] = (gr < M && gk < K) ? A[(long long)gr * lda + gk] : 0.f;
            const int gc = col0 + r;
            Bs[lk][r] = (gc < N && gk < K) ? B[(long long)gc * ldb + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][tr + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[k][tc + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gr = row0 + tr + i;
        if (gr >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gc = col0 + tc + j;
            if (gc < N) C[(long long)gr * ldc + gc] = acc[i][j];
        }
    }
}

bool sgemm_tcgen05_supported(const float* x, const float* w, int K, long long ldx, long long ldw);
long long sgemm_tcgen05_scratch_floats(int M, int N, int K);
int sgemm_tcgen05(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                  float* scratch, int* error, cudaStream_t stream);

// Floats of scratch `ts_sgemm_nt` uses for rows without gaps (sgemm_tcgen05.cu), 16-byte aligned.
TS_API long long ts_sgemm_nt_scratch_floats(int M, int N, int K) {
    return M > 0 && N > 0 && sgemm_tcgen05_supported(nullptr, nullptr, K, K, K) ? sgemm_tcgen05_scratch_floats(M, N, K) : 0;
}

// On the tensor cores where TMA takes rows and addresses, whatever M is (a row's result must not depend on what else is in
// the batch); else by multiply-adds.  `error`: an int the host can read, for waits that run out.
TS_API int ts_sgemm_nt(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, float* scratch, long long scratch_floats, int* error, cudaStream_t stream) {
    TS_REQUIRE(M >= 0 && N > 0 && K > 0, "sgemm: bad sizes M=%d N=%d K=%d", M, N, K);
    TS_REQUIRE(lda >= K && ldb >= K && ldc >= N, "sgemm: row strides smaller than the rows");
    if (M == 0) return 0;
    if (error && sgemm_tcgen05_supported(A, B, K, lda, ldb)) {
        TS_REQUIRE(scratch_floats >= sgemm_tcgen05_scratch_floats(M, N, K) && (uintptr_t)scratch % 16 == 0,
                   "sgemm: %lld floats of scratch are too few, or not aligned", scratch_floats);
        return sgemm_tcgen05(A, B, C, M, N, K, lda, ldb, ldc, scratch, error, stream);
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    TS_REQUIRE(grid.y <= 65535, "sgemm: M=%d needs more than 65535 row tiles", M);
    sgemm_nt_kernel<<<grid, 256, 0, stream>>>(A, B, C, M, N, K, lda, ldb, ldc, 0, 0, 0);
    TS_LAUNCH_CHECK("sgemm");
    return 0;
}

// `batch` products at once: product b reads A + b * batch_a and B + b * batch_b and writes C + b * batch_c
// (the per-head products of an attention that folds its key and value projections into query and output).
TS_API int ts_sgemm_nt_batched(const float* A, const float* B, float* C, int M, int N, int K, long long lda,
                               long long ldb, long long ldc, int batch, long long batch_a, long long batch_b,
                               long long batch_c, cudaStream_t stream) {
    TS_REQUIRE(M >= 0 && N > 0 && K > 0 && batch > 0, "sgemm_batched: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    TS_REQUIRE(lda >= K && ldb >= K, "sgemm_batched: row strides smaller than the rows");
    if (M == 0) return 0;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    TS_REQUIRE(grid.y <= 65535 && batch <= 65535, "sgemm_batched: grid too large");
    sgemm_nt_kernel<<<grid, 256, 0, stream>>>(A, B, C, M, N, K, lda, ldb, ldc, batch_a, batch_b, batch_c);
    TS_LAUNCH_CHECK("sgemm_batched");
    return 0;
}
