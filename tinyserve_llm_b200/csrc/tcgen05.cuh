// What the tcgen05 products share: mbarriers with bounded waits, TMA tile loads, descriptors of the fifth-generation
// tensor cores' operands.
#pragma once

#include <cuda.h>

#include "common.cuh"

constexpr long long WAIT_CYCLES = 4000000000ll;     // about two seconds at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// false: the wait ran out of time (the error word says which one); with a limit of 0 it does so without a look
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* error, int code, long long limit = WAIT_CYCLES) {
    const long long start = clock64();
    uint32_t done = 0;
    while (limit > 0) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (done) return true;
        if (clock64() - start > limit) break;
    }
    atomicExch(error, code);
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* smem, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 bfloat16 or 32 TF32 numbers) with
// the 128-byte swizzle: start address, stride between groups of 8 rows (1024 bytes), sm_100 version.
__device__ __forceinline__ uint64_t smem_desc(const void* tile) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_u32(tile) & 0x3FFFF) >> 4);          // bits 0..13: start address / 16
    d |= (uint64_t)1 << 16;                                      // bits 16..29: leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                            // bits 32..45: stride byte offset / 16
    d |= (uint64_t)1 << 46;                                      // bits 46..47: descriptor version of sm_100
    d |= (uint64_t)2 << 61;                                      // bits 61..63: 128-byte swizzle
    return d;
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Two CTAs of a cluster that work on one tile.
__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t in_first_cta(const void* local) {      // the same object in the pair's first CTA
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(0));
    return remote;
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {          // arrives on `bar` in both CTAs
    const uint16_t both = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(both) : "memory");
}
// A load into this CTA's shared memory that is counted on the first CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(void* smem, const CUtensorMap* map, uint32_t bar_in_first, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem)), "l"(map), "r"(bar_in_first), "r"(x), "r"(y) : "memory");
}
// An arrival on the other CTA's barrier that hands tensor memory over (an accumulator back, an operand on), which tcgen05's fences on both
// sides order.  It orders none of this thread's writes to shared or global memory for the other CTA: that takes a release at cluster scope,
// about a microsecond each.  What MMAs of the first CTA read from the second one's shared memory is brought there by TMA.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar_in_cluster) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_in_cluster) : "memory");
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(sym);
    }
    return fn;
}

// A [rows, cols] row-major matrix of `type` (`size` bytes an element), boxes of box_rows rows x 128 bytes, 128-byte swizzle.
static inline int make_tile_map(CUtensorMap* map, CUtensorMapDataType type, int size, const void* base, long long rows,
                                long long cols, long long ld, int box_rows, const char* who) {
    EncodeTiled encode = encode_tiled();
    if (!encode) return ts_fail("%s: the driver does not export cuTensorMapEncodeTiled", who);
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * size};
    const cuuint32_t box[2] = {(cuuint32_t)(128 / size), (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return ts_fail("%s: cuTensorMapEncodeTiled failed with %d", who, (int)r);
    return 0;
}
