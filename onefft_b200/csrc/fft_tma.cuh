// Bulk-copy building blocks shared by the TMA-staged pass kernels (fft_tma.cu) and the persistent
// one-kernel transforms (fft_long.cu): bounded mbarrier waits, tile copies, tensor maps of a pass.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

#include "fft_tiles.cuh"

namespace ofb {

constexpr unsigned kWaitLimit = 1u << 22;  // try_wait polls (each may suspend briefly): ~0.1-1 s

// Test hook of the failure path (onefft_debug_expire_waits): when non-zero, the first wait of
// every tile counts as expired without polling. The tile then takes the same path as after a
// real expiry: it records the failure in the plan's error word, lets its copy land (the normal
// bounded wait) and returns without writing. One copy per translation unit with such kernels.
static __device__ int g_expire_waits = 0;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned phase) {
    const unsigned a = smem_u32(bar);
    for (unsigned i = 0; i < kWaitLimit; ++i) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(phase)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(smem_u32(dst)),
        "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5, %6}], [%7];" ::"r"(smem_u32(dst)),
        "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3,
                                             int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];" ::"l"(
            (unsigned long long)map),
        "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// The same copies with an L2 eviction-priority hint (a createpolicy value).
__device__ __forceinline__ void tma_load_4d_hint(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                                 uint64_t* bar, unsigned long long policy) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, "
        "{%2, %3, %4, %5}], [%6], %7;" ::"r"(smem_u32(dst)),
        "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tma_load_5d_hint(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                                 int c4, uint64_t* bar, unsigned long long policy) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, "
        "{%2, %3, %4, %5, %6}], [%7], %8;" ::"r"(smem_u32(dst)),
        "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tma_store_5d_hint(const CUtensorMap* map, const void* src, int c0, int c1, int c2,
                                                  int c3, int c4, unsigned long long policy) {
    asm volatile(
        "cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group.L2::cache_hint [%0, {%2, %3, %4, %5, %6}], [%1], "
        "%7;" ::"l"((unsigned long long)map),
        "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "l"(policy)
        : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

__device__ __forceinline__ unsigned long long policy_evict_first() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// ---- host side ----------------------------------------------------------------------------------

inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

// Tensor map of the pass tile: MODE 0 {column r, row-in-box, row-box, batch} over `in`;
// MODE 1/2 {q, row-in-box, row-box, h, batch} over `out`. 8-byte elements, no swizzle.
inline bool make_map(CUtensorMap* m, const float2* base, int mode, int log2n, int log_l, int log_c, int log_s,
                     int batch) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc) return false;
    const cuuint64_t n = 1ull << log2n, L = 1ull << log_l, elo = L < 256 ? L : 256, ehi = L / elo;
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5], estr[5] = {1, 1, 1, 1, 1};
    int rank;
    if (mode == 0) {
        const cuuint64_t cols = n >> log_l;
        dims[0] = cols, dims[1] = elo, dims[2] = ehi, dims[3] = (cuuint64_t)batch;
        strides[0] = cols * 8, strides[1] = elo * cols * 8, strides[2] = n * 8;
        box[0] = 1u << log_c, box[1] = (cuuint32_t)elo, box[2] = (cuuint32_t)ehi, box[3] = 1;
        rank = 4;
    } else {
        const cuuint64_t S = 1ull << log_s, H = n >> (log_s + log_l);
        dims[0] = S, dims[1] = elo, dims[2] = ehi, dims[3] = H, dims[4] = (cuuint64_t)batch;
        strides[0] = S * 8, strides[1] = elo * S * 8, strides[2] = L * S * 8, strides[3] = n * 8;
        box[0] = 1u << log_c, box[1] = (cuuint32_t)elo, box[2] = (cuuint32_t)ehi, box[3] = 1, box[4] = 1;
        rank = 5;
    }
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t)rank, (void*)base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace ofb
