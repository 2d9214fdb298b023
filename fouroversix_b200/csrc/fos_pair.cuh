// What the CTA-pair (cta_group::2) GEMM kernels share: TMA copies that complete on either CTA's barrier, the stores of
// an epilogue, the launch (sm_100a).
#pragma once

#include "fos_tcgen05.cuh"

namespace fos {
namespace {

// A word of two rounded 16-bit outputs plus bias[0], bias[1] (`left` columns of them exist). A packed 16-bit addition
// rounds once from the exact sum, which is what adding in binary32 and rounding gives for two 16-bit numbers.
template <typename OUT> __device__ __forceinline__ uint32_t add_bias(uint32_t word, const OUT *bias, int64_t left) {
    const uint16_t *b = reinterpret_cast<const uint16_t *>(bias);
    const uint32_t lo = left > 0 ? ld_b16(b) : 0u, hi = left > 1 ? ld_b16(b + 1) : 0u, both = lo | (hi << 16);
    if constexpr (std::is_same<OUT, __half>::value) {
        const __half2 r = __hadd2_rn(*reinterpret_cast<const __half2 *>(&word), *reinterpret_cast<const __half2 *>(&both));
        return *reinterpret_cast<const uint32_t *>(&r);
    } else {
        const __nv_bfloat162 r = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162 *>(&word), *reinterpret_cast<const __nv_bfloat162 *>(&both));
        return *reinterpret_cast<const uint32_t *>(&r);
    }
}

// Whether 256 x 256 tiles on pairs of SMs finish in no more rounds than 128 x 256 tiles on single SMs: a round of either
// takes about as long (the pair's a little less), and an odd last row block leaves half of its pairs idle.
inline bool pairs_pay(int64_t tiles, int64_t pair_tiles, int sms) {
    const int64_t pairs = sms / 2 > 0 ? sms / 2 : 1;
    return (pair_tiles + pairs - 1) / pairs <= (tiles + sms - 1) / sms;
}

namespace pair {

// TMA loads whose completion is signalled on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar) : "memory");
}
// Arrive (once, on a barrier of this CTA) when the tcgen05 operations this thread issued for the pair are done.
__device__ __forceinline__ void tc_commit_pair_local(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// `N` columns (a multiple of 16) of the accumulator row of this lane, scaled, converted, a 16-bit bias added, and stored: 16
// columns (32 or 64 bytes) at a time.
template <typename OUT, int N>
__device__ __forceinline__ void store_columns(OUT *dst, const uint32_t *acc, float alpha, const OUT *bias, int64_t left, bool vec32,
                                              bool vec16) {
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        const int64_t here = left - c;
        if (here <= 0) break;
        constexpr int WORDS = 4 * static_cast<int>(sizeof(OUT));
        uint32_t pk[WORDS];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if constexpr (sizeof(OUT) == 2) {
                if (i % 2 == 0) pk[i / 2] = pack_pair<OUT>(alpha * __uint_as_float(acc[c + i]), alpha * __uint_as_float(acc[c + i + 1]));
            } else {
                pk[i] = __float_as_uint(alpha * __uint_as_float(acc[c + i]));
            }
        }
        if constexpr (sizeof(OUT) == 2) {                     // (no entry takes a bias with fp32 output)
            if (bias) {
#pragma unroll
                for (int i = 0; i < 8; ++i) pk[i] = add_bias<OUT>(pk[i], bias + c + 2 * i, here - 2 * i);
            }
        }
        OUT *at = dst + c;
        if (here >= 16 && vec32) {
#pragma unroll
            for (int i = 0; i < WORDS; i += 8) stg_32_stream(reinterpret_cast<uint8_t *>(at) + 4 * i, &pk[i]);
        } else if (here >= 16 && vec16) {
#pragma unroll
            for (int i = 0; i < WORDS; i += 4)
                reinterpret_cast<uint4 *>(at)[i / 4] = make_uint4(pk[i], pk[i + 1], pk[i + 2], pk[i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (i >= here) break;
                if constexpr (sizeof(OUT) == 2)
                    reinterpret_cast<uint16_t *>(at)[i] = static_cast<uint16_t>(pk[i >> 1] >> ((i & 1) * 16));
                else
                    reinterpret_cast<uint32_t *>(at)[i] = pk[i];
            }
        }
    }
}

// Persistent launch of clusters of two CTAs: one pair per `tiles` at most, as many as can be resident, max_ctas CTAs at
// most (0: no limit; never 1, which leaves no room for a pair); a programmatic dependent of the kernel before it in the
// stream (see launch_dependent).
template <auto KERNEL, typename... Args>
int launch(int threads, int smem_bytes, int64_t tiles, int max_ctas, cudaStream_t stream, const Args &...args) {
    static OncePerDevice configured;           // per kernel
    static int resident[64] = {};              // pairs that can be resident at once
    int dev = 0, clusters = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool kept = dev >= 0 && dev < 64;
    FOS_CUDA_TRY(configured.run(dev, [&] {
        cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        int sms = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cfg.gridDim = dim3(static_cast<unsigned>(sms & ~1));
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, KERNEL, &cfg);
        if (e == cudaSuccess && kept) resident[dev] = clusters;
        return e;
    }));
    if (kept) clusters = resident[dev];
    if (clusters < 1) clusters = 1;
    int64_t pairs = tiles < clusters ? tiles : clusters;
    if (max_ctas > 0 && pairs > max_ctas / 2) pairs = max_ctas / 2;
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs));
    cfg.numAttrs = 2;
    FOS_CUDA_TRY(cudaLaunchKernelEx(&cfg, KERNEL, args...));
    return FOS_OK;
}

}  // namespace pair
}  // namespace
}  // namespace fos
