// FP4 GEMM for at most 32 tokens (decoding; which problems: pays()): D[t, f] = alpha * sum_k X[t, k] * W[f, k] (+ bias[f]).
//
// What bounds it is the weight's way out of HBM, so the weight is the M operand (128 rows of a tile, nothing of it
// padding) and the tokens are the N operand (16 or 32 columns): per stage a CTA fetches 16 KB of weight, 2 KB of its
// scales and 4 to 6 KB for the tokens, where the general kernel would fetch and multiply a 128-row tile of padding
// for 16 tokens. Two CTAs per SM keep about 200 KB of loads in flight.
// A projection has few 128-row tiles (64 at 8192 features), so K is split over the S CTAs of a cluster, which add up
// their partial sums through distributed shared memory in the order of K: no atomics, no workspace, the same bits
// every time. S = 1 when K is short (every CTA keeps at least MIN_STAGES stages; see split_for).
// Launched as the programmatic dependent of the kernel that packs the tokens, the CTAs fetch their first
// stages of weight while that kernel still runs, and wait for it before they touch anything it writes.
//
//   warp 0     TMA producer              warp 1   scale copies and MMAs (in issue order: see the CTA-pair kernel)
//   warps 2-5  epilogue: 128 lanes = 128 features
#pragma once

#include "fos_fp4_mma.cuh"

namespace fos {
namespace {
namespace skinny {

constexpr int THREADS = 192;
constexpr int MIN_STAGES = 8;             // of a CTA, before K is split further
constexpr int MAX_SPLIT = 8;
constexpr int MAX_TOKENS = 32;

struct Params {
    const float *alpha;                   // the product's factor, or nullptr:
    const float *amax_a, *amax_b;         // then it is amax_a * amax_b / denom, 1 without amax_a
    float denom;
    const void *bias;                     // [n] of the output's type, or nullptr
    void *d;
    int32_t *status;
    int k_blocks;                         // of 64 values
    int m, n, split;
    int64_t ldd;
};

template <int N, bool MX> struct Cfg {
    static constexpr int TILES = MX ? KB_PER_STAGE / 2 : KB_PER_STAGE;    // 512-byte scale tiles of a stage per operand
    static constexpr int W_BYTES = 128 * BLOCK_K_BYTES, X_BYTES = N * BLOCK_K_BYTES, SF_BYTES = TILES * SF_TILE_BYTES;
    static constexpr int OPERAND_BYTES = W_BYTES + X_BYTES;
    static constexpr int STAGE_BYTES = OPERAND_BYTES + 2 * SF_BYTES;
    static constexpr int STAGES = N <= 16 ? 5 : 4;
    static constexpr int ACC_COLS = 32;
    static constexpr int SF_COLS = 2 * 4 * KB_PER_STAGE;                  // of a slot: weight scales, token scales
    static constexpr int TMEM = 128;
    static constexpr int BARRIER_BYTES = 128;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + BARRIER_BYTES;
    static_assert(N <= ACC_COLS && ACC_COLS + 2 * SF_COLS <= TMEM, "tensor memory");
    static_assert(2 * (SMEM_BYTES + 1024) <= 233472, "two CTAs per SM");
    static_assert(STAGES * OPERAND_BYTES >= N * 512, "the partial sums reuse the operand ring");
    static_assert(OPERAND_BYTES % 1024 == 0 && X_BYTES % 1024 == 0, "swizzle alignment");
    static_assert((2 * STAGES + 2) * 8 + 8 <= BARRIER_BYTES, "barrier area too small");
};

__device__ __forceinline__ void st_cluster_f32(uint32_t cluster_addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

template <typename OUT> __device__ __forceinline__ OUT to_out(float v) {
    if constexpr (std::is_same<OUT, __half>::value) return __float2half_rn(v);
    else if constexpr (std::is_same<OUT, __nv_bfloat16>::value) return __float2bfloat16_rn(v);
    else return v;
}

template <int N, typename OUT, bool MX>
__global__ void __launch_bounds__(THREADS, 2)
gemm_fp4_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                       const __grid_constant__ CUtensorMap map_wsf, const __grid_constant__ CUtensorMap map_xsf,
                       const Params p) {
    using C = Cfg<N, MX>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t sf_base = smem_base + C::STAGES * C::OPERAND_BYTES;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_gen + C::STAGES * C::STAGE_BYTES);
    const uint32_t full_bar = smem_u32(bars), empty_bar = full_bar + 8 * C::STAGES, acc_bar = empty_bar + 8 * C::STAGES,
                   drain_bar = acc_bar + 8;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * C::STAGES + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full_bar + 8 * s, 1);
            mbar_init(empty_bar + 8 * s, 1);
        }
        mbar_init(acc_bar, 1);
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // this CTA's tile of 128 features and its share of K
    const int split = p.split, tile = static_cast<int>(blockIdx.x) / split, part = static_cast<int>(blockIdx.x) % split;
    const int k_tiles = (p.k_blocks + KB_PER_STAGE - 1) / KB_PER_STAGE;
    const int kt0 = static_cast<int>(static_cast<int64_t>(k_tiles) * part / split);
    const int kt1 = static_cast<int>(static_cast<int64_t>(k_tiles) * (part + 1) / split);

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        const bool issue = elect_one();
        auto load_weight = [&](int s, int kt) {
            if (!issue) return;
            const uint32_t bar = full_bar + 8 * s;
            mbar_expect_tx(bar, C::STAGE_BYTES);
            tma_load_2d(smem_base + s * C::OPERAND_BYTES, &map_w, kt * BLOCK_K_BYTES, tile * 128, bar);
            tma_load_3d(sf_base + s * 2 * C::SF_BYTES, &map_wsf, 0, kt * C::TILES, tile, bar);
        };
        auto load_tokens = [&](int s, int kt) {
            if (!issue) return;
            const uint32_t bar = full_bar + 8 * s;
            tma_load_2d(smem_base + s * C::OPERAND_BYTES + C::W_BYTES, &map_x, kt * BLOCK_K_BYTES, 0, bar);
            tma_load_3d(sf_base + s * 2 * C::SF_BYTES + C::SF_BYTES, &map_xsf, 0, kt * C::TILES, 0, bar);
        };
        const int ahead = kt1 - kt0 < C::STAGES ? kt1 - kt0 : C::STAGES;
        for (int i = 0; i < ahead; ++i) load_weight(i, kt0 + i);
        asm volatile("griddepcontrol.wait;" ::: "memory");       // the packed tokens are there
        for (int i = 0; i < ahead; ++i) load_tokens(i, kt0 + i);
        __syncwarp();
        bool ok = true;
        int s = 0;
        uint32_t ph = 0;
        for (int kt = kt0 + ahead; kt < kt1; ++kt) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * s, ph, abort_flag, p.status, 1));
            if (!ok) break;
            load_weight(s, kt);
            load_tokens(s, kt);
            __syncwarp();
            if (++s == C::STAGES) { s = 0; ph ^= 1u; }
        }
        if (!ok) {
            const unsigned long long t0 = global_timer_ns();
            while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ scale copies and MMAs
        const bool issue = elect_one();
        const uint32_t idesc = mma_idesc(N);
        int s = 0;
        uint32_t ph = 0, slot = 0;
        bool ok = true;
        for (int kt = kt0; kt < kt1; ++kt) {
            ok = __all_sync(0xffffffffu, mbar_wait(full_bar + 8 * s, ph, abort_flag, p.status, 2));
            if (!ok) break;
            // (no tcgen05 fence: what was waited for are TMA copies; see the CTA-pair kernel)
            const int left = p.k_blocks - kt * KB_PER_STAGE, nkb = left < KB_PER_STAGE ? left : KB_PER_STAGE;
            const uint32_t stage = smem_base + s * C::OPERAND_BYTES;
            const uint32_t w_lo = desc_lo(stage, 16), x_lo = desc_lo(stage + C::W_BYTES, 16), sf_lo = desc_lo(sf_base + s * 2 * C::SF_BYTES);
            const uint32_t sfw = tmem_base + C::ACC_COLS + slot * C::SF_COLS, sfx = sfw + 4 * KB_PER_STAGE;
            if (issue) {
#pragma unroll
                for (int kb = 0; kb < C::TILES; ++kb) {
                    tc_copy_sf_lo(sfw + 4 * kb, sf_lo + ((kb * SF_TILE_BYTES) >> 4));
                    tc_copy_sf_lo(sfx + 4 * kb, sf_lo + ((C::SF_BYTES + kb * SF_TILE_BYTES) >> 4));
                }
#pragma unroll
                for (int kb = 0; kb < KB_PER_STAGE; ++kb) {
                    if (kb >= nkb) break;
                    const uint32_t accumulate = (kt > kt0 || kb > 0) ? 1u : 0u;
                    if constexpr (MX)
                        tc_mma_mxf4_lo(tmem_base, w_lo + 2 * kb, x_lo + 2 * kb, mma_idesc_mx(idesc, (kb & 1) * 2),
                                       sfw + 4 * (kb >> 1), sfx + 4 * (kb >> 1), accumulate);
                    else
                        tc_mma_nvf4_lo(tmem_base, w_lo + 2 * kb, x_lo + 2 * kb, idesc, sfw + 4 * kb, sfx + 4 * kb, accumulate);
                }
                tc_commit(empty_bar + 8 * s);
            }
            __syncwarp();
            if (++s == C::STAGES) { s = 0; ph ^= 1u; }
            slot ^= 1u;
        }
        if (ok) {
            if (issue) tc_commit(acc_bar);
        } else {
            // giving up: the MMAs already issued must have finished before tensor memory is released
            if (issue) tc_commit(drain_bar);
            __syncwarp();
            const long long t0 = clock64();
            while (!mbar_try_wait(drain_bar, 0) && clock64() - t0 < 20000000ll) {}   // about 10 ms
        }
    }

    // ---------------------------------------------------------------------- epilogue
    const int quad = warp & 3, feature = quad * 32 + lane;            // (warps 2..5 own quadrants 2, 3, 0, 1)
    const int n_part = N / split;                                     // token columns this CTA adds up and stores
    const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    bool ok = true;
    __syncwarp();
    if (warp >= 2) {
        asm volatile("griddepcontrol.wait;" ::: "memory");            // amax_a, and nobody reads d any more
        ok = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0, abort_flag, p.status, 4));
        tc_fence_after();
    }
    if (split > 1) {
        cluster_sync_all();       // every CTA's MMAs are done: its operand ring may take partial sums
        if (warp >= 2 && ok) {
#pragma unroll 1
            for (int c = 0; c < N; c += 16) {
                uint32_t v[16];
                tc_load_16cols_sync(t_acc + c, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int col = c + i, owner = col / n_part;
                    const uint32_t slab = smem_base + ((part * n_part + col - owner * n_part) * 128 + feature) * 4;
                    st_cluster_f32(map_to_cta(slab, owner), __uint_as_float(v[i]));
                }
            }
        }
        cluster_sync_all();       // all partial sums have arrived
    }
    if (warp >= 2 && ok) {
        const float alpha = p.alpha ? ld_float(p.alpha)
                            : !p.amax_a ? 1.0f
                                        : __fdiv_rn(__fmul_rn(ld_float(p.amax_a), ld_float(p.amax_b)), p.denom);
        const int f = tile * 128 + feature;
        const bool f_ok = f < p.n;
        const OUT *bias = static_cast<const OUT *>(p.bias);
        float b = 0.0f;
        if constexpr (sizeof(OUT) == 2) {                     // (no entry takes a bias with fp32 output)
            if (bias && f_ok) b = elem_to_float<OUT>(bias[f]);
        }
        OUT *out = static_cast<OUT *>(p.d) + f;
        const int t0 = split > 1 ? part * n_part : 0;
        auto put = [&](int c, float sum) {
            const int t = t0 + c;
            if (!f_ok || t >= p.m) return;
            OUT v = to_out<OUT>(alpha * sum);
            if constexpr (sizeof(OUT) == 2) {
                // the bias is added to the value rounded to the output's type, as a separate addition would
                if (bias) v = to_out<OUT>(elem_to_float<OUT>(v) + b);
            }
            out[t * p.ldd] = v;
        };
        if (split > 1) {
            for (int c = 0; c < n_part; ++c) {
                float sum = lds_f32(smem_base + (c * 128 + feature) * 4);
                for (int r = 1; r < split; ++r) sum += lds_f32(smem_base + ((r * n_part + c) * 128 + feature) * 4);
                put(c, sum);
            }
        } else {
#pragma unroll 1
            for (int c = 0; c < N; c += 16) {
                uint32_t v[16];
                tc_load_16cols_sync(t_acc + c, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) put(c + i, __uint_as_float(v[i]));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM) : "memory");
    }
}

// How many CTAs share a tile's K: the largest power of two that fills at most the CTAs resident at once (two per SM)
// and leaves each CTA MIN_STAGES stages.
inline int split_for(int64_t tiles, int k_tiles, int sms) {
    int split = 1;
    while (split < MAX_SPLIT && tiles * split * 2 <= 2 * sms && k_tiles / (split * 2) >= MIN_STAGES) split *= 2;
    return split;
}

// Where the kernel is taken (measured against the 128 x 128 tiles of the single-CTA kernel, in a graph, us): K split over a
// cluster, 16 x 8192 -> 8192 11.5 / 13.0, 8 x 4096 -> 2048 7.1 / 7.5, 32 x 14336 -> 4096 12.5 / 19.4, but with 32 tokens the
// exchange of the partial sums wants a long K (32 x 8192 -> 8192 12.3 / 13.0; 32 x 4096 -> 4096 8.7 / 7.8); or more tiles than
// SMs, 32 x 4096 -> 28672 14.9 / 15.6. Short K without a split: 24 x 2880 -> 2880 7.7 / 6.8, not taken.
inline bool pays(int64_t m, int64_t n_p, int64_t k_p, int sms) {
    const int k_tiles = static_cast<int>((k_p / 64 + KB_PER_STAGE - 1) / KB_PER_STAGE);
    const int64_t tiles = n_p / 128;
    return m <= MAX_TOKENS && tiles <= INT32_MAX / MAX_SPLIT &&
           (tiles >= sms || (split_for(tiles, k_tiles, sms) > 1 && (m <= 16 || k_tiles >= 32)));
}

template <int N, typename OUT, bool MX>
int launch(const CUtensorMap &mw, const CUtensorMap &mx, const CUtensorMap &mws, const CUtensorMap &mxs, const Params &p,
           int64_t tiles, bool dependent, cudaStream_t stream) {
    auto kernel = gemm_fp4_skinny_kernel<N, OUT, MX>;
    static OncePerDevice configured;   // per instantiation
    int dev = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    FOS_CUDA_TRY(configured.run(dev, [&] {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<N, MX>::SMEM_BYTES);
    }));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * p.split));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = Cfg<N, MX>::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(p.split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 2 : 1;
    FOS_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, mw, mx, mws, mxs, p));
    return FOS_OK;
}

template <int N, bool MX>
int launch_out(const CUtensorMap &mw, const CUtensorMap &mx, const CUtensorMap &mws, const CUtensorMap &mxs, const Params &p,
               int out_dtype, int64_t tiles, bool dependent, cudaStream_t stream) {
    if (out_dtype == FOS_BF16) return launch<N, __nv_bfloat16, MX>(mw, mx, mws, mxs, p, tiles, dependent, stream);
    if (out_dtype == FOS_FP16) return launch<N, __half, MX>(mw, mx, mws, mxs, p, tiles, dependent, stream);
    return launch<N, float, MX>(mw, mx, mws, mxs, p, tiles, dependent, stream);
}

template <bool MX>
int launch_n(const uint8_t *x_codes, const uint8_t *x_sf, const uint8_t *w_codes, const uint8_t *w_sf, Params p, int out_dtype,
             int64_t m_p, int64_t n_p, int64_t k_p, int sms, bool dependent, cudaStream_t stream) {
    const int tiles_k = static_cast<int>(MX ? k_p / 128 : k_p / 64);      // 512-byte scale tiles along K
    const int width = p.m <= 16 ? 16 : 32;
    p.k_blocks = static_cast<int>(k_p / 64);
    p.split = split_for(n_p / 128, (p.k_blocks + KB_PER_STAGE - 1) / KB_PER_STAGE, sms);
    constexpr int BOX = MX ? KB_PER_STAGE / 2 : KB_PER_STAGE;
    CUtensorMap mw, mx, mws, mxs;
    int st;
    if ((st = make_operand_map(&mw, w_codes, n_p, k_p / 2, 128)) != FOS_OK) return st;
    if ((st = make_operand_map(&mx, x_codes, m_p, k_p / 2, width)) != FOS_OK) return st;
    if ((st = make_scale_map(&mws, w_sf, n_p / 128, tiles_k, 1, BOX)) != FOS_OK) return st;
    if ((st = make_scale_map(&mxs, x_sf, m_p / 128, tiles_k, 1, BOX)) != FOS_OK) return st;
    const int64_t tiles = n_p / 128;
    if (width == 16) return launch_out<16, MX>(mw, mx, mws, mxs, p, out_dtype, tiles, dependent, stream);
    return launch_out<32, MX>(mw, mx, mws, mxs, p, out_dtype, tiles, dependent, stream);
}

}  // namespace skinny
}  // namespace
}  // namespace fos
