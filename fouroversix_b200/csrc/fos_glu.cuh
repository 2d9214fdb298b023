// The clamped SwiGLU of a mixture-of-experts layer on 16-bit numbers, every rounding of the reference's chain of tensor
// operations kept (src/fouroversix/model/modules/gpt_oss.py:297-335): used by the kernel that runs it on its own and by the
// epilogue of the grouped gate-up GEMM.
#pragma once

#include "fos_common.cuh"

namespace fos {
namespace {

template <typename T> struct Half16;
template <> struct Half16<__nv_bfloat16> {
    using Pair = __nv_bfloat162;
    static __device__ __forceinline__ float lo(uint32_t w) { return __uint_as_float(w << 16); }
    static __device__ __forceinline__ float hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
    static __device__ __forceinline__ float r16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
    static __device__ __forceinline__ uint32_t pack(float lo_v, float hi_v) {   // round and pack
        Pair p = __floats2bfloat162_rn(lo_v, hi_v);
        return *reinterpret_cast<uint32_t *>(&p);
    }
};
template <> struct Half16<__half> {
    using Pair = __half2;
    static __device__ __forceinline__ float lo(uint32_t w) { return __half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu))); }
    static __device__ __forceinline__ float hi(uint32_t w) { return __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16))); }
    static __device__ __forceinline__ float r16(float v) { return __half2float(__float2half_rn(v)); }
    static __device__ __forceinline__ uint32_t pack(float lo_v, float hi_v) {
        Pair p = __floats2half2_rn(lo_v, hi_v);
        return *reinterpret_cast<uint32_t *>(&p);
    }
};
template <typename P> __device__ __forceinline__ P as_pair(uint32_t w) { return *reinterpret_cast<P *>(&w); }
template <typename P> __device__ __forceinline__ uint32_t as_word(P p) { return *reinterpret_cast<uint32_t *>(&p); }

// max |value| of the eight 16-bit numbers of a 16-byte piece, folded into a running packed maximum
// (NaNs are skipped, as fmaxf skips them in the amax pass of the quantization).
template <typename P> __device__ __forceinline__ P fold_abs_max(P m, uint4 v) {
    m = __hmax2(m, __habs2(as_pair<P>(v.x)));
    m = __hmax2(m, __habs2(as_pair<P>(v.y)));
    m = __hmax2(m, __habs2(as_pair<P>(v.z)));
    return __hmax2(m, __habs2(as_pair<P>(v.w)));
}

// The warp's maximum of the lanes' packed running maxima, raised into amax[0] (a non-negative float, zeroed by the
// caller before the launch, compared as an integer). The words written are the ones the grouped amax pass would
// write: the largest magnitude of the group's values, exactly, as a float. Called by all lanes of the warp.
template <typename T>
__device__ __forceinline__ void raise_amax(typename Half16<T>::Pair m2, float *amax, int lane) {
    using H = Half16<T>;
    float m = fmaxf(H::lo(as_word(m2)), H::hi(as_word(m2)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    // (a stale smaller value read here only costs an atomic that changes nothing)
    if (lane == 0 && m > 0.0f && m > *reinterpret_cast<volatile float *>(amax)) atomicMax(reinterpret_cast<int *>(amax), __float_as_int(m));
}

// 1 / (1 + expf(-t)) of two numbers, rounded to the 16-bit type (a packed pair). The fast functions give the quotient to
// within (12 + 1.5 |t|) units of 2^-23 for |t| <= 64 (__expf: 2 + 1.173 |t| units in the last place by CUDA's own bound, the
// addition and __fdividef 3, and the binary32 sequence itself is within 4 of the true value); where both ends of that
// interval round to the same number, the binary32 sequence does too. The rest - a value within the interval of a
// rounding boundary (one in 500 in bf16, one in 60 in fp16), a large |t| - runs the sequence itself; NaN gives NaN either way.
template <typename T> __device__ __noinline__ uint32_t sigmoid16x2_sequence(float t0, float t1) {
    return Half16<T>::pack(1.0f / (1.0f + expf(-t0)), 1.0f / (1.0f + expf(-t1)));
}
// (`sure`: the result is the sequence's. The callers take the fast path of several pairs before they look: with a branch per
// pair the chains of one warp, some 300 cycles each, ran one after the other.)
template <typename T> __device__ __forceinline__ uint32_t sigmoid16x2(float t0, float t1, bool &sure) {
    using H = Half16<T>;
    const float s0 = __fdividef(1.0f, 1.0f + __expf(-t0)), s1 = __fdividef(1.0f, 1.0f + __expf(-t1));
    const float w0 = s0 * fmaf(fabsf(t0), 0x1.8p-23f, 0x1.8p-20f), w1 = s1 * fmaf(fabsf(t1), 0x1.8p-23f, 0x1.8p-20f);
    const uint32_t low = H::pack(s0 - w0, s1 - w1), high = H::pack(s0 + w0, s1 + w1);
    sure = low == high && fmaxf(fabsf(t0), fabsf(t1)) <= 64.0f;
    return low;
}

// The reference's chain on eight (gate, up) pairs, two to a word of the output, every intermediate rounded to the 16-bit type:
//   g = gate + bias_g; u = up + bias_u; g = min(g, limit); u = min(max(u, -limit), limit)   (NaN passes through)
//   out = (u + 1) * (g * sigmoid(g * alpha))
// A (gate, up) pair is one 32-bit word, and a packed 16-bit addition, multiplication or fused multiply-add
// rounds once from the exact result, which is what "compute in binary32, round to the type" gives for sums and
// products of 16-bit numbers (their exact value fits binary32, or lies so far from a rounding boundary of the
// 16-bit type that the first rounding cannot move it across). Only g * alpha (alpha is a binary32 number) and
// the sigmoid run in binary32. The _rn forms of the packed operations keep the compiler from contracting a
// multiplication and the addition after it into one fused operation, which would drop a rounding. limit2 = (r, r), floor2 = (-inf, -r) with r the limit rounded to the type:
// comparing with r selects the same values as comparing with the limit itself, because no number of the type
// lies between the two.
template <typename T>
__device__ __forceinline__ uint4 glu_words(const uint32_t (&gate_up)[8], const uint32_t (&bias)[8], float alpha,
                                           typename Half16<T>::Pair limit2, typename Half16<T>::Pair floor2,
                                           typename Half16<T>::Pair one2) {
    using H = Half16<T>;
    using P = typename H::Pair;
    uint32_t g2[4], u2[4], t2[4], s2[4], o[4];
    bool all_sure = true;
    bool sure[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        P v0 = __hadd2_rn(as_pair<P>(gate_up[2 * i]), as_pair<P>(bias[2 * i]));
        P v1 = __hadd2_rn(as_pair<P>(gate_up[2 * i + 1]), as_pair<P>(bias[2 * i + 1]));
        v0 = __hmax2_nan(__hmin2_nan(v0, limit2), floor2);
        v1 = __hmax2_nan(__hmin2_nan(v1, limit2), floor2);
        g2[i] = __byte_perm(as_word(v0), as_word(v1), 0x5410);
        u2[i] = __byte_perm(as_word(v0), as_word(v1), 0x7632);
        t2[i] = H::pack(H::lo(g2[i]) * alpha, H::hi(g2[i]) * alpha);
        s2[i] = sigmoid16x2<T>(H::lo(t2[i]), H::hi(t2[i]), sure[i]);
        all_sure = all_sure && sure[i];
    }
    if (!all_sure) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (!sure[i]) s2[i] = sigmoid16x2_sequence<T>(H::lo(t2[i]), H::hi(t2[i]));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        o[i] = as_word(__hmul2_rn(__hadd2_rn(as_pair<P>(u2[i]), one2), __hmul2_rn(as_pair<P>(g2[i]), as_pair<P>(s2[i]))));
    return make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace
}  // namespace fos
