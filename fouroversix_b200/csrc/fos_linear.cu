// A linear layer's forward pass on a packed weight as one host call: amax pass, activation quantization and the FP4 GEMM
// (which forms alpha and adds the bias itself) enqueued from C, the packed activation in a caller-provided workspace.
// What the calls do is in fos_quantize / fos_gemm_alpha / fos_gemm_nvfp4; this entry exists because a layer that is launched call by call
// from an interpreter is bound by the interpreter at decode sizes (16 x 8192 -> 8192: 109 us against 23 us of
// device time).
#include "fos_common.cuh"

namespace fos {
namespace {

struct LinearWorkspace {
    int64_t rows_p, k_p, codes, sf, amax, amax_parts, total;    // byte offsets, multiples of 256
};

LinearWorkspace linear_workspace(int64_t rows, int64_t k) {
    LinearWorkspace w{};
    w.rows_p = round_up64(rows, 128);
    w.k_p = round_up64(k, 64);
    int64_t at = 0;
    auto take = [&](int64_t bytes) { const int64_t here = at; at += round_up64(bytes, 256); return here; };
    w.amax = take(4);
    w.amax_parts = take(4 * AMAX_PARTS_WORDS);
    w.codes = take(w.rows_p * w.k_p / 2);
    w.sf = take(w.rows_p * w.k_p / 16);
    w.total = at;
    return w;
}

}  // namespace
}  // namespace fos

extern "C" int64_t fos_linear_workspace_bytes(int64_t rows, int64_t in_features) {
    if (rows <= 0 || in_features <= 0) return FOS_ERR_INVALID_ARGUMENT;
    return fos::linear_workspace(rows, in_features).total;
}

extern "C" int fos_linear_forward(const void *x, int x_dtype, int64_t rows, int64_t in_features, int64_t ld_x,
                                  int activation_rule, const uint8_t *w_codes, const uint8_t *w_sf, const float *w_amax,
                                  int weight_rule, int64_t out_features, void *out, int out_dtype, int64_t ld_out,
                                  void *workspace, int64_t workspace_bytes, const fos_gemm_opts *opts, int32_t *status,
                                  void *stream) {
    return fos_linear_forward_bias(x, x_dtype, rows, in_features, ld_x, activation_rule, w_codes, w_sf, w_amax, weight_rule,
                                   out_features, nullptr, out, out_dtype, ld_out, workspace, workspace_bytes, opts, status,
                                   stream);
}

extern "C" int fos_linear_forward_bias(const void *x, int x_dtype, int64_t rows, int64_t in_features, int64_t ld_x,
                                       int activation_rule, const uint8_t *w_codes, const uint8_t *w_sf,
                                       const float *w_amax, int weight_rule, int64_t out_features, const void *bias,
                                       void *out, int out_dtype, int64_t ld_out, void *workspace, int64_t workspace_bytes,
                                       const fos_gemm_opts *opts, int32_t *status, void *stream) {
    using namespace fos;
    if (!x || !w_codes || !w_sf || !w_amax || !out || !workspace || rows <= 0 || in_features <= 0 || out_features <= 0)
        return FOS_ERR_INVALID_ARGUMENT;
    if (bias && out_dtype == FOS_FP32) return FOS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return FOS_ERR_MISALIGNED;
    const LinearWorkspace w = linear_workspace(rows, in_features);
    if (workspace_bytes < w.total) return FOS_ERR_INVALID_ARGUMENT;
    uint8_t *base = static_cast<uint8_t *>(workspace);
    float *amax = reinterpret_cast<float *>(base + w.amax);
    const int st = quantize_activation(x, x_dtype, rows, in_features, ld_x, activation_rule, base + w.codes, base + w.sf, amax,
                                       reinterpret_cast<float *>(base + w.amax_parts), stream);
    if (st != FOS_OK) return st;
    const GemmScales scales{amax, w_amax, alpha_divisor(FOS_NVFP4, activation_rule, FOS_NVFP4, weight_rule), bias, true};
    return gemm_nvfp4_chained(base + w.codes, base + w.sf, w_codes, w_sf, scales, out, out_dtype, w.rows_p,
                              round_up64(out_features, 128), w.k_p, rows, out_features, ld_out, opts, status, stream);
}

// ---------------------------------------------------------------------------- a training step
//
// Forward and backward pass with master weights: two and four quantizations around one and two GEMMs. Launched from the
// interpreter call by call (a zeroed word, a maximum pass and a quantization each) the step was bound by the host at every
// size (365 us; 4096^3 382 us). Here each pass is one host call, and its tensors' maxima are one launch; backward,
// dy is read once for its plain and its rotated maximum.

namespace fos {
namespace {

constexpr int64_t TRAIN_WORDS_BYTES = 256;

struct OperandSlot { uint8_t *codes, *sf; };

int64_t operand_bytes(int64_t rows, int64_t cols) {                        // codes, then scales, each a multiple of 256
    const int64_t n = round_up64(rows, 128) * round_up64(cols, 64);
    return round_up64(n / 2, 256) + round_up64(n / 16, 256);
}

OperandSlot operand_slot(uint8_t *base, int64_t rows, int64_t cols) {
    return {base, base + round_up64(round_up64(rows, 128) * round_up64(cols, 64) / 2, 256)};
}

int64_t larger(int64_t a, int64_t b) { return a > b ? a : b; }

bool chain_takes(const void *p, int64_t ld, int64_t cols) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % 8 == 0 && cols % 8 == 0;
}

}  // namespace
}  // namespace fos

extern "C" int64_t fos_linear_train_forward_workspace_bytes(int64_t rows, int64_t in_features, int64_t out_features) {
    using namespace fos;
    if (rows <= 0 || in_features <= 0 || out_features <= 0) return FOS_ERR_INVALID_ARGUMENT;
    return TRAIN_WORDS_BYTES + operand_bytes(rows, in_features) + operand_bytes(out_features, in_features);
}

extern "C" int64_t fos_linear_train_backward_workspace_bytes(int64_t rows, int64_t in_features, int64_t out_features) {
    using namespace fos;
    if (rows <= 0 || in_features <= 0 || out_features <= 0) return FOS_ERR_INVALID_ARGUMENT;
    // a slot for dy and then dy^T, one for W^T and then x^T
    return TRAIN_WORDS_BYTES + larger(operand_bytes(rows, out_features), operand_bytes(out_features, rows)) +
           larger(operand_bytes(in_features, out_features), operand_bytes(in_features, rows));
}

extern "C" int64_t fos_linear_train_workspace_bytes(int64_t rows, int64_t in_features, int64_t out_features) {
    return fos::larger(fos_linear_train_forward_workspace_bytes(rows, in_features, out_features),
                       fos_linear_train_backward_workspace_bytes(rows, in_features, out_features));
}

extern "C" int fos_linear_train_forward(const void *x, const void *w, int dtype, int64_t rows, int64_t in_features, int64_t out_features,
                                        int64_t ld_x, int64_t ld_w, int activation_rule, int weight_rule, int weight_2d, void *out,
                                        int out_dtype, int64_t ld_out, void *workspace, int64_t workspace_bytes, void *stream) {
    using namespace fos;
    if (!x || !w || !out || !workspace || rows <= 0 || in_features <= 0 || out_features <= 0 || ld_x < in_features || ld_w < in_features)
        return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_INVALID_ARGUMENT;
    if (!chain_takes(x, ld_x, in_features) || !chain_takes(w, ld_w, in_features)) return FOS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return FOS_ERR_MISALIGNED;
    if (workspace_bytes < fos_linear_train_forward_workspace_bytes(rows, in_features, out_features)) return FOS_ERR_INVALID_ARGUMENT;
    int st = check_device();
    if (st != FOS_OK) return st;
    uint8_t *base = static_cast<uint8_t *>(workspace) + TRAIN_WORDS_BYTES;
    float *amax = static_cast<float *>(workspace);                          // x, W
    const OperandSlot a = operand_slot(base, rows, in_features),
                      b = operand_slot(base + operand_bytes(rows, in_features), out_features, in_features);
    const AmaxJob jobs[2] = {{x, rows, in_features, ld_x, amax, nullptr}, {w, out_features, in_features, ld_w, amax + 1, nullptr}};
    if ((st = amax_of_tensors(jobs, 2, dtype, amax, 2, stream)) != FOS_OK) return st;
    if ((st = quantize_in_chain(w, dtype, out_features, in_features, ld_w, weight_rule, weight_2d, 0, 0, 0, 0, amax + 1, b.codes, b.sf, stream)) != FOS_OK)
        return st;
    if ((st = quantize_in_chain(x, dtype, rows, in_features, ld_x, activation_rule, 0, 0, 0, 0, 0, amax, a.codes, a.sf, stream)) != FOS_OK)
        return st;
    const GemmScales scales{amax, amax + 1, alpha_divisor(FOS_NVFP4, activation_rule, FOS_NVFP4, weight_rule), nullptr, false};
    return gemm_nvfp4_chained(a.codes, a.sf, b.codes, b.sf, scales, out, out_dtype, round_up64(rows, 128), round_up64(out_features, 128),
                              round_up64(in_features, 64), rows, out_features, ld_out, nullptr, nullptr, stream);
}

extern "C" int fos_linear_train_backward(const void *dy, const void *x, const void *w, int dtype, int64_t rows, int64_t in_features,
                                         int64_t out_features, int64_t ld_dy, int64_t ld_x, int64_t ld_w, int gradient_rule,
                                         int gradient_rounding, uint64_t seed_dgrad, uint64_t seed_wgrad, int activation_rule,
                                         int weight_rule, int weight_2d, void *dx, void *dw, int out_dtype, int64_t ld_dx,
                                         int64_t ld_dw, void *workspace, int64_t workspace_bytes, void *stream) {
    using namespace fos;
    if (!dy || !x || !w || !dx || !dw || !workspace || rows <= 0 || in_features <= 0 || out_features <= 0 || ld_dy < out_features ||
        ld_x < in_features || ld_w < in_features || gradient_rounding < 0 || gradient_rounding > 2)
        return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_INVALID_ARGUMENT;
    if (rows % 16 != 0) return FOS_ERR_UNSUPPORTED;                         // the rotation takes 16 tokens at a time
    if (!chain_takes(dy, ld_dy, out_features) || !chain_takes(x, ld_x, in_features) || !chain_takes(w, ld_w, in_features))
        return FOS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return FOS_ERR_MISALIGNED;
    if (workspace_bytes < fos_linear_train_backward_workspace_bytes(rows, in_features, out_features)) return FOS_ERR_INVALID_ARGUMENT;
    int st = check_device();
    if (st != FOS_OK) return st;
    uint8_t *left = static_cast<uint8_t *>(workspace) + TRAIN_WORDS_BYTES;
    uint8_t *right = left + larger(operand_bytes(rows, out_features), operand_bytes(out_features, rows));
    float *amax = static_cast<float *>(workspace);                          // W, dy, dy^T rotated, x^T rotated
    const AmaxJob jobs[3] = {{w, out_features, in_features, ld_w, amax, nullptr},
                             {dy, rows, out_features, ld_dy, amax + 1, amax + 2},
                             {x, rows, in_features, ld_x, nullptr, amax + 3}};
    if ((st = amax_of_tensors(jobs, 3, dtype, amax, 4, stream)) != FOS_OK) return st;
    const int noisy = gradient_rounding != 0, unbiased = gradient_rounding == 2, noise_flags = unbiased ? FOS_QUANTIZE_UNBIASED : 0;
    const int64_t rows_p = round_up64(rows, 128), in_p = round_up64(in_features, 128), out_p = round_up64(out_features, 128);

    // dx[rows, in] = Q(dy) @ Q(W^T)^T
    OperandSlot a = operand_slot(left, rows, out_features), b = operand_slot(right, in_features, out_features);
    if ((st = quantize_in_chain(w, dtype, out_features, in_features, ld_w, weight_rule, weight_2d, 1, 0, 0, 0, amax, b.codes, b.sf, stream)) != FOS_OK)
        return st;
    if ((st = quantize_in_chain(dy, dtype, rows, out_features, ld_dy, gradient_rule, 0, 0, noise_flags, noisy, seed_dgrad, amax + 1, a.codes, a.sf,
                                stream)) != FOS_OK)
        return st;
    const GemmScales dgrad{amax + 1, amax, alpha_divisor(FOS_NVFP4, gradient_rule, FOS_NVFP4, weight_rule, unbiased, 0), nullptr, false};
    if ((st = gemm_nvfp4_chained(a.codes, a.sf, b.codes, b.sf, dgrad, dx, out_dtype, rows_p, in_p, round_up64(out_features, 64), rows,
                                 in_features, ld_dx, nullptr, nullptr, stream)) != FOS_OK)
        return st;

    // dW[out, in] = Q(rot(dy^T)) @ Q(rot(x^T))^T, rotated along the tokens; the slots are free once that product is done,
    // which the quantize kernels wait for
    a = operand_slot(left, out_features, rows);
    b = operand_slot(right, in_features, rows);
    if ((st = quantize_in_chain(x, dtype, rows, in_features, ld_x, activation_rule, 0, 1, FOS_QUANTIZE_RHT, 0, 0, amax + 3, b.codes, b.sf, stream)) != FOS_OK)
        return st;
    if ((st = quantize_in_chain(dy, dtype, rows, out_features, ld_dy, gradient_rule, 0, 1, FOS_QUANTIZE_RHT | noise_flags, noisy, seed_wgrad, amax + 2,
                                a.codes, a.sf, stream)) != FOS_OK)
        return st;
    const GemmScales wgrad{amax + 2, amax + 3, alpha_divisor(FOS_NVFP4, gradient_rule, FOS_NVFP4, activation_rule, unbiased, 0), nullptr, false};
    return gemm_nvfp4_chained(a.codes, a.sf, b.codes, b.sf, wgrad, dw, out_dtype, out_p, in_p, round_up64(rows, 64), out_features, in_features,
                              ld_dw, nullptr, nullptr, stream);
}
