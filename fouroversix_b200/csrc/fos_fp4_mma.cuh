// Block-scaled FP4 MMA building blocks shared by the FP4 GEMM kernels: tcgen05.mma and tcgen05.cp wrappers, descriptors,
// the tensor map of the scale tiles (sm_100a).
#pragma once

#include "fos_tcgen05.cuh"

namespace fos {
namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K_BYTES = 128;                 // 256 E2M1 values: one 128-byte swizzle row
constexpr int KB_PER_STAGE = 4;                    // MMA K-blocks (64 values, 32 bytes) per stage
constexpr int SF_TILE_BYTES = 512;                 // scales of 128 rows x 64 values

// ---------------------------------------------------------------------------- MMA wrappers

// Descriptors in two halves. The upper word of a shared-memory matrix descriptor is the same for every
// tile of a kind (stride byte offset, version, swizzle) and the lower word is the start address >> 4
// (shared-memory addresses stay below 2^18, so adding a byte offset >> 4 never carries out of the field):
// the issuing threads keep one lower word per stage and add constants, instead of rebuilding 64-bit
// descriptors for every instruction - a single thread issues every copy and every MMA of an SM, and
// what it executes between two of them is what bounds its rate.
constexpr uint32_t DESC_HI_OPERAND = (1024u >> 4) | (1u << 14) | (2u << 29);   // SBO 1024, version 1, 128-byte swizzle
constexpr uint32_t DESC_HI_SCALES = (128u >> 4) | (1u << 14);                   // SBO 128, version 1, no swizzle
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo_bytes = 0) {
    return ((addr & 0x3ffffu) >> 4) | ((lbo_bytes >> 4) << 16);
}
__device__ __forceinline__ void tc_copy_sf_lo(uint32_t taddr, uint32_t lo) {
    asm volatile("{ .reg .b64 d;\n"
                 "mov.b64 d, {%1, %2};\n"
                 "tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d; }" ::"r"(taddr), "r"(lo), "r"(DESC_HI_SCALES) : "memory");
}
__device__ __forceinline__ void tc_copy_sf_pair_lo(uint32_t taddr, uint32_t lo) {
    asm volatile("{ .reg .b64 d;\n"
                 "mov.b64 d, {%1, %2};\n"
                 "tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], d; }" ::"r"(taddr), "r"(lo), "r"(DESC_HI_SCALES) : "memory");
}
__device__ __forceinline__ void tc_mma_nvf4_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                               uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %7};\n"
        "mov.b64 db, {%2, %7};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %3, [%5], [%6], p; }\n"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem), "r"(DESC_HI_OPERAND)
        : "memory");
}
__device__ __forceinline__ void tc_mma_nvf4_pair_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                                    uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %7};\n"
        "mov.b64 db, {%2, %7};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %3, [%5], [%6], p; }\n"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem), "r"(DESC_HI_OPERAND)
        : "memory");
}

// MXFP4: two E8M0 scales per row and K-block (scale_vec::2X); which two of the four bytes of a
// scale column an instruction uses is part of its descriptor.
__device__ __forceinline__ void tc_mma_mxf4_pair_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                                    uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %7};\n"
        "mov.b64 db, {%2, %7};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], da, db, %3, [%5], [%6], p; }\n"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem), "r"(DESC_HI_OPERAND)
        : "memory");
}

__device__ __forceinline__ void tc_mma_mxf4_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                               uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %7};\n"
        "mov.b64 db, {%2, %7};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], da, db, %3, [%5], [%6], p; }\n"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem), "r"(DESC_HI_OPERAND)
        : "memory");
}

// Instruction descriptor of kind::mxf4nvf4 block-scaled MMA: A and B E2M1 (code 1 in bits
// [7,10) and [10,13)), both K-major, N >> 3 in [17,23), UE4M3 scales (bit 23 = 0), M >> 4 in
// [24,29), scale-factor byte ids 0, dense K = 64. MXFP4: E8M0 scales (bit 23 = 1) and the byte
// offset (0 or 2) of the instruction's two scales inside the 32-bit scale column in [4,6) for B
// and [29,31) for A.
__device__ __forceinline__ uint32_t mma_idesc(int n, int m = BLOCK_M) {
    return (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
__device__ __forceinline__ uint32_t mma_idesc_mx(uint32_t idesc, uint32_t sf_byte) {
    return idesc | (1u << 23) | (sf_byte << 4) | (sf_byte << 29);
}

// Scale tiles as a 3-D tensor [row groups][tiles along K][512 bytes]; box = `groups` x the tiles of one stage
// (four; two for MXFP4, whose tiles span two K-blocks).
int make_scale_map(CUtensorMap *map, const uint8_t *sf, int64_t row_groups, int64_t k_blocks, int groups,
                   int tiles_per_stage = KB_PER_STAGE) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return FOS_ERR_CUDA;
    cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(k_blocks), static_cast<cuuint64_t>(row_groups)};
    cuuint64_t strides[2] = {512, static_cast<cuuint64_t>(k_blocks) * 512};
    cuuint32_t box[3] = {128, static_cast<cuuint32_t>(tiles_per_stage), static_cast<cuuint32_t>(groups)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint8_t *>(sf), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? FOS_OK : FOS_ERR_CUDA;
}

}  // namespace
}  // namespace fos
