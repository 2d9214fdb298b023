// Block-scaled NVFP4 GEMM for sm_100a: D[m, n] = alpha * sum_k A[m, k] * B[n, k].
//
// Both operands are K-major packed E2M1 with one UE4M3 scale per 16 values, stored as
// fos_quantize writes them (scales in 128-row x 4-block tiles of 512 bytes). The kernel
// is persistent (one CTA per SM, static tile schedule) and warp specialised. Every role that
// issues TMA or tcgen05 instructions runs as a WHOLE warp with one elected lane issuing: with
// every value of its loop the same in all lanes the compiler keeps addresses and descriptors in
// uniform registers, which those instructions take directly; a lone thread's values live in
// ordinary registers and each instruction pays for moving its operands over (the single change
// from "one thread" to "one warp, one elected lane" took 8192^3 from 256 to 235 us, and the MMA
// rate of the CTA-pair kernel from 182 to 152 us).
//
//   warp 0      TMA loads: per stage the A / B tiles (128-byte swizzle, no multicast) into a ring of
//               shared-memory stages guarded by full / empty mbarriers, and - one stage AHEAD of
//               them, because their way into the MMA is longer - the two tensor copies of the
//               scale tiles into a ring of their own that is one slot longer
//   warp 1      allocates tensor memory; issues tcgen05.mma kind::mxf4nvf4.block_scale
//               (K = 64 per instruction) with the fp32 accumulator in tensor memory;
//               tcgen05.commit releases the stage
//   warps 2..9  epilogue: tcgen05.ld the accumulator (each warp owns the 32 lanes of its
//               quadrant and half of the tile's columns), multiply by alpha, convert, store
//               rows < m and columns < n. 16-bit outputs are packed while they are read, so the
//               warp's whole row segment sits in registers and the accumulator is handed back
//               to the MMA warp before the first store; stores are 32 bytes per lane.
//               (FUSED_A: the same warps first build the A tiles and their scales, see below.)
//   warps 10-11 copy each stage's scale tiles shared -> tensor memory with tcgen05.cp
//               32x128b.warpx4 (a 512-byte tile is 32 rows of 16 bytes, which every 32-lane
//               quadrant of tensor memory needs: the copy broadcasts it) into a ring of scale
//               columns, one slot per scale stage, taking stages in turn, and tcgen05.commit
//               the slot's `ready` barrier. Issued from this kernel's MMA warp, behind a wait
//               per stage, the copies queued up in line with the MMAs (372 us at 8192^3); from warps
//               of their own they overlap them, and two warps issue them faster than one (235 ->
//               219 us). (The CTA-pair kernel below does issue them from its MMA warp: two SMs share
//               that warp's waits, and its barriers are probed a stage ahead.)
//
// What bounds the kernel: 218 us at 8192^3 (K 8192, 128 x 256 tiles). Parts of it by themselves,
// before the MMA warp probed its barriers a stage ahead: MMAs alone 150 us, loads alone 148, loads
// + MMAs 176, everything 219. The scale copies are the largest single cost: twelve per stage, each
// about 30 ns of the copying warp and about 14 cycles of the tensor pipe that no MMA gets.
// Loads and MMAs together lose 26 us to the round trip of a stage (four 48 KB stages cannot cover
// it) and to the shared-memory port both use. The probes gain where few stages are in flight per tile:
// 16 x 8192 -> 8192 with 128 x 128 tiles 15.5 -> 13.0 us.
//
// Every mbarrier wait is bounded (in SM cycles). A wait that gives up records where
// in *status, raises a CTA-wide abort flag, and all roles fall through to the common exit,
// which lets in-flight copies land, releases tensor memory and returns.
#include "fos_gemm_skinny.cuh"
#include "fos_glu.cuh"
#include "fos_pair.cuh"

namespace fos {
namespace {

constexpr int A_BYTES = BLOCK_M * BLOCK_K_BYTES;   // 16 KiB
constexpr int SFA_BYTES = KB_PER_STAGE * SF_TILE_BYTES;
#ifndef FOS_GEMM_SF_LEAD
#define FOS_GEMM_SF_LEAD 1
#endif
constexpr int SF_LEAD = FOS_GEMM_SF_LEAD;   // 0 or 1: how many stages the scales are requested ahead of the operands
#ifndef FOS_GEMM_ST256
#define FOS_GEMM_ST256 1
#endif

constexpr int SF_CP_WARPS = 2;                     // warps 10 and 11 issue the scale copies, taking stages in turn
constexpr int NUM_THREADS = 384;                   // warps: 0 TMA, 1 MMA, 2-9 epilogue (FUSED_A: also the A operand), 10-11 scale copies
// Grouped launches: CTA pairs from this many rows of the buffer per group (padding included: the host knows no other number; a
// group's own share of it is 127 rows on average). In a graph, random routing, us, pairs / the better of the 128-row tiles:
//   buffer rows                 192    256    320    384    448    512    576    640    768    896    1152   1664
//   32 groups, 2880 -> 5760   72/59  76/74  79/87 106/109 137/124 140/152 143/158 168/181 203/219 231/252 292/325 412/465
//   32 groups, 2880 -> 2880   50/43  46/50  48/60  57/68  73/75  75/86  77/94  92/108 107/129 123/146 155/193 215/277
//    8 groups, 4096 -> 4096   26/22  25/27  25/27  30/33  35/33  36/38  36/40  41/41  48/48  55/56  65/72  92/99
//   16 groups, 1024 -> 2048   12/9   12/12  12/12  15/15  17/15  18/16  17/19  18/19  23/23  23/26  28/33  38/42
// From 640 on pairs are never behind by more than 2 %; below, it depends on how the groups' own rows fall (a group of 257 to
// 384 rows leaves half a pair idle), which the host does not know.
constexpr int PAIR_MIN_GROUP_ROWS = 640;
// With the SwiGLU in the epilogue, which only pairs have, they save the product's way through memory and the kernel that does it
// otherwise. But the epilogue takes some 9.5 us a tile whatever K is, against 3.5 us for the MMAs of K = 1536 and 6.7 at 2880, and
// groups of 257 to 384 rows leave half a pair idle: from 640 buffer rows per group where K is at least 1536, from 512 (385 rows
// of a group's own on average: four row tiles of 128 are two of 256) where it is at least 2048, and from 320 where it is at least
// 2880 and six rounds are sure, which leave the idle halves no more than the kernel saved. The whole layer, bf16, random routing,
// in a graph, us, fused on pairs / not:
//   rows of a group's own                          130        200        300        400        500        640       1024
//   32 experts, 1024 -> 2 x 2880 -> 1024       131/116    157/141    212/184    238/227    280/256    329/295    439/430
//   32 experts, 1536 -> 2 x 2880 -> 1536       139/125    164/157    259/208    283/256    295/293    345/337    484/502
//   32 experts, 2048 -> 2 x 2880 -> 2048       148/146    183/176    278/239    283/292    308/328    373/391    540/592
//    8 experts, 2048 -> 2 x 2048 -> 2048         54/55      64/60      78/76      85/85      93/94    108/108    146/141
//   32 experts, 2880 -> 2 x 2880 -> 2880       210/202    230/234    312/307    332/380    383/446    442/497    659/745
//    8 experts, 2880 -> 2 x 2048 -> 2880         82/79      85/85     104/97     112/114     99/105    118/130    160/170
//    8 experts, 4096 -> 2 x 2048 -> 4096         79/80      90/85     105/104    112/121    113/123    139/152    183/202
// (two experts a token with 8, four with 32). Where most tokens go to few experts: 32 experts of 2880 and 2880, 256 rows 317 / 350, 300
// rows 361 / 398; 8 of 2880 and 2048, 200 rows (one to three rounds) 91 / 82; 8 of 2048 and 1024, 130 rows 53 / 42.
inline int pair_min_glu_rows(int64_t rows_capacity, int num_groups, int64_t n_p, int64_t k_p, int sms) {
    if (k_p < 1536) return INT32_MAX;
    if (k_p < 2048) return 640;
    const int64_t sure_tiles = (rows_capacity - 127 * static_cast<int64_t>(num_groups)) / 256 * ((n_p + 255) / 256);
    return k_p >= 2880 && sure_tiles >= 6 * (sms / 2) ? 320 : 512;
}
// Up to this many rows of a group's own on average, in a buffer with the 127 spare rows per group that unknown routing needs, a
// grouped GEMM is bound by the weights (see grouped_kernel_for).
constexpr int FEW_GROUP_ROWS = 64;
constexpr int MAX_GROUPS = 256;                    // of a grouped launch (their row ranges are kept in shared memory)
constexpr int SF_COL0 = 256;                       // tensor-memory columns: accumulators first, then per
                                                   // stage 16 columns of A scales and N/8 of B scales

template <int BLOCK_N> struct Cfg {
    static constexpr int B_BYTES = BLOCK_N * BLOCK_K_BYTES;
    static constexpr int N_GROUPS = BLOCK_N / 128;                 // 128-row scale groups of B
    static constexpr int SFB_BYTES = N_GROUPS * KB_PER_STAGE * SF_TILE_BYTES;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;          // operand tiles of one stage
    static constexpr int SF_SLOT_BYTES = SFA_BYTES + SFB_BYTES;    // scale tiles of one stage
    static constexpr int STAGES = BLOCK_N == 256 ? 4 : 6;
    // The scales of a stage are requested one stage earlier than its operands and have a ring of
    // their own (shared memory and tensor memory) with one slot more than there are stages.
    static constexpr int SF_SLOTS = STAGES + SF_LEAD;
    static constexpr int ACC_STAGES = BLOCK_N == 256 ? 1 : 2;
    static constexpr int BARRIER_BYTES = 512;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + SF_SLOTS * SF_SLOT_BYTES + 1024 /*alignment slack*/ + BARRIER_BYTES;
    static constexpr int SFB_COLS = KB_PER_STAGE * (BLOCK_N / 32);  // per stage
    static constexpr int SF_STAGE_COLS = 16 + SFB_COLS;
    static_assert(STAGE_BYTES % 1024 == 0, "stages must keep the 1024-byte swizzle alignment");
    static_assert(ACC_STAGES * BLOCK_N <= SF_COL0, "accumulators overlap the scale columns");
    static_assert(SF_COL0 + SF_SLOTS * SF_STAGE_COLS <= TMEM_COLS, "scale ring does not fit tensor memory");
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
    static_assert((2 * STAGES + (SF_CP_WARPS + 1) * SF_SLOTS + 2 * ACC_STAGES + 1) * 8 + 8 <= BARRIER_BYTES, "barrier area too small");
};

struct GemmParams {
    const uint8_t *a_sf;
    const uint8_t *b_sf;
    const float *alpha;      // the product's factor, or nullptr:
    const float *amax_a;     // then it is amax_a * amax_b / alpha_denom (what fos_gemm_alpha computes), 1 without amax_a
    const float *amax_b;
    float alpha_denom;
    const void *bias;        // [n] of the output's type, added to the rounded product, or nullptr
    GluEpilogue glu;         // gemm_fp4_pair_kernel<.., GLU>: d is [rows][n / 2]
    void *d;
    int32_t *status;         // where a bounded wait that gives up records its site: the caller's word, or the sticky one
    int64_t m_p, n_p, k_p;   // padded problem (k_p in values)
    int64_t m, n, ldd;       // region of D that is written
    int out_dtype;
    int mx;                  // operands are MXFP4: E8M0 scales per 32 values, a 512-byte scale tile spans 128 values of K
    // Row-parallel layers: this rank's partial product is not stored to d but scattered, tile by tile as
    // the tiles complete, into the staging buffers of the ranks that will reduce them. Row block mb (128
    // rows) belongs to rank mb % scatter_world and is block mb / scatter_world of that rank's slab of
    // `slab_rows` rows; its staging buffer d_peer[o] (a peer mapping unless o is this rank) is
    // [world][slab_rows][ldd], and this rank writes plane scatter_rank.
    // Fused activation quantization (gemm_nvfp4_kernel<.., FUSED_A>): A is not read packed but made in the
    // kernel from x[m, k] (bf16 / fp16, row stride x_ld elements) with NVFP4 static_6 / static_4 and the
    // per-tensor amax at x_amax; a_sf is unused.
    const void *x;
    int64_t x_ld;
    const float *x_amax;
    int x_rule;
    int x_is_fp16;
    int scatter_world;       // 0: plain store to d
    int scatter_rank;
    int64_t slab_rows;
    void *d_peer[8];
    // Grouped problems (gemm_nvfp4_kernel<.., GROUPED>): A, its scales and D are the groups' rows one after
    // the other, group g at rows group_start[g] .. group_start[g + 1] (multiples of 128, read on the device: the
    // host need not know them) of which the first group_rows[g] are written to D; B and its scales are
    // num_groups matrices of n_p rows each, one after the other; alpha has one entry per group.
    const int32_t *group_start;
    const int32_t *group_rows;
    int num_groups;
};

__device__ __forceinline__ float gemm_alpha(const GemmParams &p, int group = 0) {
    if (p.alpha) return ld_float(p.alpha + group);
    if (!p.amax_a) return 1.0f;
    return __fdiv_rn(__fmul_rn(ld_float(p.amax_a + group), ld_float(p.amax_b + group)), p.alpha_denom);
}

// GROUPED: first row of every group (and one past the last group), and one past each group's last valid row.
template <bool GROUPED> struct GroupTable {
    int32_t start[GROUPED ? MAX_GROUPS + 1 : 1], end[GROUPED ? MAX_GROUPS : 1];
};

template <int THREADS> __device__ __forceinline__ void load_groups(const GemmParams &p, GroupTable<true> &groups) {
    asm volatile("griddepcontrol.wait;" ::: "memory");     // the row ranges come from an earlier kernel
    const int32_t cap = static_cast<int32_t>(p.m_p);
    // (the same number of rounds in every thread, and the warps converged again before the warp-wide
    // instructions that follow - tcgen05.alloc, elect.sync: a loop that only some lanes of a warp enter leaves
    // the warp split, and those instructions are undefined for a split warp)
    for (int g0 = 0; g0 <= p.num_groups; g0 += THREADS) {
        const int g = g0 + static_cast<int>(threadIdx.x);
        if (g <= p.num_groups) {
            int32_t s0 = ld_int(p.group_start + g);
            s0 = (s0 < 0 ? 0 : (s0 > cap ? cap : s0)) & ~127;             // never beyond the buffers
            groups.start[g] = s0;
            if (g < p.num_groups) {
                // valid rows end inside the group's own range, whatever group_rows claims
                int32_t s1 = ld_int(p.group_start + g + 1);
                s1 = (s1 < s0 ? s0 : (s1 > cap ? cap : s1)) & ~127;
                const int32_t r = ld_int(p.group_rows + g), e = s0 + (r < 0 ? 0 : r);
                groups.end[g] = e > s1 ? s1 : e;
            }
        }
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------- kernel

template <int BLOCK_N, typename OUT, bool FUSED_A = false, bool GROUPED = false>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_nvfp4_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                  const GemmParams p) {
    using C = Cfg<BLOCK_N>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    // shared memory: operand stages, scale slots, barriers
    const uint32_t sf_base = smem_base + C::STAGES * C::STAGE_BYTES;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_gen + C::STAGES * C::STAGE_BYTES + C::SF_SLOTS * C::SF_SLOT_BYTES);
    const uint32_t full_bar = smem_u32(bars);                       // [STAGES] operand tiles landed
    const uint32_t empty_bar = full_bar + 8 * C::STAGES;            // [STAGES] the stage's MMAs are done
    const uint32_t sf_full_bar = empty_bar + 8 * C::STAGES;         // [SF_CP_WARPS][SF_SLOTS] scale tiles landed
    const uint32_t sf_ready_bar = sf_full_bar + 8 * SF_CP_WARPS * C::SF_SLOTS;   // [SF_SLOTS] scales are in tensor memory
    const uint32_t acc_full_bar = sf_ready_bar + 8 * C::SF_SLOTS;   // [ACC_STAGES]
    const uint32_t acc_empty_bar = acc_full_bar + 8 * C::ACC_STAGES;
    const uint32_t drain_bar = acc_empty_bar + 8 * C::ACC_STAGES;   // only used when the CTA gives up
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * C::STAGES + (SF_CP_WARPS + 1) * C::SF_SLOTS + 2 * C::ACC_STAGES + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    __shared__ GroupTable<GROUPED> groups;
    if constexpr (GROUPED) load_groups<NUM_THREADS>(p, groups);

    if (threadIdx.x == 0) {
        // FUSED_A: besides the copy engine (B, B's scales), the eight warps that make A and its scales arrive
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full_bar + 8 * s, FUSED_A ? 9 : 1);
            mbar_init(empty_bar + 8 * s, 1);
        }
        for (int j = 0; j < C::SF_SLOTS; ++j) {
            for (int w = 0; w < SF_CP_WARPS; ++w) mbar_init(sf_full_bar + 8 * (w * C::SF_SLOTS + j), FUSED_A ? 9 : 1);
            mbar_init(sf_ready_bar + 8 * j, 1);                   // one commit by the warp that copied the slot
        }
        for (int a = 0; a < C::ACC_STAGES; ++a) {
            mbar_init(acc_full_bar + 8 * a, 1);
            mbar_init(acc_empty_bar + 8 * a, 8);   // one arrival per epilogue warp
        }
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int64_t num_m = GROUPED ? groups.start[p.num_groups] / BLOCK_M : p.m_p / BLOCK_M;
    const int64_t num_n = (p.n_p + BLOCK_N - 1) / BLOCK_N;
    // GROUPED: the group that row block mb lies in (the last g with start[g] <= row; empty groups are skipped)
    auto group_of = [&](int64_t mb) -> int {
        if constexpr (!GROUPED) return 0;
        const int32_t row = static_cast<int32_t>(mb * BLOCK_M);
        int lo = 0, hi = p.num_groups - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (groups.start[mid] <= row) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    const int64_t num_tiles = num_m * num_n;
    const int64_t k_blocks = p.k_p / 64;                       // MMA K-blocks in the problem
    const int64_t k_tiles = (k_blocks + KB_PER_STAGE - 1) / KB_PER_STAGE;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer: operands and scales
        // One warp, one elected lane: per stage the two operand tiles and, SF_LEAD stages ahead of them (their
        // way into the MMA is longer: shared memory -> tcgen05.cp -> tensor memory), the two scale copies into
        // a ring of their own that is one slot longer.
        const bool issue = elect_one();
        int64_t f_t = blockIdx.x, f_kt = 0;          // the stage whose scales are requested next
        uint32_t slot = 0, f_w = 0;                  // its ring slot, and which copying warp will take it
        int a_group = 0, b_group = 0;
        auto enter_tile = [&]() {
            if (f_t >= num_tiles) return;
            int64_t mb, nb;
            tile_coords(f_t, num_m, num_n, mb, nb);
            a_group = static_cast<int>(mb);
            b_group = static_cast<int>(nb * C::N_GROUPS) + group_of(mb) * static_cast<int>(p.n_p / 128);
        };
        auto issue_next_scales = [&]() {
            if (f_t >= num_tiles) return;
            // two tensor copies per stage: [K-blocks kb0 .. kb0+3] x [one / N_GROUPS row groups] of 512-byte tiles;
            // what lies beyond K or N is zero-filled and still counted (MXFP4: a tile spans two K-blocks, so the
            // box of its maps is two tiles per group)
            const int kb0 = static_cast<int>(f_kt * (p.mx ? KB_PER_STAGE / 2 : KB_PER_STAGE));
            const uint32_t dst = sf_base + slot * C::SF_SLOT_BYTES, bar = sf_full_bar + 8 * (f_w * C::SF_SLOTS + slot);
            if (issue) {
                if (FUSED_A) {
                    mbar_expect_tx(bar, C::SFB_BYTES);
                } else {
                    mbar_expect_tx(bar, p.mx ? C::SF_SLOT_BYTES / 2 : C::SF_SLOT_BYTES);
                    tma_load_3d(dst, &map_sfa, 0, kb0, a_group, bar);
                }
                tma_load_3d(dst + SFA_BYTES, &map_sfb, 0, kb0, b_group, bar);
            }
            if (++slot == C::SF_SLOTS) slot = 0;
            if (++f_w == SF_CP_WARPS) f_w = 0;
            if (++f_kt == k_tiles) {
                f_kt = 0;
                f_t += gridDim.x;
                enter_tile();
            }
        };
        enter_tile();
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (a dependent launch) the kernel that packs A is done
        for (int i = 0; i < SF_LEAD; ++i) issue_next_scales();
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int64_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
            int64_t mb, nb;
            tile_coords(t, num_m, num_n, mb, nb);
            const int m0 = static_cast<int>(mb * BLOCK_M);
            const int n0 = static_cast<int>(nb * BLOCK_N) + group_of(mb) * static_cast<int>(p.n_p);   // row of B
            for (int64_t kt = 0; kt < k_tiles; ++kt) {
                // the stage is free; so is the scale slot of the iteration SF_LEAD ahead (SF_SLOTS = STAGES +
                // SF_LEAD back from it: its MMAs were done before this stage's)
                ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * s, ph ^ 1u, abort_flag, p.status, 1));
                if (!ok) break;
                const uint32_t stage = smem_base + s * C::STAGE_BYTES, bar = full_bar + 8 * s;
                // rows beyond N and bytes beyond K are zero-filled by the TMA unit and still counted
                if (issue) {
                    mbar_expect_tx(bar, FUSED_A ? C::B_BYTES : C::STAGE_BYTES);
                    if (!FUSED_A) tma_load_2d(stage, &map_a, static_cast<int>(kt * BLOCK_K_BYTES), m0, bar);
                    tma_load_2d(stage + A_BYTES, &map_b, static_cast<int>(kt * BLOCK_K_BYTES), n0, bar);
                }
                issue_next_scales();
                __syncwarp();
                if (++s == C::STAGES) { s = 0; ph ^= 1u; }
            }
        }
        if (!ok) {
            // give copies that are still in flight time to land before the CTA exits
            const unsigned long long t0 = global_timer_ns();
            while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        // (The whole warp runs this loop and one elected lane issues. With every value of the loop the same in
        // all lanes the compiler keeps descriptors and addresses in uniform registers, which the tcgen05
        // instructions take directly; a lone thread's values live in ordinary registers and every instruction
        // pays for moving its operands over: 256 -> 235 us at 8192^3, the CTA-pair kernel 343 -> 249 us.)
        const bool issue = elect_one();
        // (A wait on a barrier that has completed long ago still takes some 190 cycles: the MMAs' operand reads keep shared
        // memory busy. So the next stage's barriers are probed before this stage's instructions are issued, and the
        // answer is looked at after them.)
        uint32_t s = 0, ph = 0, j = 0, jph = 0, tile_i = 0;      // operand stage / scale slot and their phases
        bool ok = true, ready = false;
        for (int64_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tile_i) {
            int64_t mb, nb;
            tile_coords(t, num_m, num_n, mb, nb);
            const int64_t n0 = nb * BLOCK_N;
            const int n_valid = static_cast<int>((p.n_p - n0) < BLOCK_N ? (p.n_p - n0) : BLOCK_N);
            const uint32_t idesc = mma_idesc(n_valid);
            const uint32_t acc = tile_i % C::ACC_STAGES, acc_ph = (tile_i / C::ACC_STAGES) & 1u;
            ok = mbar_wait(acc_empty_bar + 8 * acc, acc_ph ^ 1u, abort_flag, p.status, 3);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + acc * BLOCK_N;
            for (int64_t kt = 0; kt < k_tiles; ++kt) {
                if (!ready) {
                    ok = mbar_wait(full_bar + 8 * s, ph, abort_flag, p.status, 2);
                    if (ok) ok = mbar_wait(sf_ready_bar + 8 * j, jph, abort_flag, p.status, 5);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                tc_fence_after();
                const uint32_t s_next = s + 1 == C::STAGES ? 0 : s + 1, ph_next = s + 1 == C::STAGES ? ph ^ 1u : ph;
                const uint32_t j_next = j + 1 == C::SF_SLOTS ? 0 : j + 1, jph_next = j + 1 == C::SF_SLOTS ? jph ^ 1u : jph;
                const bool full_next = mbar_test_wait(full_bar + 8 * s_next, ph_next);
                const bool sf_next = mbar_test_wait(sf_ready_bar + 8 * j_next, jph_next);
                const int64_t kb0 = kt * KB_PER_STAGE;
                const int nkb = static_cast<int>((k_blocks - kb0) < KB_PER_STAGE ? (k_blocks - kb0) : KB_PER_STAGE);
                const uint32_t stage = smem_base + s * C::STAGE_BYTES;
                // operands: 128-byte swizzled rows, 8-row groups 1024 bytes apart; each K-block
                // of 64 values is 32 bytes further along the row. Scales: this iteration's ring slot.
                const uint32_t a_lo = desc_lo(stage, 16), b_lo = desc_lo(stage + A_BYTES, 16);
                const uint32_t sfa_tmem = tmem_base + SF_COL0 + j * C::SF_STAGE_COLS, sfb_tmem = sfa_tmem + 16;
                if (p.mx) {
                    for (int kb = 0; kb < nkb && issue; ++kb)
                        tc_mma_mxf4_lo(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, mma_idesc_mx(idesc, (kb & 1) * 2),
                                       sfa_tmem + 4 * (kb >> 1), sfb_tmem + (BLOCK_N / 32) * (kb >> 1),
                                       (kt > 0 || kb > 0) ? 1u : 0u);
                } else {
#pragma unroll
                    for (int kb = 0; kb < KB_PER_STAGE; ++kb) {
                        if (kb < nkb && issue)
                            tc_mma_nvf4_lo(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa_tmem + 4 * kb,
                                           sfb_tmem + (BLOCK_N / 32) * kb, (kt > 0 || kb > 0) ? 1u : 0u);
                    }
                }
                if (issue) tc_commit(empty_bar + 8 * s);          // stage (and scale slot) reusable once these MMAs are done
                __syncwarp();
                ready = __all_sync(0xffffffffu, full_next && sf_next);
                s = s_next;
                ph = ph_next;
                j = j_next;
                jph = jph_next;
            }
            if (ok && issue) tc_commit(acc_full_bar + 8 * acc);  // accumulator complete
        }
        if (!ok) {
            // giving up: the MMAs already issued must have finished before tensor memory is released
            if (issue) tc_commit(drain_bar);
            __syncwarp();
            const long long t0 = clock64();
            while (!mbar_try_wait(drain_bar, 0) && clock64() - t0 < 20000000ll) {}   // about 10 ms
        }
    } else if (warp >= 2 && warp < 10) {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3;                       // tensor-memory lanes 32*quad .. +31
        constexpr int COLS = BLOCK_N / 2;                // columns per warp: left or right half
        const int half = (warp - 2) >> 2;
        asm volatile("griddepcontrol.wait;" ::: "memory");   // amax_a, and whoever still reads d
        float alpha = GROUPED ? 0.0f : gemm_alpha(p);
        int64_t row_end = p.m;
        OUT *out = static_cast<OUT *>(p.d);
        const bool vec_ok = (reinterpret_cast<uintptr_t>(out) % 16 == 0) && ((p.ldd * sizeof(OUT)) % 16 == 0);
        const bool vec32_ok = FOS_GEMM_ST256 && (reinterpret_cast<uintptr_t>(out) % 32 == 0) && ((p.ldd * sizeof(OUT)) % 32 == 0);
        uint32_t tile_i = 0;
        bool ok = true;
        // FUSED_A: these eight warps are idle while a tile's MMAs run (one accumulator: the epilogue and the
        // next main loop do not overlap anyway), so they make the A operand: thread e owns row e / 2 of the
        // stage and 8 of its 16 blocks (128 values, 256 contiguous bytes of x).
        __shared__ float2 a_lut[FUSED_A ? 128 : 1];
        StaticQuantConsts qc{};
        uint32_t a_s = 0, a_ph = 0, a_j = 0, a_w = 0;
        const int e_tid = static_cast<int>(threadIdx.x) - 64, a_row = e_tid >> 1, a_half = e_tid & 1;
        if constexpr (FUSED_A) {
            qc = static_quant_consts(ld_float(p.x_amax), p.x_rule);
            if (e_tid < 128) a_lut[e_tid] = static_scale_entry(e_tid, qc.decode);
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        for (int64_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x, ++tile_i) {
            int64_t mb, nb;
            tile_coords(t, num_m, num_n, mb, nb);
            if constexpr (FUSED_A) {
                const int64_t x_row = mb * BLOCK_M + a_row;
                for (int64_t kt = 0; kt < k_tiles && ok; ++kt) {
                    // the values first (the loads do not depend on the stage), then the stage
                    uint32_t w[8][8];
                    const int64_t col0 = kt * 256 + a_half * 128;
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        const int64_t col = col0 + 16 * b;
                        if (x_row < p.m && col < p.k_p) {
                            ld_32_stream(static_cast<const uint16_t *>(p.x) + x_row * p.x_ld + col, w[b]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) w[b][i] = 0u;
                        }
                    }
                    ok = mbar_wait(empty_bar + 8 * a_s, a_ph ^ 1u, abort_flag, p.status, 8);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const uint32_t a_stage = smem_base + a_s * C::STAGE_BYTES + a_row * 128;
                    const uint32_t sfa_slot = sf_base + a_j * C::SF_SLOT_BYTES + (a_row & 31) * 16 + (a_row >> 5) * 4;
                    uint32_t sf_word = 0u, codes[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        float v[16];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float2 f = p.x_is_fp16 ? unpack2<__half>(w[b][i]) : unpack2<__nv_bfloat16>(w[b][i]);
                            v[2 * i] = f.x;
                            v[2 * i + 1] = f.y;
                        }
                        uint32_t lo, hi, sfb;
                        quantize_block_static(v, qc, a_lut, lo, hi, sfb);
                        codes[2 * (b & 1)] = lo;
                        codes[2 * (b & 1) + 1] = hi;
                        sf_word |= sfb << (8 * (b & 3));
                        if (b & 1) {
                            // blocks 2c, 2c + 1 of the row are its 16-byte chunk c, stored where the 128-byte swizzle puts it
                            const int chunk = a_half * 4 + (b >> 1);
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                         ::"r"(a_stage + ((chunk ^ (a_row & 7)) << 4)), "r"(codes[0]), "r"(codes[1]), "r"(codes[2]), "r"(codes[3]) : "memory");
                        }
                        if ((b & 3) == 3) {
                            // the four scales of one K-block (64 values): one word of that K-block's 512-byte tile
                            asm volatile("st.shared.b32 [%0], %1;" ::"r"(sfa_slot + (a_half * 2 + (b >> 2)) * SF_TILE_BYTES), "r"(sf_word) : "memory");
                            sf_word = 0u;
                        }
                    }
                    // what these threads wrote is read by the tensor core and by tcgen05.cp: make it visible to that proxy
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(full_bar + 8 * a_s);
                        mbar_arrive(sf_full_bar + 8 * (a_w * C::SF_SLOTS + a_j));
                    }
                    if (++a_s == C::STAGES) { a_s = 0; a_ph ^= 1u; }
                    if (++a_j == C::SF_SLOTS) a_j = 0;
                    if (++a_w == SF_CP_WARPS) a_w = 0;
                }
                if (!ok) break;
            }
            const int64_t row = mb * BLOCK_M + quad * 32 + lane, n0 = nb * BLOCK_N + half * COLS;
            if constexpr (GROUPED) {
                const int grp = group_of(mb);
                alpha = gemm_alpha(p, grp);
                row_end = groups.end[grp];
            }
            if (p.scatter_world > 1) {
                // row block mb belongs to rank mb % world (interleaved, so that the peer traffic is spread
                // over the whole run instead of coming in one burst per slab) and is block mb / world of
                // that rank's slab; plane `scatter_rank` of its buffer, addressed here by the global row
                const int o = static_cast<int>(mb % p.scatter_world);
                const int64_t first = static_cast<int64_t>(p.scatter_rank) * p.slab_rows + (mb / p.scatter_world) * BLOCK_M - mb * BLOCK_M;
                out = static_cast<OUT *>(p.d_peer[o]) + first * p.ldd;
            }
            const uint32_t acc = tile_i % C::ACC_STAGES, acc_ph = (tile_i / C::ACC_STAGES) & 1u;
            ok = mbar_wait(acc_full_bar + 8 * acc, acc_ph, abort_flag, p.status, 4);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BLOCK_N + half * COLS;
            const bool row_ok = row < row_end;
            if constexpr (sizeof(OUT) == 2) {
                // 16-bit outputs: scale, convert and pack while reading, so that the warp's whole
                // row segment fits in registers and the accumulator goes back to the MMA warp
                // before the first store is issued
                uint32_t pk[COLS / 2];
#pragma unroll
                for (int c = 0; c < COLS / 32; ++c) {
                    uint32_t v[32];
                    tc_load_32cols_sync(t_acc + 32 * c, v);
                    if (c + 1 == COLS / 32) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_empty_bar + 8 * acc);
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        pk[16 * c + i] = pack_pair<OUT>(alpha * __uint_as_float(v[2 * i]), alpha * __uint_as_float(v[2 * i + 1]));
                }
                const int64_t left = p.n - n0;
                if (row_ok && left > 0) {
                    OUT *dst = out + row * p.ldd + n0;
                    if (p.bias) {
                        const OUT *bias = static_cast<const OUT *>(p.bias) + n0;
#pragma unroll
                        for (int i = 0; i < COLS / 2; ++i) pk[i] = add_bias<OUT>(pk[i], bias + 2 * i, left - 2 * i);
                    }
                    if (left >= COLS && vec32_ok) {
                        // 32 bytes per store: every instruction of the warp fills whole 32-byte sectors
#pragma unroll
                        for (int i = 0; i < COLS / 16; ++i) stg_32_stream(reinterpret_cast<uint8_t *>(dst) + 32 * i, &pk[8 * i]);
                    } else if (left >= COLS && vec_ok) {
#pragma unroll
                        for (int i = 0; i < COLS / 8; ++i)
                            reinterpret_cast<uint4 *>(dst)[i] = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                    } else {
                        uint16_t *d16 = reinterpret_cast<uint16_t *>(dst);
#pragma unroll
                        for (int i = 0; i < COLS; ++i)
                            if (i < left) d16[i] = static_cast<uint16_t>(pk[i >> 1] >> ((i & 1) * 16));
                    }
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < COLS / 32; c += 2) {
                    uint32_t v0[32], v1[32];
                    tc_load_64cols_sync(t_acc + 32 * c, v0, v1);
                    if (c + 2 >= COLS / 32) {                // everything is in registers: release the accumulator
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_empty_bar + 8 * acc);
                    }
                    const int64_t col = n0 + 32 * c;
                    const int64_t left0 = p.n - col, left1 = left0 - 32;
                    if (row_ok && left0 > 0)
                        store_chunk<OUT>(out + row * p.ldd + col, v0, alpha, left0 < 32 ? static_cast<int>(left0) : 32, vec_ok);
                    if (row_ok && left1 > 0)
                        store_chunk<OUT>(out + row * p.ldd + col + 32, v1, alpha, left1 < 32 ? static_cast<int>(left1) : 32, vec_ok);
                }
            }
        }
    } else if (warp >= 10 && warp < 10 + SF_CP_WARPS) {
        // ------------------------------------------------------------------ scale copies by tcgen05.cp
        const bool issue = elect_one();
        // The warps take the stages in turn, and every (warp, slot) pair has a landing barrier of its own, which
        // the producer arms for the warp whose turn the stage will be: each barrier has one waiter, which sees
        // every one of its phases in order. (With ONE barrier per slot and an odd number of slots, a slot
        // alternated between the warps: a warp whose own stages had landed could reach its next use of a slot
        // before the other warp's stage in that slot had landed, take the barrier's not-yet-completed phase for
        // the one after it - a parity wait cannot tell them apart - and copy stale scales. Loads land out of
        // order when the kernel is bound by HBM: skinny problems computed with wrong scales and then hung.)
        const uint32_t me = static_cast<uint32_t>(warp - 10);
        uint32_t j = 0, turn = 0, seen = 0;          // bit j of `seen`: parity of this warp's next phase of slot j
        bool ok = true;
        for (int64_t t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
            for (int64_t kt = 0; kt < k_tiles; ++kt) {
                const bool mine = turn == me;
                if (++turn == SF_CP_WARPS) turn = 0;
                if (!mine) {
                    if (++j == C::SF_SLOTS) j = 0;
                    continue;
                }
                const uint32_t jph = (seen >> j) & 1u;
                seen ^= 1u << j;
                ok = mbar_wait(sf_full_bar + 8 * (me * C::SF_SLOTS + j), jph, abort_flag, p.status, 6);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t src = sf_base + j * C::SF_SLOT_BYTES, dst = tmem_base + SF_COL0 + j * C::SF_STAGE_COLS;
                // tiles: 32 rows of 16 bytes, 8-row groups 128 bytes apart, no swizzle
                // (MXFP4: a tile spans two K-blocks, so a stage has two tiles per group)
                const int ntile = p.mx ? KB_PER_STAGE / 2 : KB_PER_STAGE;
                const uint32_t src_lo = desc_lo(src);
#pragma unroll
                for (int kb = 0; kb < KB_PER_STAGE; ++kb) {
                    if (kb >= ntile || !issue) break;
                    tc_copy_sf_lo(dst + 4 * kb, src_lo + ((kb * SF_TILE_BYTES) >> 4));
#pragma unroll
                    for (int g = 0; g < C::N_GROUPS; ++g)
                        tc_copy_sf_lo(dst + 16 + (BLOCK_N / 32) * kb + 4 * g,
                                      src_lo + ((SFA_BYTES + (g * ntile + kb) * SF_TILE_BYTES) >> 4));
                }
                if (issue) tc_commit(sf_ready_bar + 8 * j);     // arrives when the copies above are done
                __syncwarp();
                if (++j == C::SF_SLOTS) j = 0;
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------- CTA-pair kernel
//
// Two CTAs of a cluster (two SMs) compute one 256 x 256 tile with cta_group::2 MMAs: CTA r of
// the pair holds rows m0 + 128 r .. of A and rows n0 + 128 r .. of B in its shared memory,
// and the tensor cores of both SMs read both halves of B. Per MMA an SM fetches a third less
// than the single-CTA kernel, whose limit that is. Only the even CTA (the leader) issues MMAs;
// both CTAs run a TMA producer and an epilogue for their own 128 rows of the tile.
//
//   warp 0     (both CTAs) TMA: per stage this CTA's tiles of A and B and its scale tiles (128 rows of A, all 256 of
//              B: each SM's tensor core needs the scales of every column); everything completes on
//              the LEADER's barriers (the cta_group::2 form of the copy)
//   warp 1     (leader) scale copies (tcgen05.cp) and MMAs, all from this one thread: the tensor pipe runs them in issue
//              order, so neither the copies nor the re-use of their tensor-memory columns need a barrier
//   warps 2..9 (both CTAs) epilogue
//
//   full[s]    leader's barrier: one arrive.expect_tx for the bytes of BOTH CTAs
//   empty[s]   one per CTA, released in both CTAs by the leader's multicast tcgen05.commit
//   acc_full   one per CTA, multicast commit
//   acc_empty  leader's barrier, 16 arrivals: 8 epilogue warps of each CTA
//
// The MMA warp issues seventeen instructions per stage of 256 K values, whose MMAs take 512 cycles, so what it does besides
// counts. Cycles per stage at 8192^3 (NVFP4 / MXFP4), measured with its waits for full[s] as: waits that poll with a
// suspend limit 716 / 669, a tight test_wait loop 730 / 686, plain try_wait 666 / 623. A wait for a barrier that completed long
// ago still costs some 190 cycles of those (its access to shared memory queues behind the MMAs' operand reads), so the next
// stage's barrier is probed before a stage's instructions are issued and the answer is looked at after them (205 -> 197 us,
// 187 -> 180 us; the single-CTA kernel: 218, 224 us). A second barrier per stage, or per group of stages, for the scales (so that they could be copied for several stages together)
// costs more than it saves. No tcgen05 fence after a wait for TMA copies: it orders tcgen05 operations of different threads, and
// only the accumulators pass between threads.
//
// Tensor memory: tiles alternate between two accumulators that OVERLAP by the columns that the scales take. The
// epilogue reads the shared columns first and then releases the barrier, so the next tile's MMAs start while the
// rest of the accumulator is still being read and stored.
namespace pair {

constexpr int TILE_N = 256;
constexpr int B_HALF_BYTES = 128 * BLOCK_K_BYTES;                         // this CTA's 128 rows of B
constexpr int OPERAND_BYTES = A_BYTES + B_HALF_BYTES;                     // 32 KiB
constexpr int THREADS = 320;
constexpr int BARRIER_BYTES = 256;

template <bool MX> struct PairCfg {
    static constexpr int TILES = MX ? KB_PER_STAGE / 2 : KB_PER_STAGE;    // 512-byte scale tiles of a stage per 128 rows
    static constexpr int SFA_BYTES = TILES * SF_TILE_BYTES;
    static constexpr int SF_BYTES = 3 * SFA_BYTES;                        // of a stage: this CTA's rows of A, all 256 rows of B
    static constexpr int STAGE_BYTES = OPERAND_BYTES + SF_BYTES;
    static constexpr int STAGES = MX ? 6 : 5;
    static constexpr int SF_COLS = 12 * TILES;                            // tensor-memory columns of a stage's scales: 4 of A, 8 of B per tile
    static constexpr int SF_COL = TMEM_COLS - 2 * 48;                     // the first of two sets, used in turn
    static constexpr int ACC1_COL = SF_COL - TILE_N;                      // first column of the odd accumulator
    static constexpr int OVERLAP = TILE_N - ACC1_COL;                     // columns that both accumulators use
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + BARRIER_BYTES;
    static_assert(SF_COLS <= 48 && OVERLAP == 96, "tensor memory");
    static_assert(SMEM_BYTES <= 232448, "more shared memory than a CTA can have");
    static_assert((2 * STAGES + 3) * 8 + 8 <= BARRIER_BYTES, "barrier area too small");
};

// GROUPED: row tiles run through each group's rows in steps of 256, so a tile never computes two groups' rows (its second
// half may reach into the next group's, or beyond the last: not stored).
//
// GLU (with GROUPED): the columns are (gate, up) pairs and what is stored is their SwiGLU, so the product itself never
// reaches memory (32768 x 5760: 377 MB less written and read, and the kernel that did it, 125 us). A lane holds
// a row of the tile, so a pair lies in neighbouring registers of one lane, and the bias is the same for all lanes.
// The accumulators overlap by 96 columns only, so the arithmetic (about 25 instructions per output, 64 outputs per thread
// and tile) runs while the next tile's MMAs do; on eight warps it takes longer than they do and bounds the kernel (32768 x
// 5760, K 2880: 382 us, without it 266 and the kernel of its own 125).
template <typename OUT, int N>
__device__ __forceinline__ void glu_columns(OUT *dst, const uint32_t *acc, float alpha, const OUT *bias, int64_t cols_left, bool row_ok,
                                            const GluEpilogue &glu, typename Half16<OUT>::Pair limit2,
                                            typename Half16<OUT>::Pair floor2, typename Half16<OUT>::Pair one2,
                                            typename Half16<OUT>::Pair &max2) {
    using H = Half16<OUT>;
    uint4 bias0[N / 16], bias1[N / 16];
#pragma unroll
    for (int i = 0; i < N / 16; ++i) {
        bias0[i] = bias1[i] = make_uint4(0u, 0u, 0u, 0u);
        if (16 * i < cols_left) {                            // (the product's width is a multiple of 16)
            bias0[i] = ld_16(bias + 16 * i);
            bias1[i] = ld_16(bias + 16 * i + 8);
        }
    }
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        if (c >= cols_left) break;
        const uint4 b0 = bias0[c / 16], b1 = bias1[c / 16];
        const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        uint32_t gate_up[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            gate_up[i] = H::pack(alpha * __uint_as_float(acc[c + 2 * i]), alpha * __uint_as_float(acc[c + 2 * i + 1]));
        const uint4 packed = glu_words<OUT>(gate_up, b, glu.alpha, limit2, floor2, one2);
        if (!row_ok) continue;
        *reinterpret_cast<uint4 *>(dst + c / 2) = packed;
        max2 = fold_abs_max(max2, packed);
    }
}

template <typename OUT, bool MX, bool GROUPED = false, bool GLU = false>
__global__ void __launch_bounds__(THREADS, 1)
gemm_fp4_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_sfa, const __grid_constant__ CUtensorMap map_sfb,
                     const GemmParams p) {
    using C = PairCfg<MX>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t sf_base = smem_base + C::STAGES * OPERAND_BYTES;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_gen + C::STAGES * C::STAGE_BYTES);
    const uint32_t full_bar = smem_u32(bars);                 // [STAGES], used in the leader only
    const uint32_t empty_bar = full_bar + 8 * C::STAGES;      // [STAGES]
    const uint32_t acc_full_bar = empty_bar + 8 * C::STAGES;
    const uint32_t acc_empty_bar = acc_full_bar + 8;          // used in the leader only
    const uint32_t drain_bar = acc_empty_bar + 8;             // only used when the leader gives up
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * C::STAGES + 3);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();                 // 0 = leader
    const bool leader = rank == 0;

    __shared__ GroupTable<GROUPED> groups;
    __shared__ int32_t first_tile[GROUPED ? MAX_GROUPS + 1 : 1];          // of each group, in 256-row tiles
    if constexpr (GROUPED) {
        load_groups<THREADS>(p, groups);
        __syncthreads();
        if (warp == 2) {
            int at = 0;                                                     // running sum, 32 groups at a time
            for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
                const int g = g0 + lane;
                int n = g < p.num_groups ? (groups.start[g + 1] - groups.start[g] + 255) / 256 : 0;
                n = n < 0 ? 0 : n;
                int sum = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += up;
                }
                if (g < p.num_groups) first_tile[g] = at + sum - n;
                at += __shfl_sync(0xffffffffu, sum, 31);
            }
            if (lane == 0) first_tile[p.num_groups] = at;
        }
        __syncwarp();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full_bar + 8 * s, 1);
            mbar_init(empty_bar + 8 * s, 1);
        }
        mbar_init(acc_full_bar, 1);
        mbar_init(acc_empty_bar, 16);
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();            // both CTAs have initialised their barriers and tensor memory
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // (the second half of a tile may lie beyond the operands: zero-filled by the copies, not stored)
    const int64_t num_m = GROUPED ? first_tile[p.num_groups] : (p.m_p + 255) / 256, num_n = (p.n_p + TILE_N - 1) / TILE_N;
    const int64_t num_tiles = num_m * num_n;
    // the group of row tile mb (the last one whose first tile is not beyond it: empty groups are skipped) and its first row
    auto locate = [&](int64_t mb, int &group) -> int64_t {
        group = 0;
        if constexpr (!GROUPED) return mb * 256;
        int lo = 0, hi = p.num_groups - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (first_tile[mid] <= mb) lo = mid; else hi = mid - 1;
        }
        group = lo;
        return groups.start[lo] + (mb - first_tile[lo]) * 256;
    };
    const int64_t k_blocks = p.k_p / 64;
    const int k_tiles = static_cast<int>((k_blocks + KB_PER_STAGE - 1) / KB_PER_STAGE);
    const int64_t pair_id = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (both CTAs)
        const bool issue = elect_one();
        const uint32_t leader_full = map_to_cta(full_bar, 0);
        asm volatile("griddepcontrol.wait;" ::: "memory");   // (a dependent launch) the kernel that packs A is done
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (int64_t t = pair_id; t < num_tiles && ok; t += num_pairs) {
            int64_t mb, nb;
            tile_coords(t, num_m, num_n, mb, nb);
            int group;
            const int m0 = static_cast<int>(locate(mb, group) + rank * 128);
            const int n0 = static_cast<int>(nb * TILE_N + rank * 128) + group * static_cast<int>(p.n_p);      // row of B
            const int a_group = m0 / 128, b_group = static_cast<int>(nb * 2) + group * static_cast<int>(p.n_p / 128);
            for (int kt = 0; kt < k_tiles; ++kt) {
                ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * s, ph ^ 1u, abort_flag, p.status, 1));
                if (!ok) break;
                const uint32_t stage = smem_base + s * OPERAND_BYTES, sf = sf_base + s * C::SF_BYTES, bar = leader_full + 8 * s;
                // out-of-range parts of a box are zero-filled and still counted: fixed byte counts.
                // The leader announces the bytes of both CTAs; its barrier may see the peer's bytes
                // first, which only makes the pending count negative for a moment.
                if (issue) {
                    if (leader) mbar_expect_tx(full_bar + 8 * s, 2 * C::STAGE_BYTES);
                    tma_load_3d_pair(sf, &map_sfa, 0, kt * C::TILES, a_group, bar);
                    tma_load_3d_pair(sf + C::SFA_BYTES, &map_sfb, 0, kt * C::TILES, b_group, bar);
                    tma_load_2d_pair(stage, &map_a, kt * BLOCK_K_BYTES, m0, bar);
                    tma_load_2d_pair(stage + A_BYTES, &map_b, kt * BLOCK_K_BYTES, n0, bar);
                }
                __syncwarp();
                if (++s == C::STAGES) { s = 0; ph ^= 1u; }
            }
        }
        // the leader's last releases arrive in both CTAs' shared memory: stay until they have
        for (int i = 0; i < C::STAGES && ok; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * s, ph ^ 1u, abort_flag, p.status, 7));
            if (++s == C::STAGES) { s = 0; ph ^= 1u; }
        }
        if (!ok) {
            const unsigned long long t0 = global_timer_ns();
            while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
    } else if (warp == 1 && leader) {
        // ------------------------------------------------------------------ scale copies and MMAs, for both CTAs
        const bool issue = elect_one();
        const uint32_t idesc = mma_idesc(TILE_N, 256);
        uint32_t s = 0, ph = 0, sf_set = 0, tile_i = 0;
        bool ok = true, ready = false;
        for (int64_t t = pair_id; t < num_tiles && ok; t += num_pairs, ++tile_i) {
            // the epilogue of the tile before has read the columns that the two accumulators share
            ok = __all_sync(0xffffffffu, mbar_wait(acc_empty_bar, (tile_i & 1u) ^ 1u, abort_flag, p.status, 3));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + ((tile_i & 1u) ? C::ACC1_COL : 0);
            for (int kt = 0; kt < k_tiles; ++kt) {
                if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(full_bar + 8 * s, ph, abort_flag, p.status, 2));
                if (!ok) break;
                // probe the next stage's barrier now (this warp has consumed the slot's phase before): the answer is back by the
                // time this stage's instructions are issued
                const uint32_t s_next = s + 1 == C::STAGES ? 0 : s + 1, ph_next = s + 1 == C::STAGES ? ph ^ 1u : ph;
                const bool next_ready = mbar_test_wait(full_bar + 8 * s_next, ph_next);
                const int left = static_cast<int>(k_blocks) - kt * KB_PER_STAGE;
                const int nkb = left < KB_PER_STAGE ? left : KB_PER_STAGE;
                const uint32_t stage = smem_base + s * OPERAND_BYTES;
                const uint32_t a_lo = desc_lo(stage, 16), b_lo = desc_lo(stage + A_BYTES, 16), sf_lo = desc_lo(sf_base + s * C::SF_BYTES);
                const uint32_t sfa = tmem_base + C::SF_COL + sf_set * 48, sfb = sfa + 4 * C::TILES;
                if (issue) {
                    // tiles: 32 rows of 16 bytes (one of 512 bytes per 128 rows and K-block; MXFP4: per two K-blocks), copied
                    // to all four 32-lane quadrants of the tensor memory of each CTA from that CTA's own shared memory
#pragma unroll
                    for (int kb = 0; kb < C::TILES; ++kb) {
                        tc_copy_sf_pair_lo(sfa + 4 * kb, sf_lo + ((kb * SF_TILE_BYTES) >> 4));
                        tc_copy_sf_pair_lo(sfb + 8 * kb, sf_lo + ((C::SFA_BYTES + kb * SF_TILE_BYTES) >> 4));
                        tc_copy_sf_pair_lo(sfb + 8 * kb + 4, sf_lo + ((C::SFA_BYTES + (C::TILES + kb) * SF_TILE_BYTES) >> 4));
                    }
#pragma unroll
                    for (int kb = 0; kb < KB_PER_STAGE; ++kb) {
                        if (kb >= nkb) break;
                        const uint32_t accumulate = (kt > 0 || kb > 0) ? 1u : 0u;
                        if constexpr (MX)
                            tc_mma_mxf4_pair_lo(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, mma_idesc_mx(idesc, (kb & 1) * 2),
                                                sfa + 4 * (kb >> 1), sfb + 8 * (kb >> 1), accumulate);
                        else
                            tc_mma_nvf4_pair_lo(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa + 4 * kb, sfb + 8 * kb, accumulate);
                    }
                    tc_commit_pair(empty_bar + 8 * s);
                }
                __syncwarp();
                sf_set ^= 1u;
                ready = __all_sync(0xffffffffu, next_ready);
                s = s_next;
                ph = ph_next;
            }
            if (ok && issue) tc_commit_pair(acc_full_bar);
        }
        if (!ok) {
            // giving up: the MMAs already issued must have finished before tensor memory is released
            if (issue) tc_commit_pair_local(drain_bar);
            __syncwarp();
            const long long t0 = clock64();
            while (!mbar_try_wait(drain_bar, 0) && clock64() - t0 < 20000000ll) {}   // about 10 ms
        }
    } else if (warp >= 2) {
        // ------------------------------------------------------------------ epilogue (both CTAs)
        const int quad = warp & 3;                       // tensor-memory lanes 32*quad .. +31
        const int half = (warp - 2) >> 2;                // which half of the shared columns, and of the others
        asm volatile("griddepcontrol.wait;" ::: "memory");   // amax_a, and whoever still reads d
        float alpha = GROUPED ? 0.0f : gemm_alpha(p);
        int64_t row_end = p.m;
        OUT *out = static_cast<OUT *>(p.d);
        const bool vec16 = (reinterpret_cast<uintptr_t>(out) % 16 == 0) && ((p.ldd * sizeof(OUT)) % 16 == 0);
        const bool vec32 = (reinterpret_cast<uintptr_t>(out) % 32 == 0) && ((p.ldd * sizeof(OUT)) % 32 == 0);
        const uint32_t leader_acc_empty = map_to_cta(acc_empty_bar, 0);
        using GluType = std::conditional_t<GLU, OUT, __half>;                  // (fp32 products have no SwiGLU)
        using GluPair = typename Half16<GluType>::Pair;
        [[maybe_unused]] GluPair limit2, floor2, one2, max2;
        if constexpr (GLU) {
            using H = Half16<GluType>;
            const float l = H::r16(p.glu.limit);
            limit2 = as_pair<GluPair>(H::pack(l, l));
            floor2 = as_pair<GluPair>(H::pack(-INFINITY, -l));
            one2 = as_pair<GluPair>(H::pack(1.0f, 1.0f));
            max2 = as_pair<GluPair>(0u);
        }
        uint32_t tile_i = 0;
        bool ok = true;
        for (int64_t t = pair_id; t < num_tiles && ok; t += num_pairs, ++tile_i) {
            int64_t mb, nb;
            tile_coords(t, num_m, num_n, mb, nb);
            int group;
            const int64_t row = locate(mb, group) + rank * 128 + quad * 32 + lane;
            if constexpr (GROUPED) {
                alpha = gemm_alpha(p, group);
                row_end = groups.end[group];
            }
            const bool odd = tile_i & 1u;
            // columns of the tile that this warp takes: half of the shared ones, then half of the others
            constexpr int FIRST = C::OVERLAP / 2, SECOND = C::ACC1_COL / 2;
            const int first = (odd ? 0 : C::ACC1_COL) + half * FIRST, second = (odd ? C::OVERLAP : 0) + half * SECOND;
            // (in the peer this barrier is arrived on from the leader's SM: one lane polls for the warp)
            if (lane == 0) ok = mbar_wait_poll(acc_full_bar, tile_i & 1u, abort_flag, p.status, 4);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (odd ? C::ACC1_COL : 0);
            OUT *dst = out + row * p.ldd + nb * TILE_N;
            const OUT *bias = p.bias ? static_cast<const OUT *>(p.bias) + nb * TILE_N : nullptr;
            const int64_t left = row < row_end ? p.n - nb * TILE_N : 0;
            auto store = [&](const uint32_t *acc, int col, auto n) {
                if constexpr (GLU) {
                    glu_columns<OUT, decltype(n)::value>(out + row * p.ldd + (nb * TILE_N + col) / 2, acc, alpha,
                                                         static_cast<const OUT *>(p.glu.bias) + group * p.n + nb * TILE_N + col,
                                                         p.n - nb * TILE_N - col, row < row_end, p.glu, limit2, floor2, one2, max2);
                } else {
                    store_columns<OUT, decltype(n)::value>(dst + col, acc, alpha, bias ? bias + col : nullptr, left - col, vec32, vec16);
                }
            };
            uint32_t v[FIRST / 48][48];
#pragma unroll
            for (int i = 0; i < FIRST / 48; ++i) tc_load_48cols_sync(t_acc + first + 48 * i, v[i]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_acc_empty);
#pragma unroll
            for (int i = 0; i < FIRST / 48; ++i) store(v[i], first + 48 * i, std::integral_constant<int, 48>{});
            if constexpr (SECOND == 80) {
                tc_load_48cols_sync(t_acc + second, v[0]);
                store(v[0], second, std::integral_constant<int, 48>{});
            }
            uint32_t w[32];
            tc_load_32cols_sync(t_acc + second + (SECOND - 32), w);
            store(w, second + (SECOND - 32), std::integral_constant<int, 32>{});
            if constexpr (GLU) {
                __syncwarp();
                raise_amax<OUT>(max2, p.glu.amax + group, lane);
                max2 = as_pair<GluPair>(0u);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync_all();            // nobody leaves while the peer may still touch this CTA's memory
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace pair

// ---------------------------------------------------------------------------- host side

template <typename OUT, bool MX, bool GROUPED, bool GLU = false>
int launch_pair(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &msa, const CUtensorMap &msb,
                const GemmParams &p, int max_ctas, cudaStream_t stream) {
    // (grouped: at most one more row tile per group than the buffer has)
    const int64_t row_tiles = (p.m_p + 255) / 256 + (GROUPED ? p.num_groups : 0);
    return pair::launch<pair::gemm_fp4_pair_kernel<OUT, MX, GROUPED, GLU>>(pair::THREADS, pair::PairCfg<MX>::SMEM_BYTES,
                                                                           row_tiles * ((p.n_p + 255) / 256), max_ctas, stream,
                                                                           ma, mb, msa, msb, p);
}

template <bool MX, bool GROUPED = false>
int launch_pair_out(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &msa, const CUtensorMap &msb,
                    const GemmParams &p, int max_ctas, cudaStream_t stream) {
    if (p.out_dtype == FOS_BF16) return launch_pair<__nv_bfloat16, MX, GROUPED>(ma, mb, msa, msb, p, max_ctas, stream);
    if (p.out_dtype == FOS_FP16) return launch_pair<__half, MX, GROUPED>(ma, mb, msa, msb, p, max_ctas, stream);
    return launch_pair<float, MX, GROUPED>(ma, mb, msa, msb, p, max_ctas, stream);
}

template <int BLOCK_N, typename OUT, bool FUSED_A = false, bool GROUPED = false>
int launch(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &msa, const CUtensorMap &msb,
           const GemmParams &p, int sms, cudaStream_t stream) {
    using C = Cfg<BLOCK_N>;
    auto kernel = gemm_nvfp4_kernel<BLOCK_N, OUT, FUSED_A, GROUPED>;
    static OncePerDevice configured;   // per instantiation
    int dev = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    FOS_CUDA_TRY(configured.run(dev, [&] {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    }));
    const int64_t tiles = (p.m_p / BLOCK_M) * ((p.n_p + BLOCK_N - 1) / BLOCK_N);
    const unsigned grid = static_cast<unsigned>(tiles < sms ? tiles : sms);
    FOS_CUDA_TRY(launch_dependent(kernel, dim3(grid), NUM_THREADS, C::SMEM_BYTES, stream, ma, mb, msa, msb, p));
    return FOS_OK;
}

template <int BLOCK_N, bool FUSED_A = false, bool GROUPED = false>
int launch_out(const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &msa, const CUtensorMap &msb,
               const GemmParams &p, int sms, cudaStream_t stream) {
    if (p.out_dtype == FOS_BF16) return launch<BLOCK_N, __nv_bfloat16, FUSED_A, GROUPED>(ma, mb, msa, msb, p, sms, stream);
    if (p.out_dtype == FOS_FP16) return launch<BLOCK_N, __half, FUSED_A, GROUPED>(ma, mb, msa, msb, p, sms, stream);
    return launch<BLOCK_N, float, FUSED_A, GROUPED>(ma, mb, msa, msb, p, sms, stream);
}

// Which kernel a problem takes (`sms`: the device's; max_ctas as in fos_gemm_opts).
constexpr int GEMM_SKINNY = 1, GEMM_PAIR = 2, GEMM_128 = 128, GEMM_256 = 256;

inline int sms_allowed(int sms, int max_ctas) { return max_ctas > 0 && max_ctas < sms ? max_ctas : sms; }

// 128 x 256 tiles unless they would fill less than half of the SMs (a 128 x 128 tile takes nine tenths of the
// time of a 128 x 256 one, so the narrow kernel only pays when it doubles the number of busy SMs); in place of
// the wide ones 256 x 256 tiles on CTA pairs wherever those need no more rounds (see pairs_pay), unless one CTA is all
// that is allowed
inline int gemm_kernel_for(int64_t m, int64_t m_p, int64_t n_p, int64_t k_p, int variant, int max_ctas, bool scatter, int sms) {
    if (variant == 128 || variant == 256) return variant;
    if (variant == 0 && max_ctas == 0 && !scatter && skinny::pays(m, n_p, k_p, sms)) return GEMM_SKINNY;
    sms = sms_allowed(sms, max_ctas);
    const int64_t tiles_256 = (m_p / BLOCK_M) * ((n_p + 255) / 256), pair_tiles = ((m_p + 255) / 256) * ((n_p + 255) / 256);
    const bool wide = n_p >= 256 && tiles_256 * 2 > sms;
    if (!scatter && max_ctas != 1 && (variant == 2 || (wide && pairs_pay(tiles_256, pair_tiles, sms)))) return GEMM_PAIR;
    return wide ? GEMM_256 : GEMM_128;
}

// 256-row tiles waste half a tile per group on average, 128-row tiles a quarter of that: pairs where groups are long.
// Groups of a few rows each (a decoding step) are bound by their weights' way out of HBM: a tile then takes the time of its
// columns, whatever its width, and the width is the one whose last round is fuller, with one row block per group. 32 groups of 32
// rows, 2880 columns: 12 wide tiles a group are 2.6 rounds, which take 3, 23 narrow ones 4.97 half rounds. (Fewer or more row
// blocks change the gain and not its sign: n narrow half rounds are never longer than the rounds of half as many wide tiles.)
// `pair_min_rows`: buffer rows per group from which pairs are taken.
inline int grouped_kernel_for(int64_t rows_capacity, int num_groups, int64_t n_p, int variant, int max_ctas, int sms,
                              int pair_min_rows = PAIR_MIN_GROUP_ROWS) {
    if (variant == 128) return GEMM_128;
    sms = sms_allowed(sms, max_ctas);
    const int64_t tiles_256 = (rows_capacity / BLOCK_M) * ((n_p + 255) / 256);
    const bool wide = n_p >= 256 && (tiles_256 * 2 > sms || variant == 256);
    if (variant == 0 && wide && max_ctas != 1 && rows_capacity / num_groups >= pair_min_rows) return GEMM_PAIR;
    // (the buffer has up to 127 rows of padding per group)
    if (variant == 0 && wide && rows_capacity <= static_cast<int64_t>(num_groups) * (127 + FEW_GROUP_ROWS)) {
        auto columns = [&](int64_t width) { return (num_groups * ((n_p + width - 1) / width) + sms - 1) / sms * width; };
        if (columns(128) < columns(256)) return GEMM_128;
    }
    return wide ? GEMM_256 : GEMM_128;
}

}  // namespace
}  // namespace fos

extern "C" int fos_gemm_fp4_kernel(int64_t m, int64_t n, int64_t k, int num_groups, const fos_gemm_opts *opts, int sms, int *k_split) {
    using namespace fos;
    const int variant = opts ? opts->variant : 0, max_ctas = opts ? opts->max_ctas : 0;
    if ((variant != 0 && variant != 128 && variant != 256 && (variant != 2 || num_groups > 0)) || max_ctas < 0 || m <= 0 || n <= 0 ||
        k <= 0 || num_groups < 0 || sms <= 0)
        return FOS_ERR_INVALID_ARGUMENT;
    const int64_t m_p = round_up64(m, 128), n_p = round_up64(n, 128), k_p = round_up64(k, 64);
    const int kernel = num_groups > 0 ? grouped_kernel_for(m_p, num_groups, n_p, variant, max_ctas, sms)
                                      : gemm_kernel_for(m, m_p, n_p, k_p, variant, max_ctas, false, sms);
    if (k_split)
        *k_split = kernel == GEMM_SKINNY ? skinny::split_for(n_p / 128, static_cast<int>((k_p / 64 + KB_PER_STAGE - 1) / KB_PER_STAGE), sms) : 1;
    return kernel;
}

extern "C" int fos_experts_glu_is_fused(int64_t rows_capacity, int64_t hidden, int64_t intermediate, int num_experts, int sms) {
    using namespace fos;
    if (rows_capacity <= 0 || rows_capacity % 128 || hidden <= 0 || hidden % 64 || intermediate <= 0 || intermediate % 64 ||
        num_experts <= 0 || num_experts > MAX_GROUPS || sms <= 0)
        return FOS_ERR_INVALID_ARGUMENT;
    const int64_t n_p = round_up64(2 * intermediate, 128);
    return grouped_kernel_for(rows_capacity, num_experts, n_p, 0, 0, sms, pair_min_glu_rows(rows_capacity, num_experts, n_p, hidden, sms)) == GEMM_PAIR;
}

static int gemm_fp4_entry(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                          const uint8_t *b_sf, const float *alpha, void *d, int out_dtype, int64_t m_p,
                          int64_t n_p, int64_t k_p, int64_t m, int64_t n, int64_t ldd, const fos_gemm_opts *opts,
                          int32_t *status, void *stream_, int mx, void *const *d_peers = nullptr, int world = 0,
                          int rank = 0, const fos::GemmScales *scales = nullptr) {
    using namespace fos;
    const int variant = opts ? opts->variant : 0, max_ctas = opts ? opts->max_ctas : 0;
    if ((variant != 0 && variant != 128 && variant != 256 && variant != 2) || max_ctas < 0) return FOS_ERR_INVALID_ARGUMENT;
    if (d_peers) {
        if (world < 2 || world > 8 || rank < 0 || rank >= world) return FOS_ERR_INVALID_ARGUMENT;
        if (m_p % (128 * static_cast<int64_t>(world)) != 0) return FOS_ERR_UNSUPPORTED;   // slabs of whole row blocks
        for (int i = 0; i < world; ++i) {
            if (!d_peers[i]) return FOS_ERR_INVALID_ARGUMENT;
            if (reinterpret_cast<uintptr_t>(d_peers[i]) % 32 != 0) return FOS_ERR_MISALIGNED;
        }
        d = d_peers[rank];
    }
    if (!a_codes || !a_sf || !b_codes || !b_sf || (!alpha && !scales) || !d) return FOS_ERR_INVALID_ARGUMENT;
    if (m_p <= 0 || n_p <= 0 || k_p < 64 || m_p % 128 || n_p % 128 || k_p % (mx ? 128 : 64)) return FOS_ERR_INVALID_ARGUMENT;
    if (m <= 0 || n <= 0 || m > m_p || n > n_p || ldd < n) return FOS_ERR_INVALID_ARGUMENT;
    if (out_dtype != FOS_BF16 && out_dtype != FOS_FP16 && out_dtype != FOS_FP32) return FOS_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(a_codes) % 16 || reinterpret_cast<uintptr_t>(b_codes) % 16 ||
        reinterpret_cast<uintptr_t>(a_sf) % 16 || reinterpret_cast<uintptr_t>(b_sf) % 16)
        return FOS_ERR_MISALIGNED;
    if (m_p > INT32_MAX || n_p > INT32_MAX || k_p / 2 > INT32_MAX) return FOS_ERR_TOO_LARGE;
    int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);

    int dev = 0, sms = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    FOS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int choice = gemm_kernel_for(m, m_p, n_p, k_p, variant, max_ctas, d_peers != nullptr, sms);
    GemmParams p{};
    p.a_sf = a_sf; p.b_sf = b_sf;
    p.alpha = alpha;
    if (scales) {
        p.amax_a = scales->amax_a;
        p.amax_b = scales->amax_b;
        p.alpha_denom = scales->denom;
        p.bias = scales->bias;
    }
    p.d = d; p.status = status;
    p.m_p = m_p; p.n_p = n_p; p.k_p = k_p; p.m = m; p.n = n; p.ldd = ldd;
    p.out_dtype = out_dtype; p.mx = mx;
    if (d_peers) {
        p.scatter_world = world;
        p.scatter_rank = rank;
        p.slab_rows = m_p / world;
        for (int i = 0; i < world; ++i) p.d_peer[i] = d_peers[i];
    }
    const int64_t sf_k_tiles = mx ? k_p / 128 : k_p / 64;     // 512-byte scale tiles along K
    if (status) {
        FOS_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int32_t), stream));
    } else {
        // no word of the caller's: a wait that gives up leaves its site in the library's sticky word
        FOS_CUDA_TRY(wait_failures_ptr(&p.status));
    }
    CUtensorMap map_a, map_b;

    if (choice == GEMM_SKINNY) {
        skinny::Params q{};
        q.alpha = alpha;
        q.amax_a = p.amax_a; q.amax_b = p.amax_b; q.denom = p.alpha_denom;
        q.d = d; q.status = p.status;
        q.bias = p.bias;
        q.m = static_cast<int>(m); q.n = static_cast<int>(n); q.ldd = ldd;
        return mx ? skinny::launch_n<true>(a_codes, a_sf, b_codes, b_sf, q, out_dtype, m_p, n_p, k_p, sms, scales && scales->chained, stream)
                  : skinny::launch_n<false>(a_codes, a_sf, b_codes, b_sf, q, out_dtype, m_p, n_p, k_p, sms, scales && scales->chained, stream);
    }

    if (choice == GEMM_PAIR) {
        CUtensorMap map_sfa, map_sfb;
        const int tiles = mx ? KB_PER_STAGE / 2 : KB_PER_STAGE;
        if ((st = make_operand_map(&map_a, a_codes, m_p, k_p / 2, 128)) != FOS_OK) return st;
        if ((st = make_operand_map(&map_b, b_codes, n_p, k_p / 2, 128)) != FOS_OK) return st;
        if ((st = make_scale_map(&map_sfa, a_sf, m_p / 128, sf_k_tiles, 1, tiles)) != FOS_OK) return st;
        if ((st = make_scale_map(&map_sfb, b_sf, n_p / 128, sf_k_tiles, 2, tiles)) != FOS_OK) return st;
        return mx ? launch_pair_out<true>(map_a, map_b, map_sfa, map_sfb, p, max_ctas, stream)
                  : launch_pair_out<false>(map_a, map_b, map_sfa, map_sfb, p, max_ctas, stream);
    }
    const bool wide = choice == GEMM_256;
    sms = sms_allowed(sms, max_ctas);                       // leave SMs to concurrent kernels
    if ((st = make_operand_map(&map_a, a_codes, m_p, k_p / 2, BLOCK_M)) != FOS_OK) return st;
    if ((st = make_operand_map(&map_b, b_codes, n_p, k_p / 2, wide ? 256 : 128)) != FOS_OK) return st;
    CUtensorMap map_sfa, map_sfb;
    const int sf_box_k = mx ? KB_PER_STAGE / 2 : KB_PER_STAGE;
    if ((st = make_scale_map(&map_sfa, a_sf, m_p / 128, sf_k_tiles, 1, sf_box_k)) != FOS_OK) return st;
    if ((st = make_scale_map(&map_sfb, b_sf, n_p / 128, sf_k_tiles, wide ? 2 : 1, sf_box_k)) != FOS_OK) return st;
    return wide ? launch_out<256>(map_a, map_b, map_sfa, map_sfb, p, sms, stream)
                : launch_out<128>(map_a, map_b, map_sfa, map_sfb, p, sms, stream);
}

cudaError_t fos::gemm_wait_failures(int32_t *host_value) { return fos::read_wait_failures(host_value); }
cudaError_t fos::gemm_wait_roles(uint32_t *host_value) { return fos::read_wait_roles(host_value); }

extern "C" int fos_gemm_nvfp4(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                              const uint8_t *b_sf, const float *alpha, void *d, int out_dtype, int64_t m_p,
                              int64_t n_p, int64_t k_p, int64_t m, int64_t n, int64_t ldd, int32_t *status,
                              void *stream) {
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, alpha, d, out_dtype, m_p, n_p, k_p, m, n, ldd, nullptr, status, stream, 0);
}

extern "C" int fos_gemm_nvfp4_ex(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                                 const uint8_t *b_sf, const float *alpha, void *d, int out_dtype, int64_t m_p,
                                 int64_t n_p, int64_t k_p, int64_t m, int64_t n, int64_t ldd, const fos_gemm_opts *opts,
                                 int32_t *status, void *stream) {
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, alpha, d, out_dtype, m_p, n_p, k_p, m, n, ldd, opts, status, stream, 0);
}

int fos::gemm_nvfp4_chained(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes, const uint8_t *b_sf,
                            const GemmScales &scales, void *d, int out_dtype, int64_t m_p, int64_t n_p, int64_t k_p,
                            int64_t m, int64_t n, int64_t ldd, const fos_gemm_opts *opts, int32_t *status, void *stream) {
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, nullptr, d, out_dtype, m_p, n_p, k_p, m, n, ldd, opts, status, stream, 0,
                          nullptr, 0, 0, &scales);
}

extern "C" int fos_gemm_nvfp4_scaled(const uint8_t *a_codes, const uint8_t *a_sf, const float *amax_a, int rule_a,
                                     int unbiased_a, const uint8_t *b_codes, const uint8_t *b_sf, const float *amax_b,
                                     int rule_b, int unbiased_b, void *d, int out_dtype, int64_t m_p, int64_t n_p,
                                     int64_t k_p, int64_t m, int64_t n, int64_t ldd, const fos_gemm_opts *opts,
                                     int32_t *status, void *stream) {
    using namespace fos;
    if (!amax_a || !amax_b) return FOS_ERR_INVALID_ARGUMENT;
    const GemmScales scales{amax_a, amax_b, alpha_divisor(FOS_NVFP4, rule_a, FOS_NVFP4, rule_b, unbiased_a, unbiased_b), nullptr, false};
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, nullptr, d, out_dtype, m_p, n_p, k_p, m, n, ldd, opts, status, stream, 0,
                          nullptr, 0, 0, &scales);
}

extern "C" int fos_gemm_mxfp4_unscaled(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes, const uint8_t *b_sf,
                                       void *d, int out_dtype, int64_t m_p, int64_t n_p, int64_t k_p, int64_t m, int64_t n,
                                       int64_t ldd, const fos_gemm_opts *opts, int32_t *status, void *stream) {
    const fos::GemmScales scales{nullptr, nullptr, 1.0f, nullptr, false};
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, nullptr, d, out_dtype, m_p, n_p, k_p, m, n, ldd, opts, status, stream, 1,
                          nullptr, 0, 0, &scales);
}

extern "C" int fos_gemm_nvfp4_fused_a(const void *x, int x_dtype, int64_t x_ld, const float *x_amax, int x_rule,
                                      const uint8_t *b_codes, const uint8_t *b_sf, const float *alpha, void *d,
                                      int out_dtype, int64_t m, int64_t n_p, int64_t k, int64_t n, int64_t ldd,
                                      int32_t *status, void *stream_) {
    using namespace fos;
    if (!x || !x_amax || !b_codes || !b_sf || !alpha || !d) return FOS_ERR_INVALID_ARGUMENT;
    if (x_dtype != FOS_BF16 && x_dtype != FOS_FP16) return FOS_ERR_INVALID_ARGUMENT;
    if (x_rule != FOS_RULE_STATIC_6 && x_rule != FOS_RULE_STATIC_4) return FOS_ERR_UNSUPPORTED;   // 4/6 stays un-fused
    if (m <= 0 || n_p <= 0 || k < 64 || n_p % 128 || n <= 0 || n > n_p || ldd < n || x_ld < k) return FOS_ERR_INVALID_ARGUMENT;
    if (k % 64) return FOS_ERR_UNSUPPORTED;          // whole scale tiles only: pad K, or quantize first
    if (out_dtype != FOS_BF16 && out_dtype != FOS_FP16 && out_dtype != FOS_FP32) return FOS_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(x) % 32 || (x_ld * 2) % 32) return FOS_ERR_MISALIGNED;   // 32-byte loads of x
    if (reinterpret_cast<uintptr_t>(b_codes) % 16 || reinterpret_cast<uintptr_t>(b_sf) % 16) return FOS_ERR_MISALIGNED;
    const int64_t m_p = round_up64(m, 128);
    if (m_p > INT32_MAX || n_p > INT32_MAX || k / 2 > INT32_MAX) return FOS_ERR_TOO_LARGE;
    int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int dev = 0, sms = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    FOS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GemmParams p{};
    p.b_sf = b_sf; p.alpha = alpha; p.d = d; p.status = status;
    p.m_p = m_p; p.n_p = n_p; p.k_p = k; p.m = m; p.n = n; p.ldd = ldd;
    p.out_dtype = out_dtype;
    p.x = x; p.x_ld = x_ld; p.x_amax = x_amax; p.x_rule = x_rule;
    p.x_is_fp16 = x_dtype == FOS_FP16 ? 1 : 0;
    if (status) {
        FOS_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int32_t), stream));
    } else {
        FOS_CUDA_TRY(wait_failures_ptr(&p.status));
    }
    const int64_t tiles_256 = (m_p / BLOCK_M) * ((n_p + 255) / 256);
    const bool wide = n_p >= 256 && tiles_256 * 2 > sms;
    CUtensorMap map_b, map_sfb;
    if ((st = make_operand_map(&map_b, b_codes, n_p, k / 2, wide ? 256 : 128)) != FOS_OK) return st;
    if ((st = make_scale_map(&map_sfb, b_sf, n_p / 128, k / 64, wide ? 2 : 1, KB_PER_STAGE)) != FOS_OK) return st;
    // (the kernel never touches the A maps in this mode; B's stand in for them)
    return wide ? launch_out<256, true>(map_b, map_b, map_sfb, map_sfb, p, sms, stream)
                : launch_out<128, true>(map_b, map_b, map_sfb, map_sfb, p, sms, stream);
}

static int gemm_grouped_entry(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes, const uint8_t *b_sf,
                              const float *alpha, const fos::GemmScales *scales, void *d, int out_dtype,
                              const int32_t *group_start, const int32_t *group_rows, int num_groups, int64_t rows_capacity,
                              int64_t n_p, int64_t k_p, int64_t n, int64_t ldd, const fos_gemm_opts *opts, int32_t *status,
                              void *stream_, const fos::GluEpilogue *glu = nullptr) {
    using namespace fos;
    const int variant = opts ? opts->variant : 0, max_ctas = opts ? opts->max_ctas : 0;
    if ((variant != 0 && variant != 128 && variant != 256) || max_ctas < 0) return FOS_ERR_INVALID_ARGUMENT;
    if (!a_codes || !a_sf || !b_codes || !b_sf || (!alpha && !scales) || !d || !group_start || !group_rows) return FOS_ERR_INVALID_ARGUMENT;
    if (num_groups <= 0 || num_groups > MAX_GROUPS) return FOS_ERR_INVALID_ARGUMENT;
    if (rows_capacity <= 0 || rows_capacity % 128 || n_p <= 0 || n_p % 128 || k_p < 64 || k_p % 64) return FOS_ERR_INVALID_ARGUMENT;
    if (n <= 0 || n > n_p || ldd < (glu ? n / 2 : n)) return FOS_ERR_INVALID_ARGUMENT;
    if (out_dtype != FOS_BF16 && out_dtype != FOS_FP16 && out_dtype != FOS_FP32) return FOS_ERR_INVALID_ARGUMENT;
    // (the epilogue's stores are 8 outputs of a row, its loads 8 numbers of the bias; in fp16 one sigmoid in 60 needs the binary32
    // sequence, in bf16 one in 500, and the few warps of an epilogue have no room for that many)
    if (glu && (out_dtype != FOS_BF16 || n % 16 || ldd % 8 || reinterpret_cast<uintptr_t>(d) % 16 || reinterpret_cast<uintptr_t>(glu->bias) % 16))
        return FOS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(a_codes) % 16 || reinterpret_cast<uintptr_t>(b_codes) % 16 ||
        reinterpret_cast<uintptr_t>(a_sf) % 16 || reinterpret_cast<uintptr_t>(b_sf) % 16)
        return FOS_ERR_MISALIGNED;
    const int64_t b_rows = n_p * num_groups;
    if (rows_capacity > INT32_MAX || b_rows > INT32_MAX || k_p / 2 > INT32_MAX) return FOS_ERR_TOO_LARGE;
    int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    int dev = 0, sms = 0;
    FOS_CUDA_TRY(cudaGetDevice(&dev));
    FOS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GemmParams p{};
    p.a_sf = a_sf; p.b_sf = b_sf; p.alpha = alpha; p.d = d; p.status = status;
    p.m_p = rows_capacity; p.n_p = n_p; p.k_p = k_p; p.m = rows_capacity; p.n = n; p.ldd = ldd;
    p.out_dtype = out_dtype;
    if (scales) {
        p.amax_a = scales->amax_a;
        p.amax_b = scales->amax_b;
        p.alpha_denom = scales->denom;
    }
    p.group_start = group_start;
    p.group_rows = group_rows;
    p.num_groups = num_groups;
    // how many row blocks are in use is known on the device only: the grid is sized for the buffers, and
    // CTAs that find no tile leave at once
    const int choice = grouped_kernel_for(rows_capacity, num_groups, n_p, variant, max_ctas, sms, glu ? pair_min_glu_rows(rows_capacity, num_groups, n_p, k_p, sms) : PAIR_MIN_GROUP_ROWS);
    if (glu) {
        if (choice != GEMM_PAIR) return FOS_ERR_UNSUPPORTED;
        p.glu = *glu;
    }
    if (status) {
        FOS_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int32_t), stream));
    } else {
        FOS_CUDA_TRY(wait_failures_ptr(&p.status));
    }
    CUtensorMap map_a, map_b, map_sfa, map_sfb;
    if (choice == GEMM_PAIR) {
        if ((st = make_operand_map(&map_a, a_codes, rows_capacity, k_p / 2, 128)) != FOS_OK) return st;
        if ((st = make_operand_map(&map_b, b_codes, b_rows, k_p / 2, 128)) != FOS_OK) return st;
        if ((st = make_scale_map(&map_sfa, a_sf, rows_capacity / 128, k_p / 64, 1, KB_PER_STAGE)) != FOS_OK) return st;
        if ((st = make_scale_map(&map_sfb, b_sf, b_rows / 128, k_p / 64, 2, KB_PER_STAGE)) != FOS_OK) return st;
        if (glu)
            return launch_pair<__nv_bfloat16, false, true, true>(map_a, map_b, map_sfa, map_sfb, p, max_ctas, stream);
        return launch_pair_out<false, true>(map_a, map_b, map_sfa, map_sfb, p, max_ctas, stream);
    }
    const bool wide = choice == GEMM_256;
    sms = sms_allowed(sms, max_ctas);
    if ((st = make_operand_map(&map_a, a_codes, rows_capacity, k_p / 2, BLOCK_M)) != FOS_OK) return st;
    if ((st = make_operand_map(&map_b, b_codes, b_rows, k_p / 2, wide ? 256 : 128)) != FOS_OK) return st;
    if ((st = make_scale_map(&map_sfa, a_sf, rows_capacity / 128, k_p / 64, 1, KB_PER_STAGE)) != FOS_OK) return st;
    if ((st = make_scale_map(&map_sfb, b_sf, b_rows / 128, k_p / 64, wide ? 2 : 1, KB_PER_STAGE)) != FOS_OK) return st;
    return wide ? launch_out<256, false, true>(map_a, map_b, map_sfa, map_sfb, p, sms, stream)
                : launch_out<128, false, true>(map_a, map_b, map_sfa, map_sfb, p, sms, stream);
}

extern "C" int fos_gemm_nvfp4_grouped(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                                      const uint8_t *b_sf, const float *alpha, void *d, int out_dtype,
                                      const int32_t *group_start, const int32_t *group_rows, int num_groups,
                                      int64_t rows_capacity, int64_t n_p, int64_t k_p, int64_t n, int64_t ldd,
                                      const fos_gemm_opts *opts, int32_t *status, void *stream) {
    return gemm_grouped_entry(a_codes, a_sf, b_codes, b_sf, alpha, nullptr, d, out_dtype, group_start, group_rows, num_groups,
                              rows_capacity, n_p, k_p, n, ldd, opts, status, stream);
}

int fos::gemm_nvfp4_grouped_scaled(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes, const uint8_t *b_sf,
                                   const GemmScales &scales, void *d, int out_dtype, const int32_t *group_start,
                                   const int32_t *group_rows, int num_groups, int64_t rows_capacity, int64_t n_p, int64_t k_p,
                                   int64_t n, int64_t ldd, int32_t *status, void *stream) {
    return gemm_grouped_entry(a_codes, a_sf, b_codes, b_sf, nullptr, &scales, d, out_dtype, group_start, group_rows, num_groups,
                              rows_capacity, n_p, k_p, n, ldd, nullptr, status, stream);
}

int fos::gemm_nvfp4_grouped_glu(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes, const uint8_t *b_sf,
                                const GemmScales &scales, const GluEpilogue &glu, void *d, int out_dtype, const int32_t *group_start,
                                const int32_t *group_rows, int num_groups, int64_t rows_capacity, int64_t n_p, int64_t k_p,
                                int64_t n, int64_t ldd, int32_t *status, void *stream) {
    return gemm_grouped_entry(a_codes, a_sf, b_codes, b_sf, nullptr, &scales, d, out_dtype, group_start, group_rows, num_groups,
                              rows_capacity, n_p, k_p, n, ldd, nullptr, status, stream, &glu);
}

extern "C" int fos_gemm_mxfp4(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                              const uint8_t *b_sf, const float *alpha, void *d, int out_dtype, int64_t m_p,
                              int64_t n_p, int64_t k_p, int64_t m, int64_t n, int64_t ldd, int32_t *status,
                              void *stream) {
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, alpha, d, out_dtype, m_p, n_p, k_p, m, n, ldd, nullptr, status, stream, 1);
}

extern "C" int fos_gemm_mxfp4_ex(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                                 const uint8_t *b_sf, const float *alpha, void *d, int out_dtype, int64_t m_p,
                                 int64_t n_p, int64_t k_p, int64_t m, int64_t n, int64_t ldd, const fos_gemm_opts *opts,
                                 int32_t *status, void *stream) {
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, alpha, d, out_dtype, m_p, n_p, k_p, m, n, ldd, opts, status, stream, 1);
}

extern "C" int fos_gemm_nvfp4_scatter(const uint8_t *a_codes, const uint8_t *a_sf, const uint8_t *b_codes,
                                      const uint8_t *b_sf, const float *alpha, void *const *d_peers, int world, int rank,
                                      int out_dtype, int64_t m_p, int64_t n_p, int64_t k_p, int64_t m, int64_t n,
                                      int64_t ldd, int32_t *status, void *stream) {
    if (!d_peers) return FOS_ERR_INVALID_ARGUMENT;
    if (out_dtype != FOS_BF16 && out_dtype != FOS_FP16) return FOS_ERR_UNSUPPORTED;
    return gemm_fp4_entry(a_codes, a_sf, b_codes, b_sf, alpha, nullptr, out_dtype, m_p, n_p, k_p, m, n, ldd, nullptr, status, stream, 0,
                          d_peers, world, rank);
}
