// The steps of a mixture-of-experts layer around the two grouped GEMMs:
//
//   fos_experts_route         routing indices -> row ranges per expert and the tables the other kernels take
//   fos_experts_gather_rows   routed tokens -> the padded row buffer the grouped quantization reads
//   fos_experts_glu           gate-up output + bias -> clamped SwiGLU, the input of the down projection
//   fos_experts_combine       down output + bias, times the routing weight, summed per token
//
// The whole layer as one call (fos_experts_forward) leaves out the second where the quantization gathers the rows itself, and the
// third where the gate-up GEMM's epilogue does it.
//
// The arithmetic follows the reference's GPT-OSS experts module
// (src/fouroversix/model/modules/gpt_oss.py:297-335), which runs it as a chain of element-wise tensor
// operations on 16-bit tensors: every operation computes in binary32 and rounds its result to the
// tensor's type. The kernels keep every one of those roundings, so the results are the bits of that
// chain; what they save is its memory traffic (each operation reads and writes the whole tensor, the
// gathers materialise the bias per row) and its launches. Gather and combine are bound by HBM, the SwiGLU
// by its arithmetic (a sigmoid with an IEEE division and six roundings per output).
#include "fos_glu.cuh"

namespace fos {
namespace {

// Every kernel of the layer starts here. In the one-call form each is launched as the programmatic dependent of the one
// before it: its CTAs may be placed while that one drains, and wait here before they touch memory. What came before
// THAT one is then complete too, because it waited the same way. (Ordinary launches: both instructions do nothing.)
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int ROW_THREADS = 256;         // of the kernels that give a row to a warp
constexpr int GATHER_CTAS = 6, GLU_CTAS = 4;     // their CTAs per SM (one wave: a warp takes rows in turn)

// The two row kernels below give a warp a row, or (few rows) a segment of one: a row is a few KB, so its own latency (look
// up the row, fetch it, reduce) dominates, and warps that do not wait for one another overlap theirs. A unit of work is
// (row, segment); in the one-call form of the layer the rows are taken in the order of the (token, slot) pairs, which
// visits the rows in use only - of 256 tokens over 32 experts a quarter of the padded buffer - and leaves the padding
// rows as they are: no row of a product depends on another, and nobody reads those.
struct RowUnits {
    int rows, segs, seg_chunks;            // rows (or pairs), segments per row, 16-byte pieces per segment
    const int32_t *pair_row, *pair_expert; // pair order: the pairs' rows (-1: none) and experts; nullptr: row order
    int top_k;
};

// out[r] = x[row_token[r]], or zeros where row_token[r] < 0, 16 bytes per lane and piece.
// With amax != nullptr also amax[row_expert[r]] = max(amax[..], max |out[r]|): the per-expert maxima the grouped
// quantization of `out` needs, so that it can skip its own pass over the buffer.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS, GATHER_CTAS)
gather_rows_kernel(const uint8_t *__restrict__ x, int64_t ld_x_bytes, const int32_t *__restrict__ row_token,
                   uint8_t *__restrict__ out, int64_t ld_out_bytes, const RowUnits units, int chunks,
                   const int32_t *__restrict__ row_expert, float *__restrict__ amax) {
    chain_begin();
    using P = typename Half16<T>::Pair;
    const int lane = threadIdx.x & 31, warps = gridDim.x * (ROW_THREADS / 32), total = units.rows * units.segs;
    for (int i = (blockIdx.x * ROW_THREADS + threadIdx.x) >> 5; i < total; i += warps) {
        const int at = units.segs == 1 ? i : i / units.segs, seg = i - at * units.segs;
        const int c_begin = seg * units.seg_chunks, c_end = min(chunks, c_begin + units.seg_chunks);
        const int r = units.pair_row ? ld_int(units.pair_row + at) : at;
        if (r < 0) continue;
        const int t = units.pair_row ? at / units.top_k : ld_int(row_token + r);
        uint4 *dst = reinterpret_cast<uint4 *>(out + r * ld_out_bytes);
        if (t < 0) {
            for (int c = c_begin + lane; c < c_end; c += 32) dst[c] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        const uint4 *src = reinterpret_cast<const uint4 *>(x + static_cast<int64_t>(t) * ld_x_bytes);
        P m2 = as_pair<P>(0u);
        for (int c0 = c_begin + lane; c0 < c_end; c0 += 32 * 4) {             // four loads in flight per lane
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = c0 + 32 * u < c_end ? ld_16(src + c0 + 32 * u) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (c0 + 32 * u < c_end) dst[c0 + 32 * u] = v[u];
                m2 = fold_abs_max<P>(m2, v[u]);
            }
        }
        __syncwarp();
        if (amax != nullptr) raise_amax<T>(m2, amax + ld_int(units.pair_row ? units.pair_expert + at : row_expert + r), lane);
    }
}

// gate_up [rows][2 * inter] with gate in the even and up in the odd columns; bias [experts][2 * inter];
// out [rows][inter]. A lane makes 8 outputs from 32 bytes of gate_up and 32 bytes of bias, two such pieces at a time.
template <typename T>
__global__ void __launch_bounds__(ROW_THREADS, GLU_CTAS)
glu_kernel(const uint8_t *__restrict__ gate_up, int64_t ld_gu_bytes, const uint8_t *__restrict__ bias, int64_t ld_bias_bytes,
           const int32_t *__restrict__ row_expert, uint8_t *__restrict__ out, int64_t ld_out_bytes, const RowUnits units, int chunks,
           float alpha, float limit, float *__restrict__ amax) {
    chain_begin();
    using H = Half16<T>;
    using P = typename H::Pair;
    const float l = H::r16(limit);
    const P limit2 = as_pair<P>(H::pack(l, l)), floor2 = as_pair<P>(H::pack(-INFINITY, -l)), one2 = as_pair<P>(H::pack(1.0f, 1.0f));
    const int lane = threadIdx.x & 31, warps = gridDim.x * (ROW_THREADS / 32), total = units.rows * units.segs;
    for (int i = (blockIdx.x * ROW_THREADS + threadIdx.x) >> 5; i < total; i += warps) {
        const int at = units.segs == 1 ? i : i / units.segs, seg = i - at * units.segs;
        const int c_begin = seg * units.seg_chunks, c_end = min(chunks, c_begin + units.seg_chunks);
        const int row = units.pair_row ? ld_int(units.pair_row + at) : at;
        if (row < 0) continue;
        const int e = ld_int(units.pair_row ? units.pair_expert + at : row_expert + row);
        uint4 *dst = reinterpret_cast<uint4 *>(out + row * ld_out_bytes);
        if (e < 0) {
            for (int c = c_begin + lane; c < c_end; c += 32) dst[c] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        const uint4 *src = reinterpret_cast<const uint4 *>(gate_up + row * ld_gu_bytes);
        const uint4 *b = reinterpret_cast<const uint4 *>(bias + e * ld_bias_bytes);
        P m2 = as_pair<P>(0u);
        for (int c0 = c_begin + lane; c0 < c_end; c0 += 64) {
            uint4 g[2][2], w[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = c0 + 32 * u < c_end ? c0 + 32 * u : c0;
                g[u][0] = ld_16_stream(src + 2 * c);
                g[u][1] = ld_16_stream(src + 2 * c + 1);
                w[u][0] = ld_16(b + 2 * c);
                w[u][1] = ld_16(b + 2 * c + 1);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (c0 + 32 * u >= c_end) break;
                const uint32_t gate_up8[8] = {g[u][0].x, g[u][0].y, g[u][0].z, g[u][0].w, g[u][1].x, g[u][1].y, g[u][1].z, g[u][1].w};
                const uint32_t bias8[8] = {w[u][0].x, w[u][0].y, w[u][0].z, w[u][0].w, w[u][1].x, w[u][1].y, w[u][1].z, w[u][1].w};
                const uint4 packed = glu_words<T>(gate_up8, bias8, alpha, limit2, floor2, one2);
                dst[c0 + 32 * u] = packed;
                m2 = fold_abs_max<P>(m2, packed);
            }
        }
        __syncwarp();
        if (amax != nullptr) raise_amax<T>(m2, amax + e, lane);     // (e is the same for the whole warp)
    }
}

constexpr int MAX_TOP_K = 8;

// out[t] = sum over the token's experts, in ascending order of the expert's index (the order in which the
// reference's host loop adds them into the 16-bit result), of (y[row] + bias[expert]) * weight, every
// operation rounded to the 16-bit type, the running sum too (packed 16-bit arithmetic: see glu_word).
template <typename T>
__global__ void __launch_bounds__(256)
combine_kernel(const uint8_t *__restrict__ y, int64_t ld_y_bytes, const uint8_t *__restrict__ bias, int64_t ld_bias_bytes,
               const int32_t *__restrict__ pair_row, const int32_t *__restrict__ pair_expert,
               const uint16_t *__restrict__ pair_weight, int top_k, uint8_t *__restrict__ out, int64_t ld_out_bytes, int tokens,
               int chunks) {
    chain_begin();
    using P = typename Half16<T>::Pair;
    __shared__ int s_row[MAX_TOP_K], s_ex[MAX_TOP_K];
    __shared__ uint32_t s_w[MAX_TOP_K];
    for (int t = blockIdx.x; t < tokens; t += gridDim.x) {
        __syncthreads();                                  // the previous token's slots have been read
        if (threadIdx.x < 32) {                           // the token's slots in the order of their experts, a lane each
            const int lane = static_cast<int>(threadIdx.x);
            int e = 0, r = -1, place = 0;
            uint32_t w = 0u;
            if (lane < top_k) {
                const int64_t i = static_cast<int64_t>(t) * top_k + lane;
                e = ld_int(pair_expert + i);
                r = ld_int(pair_row + i);
                w = ld_b16(pair_weight + i);
            }
            for (int k = 0; k < top_k; ++k) {             // (equal ones in the order of the slots)
                const int other = __shfl_sync(0xffffffffu, e, k);
                place += other < e || (other == e && k < lane) ? 1 : 0;
            }
            if (lane < top_k) {
                s_ex[place] = e;
                s_row[place] = r;
                s_w[place] = w | (w << 16);
            }
        }
        __syncthreads();
        uint4 *dst = reinterpret_cast<uint4 *>(out + t * ld_out_bytes);
        for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
            uint32_t acc[4] = {0u, 0u, 0u, 0u};
            for (int k = 0; k < top_k; ++k) {
                if (s_row[k] < 0) continue;               // a slot whose expert index was out of range
                const uint4 v = ld_16_stream(reinterpret_cast<const uint4 *>(y + s_row[k] * ld_y_bytes) + c);
                const uint4 b = ld_16(reinterpret_cast<const uint4 *>(bias + s_ex[k] * ld_bias_bytes) + c);
                const P w2 = as_pair<P>(s_w[k]);
                const uint32_t vv[4] = {v.x, v.y, v.z, v.w}, bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    acc[i] = as_word(__hadd2_rn(as_pair<P>(acc[i]), __hmul2_rn(__hadd2_rn(as_pair<P>(vv[i]), as_pair<P>(bb[i])), w2)));
            }
            dst[c] = make_uint4(acc[0], acc[1], acc[2], acc[3]);
        }
    }
}

constexpr int ROUTE_THREADS = 256, ROUTE_WARPS = ROUTE_THREADS / 32, ROUTE_MAX_EXPERTS = 256, ROUTE_MAX_SEGMENTS = 128;

// The routing tables of one layer call: a stable counting sort of the (token, slot) pairs by expert, in two
// launches of one CTA per SEGMENT of the pairs (contiguous, `seg` pairs each).
//   group_rows[e]   pairs routed to expert e           group_start[e]  first row of expert e in the padded buffer
//   pair_row[p]     the row pair p was given (ascending in p within an expert), -1 for an index outside [0, experts)
//   row_token[r], row_expert[r]   the token and the expert of row r, -1 for padding rows
// route_count_kernel: every CTA counts its segment per expert into seg_count[segment][expert], and the CTAs
// together fill the row tables with -1; CTAs beyond the segments (the one-call form) take a warp per token for its largest
// magnitude. route_place_kernel: every CTA adds up the counts of all segments (totals,
// hence the experts' first rows) and of the segments before its own (hence its own first row per expert), splits
// its segment over its warps the same way (count, running sum), and then each warp walks its pairs 32 at a
// time, ranks the pairs of one expert among themselves with match_any and advances its own counters. Rows
// ascend with the pair index because segments, warps and lanes do. With the tokens' maxima it also raises the experts', which
// the grouped quantization needs: 8192 tokens are read once for it (47 MB), not the 32768 rows that their experts get.
template <typename IDX>
__device__ __forceinline__ int route_expert_of(const IDX *__restrict__ routing, int p, int end, int experts) {
    if (p >= end) return -1;
    long long e;
    if constexpr (sizeof(IDX) == 8) asm volatile("ld.global.b64 %0, [%1];" : "=l"(e) : "l"(routing + p));
    else e = ld_int(reinterpret_cast<const int32_t *>(routing + p));
    return (e >= 0 && e < experts) ? static_cast<int>(e) : -1;
}

struct TokenMaxima {
    const uint8_t *x;                      // [tokens] rows of `chunks` 16-byte pieces, or nullptr: no maxima
    int64_t ld_bytes;
    int tokens, chunks;
    float *of_token;                       // [tokens]
};

template <typename T> __device__ __forceinline__ void token_maxima(const TokenMaxima &m, int first_warp, int warps, int lane) {
    using P = typename Half16<T>::Pair;
    for (int t = first_warp; t < m.tokens; t += warps) {
        const uint4 *src = reinterpret_cast<const uint4 *>(m.x + t * m.ld_bytes);
        P m2 = as_pair<P>(0u);
        for (int c0 = lane; c0 < m.chunks; c0 += 32 * 4) {                    // four loads in flight per lane
            uint4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = c0 + 32 * u < m.chunks ? ld_16(src + c0 + 32 * u) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int u = 0; u < 4; ++u) m2 = fold_abs_max<P>(m2, v[u]);
        }
        __syncwarp();
        float largest = fmaxf(Half16<T>::lo(as_word(m2)), Half16<T>::hi(as_word(m2)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, o));
        if (lane == 0) m.of_token[t] = largest;
    }
}

template <typename IDX, typename T>
__global__ void __launch_bounds__(ROUTE_THREADS)
route_count_kernel(const IDX *__restrict__ routing, int pairs, int seg, int segments, int experts, int rows_capacity,
                   int32_t *__restrict__ seg_count, int32_t *__restrict__ row_token, int32_t *__restrict__ row_expert,
                   float *__restrict__ amax, const TokenMaxima maxima) {
    chain_begin();
    if (static_cast<int>(blockIdx.x) >= segments) {
        const int first = ((blockIdx.x - segments) * ROUTE_THREADS + threadIdx.x) >> 5;
        token_maxima<T>(maxima, first, (gridDim.x - segments) * ROUTE_WARPS, threadIdx.x & 31);
        return;
    }
    if (amax != nullptr && blockIdx.x == 0 && threadIdx.x < 2 * experts) {        // (the one-call form: both projections' maxima)
        for (int i = threadIdx.x; i < 2 * experts; i += ROUTE_THREADS) amax[i] = 0.0f;
    }
    __shared__ int s_count[ROUTE_MAX_EXPERTS];
    const int tid = threadIdx.x;
    s_count[tid] = 0;
    for (int r = blockIdx.x * ROUTE_THREADS + tid; r < rows_capacity; r += segments * ROUTE_THREADS) {
        row_token[r] = -1;
        row_expert[r] = -1;
    }
    __syncthreads();
    const int p0 = blockIdx.x * seg, p1 = min(pairs, p0 + seg);
    for (int base = p0; base < p1; base += 4 * ROUTE_THREADS) {       // four independent loads in flight per thread
        int e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = route_expert_of(routing, base + u * ROUTE_THREADS + tid, p1, experts);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e[u] >= 0) atomicAdd(&s_count[e[u]], 1);
    }
    __syncthreads();
    if (tid < experts) seg_count[blockIdx.x * experts + tid] = s_count[tid];
}

template <typename IDX>
__global__ void __launch_bounds__(ROUTE_THREADS)
route_place_kernel(const IDX *__restrict__ routing, int pairs, int seg, int top_k, int experts,
                   const int32_t *__restrict__ seg_count, int32_t *__restrict__ group_start,
                   int32_t *__restrict__ group_rows, int32_t *__restrict__ row_token, int32_t *__restrict__ row_expert,
                   int32_t *__restrict__ pair_row, int32_t *__restrict__ pair_expert, const float *__restrict__ token_max,
                   float *__restrict__ amax) {
    chain_begin();
    __shared__ int s_max[ROUTE_MAX_EXPERTS];                 // the segment's largest magnitude per expert
    s_max[threadIdx.x] = 0;
    __shared__ int s_at[ROUTE_WARPS][ROUTE_MAX_EXPERTS];     // counts, then next rows, per (warp, expert)
    __shared__ int s_total[ROUTE_MAX_EXPERTS], s_first[ROUTE_MAX_EXPERTS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int w = 0; w < ROUTE_WARPS; ++w) s_at[w][tid] = 0;
    int before = 0;
    if (tid < experts) {
        int total = 0;
        for (int sgm = 0; sgm < static_cast<int>(gridDim.x); ++sgm) {
            const int n = ld_int(seg_count + sgm * experts + tid);
            total += n;
            if (sgm < static_cast<int>(blockIdx.x)) before += n;
        }
        s_total[tid] = total;
    }
    __syncthreads();
    if (tid == 0) {
        int at = 0;
        for (int e = 0; e < experts; ++e) {
            s_first[e] = at;
            if (blockIdx.x == 0) {
                group_start[e] = at;
                group_rows[e] = s_total[e];
            }
            at += (s_total[e] + 127) / 128 * 128;
        }
        if (blockIdx.x == 0) group_start[experts] = at;
    }
    // this CTA's segment over its warps: count ...
    const int p0 = blockIdx.x * seg, p1 = min(pairs, p0 + seg);
    const int wseg = ((p1 > p0 ? p1 - p0 : 0) + ROUTE_WARPS - 1) / ROUTE_WARPS;
    const int w0 = p0 + warp * wseg, w1 = min(p1, w0 + wseg);
    for (int base = w0; base < w1; base += 128) {
        int e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u] = route_expert_of(routing, base + 32 * u + lane, w1, experts);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e[u] >= 0) atomicAdd(&s_at[warp][e[u]], 1);
    }
    __syncthreads();
    // ... running sum from the expert's first row and the rows of the segments before this one ...
    if (tid < experts) {
        int at = s_first[tid] + before;
        for (int w = 0; w < ROUTE_WARPS; ++w) {
            const int n = s_at[w][tid];
            s_at[w][tid] = at;
            at += n;
        }
    }
    __syncthreads();
    // ... and place
    int e_next = route_expert_of(routing, w0 + lane, w1, experts);
    for (int base = w0; base < w1; base += 32) {
        const int p = base + lane, e = e_next;
        e_next = route_expert_of(routing, p + 32, w1, experts);      // the next round's load overlaps this round's work
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        const int rank = __popc(same & ((1u << lane) - 1u));
        int row = -1;
        if (e >= 0) row = s_at[warp][e] + rank;
        __syncwarp();
        if (e >= 0 && rank == 0) s_at[warp][e] += __popc(same);
        __syncwarp();
        if (p < w1) {
            pair_row[p] = row;
            pair_expert[p] = e;
            if (e >= 0) {
                const int t = p / top_k;
                row_token[row] = t;
                row_expert[row] = e;
                // (non-negative floats order like their bit patterns)
                if (token_max != nullptr) atomicMax(&s_max[e], __float_as_int(ld_float(token_max + t)));
            }
        }
    }
    if (token_max != nullptr) {
        __syncthreads();
        if (tid < experts && s_max[tid] > 0) atomicMax(reinterpret_cast<int *>(amax + tid), s_max[tid]);
    }
}

// Threads per CTA for rows of `chunks` 16-byte pieces: the multiple of 32 up to 256 that leaves the fewest
// idle threads in a row's last round (the larger on a tie).
inline unsigned threads_for(int chunks) {
    unsigned best = 256;
    double best_eff = 0.0;
    for (unsigned t = 64; t <= 256; t += 32) {
        const double eff = static_cast<double>(chunks) / (static_cast<double>((chunks + t - 1) / t) * t);
        if (eff >= best_eff) { best_eff = eff; best = t; }
    }
    return best;
}

inline bool aligned16(const void *p, int64_t ld_bytes) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld_bytes % 16 == 0;
}

// The units of `rows` rows of `chunks` 16-byte pieces: whole rows where those occupy every resident warp, else segments of
// at least 128 pieces (shorter ones only meet at the per-expert maxima); at most one wave of CTAs (a warp takes units in turn).
inline RowUnits row_units(int64_t rows, int chunks, int ctas_per_sm, unsigned *grid) {
    const int64_t warps = 148 * static_cast<int64_t>(ctas_per_sm) * (ROW_THREADS / 32);
    int64_t segs = (warps + rows - 1) / rows;
    const int64_t most = (chunks + 127) / 128;
    segs = segs < 1 ? 1 : (segs > most ? most : segs);
    RowUnits u{};
    u.rows = static_cast<int>(rows);
    u.seg_chunks = static_cast<int>(((chunks + segs - 1) / segs + 31) / 32 * 32);
    u.segs = (chunks + u.seg_chunks - 1) / u.seg_chunks;
    const int64_t ctas = (rows * u.segs + ROW_THREADS / 32 - 1) / (ROW_THREADS / 32), cap = 148 * static_cast<int64_t>(ctas_per_sm);
    *grid = static_cast<unsigned>(ctas < cap ? ctas : cap);
    return u;
}

// The (token, slot) pairs in whose order the one-call form visits the rows in use.
struct PairOrder { const int32_t *row, *expert; int64_t pairs; int top_k; };

}  // namespace
}  // namespace fos

static int gather_rows(const void *x, int dtype, int64_t ld_x, const int32_t *row_token, void *out, int64_t ld_out,
                       int64_t rows_capacity, int64_t cols, const int32_t *row_expert, float *amax,
                       const fos::PairOrder *order, void *stream_) {
    using namespace fos;
    if (!x || !row_token || !out || rows_capacity <= 0 || cols <= 0 || ld_x < cols || ld_out < cols) return FOS_ERR_INVALID_ARGUMENT;
    if ((amax != nullptr) != (row_expert != nullptr)) return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_UNSUPPORTED;
    if (cols % 8 != 0 || rows_capacity >= (int64_t(1) << 31)) return FOS_ERR_UNSUPPORTED;
    if (!aligned16(x, ld_x * 2) || !aligned16(out, ld_out * 2)) return FOS_ERR_MISALIGNED;
    const int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    unsigned g = 0;
    RowUnits units = row_units(order ? order->pairs : rows_capacity, static_cast<int>(cols / 8), GATHER_CTAS, &g);
    if (order) { units.pair_row = order->row; units.pair_expert = order->expert; units.top_k = order->top_k; }
    if (dtype == FOS_BF16)
        FOS_CUDA_TRY(launch_dependent(gather_rows_kernel<__nv_bfloat16>, dim3(g), ROW_THREADS, 0, stream,
            static_cast<const uint8_t *>(x), ld_x * 2, row_token,
            static_cast<uint8_t *>(out), ld_out * 2, units,
            static_cast<int>(cols / 8), row_expert, amax));
    else
        FOS_CUDA_TRY(launch_dependent(gather_rows_kernel<__half>, dim3(g), ROW_THREADS, 0, stream,
            static_cast<const uint8_t *>(x), ld_x * 2, row_token,
            static_cast<uint8_t *>(out), ld_out * 2, units,
            static_cast<int>(cols / 8), row_expert, amax));
    return FOS_OK;
}

extern "C" int fos_experts_gather_rows(const void *x, int dtype, int64_t ld_x, const int32_t *row_token, void *out,
                                       int64_t ld_out, int64_t rows_capacity, int64_t cols, const int32_t *row_expert,
                                       float *amax, void *stream) {
    return gather_rows(x, dtype, ld_x, row_token, out, ld_out, rows_capacity, cols, row_expert, amax, nullptr, stream);
}

static int experts_glu(const void *gate_up, int dtype, int64_t ld_gate_up, const void *bias, const int32_t *row_expert, void *out,
                       int64_t ld_out, int64_t rows_capacity, int64_t intermediate, float alpha, float limit, float *amax,
                       const fos::PairOrder *order, void *stream_) {
    using namespace fos;
    if (!gate_up || !bias || !row_expert || !out || rows_capacity <= 0 || intermediate <= 0 ||
        ld_gate_up < 2 * intermediate || ld_out < intermediate)
        return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_UNSUPPORTED;
    if (intermediate % 8 != 0 || rows_capacity >= (int64_t(1) << 31)) return FOS_ERR_UNSUPPORTED;
    if (!aligned16(gate_up, ld_gate_up * 2) || !aligned16(out, ld_out * 2) || !aligned16(bias, 2 * intermediate * 2))
        return FOS_ERR_MISALIGNED;
    const int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    unsigned g = 0;
    const int chunks = static_cast<int>(intermediate / 8);
    RowUnits units = row_units(order ? order->pairs : rows_capacity, chunks, GLU_CTAS, &g);
    if (order) { units.pair_row = order->row; units.pair_expert = order->expert; units.top_k = order->top_k; }
    if (dtype == FOS_BF16)
        FOS_CUDA_TRY(launch_dependent(glu_kernel<__nv_bfloat16>, dim3(g), ROW_THREADS, 0, stream,
            static_cast<const uint8_t *>(gate_up), ld_gate_up * 2,
            static_cast<const uint8_t *>(bias), 2 * intermediate * 2, row_expert,
            static_cast<uint8_t *>(out), ld_out * 2, units, chunks, alpha, limit, amax));
    else
        FOS_CUDA_TRY(launch_dependent(glu_kernel<__half>, dim3(g), ROW_THREADS, 0, stream,
            static_cast<const uint8_t *>(gate_up), ld_gate_up * 2,
            static_cast<const uint8_t *>(bias), 2 * intermediate * 2, row_expert,
            static_cast<uint8_t *>(out), ld_out * 2, units, chunks, alpha, limit, amax));
    return FOS_OK;
}

extern "C" int fos_experts_glu(const void *gate_up, int dtype, int64_t ld_gate_up, const void *bias, const int32_t *row_expert,
                               void *out, int64_t ld_out, int64_t rows_capacity, int64_t intermediate, float alpha,
                               float limit, float *amax, void *stream) {
    return experts_glu(gate_up, dtype, ld_gate_up, bias, row_expert, out, ld_out, rows_capacity, intermediate, alpha, limit, amax,
                       nullptr, stream);
}

extern "C" int fos_experts_combine(const void *y, int dtype, int64_t ld_y, const void *bias, const int32_t *pair_row,
                                   const int32_t *pair_expert, const void *pair_weight, int top_k, void *out,
                                   int64_t ld_out, int64_t tokens, int64_t hidden, void *stream_) {
    using namespace fos;
    if (!y || !bias || !pair_row || !pair_expert || !pair_weight || !out || tokens <= 0 || hidden <= 0 || top_k <= 0 ||
        ld_y < hidden || ld_out < hidden)
        return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_UNSUPPORTED;
    if (top_k > MAX_TOP_K || hidden % 8 != 0 || tokens >= (int64_t(1) << 31)) return FOS_ERR_UNSUPPORTED;
    if (!aligned16(y, ld_y * 2) || !aligned16(out, ld_out * 2) || !aligned16(bias, hidden * 2)) return FOS_ERR_MISALIGNED;
    const int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const unsigned g = static_cast<unsigned>(tokens < 148 * 8 ? tokens : 148 * 8);
    const int n = static_cast<int>(tokens), chunks = static_cast<int>(hidden / 8);
    if (dtype == FOS_BF16)
        FOS_CUDA_TRY(launch_dependent(combine_kernel<__nv_bfloat16>, dim3(g), threads_for(chunks), 0, stream,
            static_cast<const uint8_t *>(y), ld_y * 2,
            static_cast<const uint8_t *>(bias), hidden * 2, pair_row, pair_expert,
            static_cast<const uint16_t *>(pair_weight), top_k,
            static_cast<uint8_t *>(out), ld_out * 2, n, chunks));
    else
        FOS_CUDA_TRY(launch_dependent(combine_kernel<__half>, dim3(g), threads_for(chunks), 0, stream,
            static_cast<const uint8_t *>(y), ld_y * 2,
            static_cast<const uint8_t *>(bias), hidden * 2, pair_row, pair_expert,
            static_cast<const uint16_t *>(pair_weight), top_k,
            static_cast<uint8_t *>(out), ld_out * 2, n, chunks));
    return FOS_OK;
}

// fos_experts_route; with `amax` also zeroes amax[0 .. 2 * num_experts), and with `maxima` then raises the first num_experts to the
// largest magnitudes of the experts' tokens.
static int experts_route(const void *routing_indices, int index_bytes, int64_t tokens, int top_k, int num_experts,
                         int64_t rows_capacity, int32_t *group_start, int32_t *group_rows, int32_t *row_token,
                         int32_t *row_expert, int32_t *pair_row, int32_t *pair_expert, int32_t *workspace, float *amax,
                         const fos::TokenMaxima &maxima, int x_dtype, void *stream_) {
    using namespace fos;
    if (!routing_indices || !group_start || !group_rows || !row_token || !row_expert || !pair_row || !pair_expert ||
        !workspace || tokens <= 0 || top_k <= 0 || num_experts <= 0 || (index_bytes != 4 && index_bytes != 8))
        return FOS_ERR_INVALID_ARGUMENT;
    if (num_experts > ROUTE_MAX_EXPERTS) return FOS_ERR_UNSUPPORTED;
    const int64_t pairs64 = tokens * top_k;
    if (pairs64 >= (int64_t(1) << 30) || rows_capacity >= (int64_t(1) << 31)) return FOS_ERR_TOO_LARGE;
    if (rows_capacity % 128 != 0 || rows_capacity < round_up64(pairs64 + 127 * static_cast<int64_t>(num_experts), 128))
        return FOS_ERR_INVALID_ARGUMENT;
    const int st = check_device();
    if (st != FOS_OK) return st;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    // segments of at least 512 pairs, at most ROUTE_MAX_SEGMENTS of them
    const int pairs = static_cast<int>(pairs64), cap = static_cast<int>(rows_capacity);
    int segments = (pairs + 511) / 512;
    if (segments > ROUTE_MAX_SEGMENTS) segments = ROUTE_MAX_SEGMENTS;
    const int seg = (pairs + segments - 1) / segments;
    segments = (pairs + seg - 1) / seg;
    // (the tokens' maxima: a warp each, one wave at most)
    const int token_ctas = !maxima.x ? 0 : (maxima.tokens < 148 * 6 * ROUTE_WARPS ? (maxima.tokens + ROUTE_WARPS - 1) / ROUTE_WARPS : 148 * 6);
    auto launch = [&](auto *idx, auto element) -> int {
        using IDX = std::remove_const_t<std::remove_pointer_t<decltype(idx)>>;
        using T = decltype(element);
        FOS_CUDA_TRY(launch_dependent(route_count_kernel<IDX, T>, dim3(segments + token_ctas), ROUTE_THREADS, 0, stream, idx, pairs, seg,
                                      segments, num_experts, cap, workspace, row_token, row_expert, amax, maxima));
        FOS_CUDA_TRY(launch_dependent(route_place_kernel<IDX>, dim3(segments), ROUTE_THREADS, 0, stream, idx, pairs, seg, top_k,
                                      num_experts, workspace, group_start, group_rows, row_token, row_expert, pair_row,
                                      pair_expert, maxima.of_token, amax));
        return FOS_OK;
    };
    auto launch_index = [&](auto *idx) { return x_dtype == FOS_FP16 ? launch(idx, __half{}) : launch(idx, __nv_bfloat16{}); };
    return index_bytes == 8 ? launch_index(static_cast<const int64_t *>(routing_indices))
                            : launch_index(static_cast<const int32_t *>(routing_indices));
}

extern "C" int fos_experts_route(const void *routing_indices, int index_bytes, int64_t tokens, int top_k, int num_experts,
                                 int64_t rows_capacity, int32_t *group_start, int32_t *group_rows, int32_t *row_token,
                                 int32_t *row_expert, int32_t *pair_row, int32_t *pair_expert, int32_t *workspace,
                                 void *stream) {
    return experts_route(routing_indices, index_bytes, tokens, top_k, num_experts, rows_capacity, group_start, group_rows,
                         row_token, row_expert, pair_row, pair_expert, workspace, nullptr, fos::TokenMaxima{}, FOS_BF16, stream);
}

// ---------------------------------------------------------------------------- the whole layer in one call

namespace fos {
namespace {

struct ExpertsWorkspace {
    int64_t capacity, pairs;
    // byte offsets into the workspace, each a multiple of 256
    int64_t group_start, group_rows, row_token, row_expert, pair_row, pair_expert, route_work, amax, token_max;
    int64_t rows_x, codes_x, sf_x, gate_up, gated, codes_g, sf_g, y, total;
    int64_t apart;          // the bytes that rows_x, gate_up and y would take beyond these in places of their own
};

ExpertsWorkspace experts_workspace(int64_t tokens, int top_k, int num_experts, int64_t hidden, int64_t intermediate) {
    ExpertsWorkspace w{};
    w.pairs = tokens * top_k;
    w.capacity = round_up64(w.pairs + 127 * static_cast<int64_t>(num_experts), 128);
    int64_t at = 0;
    auto take = [&](int64_t bytes) { const int64_t here = at; at += round_up64(bytes, 256); return here; };
    w.group_start = take(4 * (num_experts + 1));
    w.group_rows = take(4 * num_experts);
    w.row_token = take(4 * w.capacity);
    w.row_expert = take(4 * w.capacity);
    w.pair_row = take(4 * w.pairs);
    w.pair_expert = take(4 * w.pairs);
    w.route_work = take(4 * static_cast<int64_t>(FOS_EXPERTS_ROUTE_WORKSPACE_INTS) * num_experts);
    w.amax = take(4 * 2 * num_experts);
    w.token_max = take(4 * tokens);
    // rows_x, gate_up and y share their place: a kernel that writes one of them writes behind its wait for the kernel before it,
    // which read, or came behind one that read, the last of the one before. (The default path writes y only.)
    const int64_t rows_bytes = round_up64(2 * w.capacity * hidden, 256), gate_up_bytes = round_up64(4 * w.capacity * intermediate, 256);
    w.rows_x = w.gate_up = w.y = take(rows_bytes > gate_up_bytes ? rows_bytes : gate_up_bytes);
    w.apart = rows_bytes + (rows_bytes > gate_up_bytes ? gate_up_bytes : rows_bytes);
    w.codes_x = take(w.capacity * hidden / 2);
    w.sf_x = take(w.capacity * hidden / 16);
    w.gated = take(2 * w.capacity * intermediate);
    w.codes_g = take(w.capacity * intermediate / 2);
    w.sf_g = take(w.capacity * intermediate / 16);
    w.total = at;
    return w;
}

}  // namespace
}  // namespace fos

extern "C" int64_t fos_experts_forward_workspace_bytes(int64_t tokens, int top_k, int num_experts, int64_t hidden, int64_t intermediate) {
    if (tokens <= 0 || top_k <= 0 || num_experts <= 0 || hidden <= 0 || intermediate <= 0) return FOS_ERR_INVALID_ARGUMENT;
    return fos::experts_workspace(tokens, top_k, num_experts, hidden, intermediate).total;
}

extern "C" int64_t fos_experts_workspace_bytes(int64_t tokens, int top_k, int num_experts, int64_t hidden, int64_t intermediate) {
    if (tokens <= 0 || top_k <= 0 || num_experts <= 0 || hidden <= 0 || intermediate <= 0) return FOS_ERR_INVALID_ARGUMENT;
    const fos::ExpertsWorkspace w = fos::experts_workspace(tokens, top_k, num_experts, hidden, intermediate);
    return w.total + w.apart;
}

extern "C" int fos_experts_forward(const void *x, int dtype, int64_t tokens, int64_t hidden, int64_t ld_x,
                                   const void *routing_indices, int index_bytes, const void *routing_weights, int top_k,
                                   int num_experts, const uint8_t *gate_up_codes, const uint8_t *gate_up_sf,
                                   const float *gate_up_amax, const void *gate_up_bias, const uint8_t *down_codes,
                                   const uint8_t *down_sf, const float *down_amax, const void *down_bias,
                                   int64_t intermediate, int weight_rule, int activation_rule, float alpha, float limit,
                                   void *out, int64_t ld_out, void *workspace, int64_t workspace_bytes, int32_t *status,
                                   void *stream_) {
    using namespace fos;
    if (!x || !routing_indices || !routing_weights || !gate_up_codes || !gate_up_sf || !gate_up_amax || !gate_up_bias ||
        !down_codes || !down_sf || !down_amax || !down_bias || !out || !workspace || tokens <= 0 || hidden <= 0 ||
        intermediate <= 0 || top_k <= 0 || num_experts <= 0)
        return FOS_ERR_INVALID_ARGUMENT;
    if (dtype != FOS_BF16 && dtype != FOS_FP16) return FOS_ERR_UNSUPPORTED;
    // whole 64-value scale tiles along both reduction dimensions (the packed weights are then not padded along K)
    if (hidden % 64 != 0 || intermediate % 64 != 0 || num_experts > 256 || top_k > MAX_TOP_K) return FOS_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return FOS_ERR_MISALIGNED;
    const ExpertsWorkspace w = experts_workspace(tokens, top_k, num_experts, hidden, intermediate);
    if (workspace_bytes < w.total) return FOS_ERR_INVALID_ARGUMENT;
    uint8_t *base = static_cast<uint8_t *>(workspace);
    auto ints = [&](int64_t off) { return reinterpret_cast<int32_t *>(base + off); };
    float *amax = reinterpret_cast<float *>(base + w.amax);
    const int64_t gate_up_rows = round_up64(2 * intermediate, 128), down_rows = round_up64(hidden, 128);

    if (ld_x < hidden || ld_out < hidden) return FOS_ERR_INVALID_ARGUMENT;
    if (!aligned16(x, ld_x * 2)) return FOS_ERR_MISALIGNED;
    // the rows are gathered by the quantization where the default rule lets it; then the maxima are the tokens'
    const bool gathered = activation_rule == FOS_RULE_MSE;
    const TokenMaxima maxima = gathered ? TokenMaxima{static_cast<const uint8_t *>(x), ld_x * 2, static_cast<int>(tokens),
                                                      static_cast<int>(hidden / 8), reinterpret_cast<float *>(base + w.token_max)}
                                        : TokenMaxima{};
    int st = experts_route(routing_indices, index_bytes, tokens, top_k, num_experts, w.capacity, ints(w.group_start),
                           ints(w.group_rows), ints(w.row_token), ints(w.row_expert), ints(w.pair_row), ints(w.pair_expert),
                           ints(w.route_work), amax, maxima, dtype, stream_);
    if (st != FOS_OK) return st;
    const PairOrder order{ints(w.pair_row), ints(w.pair_expert), w.pairs, top_k};
    st = gathered ? quantize_grouped_gathered(x, dtype, tokens, hidden, ld_x, ints(w.row_token), w.capacity, activation_rule,
                                              ints(w.group_start), ints(w.group_rows), num_experts, amax, base + w.codes_x,
                                              base + w.sf_x, stream_)
                  : FOS_ERR_UNSUPPORTED;
    if (st == FOS_ERR_UNSUPPORTED) {
        st = gather_rows(x, dtype, ld_x, ints(w.row_token), base + w.rows_x, hidden, w.capacity, hidden, ints(w.row_expert), amax,
                         &order, stream_);
        if (st != FOS_OK) return st;
        st = quantize_grouped_rows_in_use(base + w.rows_x, dtype, w.capacity, hidden, hidden, FOS_NVFP4, activation_rule, ints(w.group_start),
                                          ints(w.group_rows), num_experts, amax, base + w.codes_x, base + w.sf_x, amax, 0, stream_);
    }
    if (st != FOS_OK) return st;
    const float denom = alpha_divisor(FOS_NVFP4, activation_rule, FOS_NVFP4, weight_rule);
    // the SwiGLU in the GEMM's epilogue where that GEMM runs on CTA pairs, else in a kernel of its own
    const GemmScales gate_up_scales{amax, gate_up_amax, denom, nullptr, true};
    const GluEpilogue glu{gate_up_bias, alpha, limit, amax + num_experts};
    st = gemm_nvfp4_grouped_glu(base + w.codes_x, base + w.sf_x, gate_up_codes, gate_up_sf, gate_up_scales, glu, base + w.gated, dtype,
                                ints(w.group_start), ints(w.group_rows), num_experts, w.capacity, gate_up_rows, hidden,
                                2 * intermediate, intermediate, status, stream_);
    if (st == FOS_ERR_UNSUPPORTED) {
        st = gemm_nvfp4_grouped_scaled(base + w.codes_x, base + w.sf_x, gate_up_codes, gate_up_sf, gate_up_scales, base + w.gate_up, dtype,
                                       ints(w.group_start), ints(w.group_rows), num_experts, w.capacity, gate_up_rows, hidden,
                                       2 * intermediate, 2 * intermediate, status, stream_);
        if (st != FOS_OK) return st;
        st = experts_glu(base + w.gate_up, dtype, 2 * intermediate, gate_up_bias, ints(w.row_expert), base + w.gated, intermediate,
                         w.capacity, intermediate, alpha, limit, amax + num_experts, &order, stream_);
    }
    if (st != FOS_OK) return st;
    st = quantize_grouped_rows_in_use(base + w.gated, dtype, w.capacity, intermediate, intermediate, FOS_NVFP4, activation_rule,
                              ints(w.group_start), ints(w.group_rows), num_experts, amax + num_experts, base + w.codes_g,
                              base + w.sf_g, amax + num_experts, 0, stream_);
    if (st != FOS_OK) return st;
    st = gemm_nvfp4_grouped_scaled(base + w.codes_g, base + w.sf_g, down_codes, down_sf, {amax + num_experts, down_amax, denom, nullptr, true},
                                   base + w.y, dtype, ints(w.group_start), ints(w.group_rows), num_experts, w.capacity,
                                   down_rows, intermediate, hidden, hidden, status, stream_);
    if (st != FOS_OK) return st;
    return fos_experts_combine(base + w.y, dtype, hidden, down_bias, ints(w.pair_row), ints(w.pair_expert), routing_weights,
                               top_k, out, ld_out, tokens, hidden, stream_);
}
