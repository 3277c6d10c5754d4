// Search-side kernels: query preparation, allow-mask utilities, the block scans and top-k selection.
//
// Reference path restated: search::search (turbovec/src/search.rs:3206-4353):
//   rotate queries (:3237-3242) -> TQ+ inverse (:3154-3186) -> per-query tables (:2856-2994, :2806-2846)
//   -> block scan with whole-block mask skip (:3015-3029) and per-vector scale -> top-k under the order
//   (score desc, slot asc) (:236-252, :4285-4298).
// Integer sums are exact here as they are in every reference kernel; the float epilogue reproduces the
// reference's rounding sequence for the selected score mode.
#include <algorithm>

#include "search.cuh"

#include <cfloat>

#include "rotation.cuh"
#include "scan_common.cuh"

namespace tv {
namespace {

// =====================================================================================================
// Query preparation: one CTA per query.
// =====================================================================================================
__device__ __forceinline__ float block_max(float v, float *red, int tid, int nthreads) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFullMask, v, o));
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    float r = red[0];
    for (int w = 1; w < (nthreads >> 5); ++w) r = fmaxf(r, red[w]);
    __syncthreads();
    return r;
}

__device__ __forceinline__ int8_t round_clamp_i8(float v) {
    float r = roundf(v);                       // half away from zero, as Rust's f32::round
    r = fminf(fmaxf(r, -127.0f), 127.0f);
    return int8_t(int(r));
}

// One CTA prepares one query; with few queries nothing else runs, so the length of its dependent chain is the cost.
// The blocks of the rotation are spread over the warps, the tables of a half-byte (16 entries) belong to one thread,
// which computes its entries from the products of its coordinates and stores them as one word, and the sequential bias
// sum runs beside the table entries.  One query: dim 1536 4-bit 12.8 us before, dim 3072 2-bit 105 us before.
// The CTA also resets its query's selection state and clears the operand padding that the tensor-memory scans read
// (CTAs past the last query clear a whole row).
constexpr int kPrepThreads = 256;

template <int BITS>
__device__ __forceinline__ void half_entries(const float *q, const float *centroids, float (&e)[16]) {
    // entry = sum over the nibble's coordinates of q[d] * centroid[code] (f32, coordinate order, separately rounded)
    if constexpr (BITS == 2) {
        float p0[4], p1[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) { p0[c] = __fadd_rn(0.0f, __fmul_rn(q[0], centroids[c])); p1[c] = __fmul_rn(q[1], centroids[c]); }
#pragma unroll
        for (int nib = 0; nib < 16; ++nib) e[nib] = __fadd_rn(p0[nib >> 2], p1[nib & 3]);
    } else {
#pragma unroll
        for (int nib = 0; nib < 16; ++nib) e[nib] = __fadd_rn(0.0f, __fmul_rn(q[0], centroids[nib & ((1 << BITS) - 1)]));
    }
}

// Coordinate whose level the expansion of a filtering scan (scan_tc.cu, kLevels2 / kLevels3) puts at byte b of word i of a
// row: 16-byte chunk c of a 128-byte slab holds the byte-groups c, c + 8, c + 16, ... of the slab.
template <int BITS>
__device__ __forceinline__ int filter_coord(int i, int b) {
    const int slab = i >> 5, c = (i >> 2) & 7, w = i & 3;
    if constexpr (BITS == 2) {                                      // words 0, 1: coordinates 3 and 1 of two groups; 2, 3: 2 and 0
        const int group = c + 8 * ((w & 1) * 2 + (b >> 1));
        return slab * 128 + 4 * group + (w < 2 ? ((b & 1) ? 1 : 3) : ((b & 1) ? 0 : 2));
    } else {                                                        // two groups a word, coordinate 1 before coordinate 0
        const int group = c + 8 * (2 * w + (b >> 1));
        return slab * 128 + 2 * group + ((b & 1) ^ 1);
    }
}

// The u8 tables of a query and, for a filtering scan (scan_filter.cu), its int8 weights and the affine bound
//   isum <= alpha * sum_d W[d] * L[code[d]] + beta + D,   with the equality's two sides at most D apart,
// beta and D summed over the half-bytes from the extremes of U - alpha * (W . L) over the entries.  The entries' deviation
// is evaluated in f32 (values up to 127: 5e-5 covers it) and summed in f64; 1e-5 of the reference's own bias covers the
// roundings of its float epilogue, whose terms are that large before they cancel.
template <int BITS>
__device__ void lut_tables(const QueryPrepParams &p, const float *row, float *dev, float *mins, const float *centroids, float *red, int q, float bias_corr) {
    __shared__ double part[2][kPrepThreads / 32];
    __shared__ double batch_sum[kFilterBatches];
    __shared__ float s_bias;
    constexpr int kCoords = BITS == 2 ? 2 : 1;                     // per half-byte: 8 / BITS / 2
    const int ng = p.ngroups, tid = threadIdx.x;
    float span = 0.0f;
    for (int h = tid; h < 2 * ng; h += blockDim.x) {               // h = 2*g + half
        float e[16];
        half_entries<BITS>(row + h * kCoords, centroids, e);
        float mn = FLT_MAX, mx = -FLT_MAX;
#pragma unroll
        for (int nib = 0; nib < 16; ++nib) {
            if (e[nib] < mn) mn = e[nib];
            if (e[nib] > mx) mx = e[nib];
        }
        mins[h] = mn;
        span = fmaxf(span, __fsub_rn(mx, mn));
    }
    const float max_span = block_max(span, red, tid, blockDim.x);
    float scale = max_span > 0.0f ? __fdiv_rn(max_span, 127.0f) : 1.0f;
    float inv_scale;
    if (scale >= FLT_MIN) inv_scale = __fdiv_rn(1.0f, scale);
    else { scale = 1.0f; inv_scale = 1.0f; }
    const bool filter = BITS != 4 && p.filter.weights != nullptr;
    float w_scale = 1.0f, w_inv = 1.0f, alpha = 0.0f;
    if (filter) {
        float m = 0.0f;
        for (int d = tid; d < p.dim; d += blockDim.x) m = fmaxf(m, fabsf(row[d]));
        m = block_max(m, red, tid, blockDim.x);
        w_scale = __fdiv_rn(m, 127.0f);
        if (w_scale >= FLT_MIN) w_inv = __fdiv_rn(1.0f, w_scale);
        else w_scale = 1.0f;
        alpha = __fdiv_rn(__fmul_rn(w_scale, p.level_scale), scale);
    }
    double beta = 0.0, slack = 0.0;
    if (tid < 32) {
        if (tid == 0) {
            float bias = 0.0f;                                      // sequential in g (search.rs:2910)
            const float2 *m2 = reinterpret_cast<const float2 *>(mins);
#pragma unroll 16
            for (int g = 0; g < ng; ++g) bias = __fadd_rn(bias, __fadd_rn(m2[g].x, m2[g].y));
            p.qscale[q] = scale;
            s_bias = p.qbias[q] = __fadd_rn(bias, bias_corr);       // search.rs:3260
        }
    } else {
        uint4 *lut = reinterpret_cast<uint4 *>(p.luts + size_t(q) * p.lut_pitch);
        for (int h = tid - 32; h < 2 * ng; h += blockDim.x - 32) {
            float e[16];
            half_entries<BITS>(row + h * kCoords, centroids, e);
            const float mn = mins[h];
            uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int nib = 0; nib < 16; ++nib) {
                float r = roundf(__fmul_rn(__fsub_rn(e[nib], mn), inv_scale));
                r = fminf(fmaxf(r, 0.0f), 127.0f);
                e[nib] = r;
                w[nib >> 2] |= uint32_t(int(r)) << (8 * (nib & 3));
            }
            lut[h] = make_uint4(w[0], w[1], w[2], w[3]);
            if constexpr (BITS != 4) {
                if (filter) {
                    float wt[2];
                    for (int c = 0; c < kCoords; ++c) wt[c] = alpha * float(round_clamp_i8(__fmul_rn(row[h * kCoords + c], w_inv)));
                    float lo = FLT_MAX, hi = -FLT_MAX;
#pragma unroll
                    for (int nib = 0; nib < (BITS == 3 ? 8 : 16); ++nib) {
                        const float fit = BITS == 2 ? wt[0] * float(p.filter.levels[nib >> 2]) + wt[1] * float(p.filter.levels[nib & 3])
                                                    : wt[0] * float(p.filter.levels[nib]);
                        lo = fminf(lo, e[nib] - fit);
                        hi = fmaxf(hi, e[nib] - fit);
                    }
                    dev[h] = hi + 5e-5f;
                    beta += 0.5 * (double(hi) + double(lo));
                    slack += 0.5 * (double(hi) - double(lo)) + 5e-5;
                }
            }
        }
        if (p.pad_operands)                                         // groups past the last one, up to a whole K slab
            for (int h = 2 * ng + tid - 32; h < p.lut_pitch / 16; h += blockDim.x - 32) lut[h] = make_uint4(0, 0, 0, 0);
    }
    if (!filter) return;
    uint32_t *wrow = reinterpret_cast<uint32_t *>(p.filter.weights + size_t(q) * p.dim_pad);
    for (int i = tid; i < p.dim_pad / 4; i += blockDim.x) {
        uint32_t word = 0;
        for (int b = 0; b < 4; ++b) {
            const int d = filter_coord<BITS == 2 ? 2 : 3>(i, b);
            if (d < p.dim) word |= uint32_t(uint8_t(round_clamp_i8(__fmul_rn(row[d], w_inv)))) << (8 * b);
        }
        wrow[i] = word;
    }
    for (int o = 16; o > 0; o >>= 1) {
        beta += __shfl_xor_sync(kFullMask, beta, o);
        slack += __shfl_xor_sync(kFullMask, slack, o);
    }
    if ((tid & 31) == 0) { part[0][tid >> 5] = beta; part[1][tid >> 5] = slack; }
    __syncthreads();
    // suffix sums of the largest deviations by batches of byte-groups
    const int batches = (ng + kFilterBatch - 1) / kFilterBatch;
    for (int b = tid >> 5; b < batches; b += kPrepThreads / 32) {
        double sum = 0.0;
        for (int h = 2 * kFilterBatch * b + (tid & 31); h < min(2 * kFilterBatch * (b + 1), 2 * ng); h += 32) sum += double(dev[h]);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFullMask, sum, o);
        if ((tid & 31) == 0) batch_sum[b] = sum;
    }
    __syncthreads();
    if (tid == 0) {
        beta = slack = 0.0;
        for (int w = 0; w < kPrepThreads / 32; ++w) { beta += part[0][w]; slack += part[1][w]; }
        const double base = double(scale) * beta + double(s_bias);
        // a scale of zero marks a zero query: its scores are all zero, and the smallest slots win (bootstrap_kernel)
        p.filter.scale[q] = !(max_span > 0.0f) && s_bias == 0.0f ? 0.0f : fmaxf(float(double(scale) * double(alpha)), 1e-45f);
        double rest = 0.0;
        float *suffix = p.filter.suffix + size_t(q) * kFilterBatches;
        suffix[batches] = 0.0f;
        for (int b = batches - 1; b >= 0; --b) { rest += batch_sum[b]; suffix[b] = float(rest + 1e-2 + 1e-6 * fabs(rest)); }
        p.filter.alpha[q] = alpha;
        p.filter.bias_mid[q] = float(base);
        p.filter.bias_max[q] = float(base + double(scale) * slack * 1.000001 + 1e-5 * fabs(double(s_bias)));
    }
}

template <int LOG2B>
__global__ void __launch_bounds__(kPrepThreads) query_prep_kernel(QueryPrepParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int dim = p.dim, ng = p.ngroups, stride = dim + 8;
    float *rowA = reinterpret_cast<float *>(smem_raw);
    float *rowB = rowA + stride;
    uint16_t *perm0 = reinterpret_cast<uint16_t *>(rowB + stride);
    uint16_t *perm1 = perm0 + dim;
    float *mins = reinterpret_cast<float *>(perm0);     // reused after the rotation: 2*ng floats <= 4*dim bytes
    __shared__ float red[kPrepThreads / 32];
    __shared__ float s_scalar[2];
    __shared__ float s_centroids[16];

    const int q = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (q >= p.nq) {                                    // operand rows past the last query
        uint4 *row = reinterpret_cast<uint4 *>(p.mode == kModePermuteDot ? reinterpret_cast<uint8_t *>(p.weights) + size_t(q) * p.dim_pad
                                                                         : p.luts + size_t(q) * p.lut_pitch);
        const int words = (p.mode == kModePermuteDot ? p.dim_pad : p.lut_pitch) / 16;
        for (int i = tid; i < words; i += kPrepThreads) row[i] = make_uint4(0, 0, 0, 0);
        if (p.mode != kModePermuteDot && p.filter.weights != nullptr) {
            uint4 *w = reinterpret_cast<uint4 *>(p.filter.weights + size_t(q) * p.dim_pad);
            for (int i = tid; i < p.dim_pad / 16; i += kPrepThreads) w[i] = make_uint4(0, 0, 0, 0);
        }
        return;
    }
    if (p.cnt != nullptr) {
        if (tid == 0) { p.cnt[q] = 0; p.done[q] = 0; p.thr[q] = kEmptyKey; if (p.over != nullptr) { p.over[q] = 0; if (q == 0) { p.over[p.nq] = 0; p.over[p.nq + 1] = 0; p.over[p.nq + 2] = 0; p.over[p.nq + 3] = 0; } } if (q == 0) p.done[p.nq] = 0; }
        for (int i = tid; i < p.k; i += kPrepThreads) p.topk[size_t(q) * p.k + i] = kEmptyKey;
    }
    const float *src = p.queries + size_t(q) * dim;
    for (int i = tid; i < dim; i += kPrepThreads) {
        const float v = src[i];
        rowA[i] = v;
        if (!(fabsf(v) < 1e16f)) atomicMin(p.first_invalid, (unsigned long long)(size_t(q) * dim + i));
    }
    // both tables, 16 bytes at a time (dim is a multiple of 8)
    for (int i = tid; i < dim / 4; i += kPrepThreads) reinterpret_cast<uint4 *>(perm0)[i] = reinterpret_cast<const uint4 *>(p.perms)[i];
    if (tid < 16) s_centroids[tid] = tid < (1 << p.bits) ? p.centroids[tid] : 0.0f;
    __syncthreads();
    // Rotation::apply: no normalisation (search.rs:3237-3242)
    rotation_round<LOG2B>(rowA, rowB, perm0, dim, p.inv_sqrt_block, false, 1.0f, lane, warp, kPrepThreads / 32);
    __syncthreads();
    rotation_round<LOG2B>(rowB, rowA, perm1, dim, p.inv_sqrt_block, false, 1.0f, lane, warp, kPrepThreads / 32);
    __syncthreads();

    // TQ+ inverse (search.rs:3154-3186): q[d] / scale[d]; bias correction = -(sum q[d]*shift[d]) in f64,
    // accumulated sequentially in d.
    float bias_corr = 0.0f;
    if (p.shift != nullptr) {
        if (tid == 0) {
            double bc = 0.0;
            for (int d = 0; d < dim; ++d) bc = __dsub_rn(bc, __dmul_rn(double(rowA[d]), double(p.shift[d])));
            s_scalar[0] = __double2float_rn(bc);
        }
        __syncthreads();
        bias_corr = s_scalar[0];
        for (int d = tid; d < dim; d += kPrepThreads) rowA[d] = __fdiv_rn(rowA[d], p.scale_tq[d]);
        __syncthreads();
    }

    if (p.q_rot != nullptr)
        for (int d = tid; d < dim; d += kPrepThreads) p.q_rot[size_t(q) * dim + d] = rowA[d];

    if (p.mode == kModePermuteDot) {
        // search.rs:2806-2846: one scale for the row, weights = clamp(round(q * (1/qs)), +-127)
        float m = 0.0f;
        for (int d = tid; d < dim; d += kPrepThreads) m = fmaxf(m, fabsf(rowA[d]));
        const float qmax = block_max(m, red, tid, kPrepThreads);
        float qs = __fdiv_rn(qmax, 127.0f), inv_qs;
        if (qs >= FLT_MIN) inv_qs = __fdiv_rn(1.0f, qs);
        else { qs = 1.0f; inv_qs = 1.0f; }
        if (tid == 0) {
            p.qscale[q] = __fmul_rn(p.level_scale, qs);
            p.qbias[q] = __fadd_rn(0.0f, bias_corr);
        }
        // four weights to a word, adjacent coordinates swapped (the nibble order of a code byte)
        uint32_t *wrow = reinterpret_cast<uint32_t *>(p.weights + size_t(q) * p.dim_pad);
        const int words = p.pad_operands ? p.dim_pad / 4 : dim / 4;
        for (int i = tid; i < words; i += kPrepThreads) {
            uint32_t word = 0;
            if (4 * i < dim) {
                const float4 v = reinterpret_cast<const float4 *>(rowA)[i];
                word = uint32_t(uint8_t(round_clamp_i8(__fmul_rn(v.y, inv_qs)))) | uint32_t(uint8_t(round_clamp_i8(__fmul_rn(v.x, inv_qs)))) << 8 |
                       uint32_t(uint8_t(round_clamp_i8(__fmul_rn(v.w, inv_qs)))) << 16 | uint32_t(uint8_t(round_clamp_i8(__fmul_rn(v.z, inv_qs)))) << 24;
            }
            wrow[i] = word;
        }
        if (p.wfrag == nullptr) return;
        // mma.sync A fragments.  k-step ks covers byte-groups 16ks..16ks+15; thread t of a quad owns
        // groups 16ks + t + {0,4,8,12}; register byte order follows the nibble order of a code byte
        // (low nibble = odd coordinate 2g+1, high nibble = even coordinate 2g; search.rs:2787-2790).
        const int ksteps = (ng + 15) / 16;
        const int m_tile = q >> 4, rr = q & 15, r = rr & 7, hi_row = rr >> 3;
        for (int idx = tid; idx < ksteps * 8; idx += kPrepThreads) {
            const int ks = idx >> 3, t = (idx >> 1) & 3, half = idx & 1;
            const int ga = 16 * ks + t + 8 * half, gb = ga + 4;
            uint32_t word = 0;
            const int dims[4] = {2 * ga + 1, 2 * ga, 2 * gb + 1, 2 * gb};
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                int8_t w = 0;
                if (dims[b] < dim) w = round_clamp_i8(__fmul_rn(rowA[dims[b]], inv_qs));
                word |= uint32_t(uint8_t(w)) << (8 * b);
            }
            const size_t frag = ((size_t(ks) * p.mtiles_total + m_tile) * 32 + (r * 4 + t)) * 4 + (half * 2 + hi_row);
            p.wfrag[frag] = word;
        }
    } else if (p.bits == 2) {                                       // search.rs:2856-2994
        lut_tables<2>(p, rowA, rowB, mins, s_centroids, red, q, bias_corr);
    } else if (p.bits == 3) {
        lut_tables<3>(p, rowA, rowB, mins, s_centroids, red, q, bias_corr);
    } else {
        lut_tables<4>(p, rowA, rowB, mins, s_centroids, red, q, bias_corr);
    }
}

// =====================================================================================================
// Allow-mask utilities
// =====================================================================================================
__global__ void pack_bool_mask_kernel(const uint8_t *mask_bool, int64_t n, uint32_t *words32) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool on = i < n && mask_bool[i] != 0;
    const unsigned w = __ballot_sync(kFullMask, on);
    if ((threadIdx.x & 31) == 0 && (i >> 5) < ((n + 63) / 64) * 2) words32[i >> 5] = w;
}

__global__ void scatter_slots_kernel(const uint32_t *slots, int64_t count, uint32_t *words32) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count) atomicOr(&words32[slots[i] >> 5], 1u << (slots[i] & 31));
}

__global__ void mask_stats_kernel(uint32_t *words32, int64_t n, unsigned long long *n_allowed, uint32_t *live_blocks,
                                  uint32_t *n_live) {
    const int64_t nblocks = (n + 31) / 32;
    const int64_t b = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    unsigned w = 0;
    if (b < nblocks) {
        w = words32[b];
        const int64_t rem = n - b * 32;
        if (rem < 32) { w &= (1u << rem) - 1u; words32[b] = w; }
    }
    // ordered-within-warp append keeps neighbouring live blocks adjacent in the list
    const unsigned live = __ballot_sync(kFullMask, w != 0);
    unsigned cnt = __popc(w);
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFullMask, cnt, o);
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == 0 && live) {
        base = atomicAdd(n_live, __popc(live));
        atomicAdd(n_allowed, (unsigned long long)cnt);
    }
    base = __shfl_sync(kFullMask, base, 0);
    if (w != 0) live_blocks[base + __popc(live & ((1u << lane) - 1u))] = uint32_t(b);
}

// =====================================================================================================
// Permute-dot scan (4-bit codes): S[q][v] = sum_d W[q][d] * level[code[v][d]], exact in int32
// (search.rs:1392-1543), then fma((f32)S, scale_q, bias_q) * vec_scale[v] (search.rs:1523, 1793).
//
// CTA = 8 consumer warps + 1 producer warp.  A tile is 8 code blocks (256 vectors), one per consumer
// warp.  The producer streams the tile's codes in chunks of kChunkRows byte-group rows per block with
// bulk asynchronous copies into a ring of kStages shared-memory stages (full/empty mbarriers).  A
// consumer turns 16 rows x 4 bytes into the B fragments of four m16n8k32 MMAs: the byte of vector
// 4i+j in row g sits in byte j of the 32-bit word at (g, quad i), so one word feeds the four n-tiles
// j = 0..3 of quad i; nibbles become int8 levels with three byte-permutes per four codes.
// =====================================================================================================
constexpr int kConsumerWarps = 8;
constexpr int kChunkRows = 64;                                // byte-group rows per block per stage
constexpr int kStageBytes = kConsumerWarps * kChunkRows * kLanes;
constexpr int kStages = 4;

template <int MT, bool SPLIT>
__global__ void __launch_bounds__((kConsumerWarps + 1) * 32, MT == 1 ? (SPLIT ? 2 : 3) : (MT == 2 ? 2 : 1))
scan_pd_kernel(ScanParams p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    uint8_t *stage_mem = smem_raw;
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ng = p.ngroups;
    const int n_chunks = (ng + kChunkRows - 1) / kChunkRows;
    uint32_t pos_end = p.pos_end;
    if (p.live_blocks != nullptr) pos_end = min(pos_end, *p.n_live);
    const uint32_t pos_begin = min(p.pos_begin, pos_end);
    const uint32_t n_tiles = (pos_end - pos_begin + kConsumerWarps - 1) / kConsumerWarps;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], kConsumerWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == kConsumerWarps) {
        // ---------------- producer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                const uint32_t pos0 = pos_begin + tile * kConsumerWarps;
                const int nb = int(min(uint32_t(kConsumerWarps), pos_end - pos0));
                for (int ch = 0; ch < n_chunks && ok; ++ch, ++it) {
                    const int s = it % kStages;
                    ok = mbar_wait(&empty_bar[s], ((it / kStages) & 1) ^ 1, p.cb.error);
                    if (!ok) break;
                    const int rows = min(kChunkRows, ng - ch * kChunkRows);
                    const uint32_t bytes = uint32_t(rows) * kLanes;
                    mbar_arrive_expect_tx(&full_bar[s], bytes * nb);
                    for (int w = 0; w < nb; ++w) {
                        const uint32_t blk = p.live_blocks ? p.live_blocks[pos0 + w] : pos0 + w;
                        const uint8_t *src = p.codes + (size_t(blk) * ng + size_t(ch) * kChunkRows) * kLanes;
                        bulk_copy_g2s(stage_mem + size_t(s) * kStageBytes + size_t(w) * kChunkRows * kLanes, src,
                                      bytes, &full_bar[s]);
                    }
                }
            }
            // Drain: every copy this thread issued has to land before the CTA's shared memory is released.
            // The consumers release each stage after reading it, so waiting for the ring to come back
            // empty covers all of them; the wait is bounded like every other.
            for (int d = 0; d < kStages && ok; ++d, ++it)
                ok = mbar_wait(&empty_bar[it % kStages], ((it / kStages) & 1) ^ 1, p.cb.error);
        }
        return;
    }

    // ---------------- consumers ----------------
    const int quad = lane >> 2, t = lane & 3;
    const uint32_t T[4] = {p.level_words[0], p.level_words[1], p.level_words[2], p.level_words[3]};
    const uint32_t Tp[2] = {p.level_words[2], p.level_words[3]};
    const uint32_t Tn[2] = {negate_bytes(p.level_words[0]), negate_bytes(p.level_words[1])};
    const uint4 *wfrag = reinterpret_cast<const uint4 *>(p.wfrag);
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t pos = pos_begin + tile * kConsumerWarps + warp;
        const bool have = pos < pos_end;
        int acc[MT][4][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][j][e] = 0;
        int accn[SPLIT ? MT : 1][4][4];                       // the c < 8 half of the contraction, subtracted at the end
#pragma unroll
        for (int m = 0; m < (SPLIT ? MT : 1); ++m)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) accn[m][j][e] = 0;

        for (int ch = 0; ch < n_chunks; ++ch, ++it) {
            const int s = it % kStages;
            if (!mbar_wait(&full_bar[s], (it / kStages) & 1, p.cb.error)) return;
            if (have) {
                // lane L < 16 addresses matrix row L of the vector half 0..15, lane L >= 16 that of the half 16..31
                const uint32_t rows_addr = smem_addr(stage_mem + size_t(s) * kStageBytes + size_t(warp) * kChunkRows * kLanes) +
                                           uint32_t((((lane & 15) >> 2) + 4 * (lane & 3)) * kLanes + (lane >> 4) * 16);
                const int rows_here = min(kChunkRows, ng - ch * kChunkRows);
                const int ksteps = (rows_here + 15) / 16;
                // query fragments of this chunk's k-steps: one pointer per chunk, constant strides inside
                const uint4 *wf = wfrag + (size_t(ch) * (kChunkRows / 16) * p.mtiles_total + p.mtile_base) * 32 + lane;
                const size_t wf_step = size_t(p.mtiles_total) * 32;
                auto kstep = [&](int ks) {
                    // x[j] = the byte-groups of rows 16ks + t + {0, 4, 8, 12} (bytes 0..3) of vector 8j + quad: the
                    // load unit transposes, matrix row 4t + r being pointed at row t + 4r so that the k order of the
                    // query fragments holds
                    uint32_t x[4];
                    ldmatrix_x2_trans_b8(x, rows_addr + ks * (16 * kLanes));
                    uint32_t b0[4], b1[4], n0[SPLIT ? 4 : 1], n1[SPLIT ? 4 : 1];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if constexpr (SPLIT) expand4_split(x[j], Tp, Tn, b0[j], b1[j], n0[j], n1[j]);
                        else expand4(x[j], T, b0[j], b1[j]);
                    }
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 a = __ldg(wf + ks * wf_step + m * 32);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            mma_s8(acc[m][j], a, b0[j], b1[j]);
                            if constexpr (SPLIT) mma_s8(accn[m][j], a, n0[j], n1[j]);
                        }
                    }
                };
                if (ksteps == kChunkRows / 16) {               // a whole chunk: no loop control, constant offsets
#pragma unroll
                    for (int ks = 0; ks < kChunkRows / 16; ++ks) kstep(ks);
                } else {
                    for (int ks = 0; ks < ksteps; ++ks) kstep(ks);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[s]);
        }

        if (have) {
            const uint32_t blk = p.live_blocks ? p.live_blocks[pos] : pos;
            const int64_t base = int64_t(blk) * kLanes;
            // accumulator columns 2t, 2t+1 of n-tile j are vectors 8j + 2t and 8j + 2t + 1
            float vs[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int v = 8 * (e >> 1) + 2 * t + (e & 1);
                vs[e] = (base + v < p.n) ? p.vec_scales[base + v] : 0.0f;
            }
            uint32_t allow = 0xffffffffu;
            if (p.mask) allow = reinterpret_cast<const uint32_t *>(p.mask)[blk];
            write_block(p, pos, [&](auto put) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const int ql = 16 * (p.mtile_base + m) + quad + 8 * half;   // query within the prepared batch
                        if (ql >= p.q_base + p.nq) continue;
                        const float qs = p.qscale[ql], qb = p.qbias[ql];
                        const uint64_t thr = p.cb.thr[ql], lo = p.cb.lo ? p.cb.lo[ql] : 0ull;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                const int vl = 8 * j + 2 * t + c;
                                const bool on = base + vl < p.n && ((allow >> vl) & 1u);
                                const int isum = SPLIT ? acc[m][j][2 * half + c] - accn[SPLIT ? m : 0][j][2 * half + c] : acc[m][j][2 * half + c];
                                const float score = __fmul_rn(fmaf(float(isum), qs, qb), vs[2 * j + c]);
                                if (p.dense) put(ql, vl, on, score, uint32_t(base + vl));
                                else if (on) push_candidate(p.cb, ql, score, uint32_t(base + vl), thr, lo);
                            }
                        }
                    }
                }
            });
        }
    }
}

// =====================================================================================================
// Selection for k above kSelectMaxK (smaller k: select.cu): one CTA per query merges the previous top-k with the new candidates in shared memory.
// With few entries it is a plain bitonic sort.  With many more entries than k it is a bitonic top-k: sort
// runs of m = 2^ceil(log2 k) (at least 32) entries in alternating directions, then repeatedly take the
// element-wise minimum of each ascending/descending pair of runs (the m smallest of the pair, as a bitonic
// sequence), drop the other half, and re-sort the survivors' runs with one bitonic merge pass; the work is
// about n (log^2 m / 4 + 2 log m) compare-exchanges instead of n log^2 n / 4.  `dense_count` > 0 means the
// scan wrote exactly that many candidates per query without counting them (first chunk, see scan_tc.cu).
// =====================================================================================================
__device__ __forceinline__ void compare_exchange(uint64_t *keys, int lo, int hi, bool ascending) {
    const uint64_t a = keys[lo], b = keys[hi];
    if ((a > b) == ascending) { keys[lo] = b; keys[hi] = a; }
}

__global__ void __launch_bounds__(256) select_kernel(CandidateBuffers cb, int sort_n, int dense_count) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t *keys = reinterpret_cast<uint64_t *>(smem_raw);
    const int q = blockIdx.x, tid = threadIdx.x;
    const uint32_t raw = dense_count > 0 ? uint32_t(dense_count) : cb.cnt[q];
    const int ncand = int(min(raw, uint32_t(cb.cap)));
    if (tid == 0 && raw > uint32_t(cb.cap)) atomicExch(cb.overflow, 1u);
    // a dense first chunk has no earlier results to merge with: leaving them out keeps 4096 candidates in a
    // 4096-entry network instead of an 8192-entry one
    const int nprev = dense_count > 0 ? 0 : cb.k;
    const int total = nprev + ncand;
    // smallest power of two holding the entries
    int n2 = 32;
    while (n2 < total) n2 <<= 1;
    if (n2 > sort_n) n2 = sort_n;
    for (int i = tid; i < n2; i += blockDim.x) {
        uint64_t v = kEmptyKey;
        if (i < nprev) v = cb.topk[size_t(q) * cb.k + i];
        else if (i < total) v = cb.cand[size_t(q) * cb.cap + (i - nprev)];
        keys[i] = v;
    }
    __syncthreads();
    int m = 32;
    while (m < cb.k) m <<= 1;
    if (n2 <= 2 * m) m = n2;                                  // nothing to gain: full sort
    // runs of m entries, ascending where (index & m) == 0, descending otherwise (m == n2: one ascending run)
    for (int size = 2; size <= m; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < n2 / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1));
                compare_exchange(keys, lo, lo + stride, (lo & size) == 0);
            }
            __syncthreads();
        }
    }
    // halving rounds: live runs sit at multiples of `step` entries; run r pairs with run r + 1 (r even)
    for (int step = m; step * 2 <= n2 && m < n2; step <<= 1) {
        const int pairs = n2 / (2 * step);
        // minimum of entry j of the first run and entry j of the second: the first run keeps the m smallest
        for (int i = tid; i < pairs * m; i += blockDim.x) {
            const int pr = i / m, j = i - pr * m;
            const int lo = pr * 2 * step + j, hi = lo + step;
            const uint64_t a = keys[lo], b = keys[hi];
            if (b < a) keys[lo] = b;
        }
        __syncthreads();
        // the survivors are bitonic: one merge pass sorts them, alternating directions for the next round
        for (int stride = m >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < pairs * (m / 2); i += blockDim.x) {
                const int pr = i / (m / 2), j = i - pr * (m / 2);
                const int lo = pr * 2 * step + 2 * j - (j & (stride - 1));
                compare_exchange(keys, lo, lo + stride, (pr & 1) == 0);
            }
            __syncthreads();
        }
    }
    for (int i = tid; i < cb.k; i += blockDim.x) cb.topk[size_t(q) * cb.k + i] = keys[i];
    if (tid == 0) {
        cb.thr[q] = keys[cb.k - 1];      // kEmptyKey until k results exist: everything still passes
        cb.cnt[q] = 0;
    }
}

__global__ void finalize_kernel(CandidateBuffers cb, int nq, const unsigned long long *n_allowed, int64_t n,
                                float *scores, int64_t *slots, uint32_t *k_eff_out, int out_stride_is_k) {
    unsigned long long allowed = n_allowed ? *n_allowed : (unsigned long long)n;
    const int k_eff = int(min((unsigned long long)cb.k, min((unsigned long long)n, allowed)));
    const int stride = out_stride_is_k ? cb.k : k_eff;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i == 0) *k_eff_out = uint32_t(k_eff);
    if (i >= int64_t(nq) * cb.k) return;
    const int q = int(i / cb.k), j = int(i % cb.k);
    if (j >= k_eff) return;
    const uint64_t key = cb.topk[i];
    float s = -INFINITY;
    int64_t slot = 0;                     // (-inf, 0) padding as search.rs:4341-4352
    if (key != kEmptyKey) { s = desc_bits_to_score(uint32_t(key >> 32)); slot = int64_t(key & 0xffffffffu); }
    scores[size_t(q) * stride + j] = s;
    slots[size_t(q) * stride + j] = slot;
}

__global__ void advance_floor_kernel(const uint64_t *thr, uint64_t *lo, int nq) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < nq) lo[q] = thr[q] == kEmptyKey ? kEmptyKey : thr[q] + 1;
}

// =====================================================================================================
// Device-side id -> slot table of an id-mapped index: open addressing with linear probing over
// (u64 key, u32 slot) pairs, hash = the multiply-shift mix the reference's IdHasher uses
// (turbovec/src/id_map.rs:65-85).  The host tables stay the authority (ids never leave the host in results);
// this copy only serves large allowlists, whose resolution - one hash lookup per id, id_map.rs:670-683 - would
// otherwise run on host threads: the ids are uploaded once and one kernel turns them into mask bits.
// =====================================================================================================
constexpr uint64_t kIdEmpty = 0xffffffffffffffffull, kIdTomb = 0xfffffffffffffffeull;
__device__ __forceinline__ uint32_t id_hash(uint64_t id, int log2cap) { return uint32_t((id * 0x9E3779B97F4A7C15ull) >> (64 - log2cap)); }

// ids[i] -> slot first + i, for ids not yet in the table (a rebuild, or the rows of an add)
__global__ void idtab_insert_kernel(uint64_t *keys, uint32_t *vals, int log2cap, const uint64_t *ids, int64_t n, uint32_t first) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t id = ids[i];
    const uint32_t mask = (1u << log2cap) - 1u;
    uint32_t h = id_hash(id, log2cap);
    for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
        const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long *>(&keys[h]), kIdEmpty, id);
        if (prev == kIdEmpty || prev == id) { vals[h] = first + uint32_t(i); return; }
    }
}
// (id, slot) pairs with distinct ids: slot == 0xffffffff removes the id, otherwise sets (or inserts) its slot
__global__ void idtab_upsert_kernel(uint64_t *keys, uint32_t *vals, int log2cap, const uint64_t *ids, const uint32_t *slots, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t id = ids[i];
    const uint32_t slot = slots[i], mask = (1u << log2cap) - 1u;
    uint32_t h = id_hash(id, log2cap);
    for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
        const uint64_t k = keys[h];
        if (k == id) {
            if (slot == 0xffffffffu) keys[h] = kIdTomb; else vals[h] = slot;
            return;
        }
        if (k == kIdEmpty) {
            if (slot == 0xffffffffu) return;                  // removing an id that is not there
            const unsigned long long prev = atomicCAS(reinterpret_cast<unsigned long long *>(&keys[h]), kIdEmpty, id);
            if (prev == kIdEmpty) { vals[h] = slot; return; }
            // another new id took the place: keep probing
        }
    }
}
// allowlist ids -> mask bits; the smallest list index of an id that is not in the table goes to *first_unknown
__global__ void idtab_lookup_kernel(const uint64_t *keys, const uint32_t *vals, int log2cap, const uint64_t *ids, int64_t n,
                                    uint32_t *words32, unsigned long long *first_unknown) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t id = ids[i];
    const uint32_t mask = (1u << log2cap) - 1u;
    uint32_t h = id_hash(id, log2cap);
    for (uint32_t probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
        const uint64_t k = keys[h];
        if (k == id) { const uint32_t s = vals[h]; atomicOr(&words32[s >> 5], 1u << (s & 31)); return; }
        if (k == kIdEmpty) break;
    }
    atomicMin(first_unknown, (unsigned long long)i);
}

// Keys of a finished search with a slot offset added (the shard's first global slot); empty entries stay empty.
__global__ void export_keys_kernel(const uint64_t *topk, int64_t count, uint64_t offset, uint64_t *out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint64_t key = topk[i];
    out[i] = key == kEmptyKey ? key : key + offset;
}

// Merge of the per-shard result lists of one query: keys[list][q][k] -> the k best keys, decoded.  One CTA per
// query, bitonic sort of n_lists * k keys in shared memory (ascending keys = score descending, slot ascending).
// chunk_slots > 0: the lists hold LOCAL slots of shards that own chunks of that many slots round-robin (list r owns
// the chunks r, r + n_lists, ...); they become global slots before the sort, so ties break by the global slot.
__global__ void __launch_bounds__(256) merge_keys_kernel(const uint64_t *keys_in, int n_lists, int nq, int k, int n2,
                                                         uint32_t chunk_slots, float *scores, int64_t *slots) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t *keys = reinterpret_cast<uint64_t *>(smem_raw);
    const int q = blockIdx.x, tid = threadIdx.x;
    const int total = n_lists * k;
    for (int i = tid; i < n2; i += blockDim.x) {
        uint64_t v = kEmptyKey;
        if (i < total) {
            v = keys_in[(size_t(i / k) * nq + q) * k + (i % k)];
            if (chunk_slots != 0 && v != kEmptyKey) {
                const uint32_t local = uint32_t(v), list = uint32_t(i / k);
                const uint64_t global = (uint64_t(local / chunk_slots) * uint32_t(n_lists) + list) * chunk_slots + local % chunk_slots;
                v = (v & 0xffffffff00000000ull) | global;
            }
        }
        keys[i] = v;
    }
    __syncthreads();
    for (int size = 2; size <= n2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < n2 / 2; i += blockDim.x) {
                const int lo = 2 * i - (i & (stride - 1));
                compare_exchange(keys, lo, lo + stride, (lo & size) == 0);
            }
            __syncthreads();
        }
    }
    for (int j = tid; j < k; j += blockDim.x) {
        const uint64_t key = keys[j];
        float s = -INFINITY;
        int64_t slot = 0;                 // (-inf, 0) padding, as finalize_kernel
        if (key != kEmptyKey) { s = desc_bits_to_score(uint32_t(key >> 32)); slot = int64_t(key & 0xffffffffu); }
        scores[size_t(q) * k + j] = s;
        slots[size_t(q) * k + j] = slot;
    }
}

__global__ void gather_rows_kernel(const float *src, const uint32_t *who, int dim, float *dst) {
    const size_t from = size_t(who[blockIdx.x]) * dim, to = size_t(blockIdx.x) * dim;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) dst[to + i] = src[from + i];
}
__global__ void scatter_rows_kernel(const uint64_t *src, const uint32_t *who, int k, uint64_t *dst) {
    const size_t from = size_t(blockIdx.x) * k, to = size_t(who[blockIdx.x]) * k;
    for (int i = threadIdx.x; i < k; i += blockDim.x) dst[to + i] = src[from + i];
}

}  // namespace

// =====================================================================================================
// Host launchers
// =====================================================================================================
size_t query_prep_smem_bytes(int dim) { return size_t(2) * (dim + 8) * 4 + size_t(dim) * 4; }

cudaError_t launch_query_prep(const QueryPrepParams &p, cudaStream_t stream) {
    if (p.nq <= 0) return cudaSuccess;
    const size_t smem = query_prep_smem_bytes(p.dim);
#define TV_LAUNCH_QP(L)                                                                                        \
    case L: {                                                                                                  \
        cudaError_t e = allow_dynamic_shared(query_prep_kernel<L>, 2048);                                      \
        if (e != cudaSuccess) return e;                                                                        \
        query_prep_kernel<L><<<p.rows, kPrepThreads, smem, stream>>>(p);                                                \
        break;                                                                                                 \
    }
    switch (rotation_variant(p.dim)) {
        TV_LAUNCH_QP(3) TV_LAUNCH_QP(4) TV_LAUNCH_QP(5) TV_LAUNCH_QP(6) TV_LAUNCH_QP(7)
        TV_LAUNCH_QP(8) TV_LAUNCH_QP(9) TV_LAUNCH_QP(10) TV_LAUNCH_QP(11) TV_LAUNCH_QP(12)
        default: return cudaErrorInvalidValue;
    }
#undef TV_LAUNCH_QP
    return cudaGetLastError();
}

cudaError_t launch_pack_bool_mask(const uint8_t *mask_bool, int64_t n, uint64_t *words, cudaStream_t s) {
    const int64_t padded = ((n + 63) / 64) * 64;
    if (padded == 0) return cudaSuccess;
    pack_bool_mask_kernel<<<unsigned((padded + 255) / 256), 256, 0, s>>>(mask_bool, n, reinterpret_cast<uint32_t *>(words));
    return cudaGetLastError();
}

cudaError_t launch_scatter_slots(const uint32_t *slots, int64_t count, uint64_t *words, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    scatter_slots_kernel<<<unsigned((count + 255) / 256), 256, 0, s>>>(slots, count, reinterpret_cast<uint32_t *>(words));
    return cudaGetLastError();
}

cudaError_t launch_mask_stats(uint64_t *words, int64_t n, unsigned long long *n_allowed, uint32_t *live_blocks,
                              uint32_t *n_live, cudaStream_t s) {
    const int64_t nblocks = (n + 31) / 32;
    if (nblocks == 0) return cudaSuccess;
    mask_stats_kernel<<<unsigned((nblocks + 255) / 256), 256, 0, s>>>(reinterpret_cast<uint32_t *>(words), n, n_allowed,
                                                                        live_blocks, n_live);
    return cudaGetLastError();
}

static int sort_capacity(int cap, int k) {
    int n2 = 32;
    while (n2 < cap + k) n2 <<= 1;
    return n2;
}

cudaError_t launch_select_sort(const CandidateBuffers &cb, int nq, int dense_count, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    const int sort_n = sort_capacity(cb.cap, cb.k);
    const size_t smem = size_t(sort_n) * 8;
    // the attribute belongs to the current device: set on every launch (a host-side table write)
    cudaError_t e = cudaFuncSetAttribute(select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    select_kernel<<<nq, 256, smem, s>>>(cb, sort_n, dense_count);
    return cudaGetLastError();
}

cudaError_t launch_advance_floor(const uint64_t *thr, uint64_t *lo, int nq, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    advance_floor_kernel<<<(nq + 255) / 256, 256, 0, s>>>(thr, lo, nq);
    return cudaGetLastError();
}

cudaError_t launch_idtab_insert(uint64_t *keys, uint32_t *vals, int log2cap, const uint64_t *ids, int64_t n, uint32_t first, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    idtab_insert_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(keys, vals, log2cap, ids, n, first);
    return cudaGetLastError();
}
cudaError_t launch_idtab_upsert(uint64_t *keys, uint32_t *vals, int log2cap, const uint64_t *ids, const uint32_t *slots, int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    idtab_upsert_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(keys, vals, log2cap, ids, slots, n);
    return cudaGetLastError();
}
cudaError_t launch_idtab_lookup(const uint64_t *keys, const uint32_t *vals, int log2cap, const uint64_t *ids, int64_t n, uint64_t *words,
                                unsigned long long *first_unknown, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    idtab_lookup_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(keys, vals, log2cap, ids, n, reinterpret_cast<uint32_t *>(words), first_unknown);
    return cudaGetLastError();
}

cudaError_t launch_export_keys(const uint64_t *topk, int64_t count, uint64_t offset, uint64_t *out, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    export_keys_kernel<<<unsigned((count + 255) / 256), 256, 0, s>>>(topk, count, offset, out);
    return cudaGetLastError();
}

cudaError_t launch_merge_keys(const uint64_t *keys, int n_lists, int nq, int k, uint32_t chunk_slots, float *scores, int64_t *slots,
                              cudaStream_t s) {
    if (nq <= 0 || k <= 0 || n_lists <= 0) return cudaSuccess;
    int n2 = 32;
    while (n2 < n_lists * k) n2 <<= 1;
    if (n2 > kMergeMaxKeys) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(merge_keys_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMergeMaxKeys * 8);
    if (e != cudaSuccess) return e;
    merge_keys_kernel<<<nq, 256, size_t(n2) * 8, s>>>(keys, n_lists, nq, k, n2, chunk_slots, scores, slots);
    return cudaGetLastError();
}

cudaError_t launch_finalize(const CandidateBuffers &cb, int nq, const unsigned long long *n_allowed, int64_t n,
                            float *scores, int64_t *slots, uint32_t *k_eff_out, int out_stride_is_k, cudaStream_t s) {
    const int64_t total = int64_t(nq) * cb.k;
    finalize_kernel<<<unsigned((total + 255) / 256 + (total == 0)), 256, 0, s>>>(cb, nq, n_allowed, n, scores, slots,
                                                                                 k_eff_out, out_stride_is_k);
    return cudaGetLastError();
}

cudaError_t launch_gather_rows(const float *src, const uint32_t *who, int count, int dim, float *dst, cudaStream_t s) {
    gather_rows_kernel<<<unsigned(count), 128, 0, s>>>(src, who, dim, dst);
    return cudaGetLastError();
}
cudaError_t launch_scatter_rows(const uint64_t *src, const uint32_t *who, int count, int k, uint64_t *dst, cudaStream_t s) {
    scatter_rows_kernel<<<unsigned(count), 128, 0, s>>>(src, who, k, dst);
    return cudaGetLastError();
}

cudaError_t launch_scan_pd(const ScanParams &p, int sm_count, cudaStream_t s) {
    if (p.nq <= 0 || p.pos_end <= p.pos_begin) return cudaSuccess;
    const int mt = (p.nq + 15) / 16;
    const size_t smem = size_t(kStages) * kStageBytes;
    const uint32_t tiles = (p.pos_end - p.pos_begin + kConsumerWarps - 1) / kConsumerWarps;
    // the split lookup doubles the accumulators: with two query tiles the kernel needs 168 registers, one CTA per
    // SM, and is slower than the merged lookup (1.76 against 1.46 ms on 4 M vectors), so one tile only
    const bool split = p.pd_split != 0 && mt <= 1 && levels_split_ok(p.level_words);
    const unsigned per_sm = mt == 1 ? (split ? 2 : 3) : (mt == 2 ? 2 : 1);   // resident CTAs per SM (registers)
    const unsigned grid = unsigned(min(uint32_t(sm_count) * per_sm, tiles));
    const unsigned threads = (kConsumerWarps + 1) * 32;
#define TV_LAUNCH_PD(M, S)                                                                                          \
    {                                                                                                               \
        cudaError_t e = cudaFuncSetAttribute(scan_pd_kernel<M, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)); \
        if (e != cudaSuccess) return e;                                                                             \
        scan_pd_kernel<M, S><<<grid, threads, smem, s>>>(p);                                                        \
    }
    if (mt <= 1) { if (split) TV_LAUNCH_PD(1, true) else TV_LAUNCH_PD(1, false) }
    else if (mt <= 2) TV_LAUNCH_PD(2, false)
    else if (mt <= 4) TV_LAUNCH_PD(4, false)
    else return cudaErrorInvalidValue;
#undef TV_LAUNCH_PD
    return cudaGetLastError();
}

}  // namespace tv
