// Exact scores for the survivors of a filtering scan (2- and 3-bit codes, batches).
//
// The u8-LUT score of a vector is a sum of table entries U[g][nibble], which has no contraction narrower than 16 per
// half-byte.  But each entry is a rounded affine function of the code's levels: with int8 weights W and int8 levels L,
//     U = alpha * (W . L) + beta_h + e,   |e| <= d_h,
// where query preparation evaluates beta_h and d_h from all the entries of the half-byte.  So
//     isum <= alpha * A + beta + D,   A = sum_d W[d] * L[code[v][d]],
// and A is an int8 contraction over the coordinates (scan_tc.cu, KIND = kLevels2 / kLevels3), an eighth of the one-hot K.
// D is worth 0.2 standard deviations of a score at 200 dimensions and about one at 3,072: a vector whose bound stays
// below the k-th best score cannot be a result, and few others are left.  Those get their exact score here, by the table
// lookups and the float operations of the reference (search.rs:1176, 1596).
//
// The filter needs a k-th best score to begin with: the scan of the first chunk ranks it by the approximate score
// alpha * A + beta, the k best of that order are scored exactly, and the worst of them bounds the k-th best from below.
// They are found again by the filtering scans, which cover the first chunk as well.
//
// What bounds the scoring is the gather: a vector's bytes lie 32 apart (one per sector) in its code block, so every byte
// costs a sector.  A warp scores four survivors at a time to keep enough of them in flight, and leaves a survivor as soon
// as it can no longer reach the threshold: after every 128 byte-groups the bound is the exact sum so far, plus alpha times
// what W . L has left, plus the largest deviations of the remaining half-bytes (suffix sums from query preparation).  The
// sum of deviations is what let most survivors through, and it shrinks with every batch.
#include <algorithm>
#include <cfloat>

#include "scan_tc_common.cuh"

namespace tv {
namespace {

constexpr int kScoreThreads = 256;
constexpr int kScoreWarps = kScoreThreads / 32;
constexpr int kTogether = 4;               // survivors per warp and step
constexpr int kSample = 1024;              // vectors of the first chunk by which the next scan's survivors are estimated

// The exact keys of up to kTogether slots, valid in every lane.  EXIT: `sum` = W . L of each; a survivor that drops out on
// the way gets kEmptyKey.
template <bool EXIT, typename Emit>
__device__ __forceinline__ void exact_keys(const ScanParams &p, const uint8_t *lut, const uint32_t *wq, int q, const uint32_t (&slot)[kTogether],
                                           const int (&sum)[kTogether], uint64_t thr, int lane, Emit emit) {
    const int ng = p.ngroups;
    const uint8_t *src[kTogether];
    float facc[kTogether], vs[kTogether];
    int total[kTogether], need[kTogether], left[kTogether];
    const float qs = p.qscale[q], qb = p.qbias[q];
    const float alpha = EXIT ? p.f_alpha[q] : 0.0f;
    const float t = thr == kEmptyKey ? -INFINITY : desc_bits_to_score(uint32_t(thr >> 32));
    uint32_t alive = (1u << kTogether) - 1u;
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
        src[j] = p.codes + size_t(slot[j] >> 5) * ng * 32 + (slot[j] & 31u);
        vs[j] = p.vec_scales[slot[j]];
        facc[j] = qb; total[j] = 0; left[j] = sum[j];
        need[j] = 0;
    }
    for (int g0 = 0; g0 < ng && alive; g0 += 256) {
        int part[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j) part[j] = 0;
#pragma unroll
        for (int h0 = g0; h0 < g0 + 256; h0 += kFilterBatch) {
            if (h0 >= ng || !alive) break;
            int s[kTogether], w[kTogether];
#pragma unroll
            for (int j = 0; j < kTogether; ++j) { s[j] = 0; w[j] = 0; }
            uint32_t byte[kFilterBatch / 32][kTogether];
#pragma unroll
            for (int i = 0; i < kFilterBatch / 32; ++i)
#pragma unroll
                for (int j = 0; j < kTogether; ++j) {
                    const int g = h0 + 32 * i + lane;
                    byte[i][j] = g < ng && ((alive >> j) & 1u) ? __ldg(src[j] + size_t(g) * 32) : 0u;
                }
#pragma unroll
            for (int i = 0; i < kFilterBatch / 32; ++i) {
                const int g = h0 + 32 * i + lane;
                if (g >= ng) continue;
                const uint32_t wg = EXIT ? wq[g] : 0u;
#pragma unroll
                for (int j = 0; j < kTogether; ++j) {
                    const uint32_t b = byte[i][j];
                    s[j] += int(lut[g * 32 + (b >> 4)]) + int(lut[g * 32 + 16 + (b & 15u)]);
                    if constexpr (EXIT) {
                        // selectors of the byte's levels, in the order of wq
                        const uint32_t sel = p.bits == 2 ? (b & 0x33u) | ((b >> 2) & 0x33u) << 8 : b & 0x77u;
                        w[j] = __dp4a(int(__byte_perm(p.level_words[0], p.level_words[1], sel)), int(wg), w[j]);
                    }
                }
            }
            if (EXIT && h0 == 0) {                       // only now: the scales were requested with the first bytes
#pragma unroll
                for (int j = 0; j < kTogether; ++j) need[j] = dismissal_bound(qs, qb, t, vs[j]);
            }
            const float rest = EXIT ? p.f_suffix[size_t(q) * kFilterBatches + h0 / kFilterBatch + 1] : 0.0f;
#pragma unroll
            for (int j = 0; j < kTogether; ++j) {
                part[j] += __reduce_add_sync(kFullMask, s[j]);
                if constexpr (EXIT) {
                    left[j] -= __reduce_add_sync(kFullMask, w[j]);
                    // 1e-3 + 1e-6 of the terms: their roundings
                    const float more = alpha * float(left[j]);
                    if (float(total[j] + part[j]) + more + rest + (1e-3f + 1e-6f * (fabsf(more) + fabsf(rest))) < float(need[j])) alive &= ~(1u << j);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
            facc[j] = fmaf(qs, float(part[j]), facc[j]);
            total[j] += part[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
        const float pre = p.mode == kModeLutFlush ? facc[j] : __fadd_rn(__fmul_rn(float(total[j]), qs), qb);
        emit(j, (alive >> j) & 1u ? make_key(__fmul_rn(pre, vs[j]), slot[j]) : kEmptyKey);
    }
}

__device__ __forceinline__ void load_tables(const ScanParams &p, int q, uint4 *lut) {
    const uint4 *src = reinterpret_cast<const uint4 *>(p.luts + size_t(q) * p.lut_pitch);
    for (int i = threadIdx.x; i < p.ngroups * 2; i += kScoreThreads) lut[i] = src[i];
}

// The int8 weights of a byte-group in one word, in the order of its levels: 2-bit coordinates 3, 1, 2, 0; 3-bit 1, 0.
__device__ __forceinline__ void load_weights(const ScanParams &p, int q, uint32_t *wq) {
    const uint8_t *row = reinterpret_cast<const uint8_t *>(p.f_weights) + size_t(q) * p.f_pitch;
    for (int g = threadIdx.x; g < p.ngroups; g += kScoreThreads) {
        // rows in filter_coord order (search.cu)
        if (p.bits == 2) {
            const int c = g & 7, i = (g >> 3) & 3;
            const uint8_t *at = row + (g >> 5) * 128 + c * 16 + (i >> 1) * 4 + (i & 1) * 2;
            wq[g] = uint32_t(*reinterpret_cast<const uint16_t *>(at)) | uint32_t(*reinterpret_cast<const uint16_t *>(at + 8)) << 16;
        } else {
            wq[g] = *reinterpret_cast<const uint16_t *>(row + (g >> 6) * 128 + (g & 7) * 16 + ((g >> 3) & 7) * 2);
        }
    }
}

// Whether scoring this chunk's survivors, and redoing the queries whose lists overflowed, would take longer than the form
// without the filter saves from here on (filter_hopeless).  How many survive depends on the data (copies and tight clusters near the k-th
// result all do) and is known only now; a scan without its scoring costs a seventh of the other form, so giving up here
// costs little, and the results of the chunks before stay.  By the whole block.
__device__ bool not_worth_while(const ScanParams &p, const uint32_t *all_cnt, int all_queries) {
    __shared__ float part[2][kScoreWarps];
    if (p.f_budget_us >= FLT_MAX) return false;
    float scored = 0.0f, lost = 0.0f;
    for (int i = threadIdx.x; i < all_queries; i += kScoreThreads) {
        const uint32_t c = all_cnt[i];
        if (c > uint32_t(p.cb.cap)) lost += 1.0f;
        else scored += float(c);
    }
    for (int o = 16; o > 0; o >>= 1) {
        scored += __shfl_xor_sync(kFullMask, scored, o);
        lost += __shfl_xor_sync(kFullMask, lost, o);
    }
    if ((threadIdx.x & 31) == 0) { part[0][threadIdx.x >> 5] = scored; part[1][threadIdx.x >> 5] = lost; }
    __syncthreads();
    scored = lost = 0.0f;
    for (int w = 0; w < kScoreWarps; ++w) { scored += part[0][w]; lost += part[1][w]; }
    return filter_hopeless(p, scored, lost, all_queries, 0.0f);
}

// cand[q][i] = (W . L, slot) -> exact key, or kEmptyKey when it does not beat the k-th best.  Grid (shares of a list, queries).
// A list that overflowed is left alone: its query is searched again.
__global__ void __launch_bounds__(kScoreThreads, 3) score_survivors_kernel(ScanParams p, const uint32_t *all_cnt, int all_queries, uint32_t *stopped_at) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *wq = reinterpret_cast<uint32_t *>(smem_raw + size_t(p.ngroups) * 32);
    const int q = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n = min(p.cb.cnt[q], uint32_t(p.cb.cap));
    if (blockIdx.x * kScoreWarps * kTogether >= n) return;
    load_tables(p, q, reinterpret_cast<uint4 *>(smem_raw));
    load_weights(p, q, wq);
    if (not_worth_while(p, all_cnt, all_queries)) {       // the same outcome in every block
        if (threadIdx.x == 0) { *stopped_at = p.pos_begin + 1u; atomicOr(p.cb.overflow, kFilterStopped); }
        return;
    }
    __syncthreads();
    if (p.cb.cnt[q] > uint32_t(p.cb.cap)) return;
    uint64_t *list = p.cb.cand + size_t(q) * p.cb.cap;
    const uint64_t thr = p.cb.thr[q];
    for (uint32_t i = (blockIdx.x * kScoreWarps + warp) * kTogether; i < n; i += gridDim.x * kScoreWarps * kTogether) {
        uint32_t slot[kTogether];
        int sum[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
            const uint64_t v = list[min(i + j, n - 1)];
            slot[j] = uint32_t(v); sum[j] = int(uint32_t(v >> 32));
        }
        __syncwarp();                                     // every lane has read the slots before lane 0 puts keys there
        exact_keys<true>(p, smem_raw, wq, q, slot, sum, thr, lane, [&](int j, uint64_t key) {
            if (lane == 0 && i + j < n) list[i + j] = key < thr ? key : kEmptyKey;
        });
    }
}

// topk[q] = the k best of the first chunk by approximate score -> thr[q] just above the worst of their exact keys; the
// running top-k is empty again.  Fewer than k entries, or a k-th score that overflowed: no threshold (the filtering scans
// take an infinite one for a column without a query, and these k vectors have yet to be found).  A zero query ties with
// every vector: without a mask, whose blocks come in any order, the first k are its results, and nothing more need survive.
__device__ void bootstrap_query(const ScanParams &p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t worst[kScoreWarps];
    const int q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *top = p.cb.topk + size_t(q) * p.cb.k;
    const int k = p.cb.k;
    const bool full = top[k - 1] != kEmptyKey;
    if (full && p.f_scale[q] == 0.0f && p.live_blocks == nullptr) {
        if (threadIdx.x == 0) p.cb.thr[q] = make_key(INFINITY, 0u);
        return;
    }
    if (full) load_tables(p, q, reinterpret_cast<uint4 *>(smem_raw));
    __syncthreads();
    uint64_t mine = 0;
    if (full) {
        for (int i = warp * kTogether; i < k; i += kScoreWarps * kTogether) {
            uint32_t slot[kTogether];
#pragma unroll
            for (int j = 0; j < kTogether; ++j) slot[j] = uint32_t(top[min(i + j, k - 1)]);
            const int none[kTogether] = {};
            exact_keys<false>(p, smem_raw, nullptr, q, slot, none, kEmptyKey, lane, [&](int, uint64_t key) { mine = max(mine, key); });
        }
    }
    if (lane == 0) worst[warp] = mine;
    __syncthreads();
    for (int i = threadIdx.x; i < k; i += kScoreThreads) top[i] = kEmptyKey;
    if (threadIdx.x == 0) {
        for (int w = 0; w < kScoreWarps; ++w) mine = max(mine, worst[w]);
        worst[0] = full && fabsf(desc_bits_to_score(uint32_t(mine >> 32))) <= FLT_MAX ? mine + 1 : kEmptyKey;
        p.cb.thr[q] = worst[0];
    }
    if (p.f_budget_us >= FLT_MAX || !full) return;
    // How many vectors will the first filtering scan let through?  As large a share as of the first chunk, which the list
    // still holds: 1,024 of its vectors say it (without the places where the selection left the best of a segment).
    __syncthreads();
    const uint64_t thr = worst[0];
    if (thr == kEmptyKey) return;
    const float t = desc_bits_to_score(uint32_t(thr >> 32)), slack = p.f_max[q] - p.f_mid[q];
    const uint64_t *list = p.cb.cand + size_t(q) * p.cb.cap;
    uint32_t len = p.pos_end - p.pos_begin;
    if (p.live_blocks != nullptr) len = min(len, *p.n_live);
    len *= 32u;
    int seen = 0, through = 0;
#pragma unroll
    for (int i = 0; i < kSample / kScoreThreads; ++i) {
        const uint32_t at = uint32_t(uint64_t(i * kScoreThreads + threadIdx.x) * len / kSample);
        if (at >= len || (len > uint32_t(kSelectSegment) && (at & uint32_t(kSelectSegment - 1)) < uint32_t(kSelectMaxK))) continue;
        const uint64_t key = list[at];
        ++seen;
        if (key == kEmptyKey) continue;
        const float most = desc_bits_to_score(uint32_t(key >> 32)) + slack * p.vec_scales[uint32_t(key)];
        through += !(most < t);
    }
    seen = __reduce_add_sync(kFullMask, seen);
    through = __reduce_add_sync(kFullMask, through);
    __syncthreads();
    if (lane == 0) worst[warp] = uint64_t(uint32_t(seen)) << 32 | uint32_t(through);
    __syncthreads();
    if (threadIdx.x != 0) return;
    uint64_t both = 0;
    for (int w = 0; w < kScoreWarps; ++w) both += worst[w];
    const float share = float(uint32_t(both)) / fmaxf(float(uint32_t(both >> 32)), 1.0f);
    const float expected = share * (p.live_blocks != nullptr ? fminf(float(p.f_ahead), float(*p.n_live) * 32.0f) : float(p.f_ahead));
    if (expected > float(p.cb.cap)) {                     // as a list that has overflowed
        atomicAdd(p.f_tally + 1, 1.0f);
        p.cb.over[q] = 1u;
        atomicAdd(p.cb.overflow, 1u);
        p.cb.thr[q] = make_key(INFINITY, 0u);
    } else {
        atomicAdd(p.f_tally, expected);
    }
}

__global__ void __launch_bounds__(kScoreThreads) bootstrap_kernel(ScanParams p) {
    bootstrap_query(p);
    if (p.f_budget_us >= FLT_MAX || threadIdx.x != 0) return;
    // the block that ends last knows what all queries expect, and whether the filter is worth beginning
    __threadfence();
    if (atomicAdd(reinterpret_cast<uint32_t *>(p.f_tally + 2), 1u) != gridDim.x - 1u) return;
    __threadfence();
    const volatile float *tally = p.f_tally;
    if (filter_hopeless(p, tally[0], tally[1], int(gridDim.x), p.f_scan_us)) {
        p.cb.over[gridDim.x] = 1u;                        // given up at position 0
        atomicOr(p.cb.overflow, kFilterStopped);
    }
}

}  // namespace

bool scan_filter_supported(int bits, int mode, int ngroups, size_t smem_limit) {
    return tensor_map_encoder() != nullptr && (bits == 2 || bits == 3) && (mode == kModeLutMulAdd || mode == kModeLutFlush) && size_t(ngroups) * 36 + 1024 <= smem_limit && ngroups <= kFilterBatch * (kFilterBatches - 1);
}

cudaError_t launch_score_survivors(const ScanParams &p, int nq, int sm_count, cudaStream_t s) {
    const size_t smem = size_t(p.ngroups) * 36;
    cudaError_t e = allow_dynamic_shared(score_survivors_kernel, 1024);
    if (e != cudaSuccess) return e;
    for (int q0 = 0; q0 < nq; q0 += 32768) {
        const int here = std::min(nq - q0, 32768);
        ScanParams part = p;
        part.cb.cand += size_t(q0) * p.cb.cap; part.cb.cnt += q0; part.cb.thr += q0;
        part.luts += size_t(q0) * p.lut_pitch; part.qscale += q0; part.qbias += q0;
        part.f_alpha += q0; part.f_suffix += size_t(q0) * kFilterBatches; part.f_weights += size_t(q0) * p.f_pitch;
        // about eight CTAs per SM over all queries, at least one per query, none without a first step of its own
        const unsigned shares = unsigned(std::max(1, std::min(8 * sm_count / here, p.cb.cap / (kScoreWarps * kTogether))));
        score_survivors_kernel<<<dim3(shares, unsigned(here)), kScoreThreads, smem, s>>>(part, p.cb.cnt, nq, p.cb.over + nq);
    }
    return cudaGetLastError();
}

cudaError_t launch_bootstrap(const ScanParams &p, int nq, cudaStream_t s) {
    const size_t smem = size_t(p.ngroups) * 32;
    cudaError_t e = allow_dynamic_shared(bootstrap_kernel, 1024);
    if (e != cudaSuccess) return e;
    bootstrap_kernel<<<nq, kScoreThreads, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace tv
