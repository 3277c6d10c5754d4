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
// costs a sector.  A warp scores four survivors at a time to keep enough of them in flight.
#include <algorithm>

#include "search.cuh"
#include "tv_common.cuh"

namespace tv {
namespace {

constexpr int kScoreThreads = 256;
constexpr int kScoreWarps = kScoreThreads / 32;
constexpr int kTogether = 4;               // survivors per warp and step

// The exact keys of up to kTogether slots; valid in every lane.
template <typename Emit>
__device__ __forceinline__ void exact_keys(const ScanParams &p, const uint8_t *lut, int q, const uint32_t (&slot)[kTogether], int lane, Emit emit) {
    const int ng = p.ngroups;
    const uint8_t *src[kTogether];
#pragma unroll
    for (int j = 0; j < kTogether; ++j) src[j] = p.codes + size_t(slot[j] >> 5) * ng * 32 + (slot[j] & 31u);
    float facc[kTogether];
    int total[kTogether];
    const float qs = p.qscale[q], qb = p.qbias[q];
#pragma unroll
    for (int j = 0; j < kTogether; ++j) { facc[j] = qb; total[j] = 0; }
    for (int g0 = 0; g0 < ng; g0 += 256) {
        const int g1 = min(g0 + 256, ng);
        int sum[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j) sum[j] = 0;
#pragma unroll 4
        for (int g = g0 + lane; g < g1; g += 32) {
#pragma unroll
            for (int j = 0; j < kTogether; ++j) {
                const uint32_t byte = __ldg(src[j] + size_t(g) * 32);
                sum[j] += int(lut[g * 32 + (byte >> 4)]) + int(lut[g * 32 + 16 + (byte & 15u)]);
            }
        }
#pragma unroll
        for (int j = 0; j < kTogether; ++j) {
            sum[j] = __reduce_add_sync(kFullMask, sum[j]);
            facc[j] = fmaf(qs, float(sum[j]), facc[j]);
            total[j] += sum[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kTogether; ++j) {
        const float pre = p.mode == kModeLutFlush ? facc[j] : __fadd_rn(__fmul_rn(float(total[j]), qs), qb);
        emit(j, make_key(__fmul_rn(pre, p.vec_scales[slot[j]]), slot[j]));
    }
}

__device__ __forceinline__ void load_tables(const ScanParams &p, int q, uint4 *lut) {
    const uint4 *src = reinterpret_cast<const uint4 *>(p.luts + size_t(q) * p.lut_pitch);
    for (int i = threadIdx.x; i < p.ngroups * 2; i += kScoreThreads) lut[i] = src[i];
}

// cand[q][i] = slot -> exact key, or kEmptyKey when it does not beat the k-th best.  Grid (shares of a list, queries).
__global__ void __launch_bounds__(kScoreThreads) score_survivors_kernel(ScanParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int q = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t n = min(p.cb.cnt[q], uint32_t(p.cb.cap));
    if (blockIdx.x * kScoreWarps * kTogether >= n) return;
    load_tables(p, q, reinterpret_cast<uint4 *>(smem_raw));
    __syncthreads();
    uint64_t *list = p.cb.cand + size_t(q) * p.cb.cap;
    const uint64_t thr = p.cb.thr[q];
    for (uint32_t i = (blockIdx.x * kScoreWarps + warp) * kTogether; i < n; i += gridDim.x * kScoreWarps * kTogether) {
        uint32_t slot[kTogether];
#pragma unroll
        for (int j = 0; j < kTogether; ++j) slot[j] = uint32_t(list[min(i + j, n - 1)]);
        __syncwarp();                                     // every lane has read the slots before lane 0 puts keys there
        exact_keys(p, smem_raw, q, slot, lane, [&](int j, uint64_t key) {
            if (lane == 0 && i + j < n) list[i + j] = key < thr ? key : kEmptyKey;
        });
    }
}

// topk[q] = the k best of the first chunk by approximate score -> thr[q] just above the worst of their exact keys; the
// running top-k is empty again.  Fewer than k entries: no threshold.
__global__ void __launch_bounds__(kScoreThreads) bootstrap_kernel(ScanParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t worst[kScoreWarps];
    const int q = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *top = p.cb.topk + size_t(q) * p.cb.k;
    const int k = p.cb.k;
    const bool full = top[k - 1] != kEmptyKey;
    if (full) load_tables(p, q, reinterpret_cast<uint4 *>(smem_raw));
    __syncthreads();
    uint64_t mine = 0;
    if (full) {
        for (int i = warp * kTogether; i < k; i += kScoreWarps * kTogether) {
            uint32_t slot[kTogether];
#pragma unroll
            for (int j = 0; j < kTogether; ++j) slot[j] = uint32_t(top[min(i + j, k - 1)]);
            exact_keys(p, smem_raw, q, slot, lane, [&](int, uint64_t key) { mine = max(mine, key); });
        }
    }
    if (lane == 0) worst[warp] = mine;
    __syncthreads();
    for (int i = threadIdx.x; i < k; i += kScoreThreads) top[i] = kEmptyKey;
    if (threadIdx.x == 0) {
        for (int w = 0; w < kScoreWarps; ++w) mine = max(mine, worst[w]);
        p.cb.thr[q] = full ? mine + 1 : kEmptyKey;
    }
}

}  // namespace

bool scan_filter_supported(int bits, int mode, int ngroups, size_t smem_limit) {
    return tensor_map_encoder() != nullptr && (bits == 2 || bits == 3) && (mode == kModeLutMulAdd || mode == kModeLutFlush) && size_t(ngroups) * 32 + 1024 <= smem_limit;
}

cudaError_t launch_score_survivors(const ScanParams &p, int nq, int sm_count, cudaStream_t s) {
    const size_t smem = size_t(p.ngroups) * 32;
    cudaError_t e = cudaFuncSetAttribute(score_survivors_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    for (int q0 = 0; q0 < nq; q0 += 32768) {
        const int here = std::min(nq - q0, 32768);
        ScanParams part = p;
        part.cb.cand += size_t(q0) * p.cb.cap; part.cb.cnt += q0; part.cb.thr += q0;
        part.luts += size_t(q0) * p.lut_pitch; part.qscale += q0; part.qbias += q0;
        // about eight CTAs per SM over all queries, at least one per query, none without a first step of its own
        const unsigned shares = unsigned(std::max(1, std::min(8 * sm_count / here, p.cb.cap / (kScoreWarps * kTogether))));
        score_survivors_kernel<<<dim3(shares, unsigned(here)), kScoreThreads, smem, s>>>(part);
    }
    return cudaGetLastError();
}

cudaError_t launch_bootstrap(const ScanParams &p, int nq, cudaStream_t s) {
    const size_t smem = size_t(p.ngroups) * 32;
    cudaError_t e = cudaFuncSetAttribute(bootstrap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    bootstrap_kernel<<<nq, kScoreThreads, smem, s>>>(p);
    return cudaGetLastError();
}

}  // namespace tv
