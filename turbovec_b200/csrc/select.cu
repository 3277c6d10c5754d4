// Top-k selection over candidate keys (k up to kSelectMaxK): a histogram cut instead of a sort.
//
// The order of results is the ascending order of 64-bit keys (tv_common.cuh), so the k best entries of a list are its k
// smallest keys.  A CTA holds a segment of 4,096 keys in registers and finds an upper bound of the k-th smallest by
// counting: a linear histogram of the scores between the best and the worst key (1,024 bins; the wanted tail of a score
// distribution is sparse, so one pass nearly always leaves at most 2k keys), repeated inside the bin that holds the k-th
// key while that bin is too full.  Only the survivors are sorted, each by counting the smaller ones.
//
// What bounds it is latency: with one query the kernel is a chain of block-wide steps between two scans.  A bitonic sort
// of 4,096 keys needs 78 of them (39 us for one query, 151 us for 1,024); this form needs about ten.
//
// Lists longer than a segment are cut over `parts` CTAs of a query.  Each leaves the k best of its segment in place; the
// one that arrives last merges them with the running top-k.  Nothing waits.
#include <algorithm>
#include <cfloat>

#include "search.cuh"
#include "tv_common.cuh"

namespace tv {
namespace {

constexpr int kSelThreads = 512;
constexpr int kSelBins = 1024;
constexpr int kSelKeysPerThread = kSelectSegment / kSelThreads + 1;   // a segment and one slot for the running top-k
constexpr int kSelList = 2 * kSelectMaxK;                             // most survivors of the cut
static_assert(kSelectMaxK <= kSelThreads, "one running key per thread");

struct SelectShared {
    uint64_t list[kSelList];
    uint64_t sorted[kSelectMaxK];
    uint32_t hist[kSelBins];
    uint64_t red_lo[kSelThreads / 32], red_hi[kSelThreads / 32];
    uint32_t red_n[kSelThreads / 32];
    uint32_t n_list;
    uint32_t bin, before, within;
    uint32_t last;
};

// The min(k, valid) smallest of the block's keys (kEmptyKey = no entry), ascending in sh.sorted; returns how many.
__device__ int block_smallest(const uint64_t (&key)[kSelKeysPerThread], int k, SelectShared &sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t active = 0, taken = 0;                       // bit i: key[i] is still undecided / is below the cut
#pragma unroll
    for (int i = 0; i < kSelKeysPerThread; ++i) active |= uint32_t(key[i] != kEmptyKey) << i;
    uint32_t n_taken = 0;
    int want = 0;
    for (int pass = 0;; ++pass) {
        uint64_t lo = kEmptyKey, hi = 0;
        uint32_t cnt = __popc(active);
#pragma unroll
        for (int i = 0; i < kSelKeysPerThread; ++i)
            if ((active >> i) & 1u) { lo = min(lo, key[i]); hi = max(hi, key[i]); }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(kFullMask, lo, o));
            hi = max(hi, __shfl_xor_sync(kFullMask, hi, o));
        }
        cnt = __reduce_add_sync(kFullMask, cnt);
        if (lane == 0) { sh.red_lo[warp] = lo; sh.red_hi[warp] = hi; sh.red_n[warp] = cnt; }
        for (int b = tid; b < kSelBins; b += kSelThreads) sh.hist[b] = 0;
        if (tid == 0) sh.n_list = 0;
        __syncthreads();
        {
            const int w = lane & (kSelThreads / 32 - 1);
            lo = sh.red_lo[w]; hi = sh.red_hi[w]; cnt = lane < kSelThreads / 32 ? sh.red_n[w] : 0u;
#pragma unroll
            for (int o = kSelThreads / 64; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(kFullMask, lo, o));
                hi = max(hi, __shfl_xor_sync(kFullMask, hi, o));
            }
            cnt = __reduce_add_sync(kFullMask, cnt);
        }
        if (pass == 0) want = min(k, int(cnt));
        if (want == 0) { __syncthreads(); return 0; }
        const uint32_t enough = max(2u * uint32_t(want), 64u);         // at most kSelList survivors are sorted
        if (n_taken + cnt <= enough) { taken |= active; break; }
        // Bins: linear in the score where the scores span a finite range, else in the key's bits (equal scores, infinities).
        const float s_hi = desc_bits_to_score(uint32_t(lo >> 32)), s_lo = desc_bits_to_score(uint32_t(hi >> 32));
        const float scale = float(kSelBins - 1) / (s_hi - s_lo);
        const bool linear = s_hi > s_lo && s_hi <= FLT_MAX && s_lo >= -FLT_MAX && s_hi - s_lo <= FLT_MAX && scale <= FLT_MAX;
        const int shift = max(0, 54 - __clzll((long long)(hi - lo)));  // hi - lo < 2^(64 - clz): ten bits remain
        auto bin_of = [&](uint64_t v) -> uint32_t {
            // each rounding is monotone in the score, so bins are ordered as the keys are
            if (linear) return min(uint32_t((s_hi - desc_bits_to_score(uint32_t(v >> 32))) * scale), uint32_t(kSelBins - 1));
            return uint32_t((v - lo) >> shift);
        };
        uint32_t bins[kSelKeysPerThread];
#pragma unroll
        for (int i = 0; i < kSelKeysPerThread; ++i) {
            bins[i] = 0;
            if ((active >> i) & 1u) { bins[i] = bin_of(key[i]); atomicAdd(&sh.hist[bins[i]], 1u); }
        }
        __syncthreads();
        // the bin that holds the (want - n_taken)-th undecided key
        const uint32_t rem = uint32_t(want) - n_taken;
        const uint32_t h0 = sh.hist[2 * tid], h1 = sh.hist[2 * tid + 1];
        uint32_t sum = h0 + h1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(kFullMask, sum, o);
            if (lane >= o) sum += up;
        }
        if (lane == 31) sh.red_n[warp] = sum;
        __syncthreads();
        uint32_t base = lane < warp ? sh.red_n[lane] : 0u;              // kSelThreads / 32 <= 32 warps
        base = __reduce_add_sync(kFullMask, base);
        const uint32_t before0 = base + sum - h0 - h1, before1 = before0 + h0;
        if (before0 < rem && rem <= before0 + h0) { sh.bin = 2 * tid; sh.before = before0; sh.within = h0; }
        if (before1 < rem && rem <= before1 + h1) { sh.bin = 2 * tid + 1; sh.before = before1; sh.within = h1; }
        __syncthreads();
        const uint32_t cut = sh.bin;
        uint32_t next = 0;
#pragma unroll
        for (int i = 0; i < kSelKeysPerThread; ++i)
            if ((active >> i) & 1u) {
                if (bins[i] < cut) taken |= 1u << i;
                else if (bins[i] == cut) next |= 1u << i;
            }
        n_taken += sh.before;
        const uint32_t within = sh.within;
        active = next;
        // a bin one key wide (duplicates cannot occur) ends the search as well
        if (n_taken + within <= enough || (!linear && shift == 0)) { taken |= active; break; }
        __syncthreads();                                               // the histogram is cleared for the next pass
    }
#pragma unroll
    for (int i = 0; i < kSelKeysPerThread; ++i)
        if ((taken >> i) & 1u) {
            const uint32_t at = atomicAdd(&sh.n_list, 1u);
            if (at < uint32_t(kSelList)) sh.list[at] = key[i];
        }
    __syncthreads();
    const int c = int(min(sh.n_list, uint32_t(kSelList)));
    for (int i = tid; i < c; i += kSelThreads) {
        const uint64_t mine = sh.list[i];
        int rank = 0;
#pragma unroll 4
        for (int j = 0; j < c; ++j) rank += (sh.list[j] < mine) | ((sh.list[j] == mine) & (j < i));
        if (rank < want) sh.sorted[rank] = mine;
    }
    __syncthreads();
    return want;
}

// dense_blocks > 0: the scan wrote 32 keys per scanned block without counting them, for the first min(dense_blocks,
// *n_live) positions, and there are no earlier results.
__global__ void __launch_bounds__(kSelThreads) select_parts_kernel(CandidateBuffers cb, uint32_t dense_blocks, const uint32_t *n_live, SearchOutput out) {
    __shared__ SelectShared sh;
    const int q = blockIdx.y, tid = threadIdx.x;
    const uint32_t part = blockIdx.x;
    uint32_t raw;
    if (dense_blocks > 0) raw = (n_live ? min(dense_blocks, *n_live) : dense_blocks) * 32u;
    else raw = *reinterpret_cast<volatile uint32_t *>(&cb.cnt[q]);
    // a filtering search that was given up: these survivors were not scored, and what was found before them stands
    if (cb.over != nullptr && (*reinterpret_cast<volatile uint32_t *>(cb.overflow) & kFilterStopped) != 0u) raw = 0;
    const uint32_t ncand = min(raw, uint32_t(cb.cap));
    const uint32_t parts = max(1u, (ncand + kSelectSegment - 1) / kSelectSegment);
    if (part >= parts) return;                                          // (a late CTA may see the count already cleared: same outcome)
    // a list that the next scan is bound to fill need not be begun there: its query is searched by itself either way
    const bool spilled = raw > uint32_t(cb.cap) || (cb.over != nullptr && float(raw) > cb.unusual && float(raw) * cb.ahead > float(cb.cap));
    if (part == 0 && tid == 0 && spilled && (cb.over == nullptr || atomicExch(&cb.over[q], 1u) == 0u)) atomicAdd(cb.overflow, 1u);
    uint64_t *list = cb.cand + size_t(q) * cb.cap;
    uint64_t *seg = list + size_t(part) * kSelectSegment;
    const uint32_t here = min(uint32_t(kSelectSegment), ncand - min(ncand, part * kSelectSegment));
    uint64_t key[kSelKeysPerThread];
#pragma unroll
    for (int i = 0; i < kSelKeysPerThread - 1; ++i) {
        const uint32_t at = uint32_t(i) * kSelThreads + tid;
        key[i] = at < here ? seg[at] : kEmptyKey;
    }
    const bool with_prev = dense_blocks == 0;
    auto prev_key = [&]() { return with_prev && tid < cb.k ? cb.topk[size_t(q) * cb.k + tid] : kEmptyKey; };
    key[kSelKeysPerThread - 1] = parts == 1 ? prev_key() : kEmptyKey;
    int m = block_smallest(key, cb.k, sh);
    if (parts > 1) {
        // leave this segment's best in place; the CTA that arrives last merges all of them with the running top-k
        for (int i = tid; i < cb.k; i += kSelThreads) __stcg(seg + i, i < m ? sh.sorted[i] : kEmptyKey);
        __threadfence();
        __syncthreads();
        if (tid == 0) sh.last = atomicAdd(&cb.done[q], 1u) == parts - 1;
        __syncthreads();
        if (!sh.last) return;
        __threadfence();
        const uint32_t total = parts * uint32_t(cb.k);                  // at most kSelectSegment (launch_select)
#pragma unroll
        for (int i = 0; i < kSelKeysPerThread - 1; ++i) {
            const uint32_t at = uint32_t(i) * kSelThreads + tid;
            key[i] = at < total ? __ldcg(list + size_t(at / cb.k) * kSelectSegment + at % cb.k) : kEmptyKey;
        }
        key[kSelKeysPerThread - 1] = prev_key();
        m = block_smallest(key, cb.k, sh);
        if (tid == 0) cb.done[q] = 0;
    }
    for (int i = tid; i < cb.k; i += kSelThreads) cb.topk[size_t(q) * cb.k + i] = i < m ? sh.sorted[i] : kEmptyKey;
    if (tid == 0) {
        // kEmptyKey until k results exist: everything still passes.  A query that the filter has lost is searched again by
        // itself: until then nothing of it need survive, in this scan or a later one.
        const uint64_t nothing = make_key(INFINITY, 0u);
        if (cb.over != nullptr && (spilled || cb.thr[q] == nothing)) cb.thr[q] = nothing;
        else cb.thr[q] = m == cb.k ? sh.sorted[cb.k - 1] : kEmptyKey;
        cb.cnt[q] = 0;
    }
    if (out.scores == nullptr) return;
    const unsigned long long allowed = out.n_allowed ? *reinterpret_cast<const volatile unsigned long long *>(out.n_allowed) : (unsigned long long)out.n;
    const int k_eff = int(min((unsigned long long)cb.k, min((unsigned long long)out.n, allowed)));
    const size_t row = (size_t(q) + out.q0) * (out.stride_is_k ? cb.k : k_eff);
    for (int i = tid; i < k_eff; i += kSelThreads) {
        // (-inf, 0) padding as search.rs:4341-4352
        out.scores[row + i] = i < m ? desc_bits_to_score(uint32_t(sh.sorted[i] >> 32)) : -INFINITY;
        out.slots[row + i] = i < m ? int64_t(sh.sorted[i] & 0xffffffffu) : 0;
    }
    // (the host reads the rows after the kernel has ended; only the status words are passed on between CTAs)
    __syncthreads();
    if (tid != 0) return;
    __threadfence();
    if (atomicAdd(out.finished, 1u) != uint32_t(out.nq) - 1u) return;
    __threadfence();
    *out.finished = 0;
    volatile DeviceFlags *f = out.flags, *host = out.flags_host;
    const uint32_t overflow = f->overflow;
    host->first_invalid = f->first_invalid; host->n_allowed = f->n_allowed; host->first_unknown = f->first_unknown;
    host->n_live = f->n_live; host->overflow = overflow; host->error = f->error; host->k_eff = uint32_t(k_eff);
    if (overflow == 0) {
        f->first_invalid = ~0ull; f->n_allowed = 0; f->first_unknown = ~0ull;
        f->n_live = 0; f->error = 0; f->k_eff = 0;
    }
}

}  // namespace

int candidate_capacity(size_t k, size_t nq, size_t n) {
    if (k > size_t(kSelectMaxK)) return 8192;
    // The first chunk of a search writes every key of `capacity` vectors, so a longer list saves chunks: 131,072 keys let
    // one query over 10 M vectors finish in two scans.  Bounded by what the merge of the parts holds (parts * k keys), by
    // 2^22 keys over all queries and by the index.  2^20 / 2^22 / 2^24 keys, us: 1 M x 1536 4-bit, 128 queries 403 / 404 / 470,
    // 512 707 / 727 / 784; 1.2 M x 200 4-bit, 32 216 / 228 / 226, 128 255 / 254 / 328; 1 M x 768 2-bit, 128 630 / 597 / 675.
    size_t parts = 1;
    while (parts < 32 && 2 * parts * k <= size_t(kSelectSegment) && 2 * parts * nq * kSelectSegment <= (size_t(1) << 22) &&
           parts * kSelectSegment < n)
        parts *= 2;
    return int(parts * kSelectSegment);
}

cudaError_t launch_select(const CandidateBuffers &cb, int nq, uint32_t dense_blocks, const uint32_t *n_live, const SearchOutput *out, cudaStream_t s) {
    if (nq <= 0) return cudaSuccess;
    if (cb.k > kSelectMaxK && out != nullptr) return cudaErrorInvalidValue;
    if (cb.k > kSelectMaxK) return launch_select_sort(cb, nq, int(dense_blocks) * 32, s);
    const uint32_t list = dense_blocks > 0 ? std::min<uint32_t>(dense_blocks * 32u, uint32_t(cb.cap)) : uint32_t(cb.cap);
    const uint32_t parts = (list + kSelectSegment - 1) / kSelectSegment;
    if (parts > 1 && parts * uint32_t(cb.k) > uint32_t(kSelectSegment)) return cudaErrorInvalidValue;
    // queries on grid.y would stop at 65,535: larger batches in slices
    for (int q0 = 0; q0 < nq; q0 += 32768) {
        CandidateBuffers part = cb;
        SearchOutput o{};
        if (out != nullptr) { o = *out; o.q0 = q0; }
        part.cand += size_t(q0) * cb.cap; part.cnt += q0; part.thr += q0; part.topk += size_t(q0) * cb.k; part.done += q0;
        if (part.over != nullptr) part.over += q0;
        select_parts_kernel<<<dim3(parts, unsigned(std::min(nq - q0, 32768))), kSelThreads, 0, s>>>(part, dense_blocks, n_live, o);
    }
    return cudaGetLastError();
}

}  // namespace tv
