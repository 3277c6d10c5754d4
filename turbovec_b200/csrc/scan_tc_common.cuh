// Device-side pieces shared by the tensor-memory scans (scan_tc.cu, scan_tc_wide.cu, scan_tc_dense.cu, scan_tc_dense2.cu):
// constants of the MMA tiling, bounded mbarrier waits, the nibble -> int8 level lookup, shared-memory and
// instruction descriptors, TMA and TMEM wrappers, and the float epilogue of the score families.
#pragma once
#include <cuda.h>

#include <cfloat>
#include <climits>
#include <cstddef>

#include "search.cuh"
#include "tv_common.cuh"

namespace tv {
namespace {

constexpr int kMmaM = 128;                                    // vectors per accumulator tile (TMEM lanes)
constexpr int kMaxTileQueries = 256;                          // largest MMA N (query columns of a work item)
constexpr int kSlabK = 128;                                   // int8 elements (bytes) of K per stage
constexpr int kATileBytes = kMmaM * kSlabK;                   // 16 KB per accumulator tile and stage
constexpr int kExpandWarps = 8;
constexpr int kEpilogueWarps = 8;                             // two per TMEM lane quarter, 128 columns each
constexpr int kThreadsTc = (2 + kEpilogueWarps + kExpandWarps) * 32;   // 576
constexpr uint32_t kWaitLimitTc = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t *error_flag) {
    for (uint32_t i = 0; i < kWaitLimitTc; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(error_flag, 2u);
    return false;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// high 32 bits of a * b + c on the FMA pipe: a right shift that does not load the ALU pipe
__device__ __forceinline__ uint32_t mad_hi(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// Eight nibbles of x -> eight int8 levels; output byte i of (lo, hi) belongs to nibble i / i+4 of x.
__device__ __forceinline__ void expand8(uint32_t x, const uint32_t (&T)[4], uint32_t &lo, uint32_t &hi) {
    const uint32_t idx = x & 0x77777777u;
    const uint32_t pick = mad_hi(x & 0x88888888u, 0x80000000u, 0x32103210u);   // ((x >> 1) & 0x4..4) | 0x3210..
    lo = prmt(prmt(T[0], T[1], idx), prmt(T[2], T[3], idx), pick);
    const uint32_t idx_h = mad_hi(idx, 0x10000u, 0u), pick_h = mad_hi(pick, 0x10000u, 0u);
    hi = prmt(prmt(T[0], T[1], idx_h), prmt(T[2], T[3], idx_h), pick_h);
}

// K-major, 128-byte swizzle, 8-row groups 1024 B apart; version 1 (sm_100), base offset 0.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_byte_addr) {
    uint64_t d = 0;
    d |= uint64_t((smem_byte_addr >> 4) & 0x3fffu);           // start address
    d |= uint64_t(1) << 16;                                    // leading byte offset (unused for swizzled K-major)
    d |= uint64_t(1024 >> 4) << 32;                            // stride byte offset
    d |= uint64_t(1) << 46;                                    // descriptor version
    d |= uint64_t(2) << 61;                                    // SWIZZLE_128B
    return d;
}
// kind::i8: D = S32, A = B = signed 8-bit, both K-major, M = 128, N = NQT.
template <int NQT>
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
    constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(NQT >> 3) << 17) | (uint32_t(kMmaM >> 4) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(kIdesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// ---- CTA pairs (clusters of two, tcgen05 cta_group::2): scan_tc_dense2.cu ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Remote arrivals carry the default (CTA-scope release) semantics: what they publish was written to the arriving CTA's own
// shared memory and made visible to the asynchronous proxy by fence.proxy.async before the arrival; a cluster-scope
// release on every arrival cost more than the MMAs it guarded.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity, uint32_t *error_flag) {
    for (uint32_t i = 0; i < kWaitLimitTc; ++i)
        if (mbar_try_wait_cluster(bar, parity)) return true;
    atomicExch(error_flag, 3u);
    return false;
}
// kind::i8 across the pair: D = S32, A = B = signed 8-bit, both K-major, M = 256 (128 rows per CTA), N = 256.
__device__ __forceinline__ void umma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
    constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(256 >> 3) << 17) | (uint32_t(256 >> 4) << 24);
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(kIdesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// arrives on the barrier at `cluster_addr` (this CTA's or the peer's) once the pair's MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint32_t cluster_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_addr) : "memory");
}
// this CTA's half of a query slab; the transaction bytes are reported to the leader's barrier
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t leader_bar_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(leader_bar_addr), "r"(x), "r"(y) : "memory");
}

// Float epilogue of the score families; the integer sum is exact in all of them.  Permute-dot: fma((f32)S, scale, bias)
// (search.rs:1523, 1793).  u8-LUT, mul-add family: (f32)isum * scale + bias (search.rs:1176).  u8-LUT, flush family
// with at most 256 byte-groups (`fused`): one fma(scale, (f32)isum, bias) (search.rs:516, 577, 1596) - the same
// single rounding as the permute-dot form.  Then x vec_scale.
template <bool ONEHOT>
__device__ __forceinline__ float final_score(bool fused, uint32_t isum, float qs, float qb, float vs) {
    const float f = float(int(isum));
    if constexpr (ONEHOT) return __fmul_rn(fused ? fmaf(qs, f, qb) : __fadd_rn(__fmul_rn(f, qs), qb), vs);
    else return __fmul_rn(fmaf(f, qs, qb), vs);
}


// Integer bound that dismisses most accumulator columns without converting them to float.
// For one query (scale qs > 0, bias qb, threshold score t > 0) and every vector of a work item (vector scales
// 0 <= vs <= vs_max), a score fmul(fma((f32)isum, qs, qb), vs) can reach t only if
//     isum >= ((t / vs_max) - qb) / qs
// up to the roundings of the conversion, the fma and the multiply (each within 2^-23 relative).  The returned integer
// lies below that bound by a margin a thousand times those roundings plus two units, so `isum >= bound` is necessary
// for a candidate; the columns that satisfy it are scored exactly afterwards.  The integer compare costs one
// instruction per column where the exact score costs four, one of them (int -> float) on a quarter-rate unit; on
// L2-normalised data the vector scales of an item differ by a few percent, so hardly any column survives it.
// t <= 0 (no k-th result yet, or a non-positive one): everything is kept.  vs_max = 0 with t > 0: nothing can pass.
__device__ __forceinline__ int dismissal_bound(float qs, float qb, float t, float vs_max) {
    if (!(t > 0.0f)) return INT_MIN;
    if (!(qs > 0.0f)) return qb * vs_max >= t ? INT_MIN : INT_MAX;     // a column without a query has t = +inf
    const float g = t / vs_max;                                        // +inf when vs_max is 0
    const float bound = (g - qb) / qs;
    const float margin = 1.0e-5f * (fabsf(g) + fabsf(qb)) / qs + 2.0f;
    const float lo = bound - margin;
    if (!(lo < 2.0e9f)) return INT_MAX;
    if (lo < -2.0e9f) return INT_MIN;
    return __float2int_rd(lo);
}


// First chunk of a search: the 32 accumulator columns of a piece (queries ql0 .. ql0 + 31 of one vector) go to position `at`
// of their queries' candidate lists, every one of them (kEmptyKey for a slot that the mask does not allow).  qscale / qbias
// point at the piece's first column.
template <bool ONEHOT>
__device__ __forceinline__ void write_piece(const uint32_t (&acc)[32], const float *qscale, const float *qbias, bool fused, float vs,
                                            bool live, int64_t slot, int ql0, int nq_end, uint32_t at, const CandidateBuffers &cb) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const int ql = ql0 + j;
        if (ql < nq_end) {
            const float score = final_score<ONEHOT>(fused, acc[j], qscale[j], qbias[j], vs);
            cb.cand[size_t(ql) * cb.cap + at] = live ? make_key(score, uint32_t(slot)) : kEmptyKey;
        }
    }
}

__device__ __forceinline__ void append_candidate(const CandidateBuffers &cb, int ql, uint64_t key) {
    if (key < cb.thr[ql] && (cb.lo == nullptr || key >= cb.lo[ql])) {
        const uint32_t at = atomicAdd(&cb.cnt[ql], 1u);
        if (at < uint32_t(cb.cap)) cb.cand[size_t(ql) * cb.cap + at] = key;
    }
}

// Which runs of 8 of a piece's 32 columns hold a sum at or above the column's bound for this lane's vector (bit = run).
__device__ __forceinline__ uint32_t surviving_runs(const uint32_t (&acc)[32], const int *ibound, bool live) {
    uint32_t runs = 0;
    const int4 *pi = reinterpret_cast<const int4 *>(ibound);
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
        const int4 b = pi[j4];
        const bool may = (int(acc[4 * j4 + 0]) >= b.x) | (int(acc[4 * j4 + 1]) >= b.y) | (int(acc[4 * j4 + 2]) >= b.z) |
                         (int(acc[4 * j4 + 3]) >= b.w);
        runs |= uint32_t(may) << (j4 >> 1);
    }
    return live ? runs : 0u;
}

// Later chunks: one integer compare per column dismisses the piece unless some column could be a candidate
// (dismissal_bound).  Each lane keeps the outcome per run of 8 columns; the runs that any lane of the warp flagged are
// re-read from tensor memory (address `taddr` = the piece's first column) and scored exactly by the lanes that flagged
// them, and `push` gets the (query, key) pairs that reach the query's k-th score.  All pointers are at the piece's first
// column; every lane of the warp must call this.
template <bool ONEHOT, typename Push>
__device__ __forceinline__ void sift_piece(const uint32_t (&acc)[32], const int *ibound, const float *qscale, const float *qbias,
                                           const float *qthr, bool fused, float vs, bool live, int64_t slot, int ql0, uint32_t taddr,
                                           Push push) {
    const uint32_t runs = surviving_runs(acc, ibound, live);
    const uint32_t warp_runs = __reduce_or_sync(0xffffffffu, runs);
    if (warp_runs == 0) return;
#pragma unroll 1
    for (int c1 = 0; c1 < 32; c1 += 8) {
        if (!((warp_runs >> (c1 >> 3)) & 1u)) continue;
        uint32_t a8[8];
        tmem_ld8(taddr + c1, a8);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if ((runs >> (c1 >> 3)) & 1u) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = c1 + e;
                const float score = final_score<ONEHOT>(fused, a8[e], qscale[c], qbias[c], vs);
                if (score >= qthr[c]) push(ql0 + c, make_key(score, uint32_t(slot)));
            }
        }
    }
}

// Whether `scored` survivors of a filtering scan in the average chunk to come, and redoing `lost` queries whose lists overflow,
// would take longer than the form without the filter saves from here on (`spent`: what the filter still has to spend before).
__device__ __forceinline__ bool filter_hopeless(const ScanParams &p, float scored, float lost, int all_queries, float spent) {
    float budget = p.f_budget_us - spent;
    if (p.live_blocks != nullptr) {                       // the share of the positions that a mask leaves
        const uint32_t live = *p.n_live;
        budget *= float(live > p.pos_begin ? live - p.pos_begin : 0u) / float(p.f_positions - p.pos_begin);
    }
    if (lost > 0.5f * float(all_queries)) return true;    // most of the batch would be searched again
    const float redo = lost <= 0.0f ? 0.0f : lost < 8.0f ? p.f_redo_us * ceilf(lost * 0.25f) : p.f_redo_group_us * ceilf(lost * (1.0f / 256.0f));
    return scored * p.f_survivor_us * p.f_chunks + redo > budget + 60.0f;   // (60 us: the host's turn and a restart)
}

// ---- epilogue of scan_tc.cu and scan_tc_dense2.cu: every warp on its own ------------------------------------------
// An item with few K slabs leaves the epilogue about a thousand cycles, so it must not be a chain of barriers and
// dependent loads.  The query group of a CTA stays the same from item to item, so the parameters of its columns are read
// once; a warp derives the bounds of its columns from the largest scale of its own 32 vectors (a reciprocal and two
// multiply-adds per column, four columns to a lane), which is also a tighter bound than one over the whole tile, and meets
// no other warp.  A bound is kept negated: one add-and-max per column tells whether a run of 8 holds a survivor.
// Candidates go through a ring of the warp: appending one takes a global atomic whose result says where it goes, about a
// microsecond that the warp would sit out for every single candidate; it writes them out together, one lane each.
constexpr int kWarpColumns = 128;                             // most columns of one epilogue warp
constexpr uint32_t kRingSize = 64;
constexpr int kFar = 1 << 29;                                 // beyond every integer sum (at most 127 * 127 * 16384 in magnitude)
struct WarpRing {                    // the warp keeps the fill count in a register
    uint64_t key[kRingSize];
    uint32_t ql[kRingSize];
};
struct EpilogueShared {
    float qscale[kMaxTileQueries];    // per-query parameters of the query group
    float qbias[kMaxTileQueries];
    float qthr[kMaxTileQueries];      // score of the current k-th key (-inf while fewer than k results exist)
    uint32_t qslot[kMaxTileQueries];  // its slot: equal scores count only from smaller slots
    int nbound[kEpilogueWarps][kWarpColumns];   // per warp and column: minus the integer sum below which no vector of the warp is a candidate
    WarpRing ring[kEpilogueWarps];
};

// One column's terms of the dismissal bound (see dismissal_bound): bound = u / vs_max - w, less the margin.
__device__ __forceinline__ void column_terms(float qs, float qb, float t, float &u, float &w) {
    u = t / qs; w = qb / qs;
    if (t == INFINITY) { u = 0.0f; w = -1e30f; }                              // no query: nothing passes
    else if (!(t > 0.0f) || !(qs > 0.0f) || !(u <= FLT_MAX) || !(fabsf(w) <= FLT_MAX)) { u = 0.0f; w = 1e30f; }   // everything passes
}
__device__ __forceinline__ int negated_bound(float u, float w, float inv_vs) {
    const float x = u * inv_vs;
    const float lo = (x - w) - (1.0e-5f * (x + fabsf(w)) + 2.0f);
    return -__float2int_rd(fminf(fmaxf(lo, -float(kFar)), float(kFar)));
}

// Parameters of query group `qg` (NQT columns), by all epilogue threads; barriers on both sides are the caller's.
template <int NQT>
__device__ __forceinline__ void load_columns(EpilogueShared &es, const ScanParams &p, int qg, int et) {
    if (et >= NQT) return;
    const int ql = qg * NQT + et;
    float qs = 0.f, qb = 0.f, th = INFINITY;
    uint32_t slot = 0;
    if (ql < p.q_base + p.nq) {
        qs = p.qscale[ql]; qb = p.qbias[ql];
        const uint64_t key = p.cb.thr[ql];
        th = key == kEmptyKey ? -INFINITY : desc_bits_to_score(uint32_t(key >> 32));
        slot = uint32_t(key);
    }
    es.qscale[et] = qs; es.qbias[et] = qb; es.qthr[et] = th; es.qslot[et] = slot;
}

// RAW: a survivor of a filtering scan, appended unseen (its exact key is computed later)
template <bool RAW>
__device__ __forceinline__ void append_any(const CandidateBuffers &cb, int ql, uint64_t key) {
    if constexpr (RAW) {
        const uint32_t at = atomicAdd(&cb.cnt[ql], 1u);
        if (at < uint32_t(cb.cap)) cb.cand[size_t(ql) * cb.cap + at] = key;
    } else {
        append_candidate(cb, ql, key);
    }
}
// by the whole warp: lanes with `on` add their entry; `fill` (warp-uniform) counts the entries
template <bool RAW>
__device__ __forceinline__ void ring_push(WarpRing &ring, uint32_t &fill, const CandidateBuffers &cb, bool on, int ql, uint64_t key, int lane) {
    const uint32_t who = __ballot_sync(kFullMask, on);
    if (on) {
        const uint32_t at = fill + __popc(who & ((1u << lane) - 1u));
        if (at < kRingSize) { ring.key[at] = key; ring.ql[at] = uint32_t(ql); }
        else append_any<RAW>(cb, ql, key);
    }
    fill = min(fill + __popc(who), kRingSize);
}
// by the whole warp: writes the ring out when it holds at least `limit` entries
template <bool RAW>
__device__ __forceinline__ void ring_flush(WarpRing &ring, uint32_t &fill, const CandidateBuffers &cb, uint32_t limit, int lane) {
    if (fill < limit) return;
    __syncwarp();
    for (uint32_t i = lane; i < fill; i += 32) append_any<RAW>(cb, int(ring.ql[i]), ring.key[i]);
    __syncwarp();
    fill = 0;
}

// Which of a run's 8 columns hold a key of this lane's vector below the column's k-th key (bit = column).
template <bool ONEHOT>
__device__ __forceinline__ uint32_t better_columns(const uint32_t (&acc)[32], int r, const float *qscale, const float *qbias, const float *qthr,
                                                   const uint32_t *qslot, bool fused, float vs, uint32_t slot) {
    uint32_t better = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = 8 * r + 4 * h;
        const float4 s = *reinterpret_cast<const float4 *>(qscale + c), b = *reinterpret_cast<const float4 *>(qbias + c),
                     t = *reinterpret_cast<const float4 *>(qthr + c);
        const uint4 w = *reinterpret_cast<const uint4 *>(qslot + c);
        const float x0 = final_score<ONEHOT>(fused, acc[c], s.x, b.x, vs), x1 = final_score<ONEHOT>(fused, acc[c + 1], s.y, b.y, vs);
        const float x2 = final_score<ONEHOT>(fused, acc[c + 2], s.z, b.z, vs), x3 = final_score<ONEHOT>(fused, acc[c + 3], s.w, b.w, vs);
        better |= (uint32_t(x0 > t.x || (x0 == t.x && slot < w.x)) | uint32_t(x1 > t.y || (x1 == t.y && slot < w.y)) << 1 |
                   uint32_t(x2 > t.z || (x2 == t.z && slot < w.z)) << 2 | uint32_t(x3 > t.w || (x3 == t.w && slot < w.w)) << 3) << (4 * h);
    }
    return better;
}

// One piece (32 accumulator columns of the lane's vector) against the warp's bounds; all pointers at the piece's first
// column.  Of a run of 8 columns that any lane of the warp flags, every lane takes its own surviving columns one after the
// other (hardly ever more than one): the vector's own scale decides, by the exact score or, RAW, by the bound on it, whose
// margin covers its roundings; then (sum, slot) is appended.  Every lane must call this.
template <bool ONEHOT, bool RAW>
__device__ __forceinline__ void warp_sift(const uint32_t (&acc)[32], const int *nbound, const float *qscale, const float *qbias, const float *qthr,
                                          const uint32_t *qslot, bool fused, float vs, bool live, uint32_t slot, int ql0, WarpRing &ring,
                                          uint32_t &fill, const CandidateBuffers &cb, int lane) {
    uint32_t runs = 0;
    const int4 *pn = reinterpret_cast<const int4 *>(nbound);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int4 a = pn[2 * r], b = pn[2 * r + 1];
        int m = int(acc[8 * r]) + a.x;
        m = __viaddmax_s32(int(acc[8 * r + 1]), a.y, m);
        m = __viaddmax_s32(int(acc[8 * r + 2]), a.z, m);
        m = __viaddmax_s32(int(acc[8 * r + 3]), a.w, m);
        m = __viaddmax_s32(int(acc[8 * r + 4]), b.x, m);
        m = __viaddmax_s32(int(acc[8 * r + 5]), b.y, m);
        m = __viaddmax_s32(int(acc[8 * r + 6]), b.z, m);
        m = __viaddmax_s32(int(acc[8 * r + 7]), b.w, m);
        runs |= uint32_t(m >= 0) << r;
    }
    if (!live) runs = 0;
    const uint32_t warp_runs = __reduce_or_sync(kFullMask, runs);
    if (warp_runs == 0) return;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (!((warp_runs >> r) & 1u)) continue;
        const int4 a = pn[2 * r], b = pn[2 * r + 1];
        uint32_t mine = uint32_t(int(acc[8 * r]) + a.x >= 0) | uint32_t(int(acc[8 * r + 1]) + a.y >= 0) << 1 |
                        uint32_t(int(acc[8 * r + 2]) + a.z >= 0) << 2 | uint32_t(int(acc[8 * r + 3]) + a.w >= 0) << 3 |
                        uint32_t(int(acc[8 * r + 4]) + b.x >= 0) << 4 | uint32_t(int(acc[8 * r + 5]) + b.y >= 0) << 5 |
                        uint32_t(int(acc[8 * r + 6]) + b.z >= 0) << 6 | uint32_t(int(acc[8 * r + 7]) + b.w >= 0) << 7;
        if (!live) mine = 0;
        for (int pass = 0; __any_sync(kFullMask, mine != 0); ++pass) {
            // A second column of some vector: often a copy of a row that is among the results of many columns.  Such a tie with
            // a smaller slot is no candidate, and going through them one by one costs several times the scan (1.2 M x 200
            // 4-bit, half of the rows copies, 1,024 queries next to them: 7.9 ms, 2.9 this way).
            if constexpr (!RAW)
                if (pass == 1) {
                    mine &= better_columns<ONEHOT>(acc, r, qscale, qbias, qthr, qslot, fused, vs, slot);
                    if (!__any_sync(kFullMask, mine != 0)) break;
                }
            const int e = mine ? __ffs(int(mine)) - 1 : 0;
            uint32_t sum = acc[8 * r];
#pragma unroll
            for (int i = 1; i < 8; ++i) sum = e == i ? acc[8 * r + i] : sum;
            const int c = 8 * r + e;
            const float score = final_score<ONEHOT>(fused, sum, qscale[c], qbias[c], vs), t = qthr[c];
            bool on = mine != 0;
            uint64_t key;
            if constexpr (RAW) {
                on = on && !(score + 1.0e-5f * (fabsf(score) + fabsf(t)) < t);   // (an infinite score compares with nothing: kept)
                key = uint64_t(sum) << 32 | slot;
            } else {
                on = on && score >= t;
                key = make_key(score, slot);
            }
            ring_push<RAW>(ring, fill, cb, on, ql0 + c, key, lane);
            mine &= mine - 1;
        }
    }
}

}  // namespace
}  // namespace tv
