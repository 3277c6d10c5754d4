// u8-LUT scan for a few queries (2/3-bit codes, and every geometry the permute-dot family does not cover).
// isum = sum_g U[g][byte>>4] + U[g][16 + (byte&15)] exactly; float epilogue per mode:
//   kModeLutMulAdd: (f32)isum * scale + bias                      (search.rs:1176)
//   kModeLutFlush : acc = bias; per 256 groups acc = fma(scale, (f32)isum_batch, acc)   (search.rs:1596)
//
// With one query the scan should stream the codes; what bounds it is the two table lookups per byte.  A lookup is a byte
// permute, not a load: a 32-bit word holds the bytes of four vectors in one group, so the 16 entries of a half-byte sit in
// four registers and `prmt` picks the entries of four vectors at once.  A selector nibble above 7 asks for the sign of the
// byte it names, which is zero for table entries (at most 127), so two permutes (entries 0..7 with the nibbles as they are,
// entries 8..15 with bit 3 flipped) and an addition are an exact 16-entry lookup.  The eight nibbles of a word become the
// two selectors with one permute: h + (h >> 12) and l + (l << 12) put neighbouring nibbles side by side (on the multiply
// pipe, which is idle here).  Byte sums (at most 254 per group) are widened into 16-bit halves.  Per word and query: six
// permutes and about nine other integer operations, where loads from shared memory took eight loads and 24 operations.
// The tables of a group (two 16-byte shared-memory loads) serve NB code blocks of the warp.
#include <algorithm>

#include "scan_common.cuh"

namespace tv {
namespace {

constexpr int kLutThreads = 256;

template <int NQ, int NB>
__global__ void __launch_bounds__(kLutThreads) scan_lut_kernel(ScanParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kUnroll = 4 / NB < 2 ? 2 : 4 / NB;              // group steps whose code words are in flight
    const int ng = p.ngroups;
    uint4 *lut = reinterpret_cast<uint4 *>(smem_raw);             // [NQ][ng][high, low]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nq_here = min(NQ, p.nq);
    for (int q = 0; q < NQ; ++q) {
        const uint4 *src = reinterpret_cast<const uint4 *>(p.luts + size_t(p.q_base + min(q, nq_here - 1)) * p.lut_pitch);
        for (int i = tid; i < ng * 2; i += kLutThreads) lut[q * ng * 2 + i] = src[i];
    }
    __syncthreads();
    uint32_t pos_end = p.pos_end;
    if (p.live_blocks != nullptr) pos_end = min(pos_end, *p.n_live);
    const uint32_t pos_begin = min(p.pos_begin, pos_end);
    // A warp instruction reads 128 contiguous bytes = four group rows of a block: lane = (row lane / 8, vectors
    // 4 * (lane % 8) .. + 3).  Each lane sums its quarter of the groups for its four vectors; the four lanes that share
    // the vectors then exchange partial sums so that lane (quad, row) finishes vector 4 * quad + row.
    const int row = lane >> 3, quad = lane & 7;
    const int my_vec = 4 * quad + row;
    const uint32_t warps = gridDim.x * (kLutThreads / 32);
    const int batch = p.mode == kModeLutFlush ? 256 : 1024;       // groups per exact sum: at most 256 per lane, so 16 bits hold it
    for (uint32_t pos0 = pos_begin + (blockIdx.x * (kLutThreads / 32) + warp) * NB; pos0 < pos_end; pos0 += warps * NB) {
        const uint32_t *src[NB];
        uint32_t blk[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const uint32_t pos = min(pos0 + b, pos_end - 1);      // past the end: the last block again, not written out
            blk[b] = p.live_blocks ? p.live_blocks[pos] : pos;
            src[b] = reinterpret_cast<const uint32_t *>(p.codes + size_t(blk[b]) * ng * kLanes) + lane;
        }
        float facc[NQ][NB];
        uint32_t total[NQ][NB];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int b = 0; b < NB; ++b) { facc[q][b] = p.qbias[p.q_base + min(q, nq_here - 1)]; total[q][b] = 0; }
        for (int g0 = 0; g0 < ng; g0 += batch) {
            const int g1 = min(g0 + batch, ng);
            uint32_t even[NQ][NB], odd[NQ][NB];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
#pragma unroll
                for (int b = 0; b < NB; ++b) { even[q][b] = 0; odd[q][b] = 0; }
            auto add = [&](int g, const uint32_t (&w)[NB]) {
                uint32_t sel[NB], inv[NB], sel_l[NB], inv_l[NB];
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const uint32_t h = w[b] & 0xf0f0f0f0u, l = w[b] & 0x0f0f0f0fu;
                    // bytes 0 and 2 of the first, 1 and 3 of the second: nibbles of vectors (1, 0) and (3, 2)
                    sel[b] = prmt(mad_hi(h, 1u << 20, h), l * 0x1001u, 0x7520);
                    inv[b] = sel[b] ^ 0x88888888u;
                    sel_l[b] = mad_hi(sel[b], 0x10000u, 0u);
                    inv_l[b] = mad_hi(inv[b], 0x10000u, 0u);
                }
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    const uint4 th = lut[(q * ng + g) * 2], tl = lut[(q * ng + g) * 2 + 1];
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        const uint32_t v = prmt(th.x, th.y, sel[b]) + prmt(th.z, th.w, inv[b]) + prmt(tl.x, tl.y, sel_l[b]) + prmt(tl.z, tl.w, inv_l[b]);
                        even[q][b] += v & 0x00ff00ffu;
                        odd[q][b] = mad_hi(v, 1u << 24, odd[q][b]);   // v >> 8: byte 2 is taken out again below
                    }
                }
            };
            // every row of a full step is below g1
            const int full = (g1 - g0) / (4 * kUnroll);
            const size_t at0 = size_t(g0) * 8;
            uint32_t w[kUnroll][NB];
            if (full > 0) {
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
#pragma unroll
                    for (int b = 0; b < NB; ++b) w[u][b] = __ldg(src[b] + at0 + u * 32);
            }
            for (int s = 0; s < full; ++s) {
                uint32_t cur[kUnroll][NB];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
#pragma unroll
                    for (int b = 0; b < NB; ++b) cur[u][b] = w[u][b];
                if (s + 1 < full) {
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u)
#pragma unroll
                        for (int b = 0; b < NB; ++b) w[u][b] = __ldg(src[b] + at0 + size_t(s + 1) * (32 * kUnroll) + u * 32);
                }
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) add(g0 + (s * kUnroll + u) * 4 + row, cur[u]);
            }
            for (int g = g0 + full * 4 * kUnroll + row; g < g1; g += 4) {
                uint32_t t[NB];
#pragma unroll
                for (int b = 0; b < NB; ++b) t[b] = __ldg(src[b] + size_t(g - row) * 8);
                add(g, t);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < NQ; ++q)
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const uint32_t s1 = even[q][b] & 0xffffu, s3 = even[q][b] >> 16;      // bytes 0 and 2: vectors 1 and 3
                    const uint32_t rest = odd[q][b] - (s3 << 8);
                    const uint32_t s0 = rest & 0xffffu, s2 = rest >> 16;                  // bytes 1 and 3: vectors 0 and 2
                    const bool r0 = (row & 1) != 0, r1 = (row & 2) != 0;
                    uint32_t a = r0 ? s1 : s0, c = r0 ? s3 : s2;
                    a += __shfl_xor_sync(kFullMask, r0 ? s0 : s1, 8);
                    c += __shfl_xor_sync(kFullMask, r0 ? s2 : s3, 8);
                    uint32_t mine = r1 ? c : a;
                    mine += __shfl_xor_sync(kFullMask, r1 ? a : c, 16);
                    facc[q][b] = fmaf(p.qscale[p.q_base + min(q, nq_here - 1)], float(int(mine)), facc[q][b]);
                    total[q][b] += mine;
                }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            const uint32_t pos = pos0 + b;
            if (pos >= pos_end) continue;
            const int64_t slot = int64_t(blk[b]) * kLanes + my_vec;
            const bool on = slot < p.n && (!p.mask || ((p.mask[slot >> 6] >> (slot & 63)) & 1ull));
            const float vs = on ? p.vec_scales[slot] : 0.0f;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (q >= nq_here) continue;
                const int ql = p.q_base + q;
                const float pre = p.mode == kModeLutFlush ? facc[q][b] : __fadd_rn(__fmul_rn(float(int(total[q][b])), p.qscale[ql]), p.qbias[ql]);
                const float score = __fmul_rn(pre, vs);
                if (p.dense) p.cb.cand[size_t(ql) * p.cb.cap + size_t(pos - pos_begin) * kLanes + my_vec] = on ? make_key(score, uint32_t(slot)) : kEmptyKey;
                else if (on) push_candidate(p.cb, ql, score, uint32_t(slot), p.cb.thr[ql], p.cb.lo ? p.cb.lo[ql] : 0ull);
            }
        }
    }
}

}  // namespace

int scan_lut_width(int ngroups, size_t smem_limit) {
    const size_t table = size_t(ngroups) * 32;
    if (table == 0) return 0;
    const size_t fit = (smem_limit > 1024 ? smem_limit - 1024 : 0) / table;
    return fit >= 4 ? 4 : (fit >= 2 ? 2 : (fit >= 1 ? 1 : 0));
}

template <int NQ, int NB>
static cudaError_t launch_lut(const ScanParams &p, int sm_count, cudaStream_t s) {
    const size_t smem = size_t(NQ) * p.ngroups * 32;
    auto kern = scan_lut_kernel<NQ, NB>;
    cudaError_t e = allow_dynamic_shared(kern);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kLutThreads, smem);
    if (e != cudaSuccess) return e;
    const uint32_t tasks = (p.pos_end - p.pos_begin + NB - 1) / NB, per_cta = kLutThreads / 32;
    kern<<<std::min(uint32_t(sm_count * std::max(per_sm, 1)), (tasks + per_cta - 1) / per_cta), kLutThreads, smem, s>>>(p);
    return cudaGetLastError();
}

// Up to 4 queries; the kernel's inner loop reads all NQ tables (unused ones repeat the last query).
cudaError_t launch_scan_lut(const ScanParams &p, int sm_count, cudaStream_t s) {
    if (p.nq <= 0 || p.pos_end <= p.pos_begin) return cudaSuccess;
    if (p.nq > 4) return cudaErrorInvalidValue;
    // two blocks per warp share the table loads; below four waves of warps a block each keeps more of the chip busy
    const bool pairs = p.pos_end - p.pos_begin >= uint32_t(sm_count) * 160;
    if (p.nq == 1) return pairs ? launch_lut<1, 2>(p, sm_count, s) : launch_lut<1, 1>(p, sm_count, s);
    if (p.nq == 2) return pairs ? launch_lut<2, 2>(p, sm_count, s) : launch_lut<2, 1>(p, sm_count, s);
    return pairs ? launch_lut<4, 2>(p, sm_count, s) : launch_lut<4, 1>(p, sm_count, s);
}

}  // namespace tv
