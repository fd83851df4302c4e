// Histogram accumulation in integers for any loss: `update_hist!` / `_hist!` (src/fit-utils.jl:345-394; GPU counterpart
// `hist_kernel!`, ext/EvoTreesKernelAbstractionsExt/fit-utils.jl:57-95).  Device code of k_histg and of the quantisation in
// k_tree_begin.
//
// Numbers.  Every gradient channel is scaled by 2^s, the power of two that puts its max |g| just below 2^hb, and a row's value is
// taken apart into whole numbers: hi = rint(g 2^s), lo = rint(rest 2^(hb + 1)) -- 2 hb + 1 bits below max |g|, 37 to 43 as the
// number of rows allows (evb_hg_configure) -- and what is left after both, which is zero for every float32 that is not smaller
// than max |g| by 2^(2 hb - 23) or more.  An image cell holds two 32-bit words per channel, the sums of hi and of lo:
// 2^(31 - hb) - 32 rows fit, and one `red.shared.add.u32` per word is the whole update -- no read-modify-write chain, all warps
// of a CTA share one image.  One more word counts the rows.
// Rows with something left are queued (their ids) while the rest of a piece passes.  Few of them go to a second set of
// accumulators, 2 hb + 2 bits further down, one global reduction per feature and channel; many take the piece through the image
// once more with what is left in place of g (`accumulate`).  So every sum is the exact sum of the rows' float32 gradients (to
// 2^-63 of max |g| or less), whatever the order of the rows, however they are cut into pieces and however wide the range of a
// channel: a float sum kept 24 bits of every row, fixed point of any width alone would lose rows far below the largest.
// Least squares: unit weights pack (q >> 6, (q & 63) | 1 << 19 with the row count in the top 13 bits, |q| < 2^24) into two
// words in all; with weights, one target, all columns and up to 128 bins g is rounded to 29 bits below max |g| first.
//
// Lanes.  Lane = row of a tile of 32 rows, so a lane has its row's gradients and bins in registers and nothing is shuffled.  A
// row of bins is a sequence of 32-bit words (four features each), cut into parts of 8, then 4, 2 or 1 words.  A part owns 32
// image columns, 8 / W replicas of its W words side by side.  In step s of a part lane l adds the four features of word
// (l + s) % W into replica (l / W) % (8 / W), starting with feature l / 8.  So the 32 lanes of every reduction hit 32
// different banks (8 column groups of four lanes, each with another feature), and few features cost few reductions: ten
// features are 3 words instead of the 16 features of a 16-byte chunk.
// What bounds it is the shared-memory pipe: 4 features x planes reductions per step against two dozen other instructions.
// Measured (1.5M x 50 rows at the root, four channels + count): 138 us with the rows spread over the lanes by shuffles.
#pragma once
#include "evb_internal.cuh"
#include <float.h>

namespace evb_hg {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MAX_NQ = 5;     // channels of a CTA
constexpr int QUEUE = 384;    // rows of a piece with something left that are remembered
constexpr int QUEUE_BYTES = (QUEUE + 4) * 4; // their ids, then how many there are

struct Args {
    const uint8_t *xT;
    const int32_t *q;         // [n][NQP] words of this CTA's channels (scaled floats, packed: whole numbers)
    const uint32_t *rows;
    const LevelPlan *plan;
    const int32_t *cum, *rbase;
    unsigned long long *hsum; // [slot][bin][nq][SC]
    uint32_t *hcnt;           // [slot][bin][SC]
    unsigned long long *hlow; // [slot][SC][nq][bin]: sums of what hi and lo leave, of the slots in `low`
    uint32_t *low;            // [slot of the level] nonzero: hlow holds something; low_any: in any slot
    uint32_t *low_any;
    int hb;                   // bits of hi
    int RS, B, SC, nq, ch0;   // ch0: first channel of this CTA
    int F, word0, words;      // this CTA's words of a row
    int nfull, tails;         // parts of 8 words; bit mask of the tail parts (4, 2, 1)
    int TE;                   // tiles of 32 rows between two flushes
    int min_rows;             // rows per CTA below which fewer CTAs take part
    int pad_rows;             // what the flush of a slot costs, in rows
    long long n;              // rows of q
};

__host__ __device__ constexpr int planes(int NQ, bool CNT, bool PACK) { return PACK ? 2 : 2 * NQ + (CNT ? 1 : 0); }
__host__ __device__ constexpr int nqp(int NQ) { return NQ <= 2 ? NQ : NQ <= 4 ? 4 : 8; }
__host__ __device__ inline size_t part_bytes(int B, int P) { return (size_t)(B + 1) * P * 128; }
// words of a row -> parts of 8 and tail parts
__host__ __device__ inline void split_words(int words, int &nfull, int &tails) {
    nfull = words >> 3;
    tails = words & 7;
    if (tails == 7) { ++nfull; tails = 0; }
    if (tails == 3) tails = 4;
}
__host__ __device__ inline int nparts(int nfull, int tails) { return nfull + ((tails >> 2) & 1) + ((tails >> 1) & 1) + (tails & 1); }

template <int OFF>
__device__ __forceinline__ void red_at(uint32_t addr, uint32_t v) {
    asm volatile("red.shared.add.u32 [%0+%2], %1;" ::"r"(addr), "r"(v), "n"(OFF) : "memory");
}
template <int NQ, bool CNT, bool PACK, int C = 0>
__device__ __forceinline__ void red_cell(uint32_t addr, const uint32_t (&hi)[NQ], const uint32_t (&lo)[NQ]) {
    if constexpr (C < NQ) {
        red_at<256 * C>(addr, hi[C]);
        red_at<256 * C + 128>(addr, lo[C]);
        red_cell<NQ, CNT, PACK, C + 1>(addr, hi, lo);
    } else if constexpr (CNT && !PACK) {
        red_at<256 * NQ>(addr, 1u);
    }
}

// A scaled value -> hi and lo; returns what both leave, in units of lo.  Adding 1.5 2^23 rounds to whole numbers, half to even
// (|v| <= 2^22); every difference and product here is exact.
__device__ __forceinline__ float take_apart(float v, float two_lb, uint32_t &hi, uint32_t &lo) {
    constexpr float ONES = 12582912.0f;
    const float t = v + ONES, r = v - (t - ONES), u = fmaf(r, two_lb, ONES);
    hi = __float_as_uint(t) - 0x4b400000u;
    lo = __float_as_uint(u) - 0x4b400000u;
    return fmaf(r, two_lb, ONES - u);
}

template <int NQ>
__device__ __forceinline__ void load_q(const int32_t *p, int32_t (&q)[NQ]) {
    if constexpr (NQ == 1) q[0] = __ldg(p);
    else if constexpr (NQ == 2) { const int2 v = __ldg(reinterpret_cast<const int2 *>(p)); q[0] = v.x; q[1] = v.y; }
    else {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(p));
        q[0] = v.x; q[1] = v.y; q[2] = v.z;
        if constexpr (NQ >= 4) q[3] = v.w;
        if constexpr (NQ == 5) q[4] = __ldg(p + 4);
    }
}

// per-lane constants
struct Lane {
    uint32_t col[4];   // shared address of the image + the four features, in the lane's order
    uint32_t sel[4];   // PRMT selectors of their bins
    __device__ __forceinline__ void init(const void *smem, int lane) {
        const uint32_t img = (uint32_t)__cvta_generic_to_shared(smem);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int f = (k + (lane >> 3)) & 3;
            col[k] = img + 4u * (uint32_t)f;
            sel[k] = 0x4440u | (uint32_t)f;
        }
    }
};

// one part of W = 1 << LW words of the lane's row
template <int NQ, bool CNT, bool PACK, int LW>
__device__ __forceinline__ void part_steps(const uint8_t *xw, bool act, const uint32_t (&hi)[NQ], const uint32_t (&lo)[NQ], const Lane &ln, uint32_t poff, int lane) {
    constexpr int W = 1 << LW;
    constexpr uint32_t STRIDE = planes(NQ, CNT, PACK) * 128;
    uint32_t v[W];
    if (!act) { // past the end of the tile: all bins 0, what the lane adds lands in the guard row
#pragma unroll
        for (int s = 0; s < W; ++s) v[s] = 0u;
    } else if constexpr (W == 1) v[0] = __ldg(reinterpret_cast<const uint32_t *>(xw));
    else if constexpr (W == 2) { const uint2 t = __ldg(reinterpret_cast<const uint2 *>(xw)); v[0] = t.x; v[1] = t.y; }
    else {
#pragma unroll
        for (int h = 0; h < W / 4; ++h) {
            const uint4 t = __ldg(reinterpret_cast<const uint4 *>(xw) + h);
            v[4 * h] = t.x; v[4 * h + 1] = t.y; v[4 * h + 2] = t.z; v[4 * h + 3] = t.w;
        }
    }
    // v[s] <- word (lane + s) % W
#pragma unroll
    for (int r = 1; r < W; r <<= 1) {
        const bool on = (lane & r) != 0;
        uint32_t t[W];
#pragma unroll
        for (int s = 0; s < W; ++s) t[s] = on ? v[(s + r) & (W - 1)] : v[s];
#pragma unroll
        for (int s = 0; s < W; ++s) v[s] = t[s];
    }
    const uint32_t rep = 16u * (uint32_t)(lane & 7 & ~(W - 1)) + poff;
#pragma unroll
    for (int s = 0; s < W; ++s) {
        const uint32_t base = rep + 16u * (uint32_t)((lane + s) & (W - 1));
#pragma unroll
        for (int k = 0; k < 4; ++k) red_cell<NQ, CNT, PACK>(__byte_perm(v[s], 0u, ln.sel[k]) * STRIDE + (ln.col[k] + base), hi, lo);
    }
}

// The image -> the accumulators of a build slot; clears the image.  All warps of the CTA: one bin row of one part at a time,
// lane = image column, replicas added by shuffles.
template <int NQ, bool CNT, bool PACK, int LW>
__device__ __forceinline__ void flush_part(const Args &a, bool second, uint32_t *part, int f0, int slot) {
    constexpr int P = planes(NQ, CNT, PACK), W = 1 << LW;
    const int lane = threadIdx.x & 31, NW = blockDim.x >> 5, f = f0 + lane;
    const bool out = lane < 4 * W && f < a.F;
    auto replicas = [](auto v) {
#pragma unroll
        for (int o = 4 * W; o < 32; o <<= 1) v += __shfl_xor_sync(FULL, v, o);
        return v;
    };
    for (int bin = threadIdx.x >> 5; bin < a.B; bin += NW) {
        uint32_t *p = part + (size_t)(bin + 1) * (P * 32) + lane;
        const size_t cell = (size_t)slot * a.B + bin;
        if constexpr (PACK) {
            const uint32_t vh = p[0], vp = p[32];
            if (__ballot_sync(FULL, vp != 0u) == 0u) continue;
            p[0] = 0u; p[32] = 0u;
            const long long sum = replicas(((long long)(int32_t)vh << 6) + (long long)(vp & 0x7ffffu));
            const uint32_t cnt = replicas(vp >> 19);
            if (!out || cnt == 0u) continue;
            asm volatile("red.global.add.u64 [%0], %1;" ::"l"(a.hsum + cell * a.SC + f), "l"(sum) : "memory");
            asm volatile("red.global.add.u32 [%0], %1;" ::"l"(a.hcnt + cell * a.SC + f), "r"(cnt) : "memory");
        } else {
            if constexpr (CNT) {
                const uint32_t c = p[64 * NQ];
                if (__ballot_sync(FULL, c != 0u) == 0u) continue; // no row of these cells: all their words are zero
                p[64 * NQ] = 0u;
                const uint32_t cnt = replicas(c);
                if (out && cnt != 0u && !second) asm volatile("red.global.add.u32 [%0], %1;" ::"l"(a.hcnt + cell * a.SC + f), "r"(cnt) : "memory");
            }
            unsigned long long *sums = second ? a.hlow + (((size_t)slot * a.SC + f) * a.nq + a.ch0) * a.B + bin : a.hsum + (cell * a.nq + a.ch0) * a.SC + f;
            const size_t step = second ? a.B : a.SC;
            uint32_t hi[NQ], lo[NQ];
#pragma unroll
            for (int c = 0; c < NQ; ++c) { hi[c] = p[64 * c]; lo[c] = p[64 * c + 32]; }
#pragma unroll
            for (int c = 0; c < NQ; ++c) {
                p[64 * c] = 0u; p[64 * c + 32] = 0u;
                const long long sum = replicas(((long long)(int32_t)hi[c] << (a.hb + 1)) + (long long)(int32_t)lo[c]);
                if (out && sum != 0) asm volatile("red.global.add.u64 [%0], %1;" ::"l"(sums + c * step), "l"(sum) : "memory");
            }
        }
    }
}
template <int NQ, bool CNT, bool PACK>
__device__ __forceinline__ void flush(const Args &a, bool second, uint32_t *smem, int slot) {
    const size_t pw = (size_t)(a.B + 1) * planes(NQ, CNT, PACK) * 32; // words of a part
    int f0 = 4 * a.word0;
    for (int p = 0; p < a.nfull; ++p, smem += pw, f0 += 32) flush_part<NQ, CNT, PACK, 3>(a, second, smem, f0, slot);
    if (a.tails & 4) { flush_part<NQ, CNT, PACK, 2>(a, second, smem, f0, slot); smem += pw; f0 += 16; }
    if (a.tails & 2) { flush_part<NQ, CNT, PACK, 1>(a, second, smem, f0, slot); smem += pw; f0 += 8; }
    if (a.tails & 1) flush_part<NQ, CNT, PACK, 0>(a, second, smem, f0, slot);
}

// What is left of the queued rows -> hlow, one global reduction per feature and channel.  A warp takes a row, its lanes features.
template <int NQ>
__device__ __forceinline__ void add_left(const Args &a, const uint32_t *queue, int cnt, int slot, float two_lb) {
    constexpr int NQP = nqp(NQ);
    const int lane = threadIdx.x & 31, NW = blockDim.x >> 5, f0 = 4 * a.word0, nf = min(4 * a.words, a.F - f0);
    for (int e = threadIdx.x >> 5; e < cnt; e += NW) {
        const uint32_t rid = queue[e];
        int32_t q[NQ];
        long long v[NQ];
        load_q<NQ>(a.q + (size_t)rid * NQP, q);
#pragma unroll
        for (int c = 0; c < NQ; ++c) {
            uint32_t hi, lo;
            take_apart(take_apart(__int_as_float(q[c]), two_lb, hi, lo) * two_lb, two_lb, hi, lo);
            v[c] = ((long long)(int32_t)hi << (a.hb + 1)) + (long long)(int32_t)lo;
        }
        const uint8_t *x = a.xT + (size_t)rid * a.RS + f0;
        for (int f = lane; f < nf; f += 32) {
            unsigned long long *d = a.hlow + (((size_t)slot * a.SC + f0 + f) * a.nq + a.ch0) * a.B + (__ldg(x + f) - 1);
#pragma unroll
            for (int c = 0; c < NQ; ++c)
                if (v[c] != 0) asm volatile("red.global.add.u64 [%0], %1;" ::"l"(d + (size_t)c * a.B), "l"(v[c]) : "memory");
        }
    }
}

// Rows of the level's build nodes, cut into equal ranges; this CTA is `b` of `G`.  smem: image of all parts, zero on entry and
// on exit (guard rows excepted: nothing reads them); queue: QUEUE row ids and their number, zero on entry and on exit.
template <int NQ, bool CNT, bool PACK>
__device__ __forceinline__ void accumulate(const Args &a, uint32_t *smem, uint32_t *queue, int b, int G) {
    constexpr int P = planes(NQ, CNT, PACK), NQP = nqp(NQ);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, NW = blockDim.x >> 5;
    const int nbuild = a.plan->nbuild;
    // every slot is followed by pad_rows rows that do not exist
    const long long R = a.plan->R + (long long)nbuild * a.pad_rows;
    {
        const long long want = (R + a.min_rows - 1) / a.min_rows;
        if (want < G) G = want < 1 ? 1 : (int)want;
    }
    if (b >= G) return;
    const int lo = (int)(R * b / G), hi = (int)(R * (b + 1) / G);
    if (lo >= hi) return;
    int s;
    {
        int l = 0, r = nbuild - 1; // largest s with cum[s] + s * pad_rows <= lo
        while (l < r) { const int m = (l + r + 1) >> 1; if (a.cum[m] + m * a.pad_rows <= lo) l = m; else r = m - 1; }
        s = l;
    }
    Lane ln;
    ln.init(smem, lane);
    const uint32_t pb = (uint32_t)(a.B + 1) * P * 128;
    const float two_lb = __int_as_float((128 + a.hb) << 23); // 2^(hb + 1): lo has as many bits as hi and its sign
    const uint32_t *queued = queue + QUEUE;
    uint32_t left_rows = 0;
    for (; s < nbuild; ++s) {
        const int c0 = a.cum[s], off = s * a.pad_rows;
        if (c0 + off >= hi) break;
        const int pos = max(lo - off, c0), pe = min(hi - off, a.cum[s + 1]);
        if (pe <= pos) continue;
        const uint32_t *rows = a.rows + a.rbase[s];
        // A piece; every TE tiles the image is emptied.  second: once more, with what the first time left of each row.
        for (bool second = false;; second = true) {
            for (int p0 = pos; p0 < pe; p0 += a.TE * 32) {
                const int p1 = min(pe, p0 + a.TE * 32);
                int t = p0 + wid * 32;
                // row ids two tiles ahead; the row after the next is asked into L2 meanwhile (below the root rows are gathered)
                uint32_t ridN = t + lane < p1 ? __ldg(rows + t + lane) : 0u, ridNN = t + NW * 32 + lane < p1 ? __ldg(rows + t + NW * 32 + lane) : 0u;
                for (; t < p1; t += NW * 32) {
                    const uint32_t rid = ridN;
                    ridN = ridNN;
                    const bool act = t + lane < p1;
                    int32_t q[NQ];
#pragma unroll
                    for (int c = 0; c < NQ; ++c) q[c] = 0;
                    if (act) load_q<NQ>(a.q + (size_t)rid * NQP, q);
                    const int tn = t + 2 * NW * 32 + lane;
                    ridNN = tn < p1 ? __ldg(rows + tn) : 0u;
                    if (t + NW * 32 + lane < p1) {
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.xT + (size_t)ridN * a.RS + 4 * a.word0));
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.q + (size_t)ridN * NQP));
                    }
                    uint32_t qh[NQ], ql[NQ];
                    if constexpr (PACK) {
#pragma unroll
                        for (int c = 0; c < NQ; ++c) { qh[c] = (uint32_t)(q[c] >> 6); ql[c] = ((uint32_t)q[c] & 63u) | (1u << 19); }
                    } else {
                        uint32_t some = 0u; // nonzero: something is left of the row (an exact difference is never -0)
                        if (!second) {
#pragma unroll
                            for (int c = 0; c < NQ; ++c) some |= __float_as_uint(take_apart(__int_as_float(q[c]), two_lb, qh[c], ql[c]));
                            const unsigned who = __ballot_sync(FULL, some != 0u);
                            if (who != 0u) {
                                uint32_t at = 0;
                                if (lane == 0) at = atomicAdd(queue + QUEUE, (uint32_t)__popc(who));
                                at = __shfl_sync(FULL, at, 0) + __popc(who & ((1u << lane) - 1u));
                                if (some && at < QUEUE) queue[at] = rid;
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < NQ; ++c) {
                                const float left = take_apart(__int_as_float(q[c]), two_lb, qh[c], ql[c]);
                                some |= __float_as_uint(left);
                                take_apart(left * two_lb, two_lb, qh[c], ql[c]);
                            }
                            if (__ballot_sync(FULL, some != 0u) == 0u) continue;
                        }
                    }
                    const uint8_t *xw = a.xT + (size_t)rid * a.RS + 4 * a.word0;
                    uint32_t poff = 0;
                    for (int p = 0; p < a.nfull; ++p, poff += pb, xw += 32) part_steps<NQ, CNT, PACK, 3>(xw, act, qh, ql, ln, poff, lane);
                    if (a.tails & 4) { part_steps<NQ, CNT, PACK, 2>(xw, act, qh, ql, ln, poff, lane); poff += pb; xw += 16; }
                    if (a.tails & 2) { part_steps<NQ, CNT, PACK, 1>(xw, act, qh, ql, ln, poff, lane); poff += pb; xw += 8; }
                    if (a.tails & 1) part_steps<NQ, CNT, PACK, 0>(xw, act, qh, ql, ln, poff, lane);
                }
                __syncthreads();
                left_rows = *queued; // between the barriers: no warp queues rows of the next piece yet
                flush<NQ, CNT, PACK>(a, second, smem, s);
                __syncthreads();
            }
            if constexpr (PACK) break;
            else {
                if (left_rows == 0u) break;
                // One row in 32, by global reductions; more, through the image.  Lines at one in 8 to 128 are within 3 % of each other (300k x 30
                // gamma, log-normal target of sigma 0.7 to 2; 60k x 77, sigma 3: 0.157 ms per tree at one in 8, 0.153 at 32, 0.154 at 128).
                const bool few = left_rows <= QUEUE && left_rows * 32 <= (uint32_t)(pe - pos + a.pad_rows);
                if (!second && few) add_left<NQ>(a, queue, (int)left_rows, s, two_lb);
                if (second || few) {
                    __syncthreads();
                    if (threadIdx.x == 0) { queue[QUEUE] = 0u; a.low[s] = 1u; *a.low_any = 1u; }
                    __syncthreads();
                    break;
                }
            }
        }
    }
}

} // namespace evb_hg

// start of channel group z in the q words of n rows (16-byte aligned)
__host__ __device__ inline size_t evb_hg_qoff(const HGeom &g, long long n, int z) {
    size_t o = 0;
    for (int k = 0; k < z; ++k) o += ((size_t)n * evb_hg::nqp(min(g.per, g.nq - k * g.per)) + 3) & ~(size_t)3;
    return o;
}
__host__ __device__ inline int evb_hg_planes(const HGeom &g, int z) {
    return evb_hg::planes(min(g.per, g.nq - z * g.per), g.cnt && z == 0, g.pack);
}
// words and channels of feature group y, channel group z
__device__ __forceinline__ void evb_hg_select(const HGeom &g, evb_hg::Args &a, int y, int z) {
    a.word0 = y * g.wper;
    a.words = min(g.wper, g.W - a.word0);
    evb_hg::split_words(a.words, a.nfull, a.tails);
    a.ch0 = z * g.per;
    a.q += evb_hg_qoff(g, a.n, z);
}
namespace evb_hg {
// the words of every channel of a row (packed: q, else g 2^s as a float), and the unit of every channel's sums
struct QuantArgs {
    const float *grad;
    int32_t *q;             // channel groups one after the other, or (q2) the x words of xE
    const unsigned *gmax;   // [nq] bits of max |g|
    unsigned *signs;        // [nq] which infinities a channel has had: 1 positive, 2 negative
    double *qinv;           // [nq]
    long long n;
    int q2, bits;           // bits: g is rounded to that many below max |g|; 0: not at all
    HGeom g;
};
struct Quant {
    float sc, back;         // 2^(s of the rounding), from there to 2^s of the words
    int kind;               // QK_*
};
enum { QK_INT, QK_ROUND, QK_FLOAT, QK_INF };
__device__ __forceinline__ int32_t quant(const Quant &k, float g, unsigned *sign, double *unit) {
    if (k.kind == QK_INT) return __float2int_rn(g * k.sc);
    if (k.kind == QK_FLOAT) return __float_as_int(g * k.sc);
    if (k.kind == QK_ROUND) return __float_as_int(rintf(g * k.sc) * k.back);
    // The channel has an infinity: its rows count 2, all others nothing, in units of DBL_MAX, so that sums with one are infinite.
    // With both signs no sum means anything; whoever sees that last (here, or where the unit is written) makes the unit a NaN.
    if (!isinf(g)) return 0;
    const unsigned s = g > 0.0f ? 1u : 2u;
    if ((*(volatile unsigned *)sign & s) == 0u) {
        atomicOr(sign, s);
        __threadfence();
        if (*(volatile unsigned *)sign == 3u) *(volatile double *)unit = __longlong_as_double(0x7ff8000000000000ll);
    }
    const float v = g > 0.0f ? 2.0f : -2.0f;
    return k.back == 0.0f ? (int32_t)v : __float_as_int(v * k.back);
}
// how a channel's values become words, and the unit of its sums; bits: of its largest magnitude
__device__ __forceinline__ Quant quant_of(unsigned bits, bool pack, int hb, int round_bits, double *unit) {
    auto pow2 = [](int e) { return __int_as_float((e + 127) << 23); };
    const int ub = pack ? 24 : 2 * hb + 1; // bits of a sum's unit below max |g|
    Quant k = {1.0f, 0.0f, QK_FLOAT};      // (a channel of zeros: any scale)
    *unit = 1.0;
    if (bits - 1u < 0x7f7fffffu) {
        // max |g| = f 2^e, f in [0.5, 1); a channel of denormals keeps its scale inside the range of a float
        const int e = max((int)(bits >> 23), 1) - 126, top = pack ? 24 : hb, s = min(top - e, 127);
        k.sc = pow2(s);
        if (pack) k.kind = QK_INT;
        else if (round_bits) {
            const int sr = min(round_bits - e, 127);
            k = {pow2(sr), pow2(s - sr), QK_ROUND};
        }
        *unit = __longlong_as_double((long long)(1023 - (s + ub - top)) << 52);
    } else if (bits != 0u) {
        k.kind = QK_INF;
        k.back = pack ? 0.0f : pow2(-(hb + 1)); // in units of lo
        *unit = bits == 0x7f800000u ? DBL_MAX : __longlong_as_double(0x7ff8000000000000ll);
    }
    return k;
}
// row i of the grid's rows (blocks of adjacent rows); every thread of the block calls it
__device__ __forceinline__ void quantize(const QuantArgs &a, long long i) {
    __shared__ Quant s_k[EVB_MAX_Q];
    __shared__ float s_sc[EVB_MAX_Q];
    bool ok = true;
    for (int c = threadIdx.x; c < a.g.nq; c += blockDim.x) {
        double inv;
        const Quant k = quant_of(a.gmax[c], a.g.pack != 0, a.g.hb, a.bits, &inv);
        s_k[c] = k;
        s_sc[c] = k.sc;
        ok = k.kind == QK_FLOAT;
        if (blockIdx.x == 0) {
            *(volatile double *)(a.qinv + c) = inv;
            if (k.kind == QK_INF) {
                __threadfence();
                if (*(volatile unsigned *)(a.signs + c) == 3u) *(volatile double *)(a.qinv + c) = __longlong_as_double(0x7ff8000000000000ll);
            }
        }
    }
    const bool plain = __syncthreads_and(ok) != 0; // every channel is only scaled
    const int nq = a.g.nq;
    if (nq == 1) { // one word per row, in xE beside the row's tail features or alone
        if (i < a.n) a.q[a.q2 ? 2 * i : i] = quant(s_k[0], a.grad[i], a.signs, a.qinv);
        return;
    }
    // Word by word: the block's 256 rows are contiguous in the records and in every group of q, adjacent threads take adjacent
    // words (a thread per row would touch nq floats and nqp words at a stride of a row).
    const long long row0 = i - threadIdx.x;
    const int nr = (int)min((long long)blockDim.x, a.n - row0);
    for (int z = 0; z < a.g.ngc; ++z) {
        const int c0 = z * a.g.per, nc = min(a.g.per, nq - c0), np = nqp(nc), sh = 31 - __clz(np);
        int32_t *d = a.q + evb_hg_qoff(a.g, a.n, z) + (size_t)row0 * np;
        const float *src = a.grad + (size_t)row0 * nq + c0;
        if (sh >= 2) { // four words at a time
            for (int e = threadIdx.x; e < nr << (sh - 2); e += blockDim.x) {
                const int r = e >> (sh - 2), c = 4 * (e & ((np >> 2) - 1));
                int4 v = make_int4(0, 0, 0, 0);
                const float *g = src + (size_t)r * nq + c;
                if (plain) {
                    const float *sc = s_sc + c0 + c;
                    if (c < nc) v.x = __float_as_int(g[0] * sc[0]);
                    if (c + 1 < nc) v.y = __float_as_int(g[1] * sc[1]);
                    if (c + 2 < nc) v.z = __float_as_int(g[2] * sc[2]);
                    if (c + 3 < nc) v.w = __float_as_int(g[3] * sc[3]);
                } else {
                    const Quant *k = s_k + c0 + c;
                    unsigned *sg = a.signs + c0 + c;
                    double *un = a.qinv + c0 + c;
                    if (c < nc) v.x = quant(k[0], g[0], sg, un);
                    if (c + 1 < nc) v.y = quant(k[1], g[1], sg + 1, un + 1);
                    if (c + 2 < nc) v.z = quant(k[2], g[2], sg + 2, un + 2);
                    if (c + 3 < nc) v.w = quant(k[3], g[3], sg + 3, un + 3);
                }
                reinterpret_cast<int4 *>(d)[e] = v;
            }
        } else {
            for (int e = threadIdx.x; e < nr << sh; e += blockDim.x) {
                const int r = e >> sh, c = e & (np - 1);
                d[e] = c >= nc ? 0 : plain ? __float_as_int(src[(size_t)r * nq + c] * s_sc[c0 + c]) : quant(s_k[c0 + c], src[(size_t)r * nq + c], a.signs + c0 + c, a.qinv + c0 + c);
            }
        }
    }
}
} // namespace evb_hg
void evb_hg_quant_args(const evb_handle *h, evb_hg::QuantArgs *a);
// FN<channels, count plane, packed>(args...) for channel group z
#define EVB_HG_DISPATCH(g, z, FN, ...)                                          \
    if ((g).pack) FN<1, true, true>(__VA_ARGS__);                               \
    else {                                                                      \
        const int nc_ = min((g).per, (g).nq - (int)(z) * (g).per);              \
        if ((g).cnt && (z) == 0) switch (nc_) {                                 \
            case 1: FN<1, true, false>(__VA_ARGS__); break;                     \
            case 2: FN<2, true, false>(__VA_ARGS__); break;                     \
            case 3: FN<3, true, false>(__VA_ARGS__); break;                     \
            case 4: FN<4, true, false>(__VA_ARGS__); break;                     \
            default: FN<5, true, false>(__VA_ARGS__); break;                    \
        } else switch (nc_) {                                                   \
            case 1: FN<1, false, false>(__VA_ARGS__); break;                    \
            case 2: FN<2, false, false>(__VA_ARGS__); break;                    \
            case 3: FN<3, false, false>(__VA_ARGS__); break;                    \
            case 4: FN<4, false, false>(__VA_ARGS__); break;                    \
            default: FN<5, false, false>(__VA_ARGS__); break;                   \
        }                                                                       \
    }
void evb_hg_args(const evb_handle *h, int level, evb_hg::Args *a);
