// Fixed-point histogram build for mse with one target and unit weights: `update_hist!` / `_hist!`
// (src/fit-utils.jl:345-394; GPU counterpart `hist_kernel!`, ext/EvoTreesKernelAbstractionsExt/fit-utils.jl:57-95).
//
// Data layout.  The bins of a row live in two arrays: xH[row][RSH] holds the features in 16-byte chunks (16 features
// each) and xE[row] = {q, tail} holds the row's fixed-point gradient q = rint(g * 2^s) (written once per boosting
// round) and, when nfeats % 16 is 1..4, the bins of those last features, so that a row of 100 features is 96 + 8
// bytes: three whole sectors plus one, wherever the row is gathered from.
//
// Kernel.  Warps work on their own: there is no producer, no staging buffer and no barrier between tiles.  A warp
// takes tiles of 32 rows.  Lane l loads chunk (32 s + l) % NC of row (32 s + l) / NC in step s with one 128-bit
// load straight into registers (a row's chunks sit in adjacent lanes, so a request covers whole lines); the
// registers of a step are refilled for a later step (of this tile or of the warp's next one) as soon as they have
// been accumulated, so a few loads per lane are always in flight and no shared memory is spent on rows.
// A CTA keeps one packed image [bin][plane][column] of 32-bit words in shared memory; a row adds two
// words per feature with `red.shared.add.u32`: q >> 6 into plane 0 and (q & 0x3f) | 1 << 19 into plane 1 (the row
// count rides in the top 13 bits; |q| < 2^24).  Integer sums do not depend on the order, so all warps share the image.  The 32
// lanes of a reduction always hit 32 different banks: lanes differ in the chunk's parity, in the word of the chunk
// they work on (the four registers of a chunk are rotated by (l >> 1) & 3) and in the byte of that word
// ((l >> 3) & 3).
// The packed counters hold 8191 rows: after at most 255 tiles, and at the end of a node's rows, the CTA adds the packed
// image to the node's accumulators in global memory (`red.global.add.u64 / .u32`, cell by cell: consecutive lanes,
// consecutive addresses) and clears it.  Two CTAs share an SM, so one accumulates while the other flushes.   Every histogram entry is therefore the exact integer sum of the quantised gradients, whatever the order of
// the rows and however the rows are cut into pieces.
#include "evb_internal.cuh"
#include <stdlib.h>

namespace {

constexpr unsigned FULL = 0xffffffffu;
// Two CTAs of 384 threads per SM: while one of them flushes, the other accumulates.  Measured on B200 (10M x 100, depth 11,
// ms of this kernel per tree): 1.83; one CTA of 768 threads with 64-bit sums in shared memory between the flushes to
// global memory 1.91; three CTAs of 256: 2.28.
constexpr int Q2_THREADS = 384, Q2_WARPS = Q2_THREADS / 32;
// |q| < 2^24; plane 0 takes q >> LB, plane 1 takes (q & (2^LB - 1)) | 1 << CS, and an image cell holds 8191 rows: the signed
// plane 0 needs 24 - 6 + 13 bits, the low sums of plane 1 6 + 13 <= CS, the row count 13 bits above them.
constexpr int Q2_LB = 6, Q2_CS = 19, Q2_EPOCH = 255 / Q2_WARPS * Q2_WARPS; // tiles of 32 rows between two flushes

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

struct Q2Args {
    const uint8_t *xH;
    const uint2 *xE;
    const uint32_t *rows;
    const LevelPlan *plan;
    const int32_t *cum, *rbase;
    unsigned long long *hsum; // [slot][bin][SC] sums of q
    uint32_t *hcnt;           // [slot][bin][SC] row counts
    int RSH, B, SC;
    int nmain;                // features held in xH
    int ntail;                // features held in xE (0..4)
    int min_rows;             // rows per CTA below which fewer CTAs take part
    int pad_rows;             // what the flush of a build node costs, in rows
    uint32_t zrow;            // index of an all-zero row of xH / xE (bins 0, q 0)
};

// image geometry for NC chunks of 16 features (+ 8 replicas of the 4 tail features): NCOL columns per plane row
template <int NC, bool TAIL>
struct Q2Cfg {
    static constexpr int NEED = 16 * NC + (TAIL ? 32 : 0);
    static_assert(NEED <= 128, "at most 128 image columns per CTA");
    static constexpr int NCOL = NEED <= 32 ? 32 : NEED <= 64 ? 64 : 128;
    static constexpr int TAILCOL = NCOL - 32;
    static constexpr uint32_t ROWB = NCOL * 4; // bytes of one plane row; a bin owns two of them (plane 0, plane 1)
    static constexpr uint32_t X = NCOL / 32;   // (bin << 8 | column byte) * X = bin * 2 * ROWB + 4 * column
};

__device__ __forceinline__ uint4 ldg_chunk(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// row id: issued where it stands (a plain load may be moved next to its first use, a whole tile later)
__device__ __forceinline__ uint32_t ldg_rid(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ldg_ext(const uint2 *p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Four features (one word of bins) of one row.  u: the word; Cb: bytes {column byte of register byte k}; sel[k]: PRMT
// selector that builds (bin << 8 | column byte) of the lane's k-th feature; As: image address of the lane's column
// group in bin row 0.  (bin << 8 | column byte) * X = bin * 2 * ROWB + 4 * column.
template <uint32_t ROWB, uint32_t X>
__device__ __forceinline__ void q2_word(uint32_t u, uint32_t As, uint32_t Cb, const uint32_t (&sel)[4], uint32_t w0, uint32_t w1) {
    asm volatile(
        "{\n .reg .u32 b0, b1, b2, b3, a0, a1, a2, a3;\n"
        " prmt.b32 b0, %0, %1, %2;\n prmt.b32 b1, %0, %1, %3;\n prmt.b32 b2, %0, %1, %4;\n prmt.b32 b3, %0, %1, %5;\n"
        " mad.lo.u32 a0, b0, %10, %6;\n mad.lo.u32 a1, b1, %10, %6;\n mad.lo.u32 a2, b2, %10, %6;\n mad.lo.u32 a3, b3, %10, %6;\n"
        " red.shared.add.u32 [a0], %7;\n red.shared.add.u32 [a0+%9], %8;\n"
        " red.shared.add.u32 [a1], %7;\n red.shared.add.u32 [a1+%9], %8;\n"
        " red.shared.add.u32 [a2], %7;\n red.shared.add.u32 [a2+%9], %8;\n"
        " red.shared.add.u32 [a3], %7;\n red.shared.add.u32 [a3+%9], %8;\n}\n"
        ::"r"(u), "r"(Cb), "r"(sel[0]), "r"(sel[1]), "r"(sel[2]), "r"(sel[3]), "r"(As), "r"(w0), "r"(w1), "n"(ROWB), "n"(X)
        : "memory");
}

// iterator over the non-empty pieces (CTA row range x build slot) of a CTA, addressed by the CTA's tile index
struct PieceIt {
    int s, g0, nt, pstart, pend;
    const uint32_t *rows;
    bool end;
};
__device__ __forceinline__ void piece_load(const Q2Args &a, PieceIt &it, int lo, int hi, int nbuild) {
    for (;;) {
        if (it.s >= nbuild) { it.end = true; return; }
        const int c0 = a.cum[it.s], c1 = a.cum[it.s + 1], off = it.s * a.pad_rows;
        if (c0 + off >= hi) { it.end = true; return; }
        const int ps = max(lo - off, c0), pe = min(hi - off, c1);
        if (pe > ps) {
            it.pstart = ps; it.pend = pe; it.nt = (pe - ps + 31) >> 5;
            it.rows = a.rows + a.rbase[it.s];
            return;
        }
        ++it.s;
    }
}
__device__ __forceinline__ void piece_next(const Q2Args &a, PieceIt &it, int lo, int hi, int nbuild) {
    it.g0 += it.nt;
    ++it.s;
    piece_load(a, it, lo, hi, nbuild);
}

// register sets of chunk loads in flight per lane: step s of a tile uses set s % NSET and refills it for step s + NSET
__host__ __device__ constexpr int q2_nset(int NC) { return NC == 6 ? 3 : NC == 8 ? 4 : NC; }

template <int NC, bool TAIL>
__global__ void __launch_bounds__(Q2_THREADS, 2) k_histq2(Q2Args a) {
    using Cf = Q2Cfg<NC, TAIL>;
    constexpr int NCOL = Cf::NCOL, NSET = q2_nset(NC);
    constexpr uint32_t ROWB = Cf::ROWB, X = Cf::X;
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, wid = tid >> 5, l = tid & 31;
    constexpr int NW = Q2_WARPS, NT = Q2_THREADS;
    const int b = blockIdx.x, chunk0 = blockIdx.y * NC;
    uint32_t *img_w = reinterpret_cast<uint32_t *>(smem);
    const int nbuild = a.plan->nbuild;
    const long long R = a.plan->R + (long long)nbuild * a.pad_rows; // pad_rows rows that do not exist after every build node
    // few rows: fewer CTAs take part (every CTA costs one pass over its image)
    int G = gridDim.x;
    {
        const long long want = (R + a.min_rows - 1) / a.min_rows;
        if (want < G) G = want < 1 ? 1 : (int)want;
    }
    if (b >= G) return;
    const int lo = (int)(R * b / G), hi = (int)(R * (b + 1) / G);
    if (lo >= hi) return;
    for (int i = tid; i < (a.B + 1) * 2 * NCOL; i += NT) img_w[i] = 0u;
    __syncthreads();

    int s0;
    {
        int lft = 0, rgt = nbuild - 1; // largest s with cum[s] + s * pad_rows <= lo
        while (lft < rgt) { const int m = (lft + rgt + 1) >> 1; if (a.cum[m] + m * a.pad_rows <= lo) lft = m; else rgt = m - 1; }
        s0 = lft;
    }
    // per-lane constants
    const int rot_w = (l >> 1) & 3, rot_b = (l >> 3) & 3;
    uint32_t sel[4], Cb0 = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t cb = (uint32_t)((k + rot_b) & 3);
        Cb0 |= (cb * (4u / X)) << (8 * k);
        sel[k] = ((0xCu + k) << 12) | ((0xCu + k) << 8) | (cb << 4) | (4u + k);
    }
    const uint32_t img = smem_u32(smem);
    uint32_t A0[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) A0[p] = img + 16u * (uint32_t)((p + rot_w) & 3);
    const uint32_t At = img + 4u * (uint32_t)(Cf::TAILCOL + 4 * (l & 7));
    const bool r1 = (rot_w & 1) != 0, r2 = (rot_w & 2) != 0;
    // step s of a tile: the lane works on chunk (32 s + l) % NC of row (32 s + l) / NC.  rowsel packs the rows (5 bits
    // per step); the chunk of step 0 is ch0 and every step adds 32 % NC (mod NC).
    uint32_t rowsel = 0;
#pragma unroll
    for (int s = 0; s < NC && s < 6; ++s) rowsel |= (uint32_t)((32 * s + l) / NC) << (5 * s);
    auto row_of = [&](int s) -> int { return NC <= 6 ? (int)(rowsel >> (5 * s)) : (32 * s + l) / NC; }; // shuffles use the low 5 bits
    const int ch0 = l % NC;
    const uint8_t *xH = a.xH + (size_t)chunk0 * 16;
    const uint32_t RSH = (uint32_t)a.RSH;
    const uint32_t zrow = a.zrow; // an all-zero row: its bins land in the image's guard row

    // The packed image goes to the accumulators of build slot `slot` in global memory, at the end of a node's rows and when
    // its row counts may be full.  All threads of the CTA.
    constexpr int LB = Q2_LB, CS = Q2_CS;
    constexpr uint32_t cmask = (1u << CS) - 1u, lmask = (1u << LB) - 1u, one = 1u << CS;
    auto flush = [&](int slot) {
        __syncthreads();
        {
            // cell by cell: consecutive lanes, consecutive addresses
            const size_t base = (size_t)slot * a.B;
            constexpr int MC = 16 * NC;
            for (int c = tid; c < a.B * MC; c += NT) {
                const int bin = c / MC, col = c - bin * MC;
                uint32_t *p = img_w + (size_t)(bin + 1) * 2 * NCOL + col;
                const uint32_t vh = p[0], vp = p[NCOL];
                if ((vh | vp) == 0u) continue;
                p[0] = 0u; p[NCOL] = 0u;
                const int f = chunk0 * 16 + col;
                if (f < a.nmain) {
                    const long long sum = ((long long)(int32_t)vh << LB) + (long long)(vp & cmask);
                    const size_t o = (base + bin) * a.SC + f;
                    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(a.hsum + o), "l"(sum) : "memory");
                    asm volatile("red.global.add.u32 [%0], %1;" ::"l"(a.hcnt + o), "r"(vp >> CS) : "memory");
                }
            }
            if (TAIL) {
                for (int bin = wid; bin < a.B; bin += NW) {
                    uint32_t *p = img_w + (size_t)(bin + 1) * 2 * NCOL + Cf::TAILCOL + l;
                    const uint32_t vh = p[0], vp = p[NCOL];
                    if (__ballot_sync(FULL, (vh | vp) != 0u) == 0u) continue;
                    p[0] = 0u; p[NCOL] = 0u;
                    long long sum = ((long long)(int32_t)vh << LB) + (long long)(vp & cmask);
                    uint32_t cnt = vp >> CS;
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) { sum += __shfl_xor_sync(FULL, sum, o); cnt += __shfl_xor_sync(FULL, cnt, o); }
                    if (l < a.ntail && cnt != 0u) {
                        const size_t o = (base + bin) * a.SC + a.nmain + l;
                        asm volatile("red.global.add.u64 [%0], %1;" ::"l"(a.hsum + o), "l"(sum) : "memory");
                        asm volatile("red.global.add.u32 [%0], %1;" ::"l"(a.hcnt + o), "r"(cnt) : "memory");
                    }
                }
            }
        }
        __syncthreads();
    };

    // the two piece iterators of a warp (accumulate stage, row-id fetch stage) are warp-uniform and touched once per
    // tile: they live in shared memory so that the registers stay with the loads in flight
    __shared__ PieceIt s_it[Q2_WARPS][2];
    PieceIt &pc = s_it[wid][0], &pa = s_it[wid][1];
    pc.s = s0; pc.g0 = 0; pc.end = false;
    piece_load(a, pc, lo, hi, nbuild);
    pa = pc;
    __syncwarp();
    int ep_end = pc.end ? 0 : min(pc.nt, Q2_EPOCH);

    // row ids of tile g of this CTA (lane = row of the tile); rows past the end of the tile read the zero row
    auto fetch = [&](int g) -> uint32_t {
        while (!pa.end && g >= pa.g0 + pa.nt) piece_next(a, pa, lo, hi, nbuild);
        if (pa.end) return zrow;
        const int off = pa.pstart + ((g - pa.g0) << 5);
        return off + l < pa.pend ? ldg_rid(pa.rows + off + l) : zrow;
    };
    // chunk of step s for the tile whose row ids are `rid`; ch = the lane's chunk in that step
    auto load_chunk = [&](uint32_t rid, int s, int ch) -> uint4 {
        const uint32_t r = __shfl_sync(FULL, rid, row_of(s));
        return ldg_chunk(xH + (size_t)(r * RSH + (uint32_t)ch * 16u));
    };
    auto ch_of = [&](int s) -> int { return (ch0 + (32 * s) % NC) % NC; };

    uint32_t ridC, ridB;
    uint4 v[NSET];
    uint2 extC;
    ridC = fetch(wid);
    ridB = fetch(wid + NW);
    extC = ldg_ext(a.xE + ridC);
#pragma unroll
    for (int s = 0; s < NSET; ++s) v[s] = load_chunk(ridC, s, ch_of(s));
    for (int g = wid;; g += NW) {
        bool done = false;
        for (;;) {
            if (pc.end) { done = true; break; }
            if (g < pc.g0 + ep_end) break;
            flush(pc.s);
            if (ep_end == pc.nt) { piece_next(a, pc, lo, hi, nbuild); if (!pc.end) ep_end = min(pc.nt, Q2_EPOCH); }
            else ep_end = min(pc.nt, ep_end + Q2_EPOCH);
        }
        if (done) break;
        const uint2 extN = ldg_ext(a.xE + ridB);
        const uint32_t ridA = fetch(g + 2 * NW);
#pragma unroll
        for (int s = 0; s < NC; ++s) {
            const int ch = ch_of(s);
            const uint32_t q = __shfl_sync(FULL, extC.x, row_of(s));
            const uint32_t w0 = (uint32_t)((int32_t)q >> LB), w1 = (q & lmask) | one;
            const uint4 c = v[s % NSET];
            const uint32_t t0 = r1 ? c.y : c.x, t1 = r1 ? c.z : c.y, t2 = r1 ? c.w : c.z, t3 = r1 ? c.x : c.w;
            const uint32_t u0 = r2 ? t2 : t0, u1 = r2 ? t3 : t1, u2 = r2 ? t0 : t2, u3 = r2 ? t1 : t3;
            const uint32_t Cb = Cb0 + (uint32_t)ch * ((64u / X) * 0x01010101u); // column byte += 16 columns per chunk
            q2_word<ROWB, X>(u0, A0[0], Cb, sel, w0, w1);
            q2_word<ROWB, X>(u1, A0[1], Cb, sel, w0, w1);
            q2_word<ROWB, X>(u2, A0[2], Cb, sel, w0, w1);
            q2_word<ROWB, X>(u3, A0[3], Cb, sel, w0, w1);
            // the same registers, for step s + NSET: of this tile, or of the warp's next tile
            if (s + NSET < NC) v[s % NSET] = load_chunk(ridC, s + NSET, ch_of(s + NSET));
            else v[s % NSET] = load_chunk(ridB, s + NSET - NC, ch_of(s + NSET - NC));
        }
        if (TAIL) { // lane = row of the tile
            const uint32_t q = extC.x;
            const uint32_t w0 = (uint32_t)((int32_t)q >> LB), w1 = (q & lmask) | one;
            q2_word<ROWB, X>(extC.y, At, Cb0, sel, w0, w1);
        }
        extC = extN;
        ridC = ridB; ridB = ridA;
    }
}

// tail features of every row: xE[i].y = bins of features nmain .. nmain + ntail - 1 (one byte each, zero padded)
__global__ void __launch_bounds__(256) k_q2_tail(const uint8_t *xC, long long n, int nmain, int ntail, uint2 *xE) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t t = 0;
    for (int k = 0; k < ntail; ++k) t |= (uint32_t)xC[(size_t)(nmain + k) * n + i] << (8 * k);
    xE[i] = make_uint2(0u, t);
}

template <int NC, bool TAIL>
int q2_instance(bool launch, const Q2Args *a, dim3 grid, size_t smem, cudaStream_t st) {
    static size_t attr_set[64] = {}; // dynamic shared memory the kernel has been allowed on each device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && attr_set[dev] < smem) {
        cudaError_t e = cudaFuncSetAttribute(k_histq2<NC, TAIL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return launch ? (int)e : 0;
        attr_set[dev] = smem;
    }
    if (!launch) {
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_histq2<NC, TAIL>, Q2_THREADS, smem) != cudaSuccess) nb = 0;
        return nb;
    }
    return (int)evb_launch(k_histq2<NC, TAIL>, grid, dim3(Q2_THREADS), smem, st, *a);
}
template <bool TAIL>
int q2_dispatch_nc(int NC, bool launch, const Q2Args *a, dim3 grid, size_t smem, cudaStream_t st) {
    switch (NC) {
    case 1: return q2_instance<1, TAIL>(launch, a, grid, smem, st);
    case 2: return q2_instance<2, TAIL>(launch, a, grid, smem, st);
    case 3: return q2_instance<3, TAIL>(launch, a, grid, smem, st);
    case 4: return q2_instance<4, TAIL>(launch, a, grid, smem, st);
    case 5: return q2_instance<5, TAIL>(launch, a, grid, smem, st);
    default: return q2_instance<6, TAIL>(launch, a, grid, smem, st);
    }
}
int q2_dispatch(int NC, bool tail, bool launch, const Q2Args *a, dim3 grid, size_t smem, cudaStream_t st) {
    if (tail) return q2_dispatch_nc<true>(NC, launch, a, grid, smem, st);
    switch (NC) {
    case 7: return q2_instance<7, false>(launch, a, grid, smem, st);
    case 8: return q2_instance<8, false>(launch, a, grid, smem, st);
    default: return q2_dispatch_nc<false>(NC, launch, a, grid, smem, st);
    }
}
int q2_ncol(int NC, bool tail) { const int need = 16 * NC + (tail ? 32 : 0); return need <= 32 ? 32 : need <= 64 ? 64 : 128; }
size_t q2_smem(int B, int NC, bool tail) { return (size_t)(B + 1) * 2 * q2_ncol(NC, tail) * 4; } // packed image [B + 1][2][NCOL] words

} // namespace

// Least squares with one target and unit weights on many rows.  Below Q2_MIN_ROWS the general integer kernel is as fast (it
// does less for features that do not fill a 16-byte chunk and has the smaller image to flush), and the training predict has
// to be able to read the chunk rows: tree, leaf values and two tiles of rows within 100 KB.
bool evb_q2_wanted(const evb_handle *h) {
    if (h->p.loss != EVB_MSE || h->nq != 1) return false; // (hessians left out as well)
    if (const char *e = getenv("EVB_HIST_Q2")) { if (atoi(e) == 0) return false; }
    else if (h->n < 300000) return false;
    const int words = (h->nfeats + 15) / 16 * 4 + 8;
    return (size_t)(h->nn + 4) * 8 + (size_t)2 * 256 * words * 4 <= (size_t)100 * 1024 && words <= 64;
}

// Chooses the layout: chunks per CTA group, number of groups, tail features.  Returns EVB_ERR_LIMIT when the shape
// does not fit (the caller then uses the other histogram kernels).
int32_t evb_q2_configure(evb_handle *h) {
    const int nf = h->nfeats, B = h->B;
    Q2Geom &g = h->q2;
    const size_t smem_max = 224 * 1024; // the kernel also holds a few KB of static shared memory
    const int t = nf % 16;
    const int nc_all = (nf + 15) / 16;
    // one group with the tail in xE if it fits
    g.ntail = 0;
    g.NC = 0;
    if (t >= 1 && t <= 4 && nf / 16 >= 1 && nf / 16 <= 6) {
        const int NC = nf / 16;
        if (q2_smem(B, NC, true) <= smem_max) { g.NC = NC; g.ngroups = 1; g.ntail = t; }
    }
    if (g.NC == 0) {
        // groups of equal chunk counts; the widest image that fits shared memory
        int ncmax = 8;
        while (ncmax > 1 && q2_smem(B, ncmax, false) > smem_max) ncmax >>= 1;
        if (q2_smem(B, ncmax, false) > smem_max) return EVB_ERR_LIMIT;
        g.ngroups = (nc_all + ncmax - 1) / ncmax;
        g.NC = (nc_all + g.ngroups - 1) / g.ngroups;
    }
    if (g.ngroups > 64) return EVB_ERR_LIMIT;
    g.nmain = nf - g.ntail;
    g.RSH = g.ngroups * g.NC * 16;
    if ((unsigned long long)(h->n + 1) * g.RSH >= (1ull << 32)) return EVB_ERR_LIMIT; // 32-bit byte offsets into xH
    g.smem = q2_smem(B, g.NC, g.ntail > 0);
    const int occ = q2_dispatch(g.NC, g.ntail > 0, false, nullptr, dim3(), g.smem, 0);
    if (occ < 1) { evb_set_error("fixed-point histogram kernel cannot be resident (smem=%zu)", g.smem); return EVB_ERR_CUDA; }
    g.G = occ * h->num_sms;
    g.min_rows = 512; // measured: 100k x 10 rows 0.054 ms per tree at 512, 0.059 at 1024, 0.088 at 4096; no difference at 10M rows.
    // evb_pad_rows: 1M x 100, half of the rows, 0.239 -> 0.233 ms per tree, 10M x 100 3.11 -> 3.10
    return EVB_OK;
}

// xH / xE from the feature-major matrix on the device (h->xC), once at create time
int32_t evb_q2_build_layout(evb_handle *h) {
    const Q2Geom &g = h->q2;
    EVB_CUDA(cudaMemsetAsync(h->xH, 0, (size_t)(h->n + 1) * g.RSH, h->st)); // row n: the all-zero row
    EVB_CUDA(cudaMemsetAsync(h->xE + h->n, 0, sizeof(uint2), h->st));
    EVB_CHECK(evb_launch_transpose(h, h->xC, h->n, h->n, 0, g.nmain, h->xH, g.RSH, h->st));
    k_q2_tail<<<(unsigned)((h->n + 255) / 256), 256, 0, h->st>>>(h->xC, h->n, g.nmain, g.ntail, h->xE);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

// what the binarize kernel does not write: the all-zero row n, and the xE words when no feature lives there
int32_t evb_q2_clear_layout(evb_handle *h) {
    const Q2Geom &g = h->q2;
    EVB_CUDA(cudaMemsetAsync(h->xH + (size_t)h->n * g.RSH, 0, g.RSH, h->st));
    EVB_CUDA(cudaMemsetAsync(h->xE + (g.ntail > 0 ? h->n : 0), 0, sizeof(uint2) * (g.ntail > 0 ? 1 : (size_t)h->n + 1), h->st));
    return EVB_OK;
}

int32_t evb_launch_histq2(evb_handle *h, int level) {
    const Q2Geom &g = h->q2;
    Q2Args a;
    a.xH = h->xH; a.xE = h->xE; a.rows = h->rows[(level - 1) & 1];
    a.plan = h->plan + level; a.cum = h->cum; a.rbase = h->rbase;
    a.hsum = h->hsum_q; a.hcnt = h->hcnt_q;
    a.RSH = g.RSH; a.B = h->B; a.SC = h->SC; a.nmain = g.nmain; a.ntail = g.ntail; a.min_rows = g.min_rows; a.pad_rows = evb_pad_rows(h); a.zrow = (uint32_t)h->n;
    evb_tic(h, EVB_T_HIST);
    const cudaError_t e = (cudaError_t)q2_dispatch(g.NC, g.ntail > 0, true, &a, dim3(g.G, g.ngroups), g.smem, h->st);
    evb_toc(h, EVB_T_HIST);
    EVB_CUDA(e);
    return EVB_OK;
}
