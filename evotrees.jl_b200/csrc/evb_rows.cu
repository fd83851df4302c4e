// Row-parallel kernels: layout conversion of the binned matrix, loss gradients (`update_grads!`,
// src/loss.jl:100-128, 219-236; GPU counterparts ext/EvoTreesKernelAbstractionsExt/loss.jl:106-191), row
// subsampling (`subsample`, src/subsample.jl:6-38), the training `predict!` (src/predict.jl:1-62) fused with
// the gradients of the next round and `binarize` (src/fit-utils.jl:66-72).
#include "evb_device.cuh"
#include <float.h>
#include <algorithm>
#include <mutex>

namespace {

constexpr unsigned FULL = 0xffffffffu;

// ---------------------------------------------------------------------------------- layout
// xT[row][j] = xcol[j][row] for a block of columns; one thread = one row x 4 consecutive features
__global__ void k_transpose(const uint8_t *xcol, long long ld, long long nrows, int j0, int nj, uint8_t *xT, int RS) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int jj = blockIdx.y * 4;
    if (i >= nrows || jj >= nj) return;
    uint8_t v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (jj + q < nj) v[q] = xcol[(size_t)(jj + q) * ld + i];
    uint8_t *dst = xT + (size_t)i * RS + j0 + jj;
    if (((j0 + jj) & 3) == 0 && jj + 4 <= nj) {
        *reinterpret_cast<uint32_t *>(dst) = (uint32_t)v[0] | ((uint32_t)v[1] << 8) | ((uint32_t)v[2] << 16) | ((uint32_t)v[3] << 24);
    } else {
        for (int q = 0; q < 4 && jj + q < nj; ++q) dst[q] = v[q];
    }
}

// range check of the binned matrix
__global__ void k_check_bins(const uint8_t *xC, size_t total, int nbins, int *err) {
    bool bad = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) { const int v = xC[i]; bad |= v < 1 || v > nbins; }
    if (bad) atomicCAS(err, 0, EVB_DERR_BIN_RANGE);
}

// wmax: null, or the maximum of the weights goes there (they are a channel of the histograms then)
__global__ void __launch_bounds__(256) k_init_state(float *grad, float *pred, const float *w, const float *pred0, const float *mu, long long n, int K, int nq, unsigned *wmax) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (wmax) {
        const unsigned m = __reduce_max_sync(0xffffffffu, i < n ? __float_as_uint(w[i]) : 0u);
        if ((threadIdx.x & 31) == 0 && m > *(volatile unsigned *)wmax) atomicMax(wmax, m);
    }
    if (i >= n) return;
    if (w) grad[(size_t)i * nq + nq - 1] = w[i]; // ∇[end, :] .= w (src/init.jl:173-174)
    for (int k = 0; k < K; ++k) pred[(size_t)i * K + k] = pred0 ? pred0[(size_t)i * K + k] : mu[k];
}

// ---------------------------------------------------------------------------------- gradients
// max |g| of every changing channel over the rows of a 256-thread block -> global maxima (bit patterns of non-negative
// floats, which order like unsigned integers).  rec: the thread's gradient record, or null.  Every thread calls it.
__device__ __forceinline__ void block_absmax(const float *rec, int ng, unsigned *gmax) {
    __shared__ unsigned s_max[EVB_MAX_Q];
    if (threadIdx.x < ng) s_max[threadIdx.x] = 0u;
    __syncthreads();
    for (int c = 0; c < ng; ++c) {
        const unsigned m = __reduce_max_sync(FULL, rec ? __float_as_uint(fabsf(rec[c])) : 0u);
        if ((threadIdx.x & 31) == 0 && m > *(volatile unsigned *)(s_max + c)) atomicMax(s_max + c, m);
    }
    __syncthreads();
    if (threadIdx.x < ng && s_max[threadIdx.x] > *(volatile unsigned *)(gmax + threadIdx.x)) atomicMax(gmax + threadIdx.x, s_max[threadIdx.x]);
}
__global__ void __launch_bounds__(256) k_grads(int loss, int K, int nq, int unit_w, int elided, int ycols, long long n, const float *pred, const void *y, float *grad, unsigned *gmax,
                                               int ng, AlphaSet alpha) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float *rec = i < n ? grad + (size_t)i * nq : nullptr;
    if (rec) grad_row(loss, K, elided != 0, pred + (size_t)i * K, y, ycols, i, unit_w ? 1.0f : rec[nq - 1], rec, alpha);
    block_absmax(rec, ng, gmax);
}

// ---------------------------------------------------------------------------------- row sampling
constexpr int SEL_CHUNK = 2048, SEL_THREADS = 256;
__global__ void __launch_bounds__(SEL_THREADS) k_sel_count(const uint8_t *mask, uint8_t cond, long long n, int32_t *bcnt) {
    __shared__ int s[SEL_THREADS / 32];
    const long long base = (long long)blockIdx.x * SEL_CHUNK;
    int c = 0;
    for (int i8 = 0; i8 < SEL_CHUNK / SEL_THREADS; ++i8) {
        const long long i = base + i8 * SEL_THREADS + threadIdx.x;
        const bool sel = i < n && mask[i] <= cond;
        c += __popc(__ballot_sync(FULL, sel));
    }
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < SEL_THREADS / 32; ++w) t += s[w];
        bcnt[blockIdx.x] = t;
    }
}
// Row mask bytes from the caller's generator: PCG64 (O'Neill, "PCG: A Family of Simple Fast Space-Efficient Statistically
// Good Algorithms for Random Number Generation", 2014: 128-bit LCG, XSL-RR output), whose 64-bit outputs are used as two
// 32-bit words, low one first, of four bytes each.  An LCG can be advanced by any distance in logarithmic time, so every
// thread makes the eight bytes of its own rows: the bytes of a generator on the host (0.75 ms per million rows, plus the
// copy over PCIe: 0.85 of the 1.0 ms per tree at 1M rows) without the host.
// state' after 2^k steps = state * M[k] + inc * G[k]; filled by the host once per device
typedef unsigned __int128 u128;
__constant__ u128 c_pcg_m[32], c_pcg_g[32];
constexpr uint64_t PCG_MULT_HI = 2549297995355413924ull, PCG_MULT_LO = 4865540595714422341ull;
__device__ __forceinline__ uint64_t pcg_out(u128 s) {
    const uint64_t hi = (uint64_t)(s >> 64), x = hi ^ (uint64_t)s;
    const unsigned r = (unsigned)(hi >> 58);
    return (x >> r) | (x << ((64u - r) & 63u));
}
// gen: {state lo, hi, increment lo, hi, left, left word}: left = 1 when the high half of the last output is still to be used
__global__ void __launch_bounds__(SEL_THREADS) k_sel_pcg(const uint64_t *gen, uint8_t cond, long long n, uint8_t *mask, int32_t *bcnt) {
    static_assert(SEL_CHUNK == 8 * SEL_THREADS, "eight rows per thread");
    __shared__ int s[SEL_THREADS / 32];
    const u128 inc = ((u128)gen[3] << 64) | gen[2];
    u128 st = ((u128)gen[1] << 64) | gen[0];
    const unsigned left = (unsigned)gen[4];
    const long long t = (long long)blockIdx.x * SEL_THREADS + threadIdx.x;
    // outputs t - left and, when a word is left over, t; output d is made from the state after d + 1 steps
    uint32_t skip = (uint32_t)(t + 1 - left);
    for (int k = 0; skip; ++k, skip >>= 1)
        if (skip & 1u) st = st * c_pcg_m[k] + inc * c_pcg_g[k];
    uint64_t w = pcg_out(st);
    if (left) {
        const uint32_t lo = t == 0 ? (uint32_t)gen[5] : (uint32_t)(w >> 32);
        st = st * c_pcg_m[0] + inc;
        w = (uint64_t)lo | ((uint64_t)(uint32_t)pcg_out(st) << 32);
    }
    int c = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const uint8_t b = (uint8_t)(w >> (8 * q));
        if (8 * t + q < n) c += b <= cond;
    }
    if (8 * t + 8 <= n) *reinterpret_cast<uint64_t *>(mask + 8 * t) = w;
    else for (int q = 0; 8 * t + q < n && q < 8; ++q) mask[8 * t + q] = (uint8_t)(w >> (8 * q));
    c = __reduce_add_sync(FULL, c);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int q = 0; q < SEL_THREADS / 32; ++q) tot += s[q];
        bcnt[blockIdx.x] = tot;
    }
}
struct RootPlan { int32_t *seg_cnt, *cum, *slot_node, *rbase; int4 *pl; uint8_t *kind; LevelPlan *plan; };
__global__ void __launch_bounds__(1024) k_sel_scan(int32_t *bcnt, int nblocks, RootPlan r) {
    __shared__ int sm[33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < nblocks; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < nblocks ? bcnt[i] : 0;
        int incl = v;
        for (int d = 1; d < 32; d <<= 1) { int t = __shfl_up_sync(FULL, incl, d); if (lane >= d) incl += t; }
        __syncthreads();
        if (lane == 31) sm[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int w = sm[lane], wi = w;
            for (int d = 1; d < 32; d <<= 1) { int t = __shfl_up_sync(FULL, wi, d); if (lane >= d) wi += t; }
            sm[lane] = wi - w;
            if (lane == 31) sm[32] = wi;
        }
        __syncthreads();
        if (i < nblocks) bcnt[i] = carry + sm[wid] + incl - v;
        carry += sm[32];
        __syncthreads();
    }
    if (threadIdx.x == 0) { // the root: its rows are the sampled ones
        r.seg_cnt[1] = carry; r.kind[1] = EVB_KIND_BUILD;
        r.cum[0] = 0; r.cum[1] = carry; r.slot_node[0] = 1; r.rbase[0] = 0;
        r.pl[0] = make_int4(1, 0, carry, 0); r.pl[1] = make_int4(0, carry, 0, 0);
        r.plan[1].nbuild = 1; r.plan[1].npl = 1; r.plan[1].R = carry; r.plan[1].n_sel = carry; r.plan[1].total = carry;
    }
}
__global__ void __launch_bounds__(SEL_THREADS) k_sel_scatter(const uint8_t *mask, uint8_t cond, long long n, const int32_t *boff, uint32_t *rows) {
    constexpr int NW = SEL_CHUNK / 32;
    __shared__ uint32_t s_bits[NW];
    __shared__ int s_pref[NW];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long base = (long long)blockIdx.x * SEL_CHUNK;
    for (int i8 = 0; i8 < SEL_CHUNK / SEL_THREADS; ++i8) {
        const long long i = base + i8 * SEL_THREADS + threadIdx.x;
        const bool sel = i < n && mask[i] <= cond;
        const unsigned bal = __ballot_sync(FULL, sel);
        if (lane == 0) s_bits[i8 * (SEL_THREADS / 32) + wid] = bal;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int c0 = __popc(s_bits[2 * lane]), c1 = __popc(s_bits[2 * lane + 1]);
        int incl = c0 + c1;
        for (int d = 1; d < 32; d <<= 1) { int t = __shfl_up_sync(FULL, incl, d); if (lane >= d) incl += t; }
        s_pref[2 * lane] = incl - c0 - c1;
        s_pref[2 * lane + 1] = incl - c1;
    }
    __syncthreads();
    const int off = boff[blockIdx.x];
    for (int i8 = 0; i8 < SEL_CHUNK / SEL_THREADS; ++i8) {
        const int pos = i8 * SEL_THREADS + threadIdx.x;
        const uint32_t word = s_bits[pos >> 5];
        if ((word >> lane) & 1u) rows[off + s_pref[pos >> 5] + __popc(word & ((1u << lane) - 1u))] = (uint32_t)(base + pos);
    }
}
static_assert(SEL_CHUNK / 32 == 64, "k_sel_scatter assumes 64 ballot words");

// ---------------------------------------------------------------------------------- training predict (+ next gradients)
struct FinArgs {
    const uint8_t *xT;
    const uint32_t *t_packed;
    const float *t_pred;
    float *pred, *grad;
    const void *y;
    uint32_t *nidx;
    unsigned *gmax; // [ng] max |g| of the gradients computed here
    int ng;
    long long n;
    int RS, K, nq, unit_w, elided, loss, nn, ycols, compute_grads, packed_in_smem;
    AlphaSet alpha;
    int mode; // 0: traverse, add the leaf, next gradients; 1: traverse only (leaf ids); 2: leaf ids are in nidx, add + gradients
    const uint4 *pub_src; // the finished tree goes to pinned host memory from here (pub_n 16-byte words; 0: a later kernel does it)
    uint4 *pub_dst;
    int pub_n;
};
__global__ void __launch_bounds__(256) k_finalize(FinArgs a) {
    extern __shared__ uint32_t s_packed[];
    if (blockIdx.x == 0) publish(a.pub_src, a.pub_dst, a.pub_n);
    const uint32_t *packed = a.t_packed;
    if (a.packed_in_smem) {
        for (int i = threadIdx.x; i < a.nn; i += blockDim.x) s_packed[i] = a.t_packed[i];
        __syncthreads();
        packed = s_packed;
    }
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float *rec = nullptr;
    if (i < a.n) {
        const int nid = a.mode == 2 ? (int)a.nidx[i] : traverse(packed, a.xT + (size_t)i * a.RS);
        a.nidx[i] = (uint32_t)nid;
        float *p = a.pred + (size_t)i * a.K;
        if (a.mode != 1) pred_add(a.loss, a.K, p, a.t_pred + (size_t)(nid - 1) * a.K);
        if (a.compute_grads && a.mode != 1) {
            rec = a.grad + (size_t)i * a.nq;
            grad_row(a.loss, a.K, a.elided != 0, p, a.y, a.ycols, i, a.unit_w ? 1.0f : rec[a.nq - 1], rec, a.alpha);
        }
    }
    if (a.compute_grads && a.mode != 1) block_absmax(rec, a.ng, a.gmax);
}

// The same update with everything a CTA's 256 rows hold staged through shared memory: bins, predictions and gradient records are
// contiguous in memory per CTA but strided per row (K and nq words), so they are copied with coalesced accesses of 16 bytes
// and every thread works on its own row out of shared memory.  Rows of bins are padded by one word so that equal byte offsets
// of different rows fall into different banks.  Used when it all fits; KT: outputs known at compile time (0: up to 32), so that a
// row's predictions and gradients stay in registers.
// Bound by HBM: per row RS + 8 K + 4 nq + 8 bytes (and y).  Measured before the records went through shared memory: 2M x 28, five
// outputs 0.140 ms, 5M x 50, two outputs 0.177 ms.
__device__ __forceinline__ void copy_floats(float *dst, const float *src, int n) { // both 16-byte aligned
    for (int i = threadIdx.x; i < n >> 2; i += 256) reinterpret_cast<float4 *>(dst)[i] = reinterpret_cast<const float4 *>(src)[i];
    for (int i = (n & ~3) + threadIdx.x; i < n; i += 256) dst[i] = src[i];
}
template <int KT>
__global__ void __launch_bounds__(256) k_finalize_staged(FinArgs a) {
    extern __shared__ __align__(16) uint32_t s_fin[]; // predictions [256][K], records [256][nq], packed tree [nn], bins [256][RS / 4 + 1]
    constexpr int KM = KT ? KT : 32;
    const int K = KT ? KT : a.K, nq = a.nq;
    float *s_p = reinterpret_cast<float *>(s_fin), *s_g = s_p + 256 * K;
    uint32_t *s_tree = reinterpret_cast<uint32_t *>(s_g + 256 * nq);
    uint32_t *s_rows = s_tree + a.nn;
    if (blockIdx.x == 0) publish(a.pub_src, a.pub_dst, a.pub_n);
    const int rw = a.RS >> 2, rwp = rw + 1; // words per row, padded
    for (int i = threadIdx.x; i < a.nn; i += 256) s_tree[i] = a.t_packed[i];
    const long long row0 = (long long)blockIdx.x * 256;
    const int nr = (int)min((long long)256, a.n - row0);
    const uint4 *src = reinterpret_cast<const uint4 *>(a.xT + (size_t)row0 * a.RS);
    const int cpr = a.RS >> 4, nchunk = nr * cpr;
    for (int c = threadIdx.x; c < nchunk; c += 256) {
        const uint4 v = src[c];
        const int r = c / cpr, part = c - r * cpr;
        uint32_t *d = s_rows + r * rwp + part * 4;
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
    copy_floats(s_p, a.pred + (size_t)row0 * K, nr * K);
    const long long i = row0 + threadIdx.x;
    float w = 1.0f;
    if (a.compute_grads && !a.unit_w && i < a.n) w = a.grad[(size_t)i * nq + nq - 1];
    __syncthreads();
    float *rec = nullptr;
    if (i < a.n) {
        const int nid = traverse(s_tree, reinterpret_cast<const uint8_t *>(s_rows + threadIdx.x * rwp));
        a.nidx[i] = (uint32_t)nid;
        float p[KM], leaf[KM], g[2 * KM];
        float *sp = s_p + threadIdx.x * K;
#pragma unroll
        for (int k = 0; k < KM; ++k) if (k < K) { p[k] = sp[k]; leaf[k] = __ldg(a.t_pred + (size_t)(nid - 1) * K + k); }
        pred_add(a.loss, K, p, leaf);
#pragma unroll
        for (int k = 0; k < KM; ++k) if (k < K) sp[k] = p[k];
        if (a.compute_grads) {
            grad_row(a.loss, K, a.elided != 0, p, a.y, a.ycols, i, w, g, a.alpha);
            rec = s_g + threadIdx.x * nq;
#pragma unroll
            for (int c = 0; c < 2 * KM; ++c) if (c < a.ng) rec[c] = g[c];
            if (!a.unit_w) rec[nq - 1] = w;
        }
    }
    __syncthreads();
    copy_floats(a.pred + (size_t)row0 * K, s_p, nr * K);
    if (a.compute_grads) {
        copy_floats(a.grad + (size_t)row0 * nq, s_g, nr * nq);
        block_absmax(rec, a.ng, a.gmax);
    }
}

// The same update as a pipeline: a few CTAs per SM stay resident and walk over tiles of 256 rows.  The tree and its leaf values are loaded into shared memory once per CTA; the bins of tile t + 1 are copied into the
// other of two shared-memory buffers (`cp.async`, 16 bytes per copy; rows sit at an odd number of 16-byte chunks, so
// the same feature of 8 adjacent rows falls into different banks) while tile t is traversed, and the row's prediction
// and target are requested before the traversal starts, so that a tile costs one memory round trip, not three.
// Rows come from xT ([n][RS]) or, on the fixed-point histogram path, from the 16-byte chunk rows xH ([n][RSH], feature f
// at byte f) plus the word of tail features kept in xE: 104 instead of 128 bytes per row at 100 features.
struct FinPipeArgs {
    FinArgs f;
    const uint8_t *rowsA; // xT or xH
    const uint2 *xE;      // non-null: word y of xE[row] follows the row's bytes (tail features)
    int strideA;          // bytes between rows of rowsA
    int wordsA;           // words copied per row from rowsA
    int S;                // words per row in shared memory: a multiple of 4, an odd number of 16-byte chunks
    int ntiles;
};
// One output.  MSE1: mse with unit weights (the record is g alone): loss and record layout are compile-time constants
template <bool MSE1>
__global__ void __launch_bounds__(256) k_finalize_pipe(FinPipeArgs a) {
    // [nnp] packed tree, [nnp] leaf values, 2 x [256][S] words of bins; nnp = nn rounded up to four
    // words, so that the row buffers start on a 16-byte boundary (the copies into them are 16 bytes wide)
    extern __shared__ __align__(16) uint32_t s_fp[];
    const FinArgs &f = a.f;
    if (blockIdx.x == 0) publish(f.pub_src, f.pub_dst, f.pub_n);
    const int nnp = (f.nn + 3) & ~3;
    uint32_t *s_tree = s_fp;
    float *s_leaf = reinterpret_cast<float *>(s_fp + nnp);
    uint32_t *s_rows = s_fp + 2 * nnp;
    const int S = a.S, wA = a.wordsA;
    for (int i = threadIdx.x; i < f.nn; i += 256) {
        s_tree[i] = f.t_packed[i];
        s_leaf[i] = f.t_pred[i];
    }
    const int cpr = wA >> 2;                     // 16-byte chunks per row
    const uint32_t magic = 65536u / (uint32_t)cpr + 1u; // (c * magic) >> 16 == c / cpr for c < 4096, cpr <= 16
    auto stage = [&](int tile, int buf) {
        if (tile < a.ntiles) {
            const long long row0 = (long long)tile * 256;
            const int nr = (int)min((long long)256, f.n - row0);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_rows + (size_t)buf * 256 * S);
            const uint8_t *src = a.rowsA + (size_t)row0 * a.strideA;
            const int total = nr * cpr;
            for (int c = threadIdx.x; c < total; c += 256) {
                const int r = (int)(((uint32_t)c * magic) >> 16), part = c - r * cpr;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(r * S + part * 4) * 4u),
                             "l"(src + (size_t)r * a.strideA + part * 16) : "memory");
            }
            if (a.xE && (int)threadIdx.x < nr)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (uint32_t)(threadIdx.x * S + wA) * 4u),
                             "l"(reinterpret_cast<const uint32_t *>(a.xE + row0 + threadIdx.x) + 1) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned gm = 0u, hm = 0u; // bits of the largest |g|, |h| of this thread's rows (a NaN is larger than all numbers)
    int buf = 0;
    stage(blockIdx.x, 0);
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, buf ^= 1) {
        stage(tile + gridDim.x, buf ^ 1);
        const long long i = (long long)tile * 256 + threadIdx.x;
        const bool act = i < f.n;
        float *p = f.pred + i;
        float pv = 0.0f;
        if (act) {
            pv = *p;
            if (f.compute_grads) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(f.y) + (size_t)i * 4));
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads(); // tile `tile` (and, the first time, the tree) is in place
        if (act) {
            const int nid = traverse(s_tree, reinterpret_cast<const uint8_t *>(s_rows + ((size_t)buf * 256 + threadIdx.x) * S));
            f.nidx[i] = (uint32_t)nid;
            const int loss = MSE1 ? (int)EVB_MSE : f.loss;
            pred_add(loss, 1, &pv, s_leaf + (nid - 1));
            *p = pv;
            if (f.compute_grads) {
                const int nq = MSE1 ? 1 : f.nq;
                float *rec = f.grad + (size_t)i * nq, g[2]; // one output: g, h and the weight at most
                const float w = MSE1 || f.unit_w ? 1.0f : rec[nq - 1];
                grad_row(loss, 1, MSE1 ? true : f.elided != 0, &pv, f.y, 1, i, w, g, f.alpha);
                rec[0] = g[0];
                gm = max(gm, __float_as_uint(fabsf(g[0])));
                if (!MSE1 && f.ng > 1) { rec[1] = g[1]; hm = max(hm, __float_as_uint(fabsf(g[1]))); }
            }
        }
        __syncthreads(); // everybody is done with this buffer: the next iteration refills it
    }
    if (f.compute_grads) {
        const float m2[2] = {__uint_as_float(gm), __uint_as_float(hm)};
        block_absmax(m2, f.ng, f.gmax); // K == 1: one or two channels
    }
}

// ---------------------------------------------------------------------------------- quantile leaves
// Leaf values of the quantile loss: the alpha-quantile (linear interpolation between the two neighbouring order
// statistics, `Statistics.quantile`) of the residuals of the sampled rows of every leaf (src/predict.jl:264-272).
// The order statistics of all leaves are found together by a radix selection on the order-preserving bit pattern of
// the residual: four passes of 8 bits, each a counting kernel over the rows (one shared-memory-free atomic per row
// and wanted rank into the leaf's 256 counters) and a pick kernel (one warp per leaf walks its counters).
struct QselArgs {
    const uint32_t *nidx;
    const float *grad;        // residual of row i: grad[i * GS + roff]
    const uint8_t *mask;      // rows with mask <= cond are sampled; null: all
    uint32_t *cnt;            // [2][nn + 1][256]
    uint32_t *prefix;         // [2][nn + 1] bits decided so far
    uint32_t *rank;           // [2][nn + 1] rank still to find inside the current prefix
    float *gamma;             // [nn + 1] interpolation weight
    const uint8_t *t_split;
    const double *nsum;
    float *t_pred;
    long long n;
    int GS, roff, nn, C, pass, K, k, clamp; // k: output row being filled; clamp: max(eps, .) on the denominator (quantile)
    uint8_t cond;
    double alpha, eb, lambda, L2; // eb = eta / bagging_size
};
__device__ __forceinline__ uint32_t float_key(float v) { const uint32_t b = __float_as_uint(v); return (b & 0x80000000u) ? ~b : b | 0x80000000u; }
__device__ __forceinline__ float key_float(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? k & 0x7fffffffu : ~k); }
__global__ void __launch_bounds__(256) k_qsel_count(QselArgs a) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || (a.mask && a.mask[i] > a.cond)) return;
    const uint32_t leaf = a.nidx[i];
    const uint32_t key = float_key(a.grad[(size_t)i * a.GS + a.roff]);
    const int shift = 24 - 8 * a.pass;
    const uint32_t digit = (key >> shift) & 0xffu;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const size_t e = (size_t)r * (a.nn + 1) + leaf;
        // pass 0 counts every row; later passes only the rows that share the bits decided so far
        if (a.pass == 0 || (key >> (shift + 8)) == (a.prefix[e] >> (shift + 8))) atomicAdd(&a.cnt[e * 256 + digit], 1u);
        if (a.pass == 0) break; // the first pass is the same for both ranks: counted once, in the counters of rank 0
    }
}
__global__ void __launch_bounds__(256) k_qsel_pick(QselArgs a) {
    const int leaf = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (leaf < 1 || leaf > a.nn) return;
    const int shift = 24 - 8 * a.pass;
    for (int r = 0; r < 2; ++r) {
        const size_t e = (size_t)r * (a.nn + 1) + leaf;
        uint32_t *cnt = a.cnt + (a.pass == 0 ? (size_t)leaf : e) * 256;
        uint32_t c[8], tot = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) { c[q] = cnt[lane * 8 + q]; tot += c[q]; }
        uint32_t incl = tot;
        for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += v; }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        uint32_t want;
        if (a.pass == 0) {
            // ranks of the two order statistics: h = (n - 1) alpha, lo = floor(h), hi = lo + 1 (clamped)
            const double hpos = total > 0 ? (double)(total - 1) * a.alpha : 0.0;
            const uint32_t lo = (uint32_t)floor(hpos), hi = lo + 1 < total ? lo + 1 : lo;
            if (r == 0 && lane == 0) a.gamma[leaf] = total > 0 ? (float)(hpos - floor(hpos)) : -1.0f; // -1: no sampled row
            want = r == 0 ? lo : hi;
        } else {
            want = a.rank[e];
        }
        // the digit whose cumulative count first exceeds `want`
        const uint32_t excl = incl - tot;
        int found = -1;
        uint32_t before = 0;
        if (total > 0 && want >= excl && want < incl) {
            uint32_t run = excl;
#pragma unroll
            for (int q = 0; q < 8; ++q) { if (found < 0 && want < run + c[q]) { found = lane * 8 + q; before = run; } run += c[q]; }
        }
        const unsigned who = __ballot_sync(FULL, found >= 0);
        if (who) {
            const int src = __ffs(who) - 1;
            found = __shfl_sync(FULL, found, src);
            before = __shfl_sync(FULL, before, src);
            if (lane == 0) {
                a.prefix[e] = (a.pass == 0 ? 0u : a.prefix[e]) | ((uint32_t)found << shift);
                a.rank[e] = want - before;
            }
        } else if (lane == 0) { a.prefix[e] = 0u; a.rank[e] = 0u; }
        __syncwarp();
    }
    // the counters are used again by the next pass
    for (int r = 0; r < 2; ++r) {
        uint32_t *cnt = a.cnt + ((size_t)r * (a.nn + 1) + leaf) * 256;
        for (int q = lane; q < 256; q += 32) cnt[q] = 0u;
    }
}
// leaf value from the two order statistics (their full keys are in `prefix` after the last pass)
__global__ void k_qsel_leaf(QselArgs a) {
    const int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf < 1 || leaf > a.nn || a.t_split[leaf - 1]) return;
    const float g = a.gamma[leaf];
    if (g < 0.0f) return; // not a leaf of this tree (or no sampled row reached it): keeps its zero
    const float lo = key_float(a.prefix[leaf]), hi = key_float(a.prefix[(size_t)(a.nn + 1) + leaf]);
    const double q = (double)lo + (double)g * ((double)hi - (double)lo);
    const double w = a.nsum[(size_t)leaf * a.C + a.C - 1];
    const double denom = 1.0 + a.lambda + a.L2 / w;
    a.t_pred[(size_t)(leaf - 1) * a.K + a.k] = (float)(a.eb * q / (a.clamp ? fmax(DBL_EPSILON, denom) : denom));
}

// node of every sampled row from the row lists left by the partition kernels; one CTA per node
__global__ void k_nidx_from_partition(const uint32_t *rows0, const uint32_t *rows1, const int32_t *seg_start,
                                      const int32_t *seg_cnt, const uint8_t *t_split, int nn, uint32_t *out) {
    for (int n = 1 + blockIdx.x; n <= nn; n += gridDim.x) {
        const int cnt = seg_cnt[n];
        if (cnt <= 0 || t_split[n - 1]) continue;
        const int depth = 32 - __clz(n); // root = 1
        const uint32_t *rows = ((depth - 1) & 1) ? rows1 : rows0;
        const int s0 = seg_start[n];
        for (int r = threadIdx.x; r < cnt; r += blockDim.x) out[rows[s0 + r]] = (uint32_t)n;
    }
}

// ---------------------------------------------------------------------------------- binarize
// searchsortedfirst(edges[j], x): 1 + number of edges strictly below x
template <typename T>
__global__ void __launch_bounds__(256) k_binarize(const T *x, long long ld, long long n, const T *edges, int nedges, uint8_t *out, long long ldo,
                                                   int *nan_err = nullptr) {
    extern __shared__ unsigned char s_raw[];
    T *e = reinterpret_cast<T *>(s_raw);
    const int j = blockIdx.y;
    for (int q = threadIdx.x; q < nedges; q += blockDim.x) e[q] = edges[(size_t)j * nedges + q];
    __syncthreads();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const T v = x[(size_t)j * ld + i];
        if (nan_err && v != v) atomicCAS(nan_err, 0, EVB_DERR_NAN); // missing values are not supported (test/missings.jl)
        int lo = 0, hi = nedges;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (e[mid] < v) lo = mid + 1; else hi = mid; }
        out[(size_t)j * ldo + i] = (uint8_t)(lo + 1);
    }
}

// ---------------------------------------------------------------------------------- evaluation data
struct EvalArgs {
    const uint8_t *xT;
    const uint32_t *t_packed;
    const float *t_pred;
    const float *fixed_leaf; // non-null: every row receives this leaf (the one-node bias tree), no traversal
    float *pred;
    const void *y;
    const float *w;
    double *part; // [gridDim.x][2]
    long long n;
    int RS, K, loss, metric, nn, ycols, packed_in_smem;
    AlphaSet alpha;
};
// `predict!(cb.p, tree, cb.x_bin, cb.feattypes)` followed by the per-row metric (src/callback.jl:123-128).  Every
// block owns a fixed set of rows and sums them in a fixed order, so the result does not depend on scheduling.
__global__ void __launch_bounds__(256) k_eval_tree(EvalArgs a) {
    extern __shared__ uint32_t s_packed[];
    __shared__ double s_red[2][8];
    const uint32_t *packed = a.t_packed;
    if (a.packed_in_smem && !a.fixed_leaf) {
        for (int i = threadIdx.x; i < a.nn; i += blockDim.x) s_packed[i] = a.t_packed[i];
        __syncthreads();
        packed = s_packed;
    }
    double sv = 0.0, sw = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (long long)gridDim.x * blockDim.x) {
        float *p = a.pred + (size_t)i * a.K;
        const float *leaf = a.fixed_leaf ? a.fixed_leaf : a.t_pred + (size_t)(traverse(packed, a.xT + (size_t)i * a.RS) - 1) * a.K;
        pred_add(a.loss, a.K, p, leaf);
        const float w = a.w ? a.w[i] : 1.0f;
        sv += (double)metric_row(a.metric, a.K, p, a.y, a.ycols, i, w, a.alpha);
        sw += (double)w;
    }
    for (int o = 16; o > 0; o >>= 1) { sv += __shfl_down_sync(FULL, sv, o); sw += __shfl_down_sync(FULL, sw, o); }
    if ((threadIdx.x & 31) == 0) { s_red[0][threadIdx.x >> 5] = sv; s_red[1][threadIdx.x >> 5] = sw; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tv = 0.0, tw = 0.0;
        for (int q = 0; q < 8; ++q) { tv += s_red[0][q]; tw += s_red[1][q]; }
        a.part[2 * blockIdx.x] = tv;
        a.part[2 * blockIdx.x + 1] = tw;
    }
}
__global__ void __launch_bounds__(256) k_eval_sum(const double *part, int nblocks, double *out, const uint4 *pub_src, uint4 *pub_dst, int pub_n) {
    __shared__ double s_red[2][256];
    double tv = 0.0, tw = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 256) { tv += part[2 * b]; tw += part[2 * b + 1]; }
    s_red[0][threadIdx.x] = tv; s_red[1][threadIdx.x] = tw;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) { s_red[0][threadIdx.x] += s_red[0][threadIdx.x + o]; s_red[1][threadIdx.x] += s_red[1][threadIdx.x + o]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) { out[0] = s_red[0][0]; out[1] = s_red[1][0]; }
    __syncthreads(); // the sums are part of the block
    publish(pub_src, pub_dst, pub_n);
}

} // namespace

// =====================================================================================================
int32_t evb_launch_transpose(evb_handle *, const uint8_t *xcol_dev, int64_t ld, int64_t nrows, int j0, int nj, uint8_t *xT,
                             int RS, cudaStream_t st) {
    dim3 grid((unsigned)((nrows + 255) / 256), (unsigned)((nj + 3) / 4));
    k_transpose<<<grid, 256, 0, st>>>(xcol_dev, ld, nrows, j0, nj, xT, RS);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_check_bins(evb_handle *h) {
    const size_t total = (size_t)h->n * h->nfeats;
    k_check_bins<<<(unsigned)std::min<size_t>((total + 255) / 256, (size_t)h->num_sms * 16), 256, 0, h->st>>>(h->xC, total, h->B, h->d_err);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_init_state(evb_handle *h, const float *w_dev, const float *pred0_dev, const float *mu_dev) {
    k_init_state<<<(unsigned)((h->n + 255) / 256), 256, 0, h->st>>>(h->grad, h->pred, w_dev, pred0_dev, mu_dev, h->n, h->K, h->nq,
                                                                      h->unit_w ? nullptr : h->d_gmax + h->nq - 1);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_grads(evb_handle *h) {
    EVB_CUDA(cudaMemsetAsync(evb_gmax(h, false), 0, sizeof(unsigned) * h->ng, h->st));
    evb_tic(h, EVB_T_GRADS);
    k_grads<<<(unsigned)((h->n + 255) / 256), 256, 0, h->st>>>(h->p.loss, h->K, h->nq, h->unit_w ? 1 : 0, h->Ce != h->C, h->ycols, h->n, h->pred, h->y, h->grad,
                                                                evb_gmax(h, false), h->ng, evb_alpha_set(h));
    evb_toc(h, EVB_T_GRADS);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_pcg_tables(int dev) { // once per device, outside any capture
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> g(mu);
    if (dev < 64 && done[dev]) return EVB_OK;
    u128 m[32], a[32];
    m[0] = ((u128)PCG_MULT_HI << 64) | PCG_MULT_LO;
    a[0] = 1;
    for (int k = 1; k < 32; ++k) { m[k] = m[k - 1] * m[k - 1]; a[k] = (m[k - 1] + 1) * a[k - 1]; }
    EVB_CUDA(cudaMemcpyToSymbol(c_pcg_m, m, sizeof(m)));
    EVB_CUDA(cudaMemcpyToSymbol(c_pcg_g, a, sizeof(a)));
    if (dev < 64) done[dev] = true;
    return EVB_OK;
}
// the generator after the words of n bytes have been taken from it (same six words as k_sel_pcg reads)
void evb_pcg_advance(uint64_t gen[6], int64_t n) {
    const u128 inc = ((u128)gen[3] << 64) | gen[2], mult = ((u128)PCG_MULT_HI << 64) | PCG_MULT_LO;
    u128 st = ((u128)gen[1] << 64) | gen[0];
    const uint64_t words = (uint64_t)(n + 3) / 4;
    if (words == 0) return;
    const uint64_t fresh = words - gen[4], outputs = (fresh + 1) / 2;
    u128 m = mult, g = 1, am = 1, ag = 0; // am, ag: the steps taken so far
    for (uint64_t k = outputs; k; k >>= 1) {
        if (k & 1) { am = am * m; ag = ag * m + g; }
        g = (m + 1) * g;
        m = m * m;
    }
    st = st * am + inc * ag;
    gen[0] = (uint64_t)st; gen[1] = (uint64_t)(st >> 64);
    gen[4] = fresh & 1;
    if (outputs) {
        const uint64_t hi = (uint64_t)(st >> 64), x = hi ^ (uint64_t)st;
        const unsigned r = (unsigned)(hi >> 58);
        gen[5] = ((x >> r) | (x << ((64u - r) & 63u))) >> 32;
    }
}

// the sampled rows of a tree, after k_tree_begin
int32_t evb_launch_rows_init(evb_handle *h, int use_mask, uint8_t mask_cond) {
    if (!use_mask) return EVB_OK;
    const int nblocks = (int)((h->n + SEL_CHUNK - 1) / SEL_CHUNK);
    const RootPlan r{h->seg_cnt, h->cum, h->slot_node, h->rbase, h->pl, h->kind, h->plan};
    evb_tic(h, EVB_T_ROWS_INIT);
    if (use_mask == EVB_MASK_PCG) EVB_CUDA(evb_launch(k_sel_pcg, dim3(nblocks), dim3(SEL_THREADS), 0, h->st, h->gen_d, mask_cond, h->n, h->mask_d, h->scan_tmp));
    else EVB_CUDA(evb_launch(k_sel_count, dim3(nblocks), dim3(SEL_THREADS), 0, h->st, h->mask_d, mask_cond, h->n, h->scan_tmp));
    EVB_CUDA(evb_launch(k_sel_scan, dim3(1), dim3(1024), 0, h->st, h->scan_tmp, nblocks, r));
    EVB_CUDA(evb_launch(k_sel_scatter, dim3(nblocks), dim3(SEL_THREADS), 0, h->st, h->mask_d, mask_cond, h->n, h->scan_tmp, h->rows[0]));
    evb_toc(h, EVB_T_ROWS_INIT);
    h->tm.launches[EVB_T_ROWS_INIT] += 2;
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_finalize(evb_handle *h, bool compute_grads, int mode, void *publish_to) {
    FinArgs a;
    a.xT = h->xT; a.t_packed = h->t_packed; a.t_pred = h->t_pred; a.pred = h->pred; a.grad = h->grad; a.y = h->y;
    a.nidx = h->nidx; a.n = h->n; a.RS = h->RS; a.K = h->K; a.nq = h->nq; a.unit_w = h->unit_w ? 1 : 0; a.elided = h->Ce != h->C; a.loss = h->p.loss; a.nn = h->nn;
    a.gmax = evb_gmax(h, true); a.ng = h->ng; // cleared by the root's scan or the tree kernel
    a.ycols = h->ycols; a.compute_grads = compute_grads ? 1 : 0; a.alpha = evb_alpha_set(h); a.mode = mode;
    a.pub_src = reinterpret_cast<const uint4 *>(h->plan); a.pub_dst = static_cast<uint4 *>(publish_to); a.pub_n = publish_to ? (int)(h->h_tree_bytes / 16) : 0;
    const size_t smem = (size_t)h->nn * 4;
    a.packed_in_smem = smem <= 40 * 1024 ? 1 : 0;
    const size_t staged = smem + (size_t)256 * (h->RS + 4) + (size_t)1024 * (h->K + h->nq);
    static bool attr_pipe[64] = {};
    static const bool direct = getenv("EVB_FINALIZE_DIRECT") != nullptr;
    static const bool no_pipe = getenv("EVB_FINALIZE_PIPE") != nullptr && atoi(getenv("EVB_FINALIZE_PIPE")) == 0;
    // pipelined kernel: rows from the chunk layout of the fixed-point histogram kernel when it exists, else from xT
    FinPipeArgs pa;
    pa.f = a;
    const bool from_q2 = h->use_q2; // evb_create sees to it that this kernel can run then; xH holds feature f at byte f of the row, the tail features follow in xE
    pa.rowsA = from_q2 ? h->xH : h->xT;
    pa.xE = from_q2 && h->q2.ntail > 0 ? h->xE : nullptr;
    pa.strideA = from_q2 ? h->q2.RSH : h->RS;
    pa.wordsA = pa.strideA / 4;
    pa.S = pa.wordsA + 4; // one more chunk: room for the tail word, and an odd chunk count (wordsA / 4 is even or RSH-odd)
    if (((pa.S >> 2) & 1) == 0) pa.S += 4;
    pa.ntiles = (int)((h->n + 255) / 256);
    const size_t pipe_smem = (size_t)((h->nn + 3) & ~3) * 8 + (size_t)2 * 256 * pa.S * 4;
    evb_tic(h, EVB_T_FINALIZE);
    // measured (B200): 0.33 instead of 0.42 ms per 10M rows x 100 features with one output; with several outputs the
    // prediction and gradient streams outweigh the bins and the one-tile-per-CTA kernel below is faster
    if (mode == 0 && h->K == 1 && pipe_smem <= 100 * 1024 && pa.wordsA <= 64 && !direct && !no_pipe && h->dev < 64) {
        if (!attr_pipe[h->dev]) {
            cudaFuncSetAttribute(k_finalize_pipe<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
            cudaFuncSetAttribute(k_finalize_pipe<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
            attr_pipe[h->dev] = true;
        }
        int per_sm = (int)((227 * 1024) / (pipe_smem + 1024)); // 1 KB per resident CTA is reserved
        if (per_sm > 6) per_sm = 6;
        if (per_sm < 1) per_sm = 1;
        int grid = h->num_sms * per_sm;
        if (grid > pa.ntiles) grid = pa.ntiles;
        if (h->p.loss == EVB_MSE && h->nq == 1) EVB_CUDA(evb_launch(k_finalize_pipe<true>, dim3(grid), dim3(256), pipe_smem, h->st, pa));
        else EVB_CUDA(evb_launch(k_finalize_pipe<false>, dim3(grid), dim3(256), pipe_smem, h->st, pa));
    } else if (mode == 0 && h->RS <= 256 && staged <= 100 * 1024 && !direct && h->dev < 64) {
        const dim3 tiles((unsigned)((h->n + 255) / 256));
#define EVB_FIN(KT) do { \
            if (staged > 48 * 1024) EVB_CUDA(cudaFuncSetAttribute(k_finalize_staged<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024)); \
            EVB_CUDA(evb_launch(k_finalize_staged<KT>, tiles, dim3(256), staged, h->st, a)); } while (0)
        switch (h->K) {
        case 1: EVB_FIN(1); break;
        case 2: EVB_FIN(2); break;
        case 3: EVB_FIN(3); break;
        case 4: EVB_FIN(4); break;
        case 5: EVB_FIN(5); break;
        case 6: EVB_FIN(6); break;
        case 7: EVB_FIN(7); break;
        case 8: EVB_FIN(8); break;
        default: EVB_FIN(0);
        }
#undef EVB_FIN
    } else {
        EVB_CUDA(evb_launch(k_finalize, dim3((unsigned)((h->n + 255) / 256)), dim3(256), a.packed_in_smem ? smem : 0, h->st, a));
    }
    evb_toc(h, EVB_T_FINALIZE);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

// applies the current tree (or, with `fixed_leaf_dev`, one leaf for every row) to the evaluation predictions and
// leaves the metric sums in h->d_evsum
int32_t evb_launch_eval(evb_handle *h, const float *fixed_leaf_dev, void *publish_to) {
    EvalArgs a;
    a.xT = h->ev_xT; a.t_packed = h->t_packed; a.t_pred = h->t_pred; a.fixed_leaf = fixed_leaf_dev; a.pred = h->ev_pred;
    a.y = h->ev_y; a.w = h->ev_w; a.part = h->ev_part; a.n = h->ev_n; a.RS = h->RS; a.K = h->K; a.loss = h->p.loss;
    a.metric = h->ev_metric; a.nn = h->nn; a.ycols = h->ycols; a.alpha = evb_alpha_set(h);
    const size_t smem = (size_t)h->nn * 4;
    a.packed_in_smem = smem <= 40 * 1024 ? 1 : 0;
    evb_tic(h, EVB_T_FINALIZE);
    k_eval_tree<<<h->ev_blocks, 256, (a.packed_in_smem && !fixed_leaf_dev) ? smem : 0, h->st>>>(a);
    k_eval_sum<<<1, 256, 0, h->st>>>(h->ev_part, h->ev_blocks, h->d_evsum, reinterpret_cast<const uint4 *>(h->plan), static_cast<uint4 *>(publish_to),
                                     publish_to ? (int)(h->h_tree_bytes / 16) : 0);
    evb_toc(h, EVB_T_FINALIZE);
    h->tm.launches[EVB_T_FINALIZE] += 1; // two kernels inside one timed bracket
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

// quantile loss, K = 1: leaf ids are in h->nidx (finalize mode 1); fills the leaf values of the tree
int32_t evb_launch_quantile_leaves(evb_handle *h, bool use_mask, uint8_t mask_cond) {
    QselArgs a;
    a.nidx = h->nidx; a.grad = h->grad; a.mask = use_mask ? h->mask_d : nullptr; a.cnt = h->qs_cnt; a.prefix = h->qs_prefix;
    a.rank = h->qs_rank; a.gamma = h->qs_gamma; a.t_split = h->t_split; a.nsum = h->nsum; a.t_pred = h->t_pred; a.n = h->n;
    a.GS = h->nq; a.nn = h->nn; a.C = h->C; a.cond = mask_cond;
    a.eb = h->p.eta / (double)h->p.bagging_size; a.lambda = h->p.lambda; a.L2 = h->p.L2; a.K = h->K;
    a.clamp = h->p.loss == EVB_QUANTILE ? 1 : 0; // src/predict.jl:270 has the max(eps, .), :279 has not
    evb_tic(h, EVB_T_FINALIZE);
    for (int k = 0; k < h->K; ++k) { // one selection per output row: the residual of row k sits in the slot of h_k
        const int c = h->K + k;
        a.k = k; a.roff = c;
        a.alpha = h->p.loss == EVB_QUANTILE ? h->p.alpha : h->p.alphas[k];
        for (int pass = 0; pass < 4; ++pass) {
            a.pass = pass;
            k_qsel_count<<<(unsigned)((h->n + 255) / 256), 256, 0, h->st>>>(a);
            if (h->world > 1) {
                // row-sharded: the digit counts of all ranks are added, so every rank walks to the same order
                // statistics of the leaf's rows on all ranks (integer sums: the same leaves as on one GPU)
                int32_t *c32 = reinterpret_cast<int32_t *>(h->qs_cnt);
                EVB_CHECK(evb_nccl_allreduce_i32(h, c32, c32, (size_t)2 * (h->nn + 1) * 256));
            }
            k_qsel_pick<<<(h->nn + 8) / 8, 256, 0, h->st>>>(a);
        }
        k_qsel_leaf<<<(h->nn + 256) / 256, 256, 0, h->st>>>(a);
    }
    evb_toc(h, EVB_T_FINALIZE);
    h->tm.launches[EVB_T_FINALIZE] += 9 * h->K - 1;
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_nidx_from_partition(evb_handle *h, uint32_t *out_dev) {
    EVB_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(uint32_t) * h->n, h->st));
    int blocks = h->nn < 1024 ? h->nn : 1024;
    k_nidx_from_partition<<<blocks, 256, 0, h->st>>>(h->rows[0], h->rows[1], h->seg_start, h->seg_cnt, h->t_split, h->nn, out_dev);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

// ---- training matrix from raw features -----------------------------------------------------------------
struct DevBufT {
    void *p = nullptr;
    ~DevBufT() { evb_dev_free(p); }
};
// `binarize(x_train; edges)` of `init_core` (ext/EvoTreesKernelAbstractionsExt/init.jl:3-6, src/fit-utils.jl:66-72) on the
// device: the raw column-major matrix travels in blocks of whole features (each at most 256 MB) and every block is
// binarized straight into the feature-major bin matrix h->xC; the bins never visit the host.  NaN sets the error word.
int32_t evb_upload_binarize(evb_handle *h, const void *x, int32_t dtype, const void *edges, int32_t nedges) {
    const size_t es = dtype == EVB_F64 ? 8 : 4;
    const int64_t n = h->n;
    const int nfeats = h->nfeats;
    int cf = (int)std::max<int64_t>(1, std::min<int64_t>(nfeats, ((int64_t)256 << 20) / (int64_t)(n * es)));
    DevBufT d_x, d_e;
    EVB_CUDA(evb_dev_alloc(&d_x.p, (size_t)cf * n * es));
    EVB_CUDA(evb_dev_alloc(&d_e.p, (size_t)nedges * nfeats * es));
    EVB_CUDA(cudaMemcpyAsync(d_e.p, edges, (size_t)nedges * nfeats * es, cudaMemcpyHostToDevice, h->st));
    unsigned bx = (unsigned)((n + 255) / 256);
    if (bx > 4096) bx = 4096;
    for (int j0 = 0; j0 < nfeats; j0 += cf) {
        const int nj = std::min(cf, nfeats - j0);
        // no wait at the end of a block: its last chunks travel while the host gathers the next block's first ones
        EVB_CHECK(evb_h2d_staged(d_x.p, (const char *)x + (size_t)j0 * n * es, (size_t)nj * n * es, h->st, false));
        dim3 grid(bx, (unsigned)nj);
        if (dtype == EVB_F32)
            k_binarize<float><<<grid, 256, (size_t)nedges * 4, h->st>>>((const float *)d_x.p, n, n, (const float *)d_e.p + (size_t)j0 * nedges, nedges,
                                                                           h->xC + (size_t)j0 * n, n, h->d_err);
        else
            k_binarize<double><<<grid, 256, (size_t)nedges * 8, h->st>>>((const double *)d_x.p, n, n, (const double *)d_e.p + (size_t)j0 * nedges, nedges,
                                                                            h->xC + (size_t)j0 * n, n, h->d_err);
        EVB_CUDA(cudaGetLastError());
    }
    EVB_CUDA(cudaStreamSynchronize(h->st)); // the staging buffers are freed on return
    return EVB_OK;
}

// ---- stateless entry points -----------------------------------------------------------------------
int32_t evb_check_device(int device) {
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        evb_set_error("no CUDA device available (%s): this library has no CPU fallback", cudaGetErrorString(e));
        return EVB_ERR_CUDA;
    }
    if (device < 0 || device >= ndev) { evb_set_error("device %d out of range (0..%d)", device, ndev - 1); return EVB_ERR_ARG; }
    EVB_CUDA(cudaSetDevice(device));
    return EVB_OK;
}

struct DevBuf {
    void *p = nullptr;
    ~DevBuf() { evb_dev_free(p); }
    cudaError_t alloc(size_t bytes) { return evb_dev_alloc(&p, bytes ? bytes : 1); }
    template <typename T> T *as() { return reinterpret_cast<T *>(p); }
};

// Diagnostic: the quotients of a split scan
static __global__ void __launch_bounds__(256) k_quotients(const double *a, const double *b, double *q, uint8_t *ok, long long n) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    ok[i] = quot_ok(x, y) ? 1 : 0;
    q[i] = quot_ok(x, y) ? quot(x, y) : x / y;
}
extern "C" int32_t evb_test_quotients(int32_t device, int64_t n, const double *a, const double *b, double *q, uint8_t *ok) {
    if (n < 1 || n > (int64_t)1 << 26 || !a || !b || !q || !ok) { evb_set_error("evb_test_quotients: invalid argument"); return EVB_ERR_ARG; }
    EVB_CHECK(evb_check_device(device));
    DevBuf d_a, d_b, d_q, d_ok;
    EVB_CUDA(d_a.alloc((size_t)n * 8)); EVB_CUDA(d_b.alloc((size_t)n * 8)); EVB_CUDA(d_q.alloc((size_t)n * 8)); EVB_CUDA(d_ok.alloc((size_t)n));
    EVB_CUDA(cudaMemcpy(d_a.p, a, (size_t)n * 8, cudaMemcpyHostToDevice));
    EVB_CUDA(cudaMemcpy(d_b.p, b, (size_t)n * 8, cudaMemcpyHostToDevice));
    k_quotients<<<(unsigned)((n + 255) / 256), 256>>>(d_a.as<double>(), d_b.as<double>(), d_q.as<double>(), d_ok.as<uint8_t>(), n);
    EVB_CUDA(cudaGetLastError());
    EVB_CUDA(cudaMemcpy(q, d_q.p, (size_t)n * 8, cudaMemcpyDeviceToHost));
    EVB_CUDA(cudaMemcpy(ok, d_ok.p, (size_t)n, cudaMemcpyDeviceToHost));
    return EVB_OK;
}

extern "C" int32_t evb_binarize(int32_t device, const void *x, int32_t dtype, int64_t nobs, int32_t nfeats, const void *edges,
                                int32_t nedges, uint8_t *x_bin) {
    if (!x || !edges || !x_bin || nobs < 0 || nfeats < 1 || nedges < 1 || nedges > 254 || (dtype != EVB_F32 && dtype != EVB_F64)) {
        evb_set_error("evb_binarize: invalid argument");
        return EVB_ERR_ARG;
    }
    EVB_CHECK(evb_check_device(device));
    if (nobs == 0) return EVB_OK;
    const size_t es = dtype == EVB_F32 ? 4 : 8;
    cudaStream_t st;
    EVB_CUDA(cudaStreamCreate(&st));
    const int64_t chunk = nobs < (int64_t)4 << 20 ? nobs : (int64_t)4 << 20;
    DevBuf d_x, d_e, d_o;
    auto body = [&]() -> int32_t {
        EVB_CUDA(d_x.alloc((size_t)chunk * nfeats * es)); EVB_CUDA(d_e.alloc((size_t)nedges * nfeats * es)); EVB_CUDA(d_o.alloc((size_t)chunk * nfeats));
        EVB_CUDA(cudaMemcpyAsync(d_e.p, edges, (size_t)nedges * nfeats * es, cudaMemcpyHostToDevice, st));
        for (int64_t r0 = 0; r0 < nobs; r0 += chunk) {
            const int64_t nr = nobs - r0 < chunk ? nobs - r0 : chunk;
            EVB_CUDA(cudaMemcpy2DAsync(d_x.p, (size_t)chunk * es, (const char *)x + (size_t)r0 * es, (size_t)nobs * es, (size_t)nr * es,
                                       (size_t)nfeats, cudaMemcpyHostToDevice, st));
            unsigned bx = (unsigned)((nr + 255) / 256);
            if (bx > 4096) bx = 4096;
            dim3 grid(bx, (unsigned)nfeats);
            if (dtype == EVB_F32)
                k_binarize<float><<<grid, 256, (size_t)nedges * 4, st>>>(d_x.as<float>(), chunk, nr, d_e.as<float>(), nedges, d_o.as<uint8_t>(), chunk);
            else
                k_binarize<double><<<grid, 256, (size_t)nedges * 8, st>>>(d_x.as<double>(), chunk, nr, d_e.as<double>(), nedges, d_o.as<uint8_t>(), chunk);
            EVB_CUDA(cudaGetLastError());
            EVB_CUDA(cudaMemcpy2DAsync(x_bin + r0, (size_t)nobs, d_o.p, (size_t)chunk, (size_t)nr, (size_t)nfeats, cudaMemcpyDeviceToHost, st));
        }
        EVB_CUDA(cudaStreamSynchronize(st));
        return EVB_OK;
    };
    int32_t rc = body();
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}
