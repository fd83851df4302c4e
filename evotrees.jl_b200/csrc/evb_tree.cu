// Per-level tree growth on the device: sibling subtraction + split scan + split application
// (`subtract_hist!`, `get_best_split`/`_scan_node!`, `_child_sums!`, `pred_leaf_cpu!`: src/fit-utils.jl:321-332,
// 403-486, src/split.jl:1-117, src/predict.jl:198-247, src/fit.jl:85-137) and the stable row partition
// (`split_set!`, src/fit-utils.jl:93-312; GPU counterpart `update_nodes_idx_kernel!`,
// ext/EvoTreesKernelAbstractionsExt/fit-utils.jl:9-31).  Everything a level needs (active nodes, segment
// bounds, build/subtract choice, work lists) lives in device memory, so the host enqueues a fixed sequence of
// launches per level and never reads anything back until the tree is complete.
#include "evb_histg.cuh"
#include "evb_device.cuh"
#include <float.h>
#include <algorithm>

namespace {

constexpr unsigned FULL = 0xffffffffu;

// exclusive scan over the threads of a block (blockDim.x <= 1024, multiple of 32); returns the exclusive
// prefix of v and writes the block total to *total.  `sm` is 33 ints of shared memory.
__device__ __forceinline__ int block_excl_scan(int v, int *sm, int *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int incl = warp_incl_scan_i(v, lane);
    __syncthreads();
    if (lane == 31) sm[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = lane < nw ? sm[lane] : 0;
        int wi = warp_incl_scan_i(w, lane);
        sm[lane] = wi - w;
        if (lane == 31) sm[32] = wi;
    }
    __syncthreads();
    *total = sm[32];
    return incl - v + sm[wid];
}

// ------------------------------------------------------------------------------------------ begin of a tree
struct BeginArgs {
    int32_t *seg_start, *seg_cnt, *bslot, *t_feat, *cum, *slot_node, *rbase;
    int4 *pl;
    uint8_t *kind, *t_bin, *t_split;
    float *t_gain, *t_w, *t_pred;
    uint32_t *t_packed;
    double *nsum;
    LevelPlan *plan;
    uint32_t *ticket, *rows, *low;
    const uint32_t *gen_js_host; // pinned: generator state and column sample of this tree
    uint32_t *gen_js;
    int ngen_js;
    int nids, nn, K, C, D, all_rows;
    evb_hg::QuantArgs q; // q.grad null: the fixed-point gradients are those of the last tree
};
// One thread per row and per node: clears the tree, lists all rows and plans the root (without a row sample), and turns the
// gradients into fixed-point numbers.
__global__ void __launch_bounds__(256) k_tree_begin(BeginArgs a) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i < a.ngen_js) a.gen_js[i] = __ldcv(a.gen_js_host + i);
    if (a.q.grad) evb_hg::quantize(a.q, i);
    if (a.all_rows && i < a.q.n) a.rows[i] = (uint32_t)i;
    if (i < a.nids) {
        const bool root = i == 1 && a.all_rows;
        a.seg_start[i] = 0; a.seg_cnt[i] = root ? (int32_t)a.q.n : 0; a.kind[i] = root ? EVB_KIND_BUILD : EVB_KIND_NONE; a.bslot[i] = 0; a.ticket[i] = 0u; a.low[i] = 0u;
        for (int c = 0; c < a.C; ++c) a.nsum[(size_t)i * a.C + c] = 0.0;
        if (root) {
            a.cum[0] = 0; a.cum[1] = (int32_t)a.q.n; a.slot_node[0] = 1; a.rbase[0] = 0;
            a.pl[0] = make_int4(1, 0, (int32_t)a.q.n, 0); a.pl[1] = make_int4(0, (int32_t)a.q.n, 0, 0);
            a.plan[1].nbuild = 1; a.plan[1].npl = 1; a.plan[1].R = a.q.n; a.plan[1].n_sel = (int32_t)a.q.n; a.plan[1].total = (int32_t)a.q.n;
        }
    }
    if (i < a.nn) {
        a.t_feat[i] = 0; a.t_bin[i] = 0; a.t_split[i] = 0; a.t_gain[i] = 0.f; a.t_w[i] = 0.f; a.t_packed[i] = 0u;
        for (int k = 0; k < a.K; ++k) a.t_pred[(size_t)i * a.K + k] = 0.f;
    }
    if (i >= 2 && i <= a.D) { a.plan[i].nbuild = 0; a.plan[i].npl = 0; a.plan[i].R = 0; a.plan[i].total = 0; }
}

// ------------------------------------------------------------------------------------------ split scan
constexpr int EVB_MAX_PEERS = 8;

struct ScanArgs {
    const double *hcomp;
    double *hist, *nsum;
    const uint8_t *kind;
    const int32_t *bslot;
    const uint32_t *js0;
    const uint8_t *feattypes;
    const int32_t *mono;
    int32_t *t_feat;
    uint8_t *t_bin, *t_split;
    float *t_gain, *t_w, *t_pred;
    uint32_t *t_packed;
    double *fbest_gain; // [nodes of the level][F] best gain of each feature
    int32_t *fbest_bin; // [nodes of the level][F] its bin (0-based) or -1
    double *fbest_left; // [nodes of the level][F][3] its left sums (one output)
    // oblivious trees (null otherwise): [nodes of the level + 1][F * B] gain of every candidate (0: not eligible),
    // the last row receives the level totals; obl_best = {gain, candidate index or -1} of the shared split
    double *obl_gain, *obl_best;
    const LevelPlan *plan;
    const int32_t *slot_node;
    int slots; // build slots the level can have
    // Row-sharded runs with peer access: every rank scans the feature slots f with f % world == rank (`hcomp` then
    // points at the sums made by k_peer_reduce) and publishes one candidate per node to every rank.
    double *peer_cand[EVB_MAX_PEERS];
    const double *cand_local; // [nodes of the level][world][3 + C]: gain, feature slot, bin, left sums
    int world, rank;          // world == 1: no peers (single GPU, or histograms already summed by NCCL)
    int F, C, K, B, level, D, hist_nodes, loss;
    int elide_h;        // mse: the h channels equal twice the w channel and are rebuilt instead of read
    // non-null: the built histograms are read straight from the integer accumulators of the fixed-point kernel
    // ([slot][bin][channel][SC] sums of q, [slot][bin][SC] row counts) instead of from hcomp
    const unsigned long long *qsum;
    const uint32_t *qcnt;
    const double *qinv;
    const unsigned long long *qlow; // [slot][SC][channel][bin], low_unit times as fine as qsum: of the build slots in `low`
    const uint32_t *low;
    double low_unit;
    int SC, nq, unit_w;
    // non-null: the last feature of a node to be scanned decides the node (one GPU, binary trees)
    uint32_t *ticket;
    unsigned *gmax;           // [ng] cleared by the root's scan: the gradient kernels of this tree start from zero
    int ng;
    int32_t *cur_l, *cur_r;   // where the partition puts the next left / right rows of a split node
    const int32_t *seg_start, *seg_cnt;
    double neb; // -eta / bagging_size
    double lambda, L2, gamma, min_weight;
};

// a load that is issued where it stands, not moved behind the branch its value is used in
__device__ __forceinline__ int load_now(const int32_t *p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
// mae: |mean of the side - mean of the parent| * weight / (1 + lambda + L2 / w)   (src/split.jl:2, 119-130)
__device__ __forceinline__ double term_shift(double g, double w, double mu_p, double d) { return fabs(g / w - mu_p) * w / d; }
// credibility losses: Z * |m1| / (1 + L2 / w), Z from the ratio of variances or of standard deviations
// (src/split.jl:3-4, src/loss.jl:275-289)
__device__ __forceinline__ double term_cred(int loss, double m1, double m2, double w, double L2) {
    const double vhm = (m1 / w) * (m1 / w);
    const double evpv = fmax(DBL_EPSILON, m2 / w - vhm);
    const double z = loss == EVB_CRED_VAR ? vhm / (vhm + evpv) : sqrt(vhm) / (sqrt(vhm) + sqrt(evpv));
    return z * fabs(m1) / (1.0 + L2 / w);
}
__device__ __forceinline__ bool own_gain(int loss) { return loss >= EVB_MAE; }
// gain of one output row of a candidate split: left sums (gl, hl, w_l), parent sums (sg, sh, w_p)
__device__ __forceinline__ double side_gain(const ScanArgs &a, double gl, double hl, double w_l, double sg, double sh, double w_p) {
    const double w_r = w_p - w_l;
    if ((a.loss == EVB_MAE || a.loss == EVB_QUANTILE || a.loss == EVB_MULTIQUANTILE)) {
        const double d_l = fmax(DBL_EPSILON, 1.0 + a.lambda + a.L2 / w_l), d_r = fmax(DBL_EPSILON, 1.0 + a.lambda + a.L2 / w_r);
        const double mu_p = sg / w_p;
        return term_shift(gl, w_l, mu_p, d_l) + term_shift(sg - gl, w_r, mu_p, d_r);
    }
    return term_cred(a.loss, gl, hl, w_l, a.L2) + term_cred(a.loss, sg - gl, sh - hl, w_r, a.L2);
}
// pred_scalar of the three losses (src/predict.jl:219-222, 257-261): the sign is the gradient's, not minus it
__device__ __forceinline__ double own_scalar(const ScanArgs &a, double g, double w) {
    return -a.neb * g / ((a.loss == EVB_MAE || a.loss == EVB_QUANTILE || a.loss == EVB_MULTIQUANTILE) ? fmax(DBL_EPSILON, w + a.lambda * w + a.L2) : (w + a.L2));
}
// pred_leaf_cpu! for output row k (src/predict.jl:198-204, 224-234, 241-247; mae :250-257, cred :211-218)
__device__ __forceinline__ float leaf_value(const ScanArgs &a, const double *s, int k) {
    const int K = a.K, C = a.C;
    if (own_gain(a.loss)) return (float)own_scalar(a, s[k], s[C - 1]);
    double g, h;
    if (a.loss == EVB_GAUSSIAN_MLE || a.loss == EVB_LOGISTIC_MLE) {
        const int Y = K / 2, t = k >> 1, j = k & 1;
        g = s[2 * t + j];
        h = s[2 * Y + 2 * t + j];
    } else {
        g = s[k];
        h = s[K + k];
    }
    return (float)(a.neb * g / fmax(DBL_EPSILON, h + a.lambda * s[C - 1] + a.L2));
}

// Entries of the histogram built for a slot, channel by channel.  A channel's loads are issued together (`load`, raw bits) and
// turned into doubles where they are used (`value`): a conversion or a branch between two loads would make each of them
// wait for the one before it (measured at five classes: 20 us per node and level for a scan, 17 us for a decision).
struct Chan {
    bool cnt;          // row counts
    int idx;           // quantised channel
    double mul;
};
__device__ __forceinline__ Chan chan_of(const ScanArgs &a, int c, int K, int C) {
    const bool h2w = a.elide_h && c >= K && c < 2 * K; // h = 2w (src/loss.jl:52)
    const bool w = c == C - 1 || h2w;
    Chan ch;
    ch.cnt = w && a.unit_w;
    ch.idx = w ? a.nq - 1 : c;
    ch.mul = (h2w ? 2.0 : 1.0) * (ch.cnt || !a.qsum ? 1.0 : __ldg(a.qinv + ch.idx));
    return ch;
}
// bins b0 + j * stride, j < N (past the last one: the last one again), of feature slot f / feature `feat`
template <int N>
__device__ __forceinline__ void chan_load(const ScanArgs &a, const Chan &ch, int slot, int f, uint32_t feat, int c, int b0, int stride, int C, long long (&raw)[N]) {
    if (!a.qsum) {
        const double *p = a.hcomp + (((size_t)slot * a.F + f) * C + c) * a.B;
#pragma unroll
        for (int j = 0; j < N; ++j) raw[j] = __double_as_longlong(p[min(b0 + j * stride, a.B - 1)]);
    } else if (ch.cnt) {
        const uint32_t *p = a.qcnt + (size_t)slot * a.B * a.SC + feat;
#pragma unroll
        for (int j = 0; j < N; ++j) raw[j] = (long long)__ldg(p + (size_t)min(b0 + j * stride, a.B - 1) * a.SC);
    } else {
        const unsigned long long *p = a.qsum + ((size_t)slot * a.B * a.nq + ch.idx) * a.SC + feat;
#pragma unroll
        for (int j = 0; j < N; ++j) raw[j] = (long long)__ldg(p + (size_t)min(b0 + j * stride, a.B - 1) * a.nq * a.SC);
    }
}
__device__ __forceinline__ double chan_value(const ScanArgs &a, const Chan &ch, long long raw) {
    return a.qsum ? (double)raw * ch.mul : __longlong_as_double(raw);
}
// The build slot has sums below those of qsum, bin after bin so that a scan reads whole sectors (in the layout of qsum, 32 bytes for
// every 8 used, they cost a scan half of its time again: 1.6M x 69, 255 bins 0.147 -> 0.217 ms per tree).
__device__ __forceinline__ bool slot_low(const ScanArgs &a, int slot) { return a.qlow && load_now(reinterpret_cast<const int32_t *>(a.low) + slot) != 0; }
template <int N>
__device__ __forceinline__ void chan_load_low(const ScanArgs &a, const Chan &ch, int slot, uint32_t feat, int b0, int stride, long long (&raw)[N]) {
    const unsigned long long *p = a.qlow + (((size_t)slot * a.SC + feat) * a.nq + (ch.cnt ? 0 : ch.idx)) * a.B;
#pragma unroll
    for (int j = 0; j < N; ++j) raw[j] = (long long)__ldg(p + min(b0 + j * stride, a.B - 1));
}
template <int N>
__device__ __forceinline__ void chan_add_low(const ScanArgs &a, const Chan &ch, const long long (&raw)[N], double (&v)[N]) {
    const double unit = ch.cnt ? 0.0 : ch.mul * a.low_unit; // (row counts have none: whatever was loaded is finite)
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] += (double)raw[j] * unit;
}

// Root sum of a channel from the whole numbers of the bins of any feature, raw[j]: bin b0 + j * stride (every sampled row has
// exactly one bin; the reference sums the gradients of the sampled rows directly, src/fit.jl:66).  The total of the whole numbers is
// the same for every feature and converted once, so that all features' scans and the decision work with the same parent.
template <int N>
__device__ __forceinline__ double chan_total(const ScanArgs &a, const Chan &ch, int slot, uint32_t feat, bool low, int b0, int stride, const long long (&raw)[N]) {
    long long t = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) if (b0 + j * stride < a.B) t += raw[j];
    double v = (double)warp_sum(t) * ch.mul;
    if (low && !ch.cnt) {
        const unsigned long long *p = a.qlow + (((size_t)slot * a.SC + feat) * a.nq + ch.idx) * a.B;
        t = 0;
        for (int j = 0; j < N; ++j) if (b0 + j * stride < a.B) t += (long long)__ldg(p + b0 + j * stride);
        v += (double)warp_sum(t) * (ch.mul * a.low_unit);
    }
    return v;
}

// Sharded with peer access: sums the ranks' freshly built histograms for the feature slots this rank owns, by
// loads from the peers' memory past the caches, in rank order (so the result does not depend on timing).  One CTA
// per (build slot, owned feature); at the root level feature slot 0 is summed on every rank (it gives the root sums).
struct PeerReduceArgs {
    const double *peer_hcomp[EVB_MAX_PEERS];
    double *hsum;
    const LevelPlan *plan;
    int world, rank, F, CB, level;
    int K, elided; // elided: mse, every rank's hessian channels are exactly 2 x its weight channel -- they are not fetched
};
__global__ void __launch_bounds__(256) k_peer_reduce(PeerReduceArgs a) {
    const int Fown = (a.F - a.rank + a.world - 1) / a.world;
    const int per = Fown + 1; // last index of a slot: feature slot 0 (root level only)
    const int s = blockIdx.x / per, fi = blockIdx.x % per;
    if (s >= a.plan->nbuild) return;
    int f;
    if (fi < Fown) f = fi * a.world + a.rank;
    else { if (a.level != 1 || a.rank == 0) return; f = 0; }
    const size_t base = ((size_t)s * a.F + f) * a.CB;
    const int B = a.CB / (2 * a.K + 1);
    for (int idx = threadIdx.x; idx < a.CB; idx += blockDim.x) {
        const int c = idx / B;
        if (a.elided && c >= a.K && c < 2 * a.K) continue;
        double v = 0.0;
#pragma unroll 8
        for (int q = 0; q < a.world; ++q) v += __ldcv(a.peer_hcomp[q] + base + idx);
        a.hsum[base + idx] = v;
        if (a.elided && c == 2 * a.K) // h_k = 2w (src/loss.jl:52): doubling commutes with the rounding of the sum
            for (int k = 0; k < a.K; ++k) a.hsum[base + (size_t)(a.K + k) * B + (idx - c * B)] = 2.0 * v;
    }
}

// Scan of one (node, feature): applies the sibling subtraction (`subtract_hist!`, fit-utils.jl:321-332) to the
// staged histogram `sm` of the build node, stores the node's histogram if its children will need it, scans the
// bins (`_scan_node!`, fit-utils.jl:403-436) and records the best split of this feature.
template <int MAXCHK, bool OWN, bool OBL, bool K1, bool LOW>
__device__ __forceinline__ void scan_one(const ScanArgs &a, int n, bool sub, int f, uint32_t feat, int slot, double *s_sum, int lane, bool first_owned) {
    // K1: one output with gradient, hessian and weight channels (C = 3), known at compile time: the loops over the
    // outputs and the channel tests fold away
    const int C = K1 ? 3 : a.C, K = K1 ? 1 : a.K, B = a.B, F = a.F;
    const int m = 1 << (a.level - 1);
    const size_t FCB = (size_t)F * C * B;
    const double *__restrict__ hp = a.hist + (size_t)(n >> 1) * FCB;
    const bool keep = n < a.hist_nodes;
    double *__restrict__ hn = a.hist + (size_t)n * FCB;
    if (n == 1) {
        constexpr int NB = K1 ? 3 : 1; // channels whose loads are issued together
        for (int c0 = 0; c0 < C; c0 += NB) {
            Chan ch[NB];
            long long raw[NB][MAXCHK];
#pragma unroll
            for (int u = 0; u < NB; ++u) {
                ch[u] = chan_of(a, c0 + u, K, C);
                chan_load<MAXCHK>(a, ch[u], slot, f, feat, c0 + u, lane, 32, C, raw[u]);
            }
            double v[NB];
            if (a.qsum) {
#pragma unroll
                for (int u = 0; u < NB; ++u) v[u] = chan_total<MAXCHK>(a, ch[u], slot, feat, LOW, lane, 32, raw[u]);
            } else { // sharded: the bins of feature slot 0, in doubles
#pragma unroll
                for (int u = 0; u < NB; ++u) {
                    v[u] = 0.0;
#pragma unroll
                    for (int j = 0; j < MAXCHK; ++j) if (lane + 32 * j < B) v[u] += __longlong_as_double(raw[u][j]);
                    v[u] = warp_sum(v[u]);
                }
            }
            if (lane == 0) {
#pragma unroll
                for (int u = 0; u < NB; ++u) { s_sum[c0 + u] = v[u]; if (first_owned) a.nsum[(size_t)C + c0 + u] = v[u]; }
            }
        }
    } else {
        for (int c = lane; c < C; c += 32) s_sum[c] = a.nsum[(size_t)n * C + c];
    }
    __syncwarp();
    double gain_p = 0.0;
    const double w_p = s_sum[C - 1];
    if (!OWN) {
        for (int k = 0; k < K; ++k) gain_p += term_gh(s_sum[k], s_sum[K + k], w_p, a.lambda, a.L2); // node_gain, split.jl:58-66
    } else if (a.loss != EVB_MAE && a.loss != EVB_QUANTILE && a.loss != EVB_MULTIQUANTILE) {
        for (int k = 0; k < K; ++k) gain_p += term_cred(a.loss, s_sum[k], s_sum[K + k], w_p, a.L2);   // split.jl:70-78; mae: 0
    }

    // lane l holds the CH adjacent bins l * CH .. l * CH + CH - 1 (CH * 32 >= B): a running sum over the bins is a
    // running sum inside the lane plus ONE warp scan of the lanes' totals, whatever CH is
    constexpr int CH = MAXCHK;
    const int bin0 = lane * CH;
    const bool numeric = a.feattypes[feat] != 0;
    const int constraint = a.mono[feat];
    const int b_max = numeric ? B - 1 : B;
    const size_t fo = (size_t)f * C * B;
    const bool elide = a.elide_h != 0; // mse: every h entry is exactly twice the w entry (src/loss.jl:52), it is not read
    // entries of channel c in the lane's bins: the loads (`fetch`) run ahead of their use (`take`), which subtracts from the
    // parent's histogram and keeps the result for the children
    struct Raw { Chan ch; long long b[CH], low[LOW ? CH : 1]; double p[CH]; };
    auto fetch = [&](int c, Raw &r) {
        r.ch = chan_of(a, c, K, C);
        chan_load<CH>(a, r.ch, slot, f, feat, c, bin0, 1, C, r.b);
        if constexpr (LOW) chan_load_low<CH>(a, r.ch, slot, feat, bin0, 1, r.low);
        if (sub) {
#pragma unroll
            for (int j = 0; j < CH; ++j) r.p[j] = __ldg(hp + fo + (size_t)c * B + min(bin0 + j, B - 1));
        }
    };
    auto take = [&](int c, const Raw &r, double (&v)[CH]) {
#pragma unroll
        for (int j = 0; j < CH; ++j) v[j] = chan_value(a, r.ch, r.b[j]);
        if constexpr (LOW) chan_add_low<CH>(a, r.ch, r.low, v);
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int b = bin0 + j;
            if (sub) v[j] = r.p[j] - v[j];
            if (b >= B) v[j] = 0.0;
            if (keep && b < B) hn[fo + (size_t)c * B + b] = v[j];
        }
    };
    auto running = [&](double (&v)[CH]) { // inclusive running sum over the bins (numeric features only)
        if (!numeric) return;
#pragma unroll
        for (int j = 1; j < CH; ++j) v[j] += v[j - 1];
        const double incl = warp_incl_scan(v[CH - 1], lane);
        double before = __shfl_up_sync(FULL, incl, 1);
        if (lane == 0) before = 0.0;
#pragma unroll
        for (int j = 0; j < CH; ++j) v[j] += before;
    };
    double best_g = 0.0, best_h = 0.0, best_w = 0.0; // left sums of the lane's candidate (K1)
    double lg = a.gamma; // get_best_split starts at gamma and takes strict improvements (fit-utils.jl:444-450)
    int lb = 0x7fffffff;
    if (a.level < a.D) {
        double wl[CH], gacc[CH], g1[CH], h1[CH];
        unsigned okmask = 0xffu;
        Raw rw, rg, rh;
        fetch(C - 1, rw);
        fetch(0, rg);
        if (!elide) fetch(K, rh);
        take(C - 1, rw, wl);
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            gacc[j] = 0.0;
            const int b = bin0 + j;
            if (elide && keep && b < B)
                for (int k = 0; k < K; ++k) hn[fo + (size_t)(K + k) * B + b] = 2.0 * wl[j];
        }
        running(wl);
        for (int k = 0; k < K; ++k) {
            const double sg = s_sum[k], sh = s_sum[K + k];
            double gl[CH], hl[CH];
            take(k, rg, gl);
            if (!elide) take(K + k, rh, hl);
            if (!K1 && k + 1 < K) { // the next output's entries are on their way while this one is scanned
                fetch(k + 1, rg);
                if (!elide) fetch(K + k + 1, rh);
            }
            running(gl);
            if (!elide) running(hl);
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                if (elide) hl[j] = 2.0 * wl[j];
                if (K1) { g1[j] = gl[j]; h1[j] = hl[j]; }
                const double w_l = wl[j], w_r = w_p - w_l;
                if (!OWN) gacc[j] += terms_gh(gl[j], hl[j], w_l, sg - gl[j], sh - hl[j], w_r, a.lambda, a.L2);
                else gacc[j] += side_gain(a, gl[j], hl[j], w_l, sg, sh, w_p);
                if (k == 0 && constraint != 0) {
                    // pred_scalar on left / right sums (src/predict.jl:205-208, 235-238)
                    const double pl = OWN ? own_scalar(a, gl[j], w_l) : a.neb * gl[j] / fmax(DBL_EPSILON, hl[j] + a.lambda * w_l + a.L2);
                    const double pr = OWN ? own_scalar(a, sg - gl[j], w_r)
                                          : a.neb * (sg - gl[j]) / fmax(DBL_EPSILON, (sh - hl[j]) + a.lambda * w_r + a.L2);
                    const bool ok = (constraint == -1 && pl > pr) || (constraint == 1 && pl < pr);
                    if (!ok) okmask &= ~(1u << j);
                }
            }
        }
        // candidate of this lane: lowest bin among its strict maxima
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int b = bin0 + j;
            const double w_l = wl[j], w_r = w_p - w_l;
            double g = 0.0;
            const bool elig = b < b_max && w_l > a.min_weight && w_r > a.min_weight && ((okmask >> j) & 1u);
            if (elig) {
                g = gacc[j] - gain_p;
                if (g > lg) { lg = g; lb = b; if (K1) { best_g = g1[j]; best_h = h1[j]; best_w = wl[j]; } }
            }
            if (OBL && b < B) a.obl_gain[((size_t)(n - m) * F + f) * B + b] = g; // update_gains!, fit-utils.jl:457-463
        }
        const int mine = lb;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const double og = __shfl_xor_sync(FULL, lg, d);
            const int ob = __shfl_xor_sync(FULL, lb, d);
            if (og > lg || (og == lg && ob < lb)) { lg = og; lb = ob; }
        }
        if (K1 && mine == lb && lb != 0x7fffffff) { // a bin is one lane's
            double *l = a.fbest_left + ((size_t)(n - m) * F + f) * 3;
            l[0] = best_g; l[1] = best_h; l[2] = best_w;
        }
    }
    __syncwarp();
    if (lane == 0) {
        a.fbest_gain[(size_t)(n - m) * F + f] = lg;
        a.fbest_bin[(size_t)(n - m) * F + f] = lb == 0x7fffffff ? -1 : lb;
    }
    __syncwarp();
}

// Oblivious trees, stage 1b: one thread per candidate (feature slot, bin) adds the gains of the level's nodes in
// ascending node order and drops the candidate if any node holds no positive gain for it (src/fit.jl:196-211; at
// the root level the reference applies no mask, which changes nothing for gamma >= 0).  Sharded with peer access,
// every rank does this for its own feature slots; k_scan_node then publishes the rank's best split with each
// node's left sums and k_scan_final takes the best of the ranks (the same for every node: the gains are level totals).
__global__ void __launch_bounds__(128) k_obl_sum(ScanArgs a) {
    const int m = 1 << (a.level - 1);
    const size_t FB = (size_t)a.F * a.B;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= FB) return;
    double tot = 0.0;
    // sharded with peer access: only the feature slots this rank scans hold gains; the others never win here
    bool ok = (int)(e / a.B) % a.world == a.rank;
    for (int i = 0; ok && i < m; ++i) {
        const double g = a.obl_gain[(size_t)i * FB + e];
        tot += g;
        ok = ok && g > 0.0;
    }
    a.obl_gain[(size_t)m * FB + e] = ok ? tot : 0.0;
}

// Oblivious trees, stage 1c: first maximum of the level totals in (feature slot, bin) order (`findmax`,
// src/fit.jl:213-217); it is the level's split if it exceeds gamma.  One CTA.
__global__ void __launch_bounds__(1024) k_obl_pick(ScanArgs a) {
    __shared__ double s_g[32];
    __shared__ int s_e[32];
    const int m = 1 << (a.level - 1);
    const int FB = a.F * a.B;
    const double *tot = a.obl_gain + (size_t)m * FB;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double bg = a.gamma;
    int be = 0x7fffffff;
    for (int e = threadIdx.x; e < FB; e += blockDim.x) {
        const double g = tot[e];
        if (g > bg) { bg = g; be = e; }
    }
    auto red = [&]() {
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const double og = __shfl_xor_sync(FULL, bg, d);
            const int oe = __shfl_xor_sync(FULL, be, d);
            if (oe != 0x7fffffff && (og > bg || (og == bg && oe < be))) { bg = og; be = oe; }
        }
    };
    red();
    if (lane == 0) { s_g[wid] = bg; s_e[wid] = be; }
    __syncthreads();
    if (wid == 0) {
        bg = s_g[lane]; be = s_e[lane];
        red();
        if (lane == 0) { a.obl_best[0] = bg; a.obl_best[1] = be == 0x7fffffff ? -1.0 : (double)be; }
    }
}

// Writes everything that follows from the split decision of node n: child sums, tree arrays, leaf values
// (`_child_sums!` result, src/fit.jl:90-98, 120-121, 74-82, 131-135).  One warp; s_left holds the left sums.
__device__ __forceinline__ void apply_split(const ScanArgs &a, int n, bool has, double gain, int slot, int bin, const double *s_sum,
                                            double *s_left, double *s_right, int lane) {
    const int C = a.C, K = a.K;
    if (has) {
        const uint32_t feat = a.js0[slot];
        const bool numeric = a.feattypes[feat] != 0;
        for (int c = lane; c < C; c += 32) s_right[c] = s_sum[c] - s_left[c];
        __syncwarp();
        const int nl = n << 1, nr = nl + 1;
        for (int c = lane; c < C; c += 32) {
            a.nsum[(size_t)nl * C + c] = s_left[c];
            a.nsum[(size_t)nr * C + c] = s_right[c];
        }
        if (lane == 0) {
            a.t_w[n - 1] = (float)s_sum[C - 1];
            a.t_gain[n - 1] = (float)gain;
            a.t_bin[n - 1] = (uint8_t)(bin + 1);
            a.t_feat[n - 1] = (int32_t)feat + 1;
            a.t_split[n - 1] = 1;
            a.t_packed[n - 1] = feat | ((uint32_t)(bin + 1) << 16) | (1u << 24) | ((numeric ? 1u : 0u) << 25);
        }
        if (a.level + 1 == a.D) {
            // children sit at max depth: they are leaves (src/fit.jl:74-82)
            for (int k = lane; k < K; k += 32) {
                a.t_pred[(size_t)(nl - 1) * K + k] = leaf_value(a, s_left, k);
                a.t_pred[(size_t)(nr - 1) * K + k] = leaf_value(a, s_right, k);
            }
            if (lane == 0) { a.t_w[nl - 1] = (float)s_left[C - 1]; a.t_w[nr - 1] = (float)s_right[C - 1]; }
        }
    } else {
        if (lane == 0) a.t_w[n - 1] = (float)s_sum[C - 1];
        for (int k = lane; k < K; k += 32) a.t_pred[(size_t)(n - 1) * K + k] = leaf_value(a, s_sum, k);
    }
}

// Stage 2: one warp per node: first strict maximum over the (owned) features in ascending feature order and the
// left-child sums of the winner (`_child_sums!`, fit-utils.jl:472-486).  Single GPU: the split is applied at once.
// Sharded with peer access: the rank's candidate is written into every rank's candidate table instead.
template <int MAXCHK, bool K1>
__device__ __forceinline__ void node_select(const ScanArgs &a, int n, double *s_sum, double *s_left, double *s_right, int lane) {
    const int C = K1 ? 3 : a.C, K = K1 ? 1 : a.K, B = a.B, F = a.F; // K1: one output, channels g, h, w known at compile time
    const int m = 1 << (a.level - 1), i = n - m;
    const int Fown = (F - a.rank + a.world - 1) / a.world;
    const int slot_n = a.bslot[n];
    const bool sub = a.kind[n] == EVB_KIND_SUB;
    const bool low = a.world == 1 && slot_low(a, slot_n);
    double fg[4];
    int fb[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int fi = lane + 32 * u;
        fb[u] = -1; fg[u] = 0.0;
        if (fi < Fown && !a.obl_gain) { // written by other warps of this launch when the scan is fused: past L1
            const int f = fi * a.world + a.rank;
            fg[u] = __ldcg(a.fbest_gain + (size_t)i * F + f);
            fb[u] = __ldcg(a.fbest_bin + (size_t)i * F + f);
        }
    }
    for (int c = lane; c < C; c += 32) s_sum[c] = __ldcg(a.nsum + (size_t)n * C + c);
    const size_t FCB = (size_t)F * C * B;
    const double *hp = a.hist + (size_t)(n >> 1) * FCB;
    const double *hn = a.hist + (size_t)n * FCB;
    __syncwarp();

    double bg = a.gamma;
    int bs = 0x7fffffff, bb = -1;
    if (a.obl_gain) { // oblivious: every node of the level takes the split k_obl_pick chose (src/fit.jl:213-225)
        const double e = a.obl_best[1];
        if (e >= 0.0) { bg = a.obl_best[0]; bs = (int)e / B; bb = (int)e % B; }
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (fb[u] >= 0 && fg[u] > bg) { bg = fg[u]; bs = (lane + 32 * u) * a.world + a.rank; bb = fb[u]; }
        for (int fi = lane + 128; fi < Fown; fi += 32) {
            const int f = fi * a.world + a.rank;
            const double g = __ldcg(a.fbest_gain + (size_t)i * F + f);
            const int b = __ldcg(a.fbest_bin + (size_t)i * F + f);
            if (b >= 0 && g > bg) { bg = g; bs = f; bb = b; }
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const double og = __shfl_xor_sync(FULL, bg, d);
            const int os = __shfl_xor_sync(FULL, bs, d), ob = __shfl_xor_sync(FULL, bb, d);
            if (os != 0x7fffffff && (og > bg || (og == bg && os < bs))) { bg = og; bs = os; bb = ob; }
        }
    }
    const bool has = bs != 0x7fffffff;
    if (has && K1 && !a.obl_gain) { // kept by the feature's scan
        if (lane < 3) s_left[lane] = __ldcg(a.fbest_left + ((size_t)i * F + bs) * 3 + lane);
        __syncwarp();
    } else if (has) {
        const uint32_t feat = a.js0[bs];
        const bool numeric = a.feattypes[feat] != 0;
        const size_t fo = (size_t)bs * C * B;
        // channels side by side: their loads and their sums over the lanes overlap
        constexpr int NC = MAXCHK <= 2 ? 6 : 2;
        for (int c0 = 0; c0 < C; c0 += NC) {
            long long rb[NC][MAXCHK];
            double rp[NC][MAXCHK], v[NC];
            Chan ch[NC];
#pragma unroll
            for (int u = 0; u < NC; ++u) {
                const int c = min(c0 + u, C - 1);
                ch[u] = chan_of(a, c, K, C);
                if (a.world > 1) { // sharded: the summed histogram of every scanned node is retained locally for the owned features
#pragma unroll
                    for (int j = 0; j < MAXCHK; ++j) rp[u][j] = hn[fo + (size_t)c * B + min(lane + 32 * j, B - 1)];
                } else {
                    chan_load<MAXCHK>(a, ch[u], slot_n, bs, feat, c, lane, 32, C, rb[u]);
                    if (sub) {
#pragma unroll
                        for (int j = 0; j < MAXCHK; ++j) rp[u][j] = hp[fo + (size_t)c * B + min(lane + 32 * j, B - 1)];
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < NC; ++u) {
                v[u] = 0.0;
                double built[MAXCHK];
                if (a.world == 1) {
#pragma unroll
                    for (int j = 0; j < MAXCHK; ++j) built[j] = chan_value(a, ch[u], rb[u][j]);
                    if (low) {
                        long long raw[MAXCHK];
                        chan_load_low<MAXCHK>(a, ch[u], slot_n, feat, lane, 32, raw);
                        chan_add_low<MAXCHK>(a, ch[u], raw, built);
                    }
                }
#pragma unroll
                for (int j = 0; j < MAXCHK; ++j) {
                    const int b = lane + 32 * j;
                    double e = rp[u][j];
                    if (a.world == 1) e = sub ? rp[u][j] - built[j] : built[j];
                    if (b < B && (numeric ? b <= bb : b == bb)) v[u] += e;
                }
            }
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) {
#pragma unroll
                for (int u = 0; u < NC; ++u) v[u] += __shfl_xor_sync(FULL, v[u], d);
            }
            if (lane == 0) {
#pragma unroll
                for (int u = 0; u < NC; ++u) if (c0 + u < C) s_left[c0 + u] = v[u];
            }
        }
        __syncwarp();
    }
    if (a.world == 1) {
        apply_split(a, n, has, bg, bs, bb, s_sum, s_left, s_right, lane);
        if (has && lane == 0) { const int s0 = a.seg_start[n]; a.cur_l[n] = s0; a.cur_r[n] = s0 + a.seg_cnt[n]; }
        return;
    }
    const int RC = 3 + C;
    for (int q = 0; q < a.world; ++q) {
        double *rec = a.peer_cand[q] + ((size_t)i * a.world + a.rank) * RC;
        if (lane == 0) { rec[0] = bg; rec[1] = has ? (double)bs : -1.0; rec[2] = (double)bb; }
        if (has) for (int c = lane; c < C; c += 32) rec[3 + c] = s_left[c];
    }
}
// The same on one GPU where the scans keep their candidates' left sums, by the warp that scanned the node's last feature: the node
// sums are in s_sum already, gains and bins are requested at once (K1: the left sums of up to 32 features too) -- one trip to L2
// and one reduction, for several outputs a second trip for the winner's sums.
template <bool K1>
__device__ __forceinline__ void node_decide(const ScanArgs &a, int n, const double *s_sum, double *s_left, double *s_right, int lane) {
    const int F = a.F, C = K1 ? 3 : a.C, i = n - (1 << (a.level - 1));
    const double *gains = a.fbest_gain + (size_t)i * F;
    const int32_t *bins = a.fbest_bin + (size_t)i * F;
    const double *lefts = a.fbest_left + (size_t)i * F * C;
    const int s0 = a.seg_start[n], c0 = a.seg_cnt[n];
    double l0 = 0.0, l1 = 0.0, l2 = 0.0;
    if (K1 && lane < F) { l0 = __ldcg(lefts + lane * 3); l1 = __ldcg(lefts + lane * 3 + 1); l2 = __ldcg(lefts + lane * 3 + 2); }
    double bg = a.gamma;
    int bs = 0x7fffffff, bb = -1;
#pragma unroll 4
    for (int f = lane; f < F; f += 32) {
        const double g = __ldcg(gains + f);
        const int b = __ldcg(bins + f);
        if (b >= 0 && g > bg) { bg = g; bs = f; bb = b; }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const double og = __shfl_xor_sync(FULL, bg, d);
        const int os = __shfl_xor_sync(FULL, bs, d), ob = __shfl_xor_sync(FULL, bb, d);
        if (os != 0x7fffffff && (og > bg || (og == bg && os < bs))) { bg = og; bs = os; bb = ob; }
    }
    const bool has = bs != 0x7fffffff;
    if (has) {
        if (!K1 || bs >= 32) { if (lane < C) s_left[lane] = __ldcg(lefts + (size_t)bs * C + lane); } // C <= 2 * EVB_MULTI_K + 1 < 32
        else if (lane == bs) { s_left[0] = l0; s_left[1] = l1; s_left[2] = l2; }
        if (lane == 0) { a.cur_l[n] = s0; a.cur_r[n] = s0 + c0; }
        __syncwarp();
    }
    apply_split(a, n, has, bg, bs, bb, s_sum, s_left, s_right, lane);
}

template <bool K1>
__global__ void __launch_bounds__(256) k_scan_node(ScanArgs a) {
    __shared__ double s_sum[8][72], s_left[8][72], s_right[8][72];
    const int wid = threadIdx.x >> 5, m = 1 << (a.level - 1), i = blockIdx.x * 8 + wid;
    if (i >= m || a.kind[m + i] == EVB_KIND_NONE) return;
    node_select<8, K1>(a, m + i, s_sum[wid], s_left[wid], s_right[wid], threadIdx.x & 31);
}

// Stage 1: one warp per (node, owned feature slot), lanes over bins.  The nodes of a level come in pairs sharing a
// build slot: the build node reads the slot's histogram, its sibling subtracts it from the parent's.  Warps are
// independent, so even the root level (one node) spreads over many SMs.
// OWN: the loss brings its own split gain (mae, credibility); OBL: oblivious trees, the gain of every candidate is
// stored as well; LOW: histograms may have a second set of sums (ScanArgs::qlow).  The default instance carries none of that code.
// Registers: with both sets of sums the loads of three channels are in flight twice, and a compiler that is short of registers waits
// for them one after the other.  ms of scans per tree with 64 and 80 (64 bins): 3M x 20 poisson 0.087 and 0.078, 60k x 77 0.074 and 0.072;
// with 128 and 170, in CTAs of half the size: 1M x 40 gamma, 128 bins 0.097 and 0.087, 2M x 10 logloss, 255 bins 0.141 and 0.126.
constexpr int scan_threads(int CH, bool K1, bool LOW) { return K1 && LOW && CH > 2 ? 128 : 256; }
template <int MAXCHK, bool OWN, bool OBL, bool K1, bool LOW>
__global__ void __launch_bounds__(scan_threads(MAXCHK, K1, LOW), MAXCHK <= 2 ? (K1 && !LOW ? 4 : 3) : K1 && LOW ? 3 : 2) k_scan_feat(ScanArgs a) {
    constexpr int NCH = K1 ? 3 : 72;
    __shared__ double s_sum_all[8][NCH], s_left_all[8][NCH], s_right_all[8][NCH];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int F = a.F;
    const int Fown = (F - a.rank + a.world - 1) / a.world;
    if (blockIdx.x == 0 && a.level == 1 && threadIdx.x < a.ng) a.gmax[threadIdx.x] = 0u;
    if (Fown <= 0) return;
    long long gw = (long long)blockIdx.x * wpb + wid;
    const int which = a.level > 1 ? (int)(gw & 1) : 0;
    if (a.level > 1) gw >>= 1;
    const int s = (int)(gw / Fown), fi = (int)(gw % Fown);
    const int f = fi * a.world + a.rank;
    const int nbuild = load_now(&a.plan->nbuild), nb = load_now(a.slot_node + min(s, a.slots - 1)), feat = load_now(reinterpret_cast<const int32_t *>(a.js0) + f);
    const bool low = LOW && slot_low(a, min(s, a.slots - 1));
    if (s >= nbuild) return;
    const int n = which ? nb ^ 1 : nb;
    // two bodies: a test between the loads of the channels costs a level 0.5 us
    if (LOW && low) scan_one<MAXCHK, OWN, OBL, K1, true>(a, n, which != 0, f, (uint32_t)feat, s, s_sum_all[wid], lane, fi == 0);
    else scan_one<MAXCHK, OWN, OBL, K1, false>(a, n, which != 0, f, (uint32_t)feat, s, s_sum_all[wid], lane, fi == 0);
    if (!OBL && a.ticket) {
        // the warp that scans the node's last feature decides the node: no launch of its own for that
        unsigned last = 0;
        if (lane == 0) last = arrive(a.ticket + n) == (unsigned)(F - 1);
        if (!__shfl_sync(FULL, last, 0)) return;
        __syncwarp();
        if constexpr (K1) node_decide<true>(a, n, s_sum_all[wid], s_left_all[wid], s_right_all[wid], lane);
        else node_select<MAXCHK, false>(a, n, s_sum_all[wid], s_left_all[wid], s_right_all[wid], lane);
    }
}

// Stages 1 and 2 for 2 to EVB_MULTI_K outputs with gradients and hessians on one GPU: one CTA per (node, feature), one warp per
// output.  The gain is a sum over the outputs, so the warps load, sum and rate their outputs side by side and warp 0 adds the
// gains up in output order; a warp still holds its running sums when the best bin is known and leaves the left sums for the
// decision.  One warp for all outputs is a chain of 2 K + 1 channels and pairs of divisions, and the decision had to sum the
// winner's bins again: a level of the scan took 42 us at 28 features and five classes, 18 now (2 outputs, 50 features: 23 and 14).
template <int CH>
__global__ void __launch_bounds__(32 * EVB_MULTI_K, CH <= 2 ? 3 : 2) k_scan_multi(ScanArgs a) {
    __shared__ double s_gain[EVB_MULTI_K][32 * CH]; // [output][j * 32 + lane] of bin lane * CH + j
    __shared__ double s_gp[EVB_MULTI_K], s_sum[2 * EVB_MULTI_K + 1], s_left[2 * EVB_MULTI_K + 1], s_right[2 * EVB_MULTI_K + 1];
    __shared__ int s_bin, s_last;
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int C = a.C, K = a.K, B = a.B, F = a.F;
    if (blockIdx.x == 0 && a.level == 1 && threadIdx.x < a.ng) a.gmax[threadIdx.x] = 0u;
    int gw = blockIdx.x;
    const int which = a.level > 1 ? gw & 1 : 0;
    if (a.level > 1) gw >>= 1;
    const int s = gw / F, f = gw % F;
    const int nbuild = load_now(&a.plan->nbuild), nb = load_now(a.slot_node + min(s, a.slots - 1));
    const uint32_t feat = (uint32_t)load_now(reinterpret_cast<const int32_t *>(a.js0) + f);
    const bool low = slot_low(a, min(s, a.slots - 1));
    if (s >= nbuild) return;
    const int n = which ? nb ^ 1 : nb, i = n - (1 << (a.level - 1));
    const bool numeric = a.feattypes[feat] != 0, sub = which != 0, keep = n < a.hist_nodes, elide = a.elide_h != 0;
    const int constraint = k == 0 ? a.mono[feat] : 0;
    const int bin0 = lane * CH, b_max = numeric ? B - 1 : B;
    const size_t FCB = (size_t)F * C * B, fo = (size_t)f * C * B;
    const double *__restrict__ hp = a.hist + (size_t)(n >> 1) * FCB + fo;
    double *__restrict__ hn = a.hist + (size_t)n * FCB + fo;
    // own gradient and hessian channels and the weights, which every warp needs
    const Chan cg = chan_of(a, k, K, C), chs = chan_of(a, K + k, K, C), cw = chan_of(a, C - 1, K, C);
    double gl[CH], hl[CH], wl[CH];
    double sg, sh, w_p;
    {
        long long rg[CH], rh[CH], rw[CH];
        chan_load<CH>(a, cw, s, f, feat, C - 1, bin0, 1, C, rw);
        chan_load<CH>(a, cg, s, f, feat, k, bin0, 1, C, rg);
        if (!elide) chan_load<CH>(a, chs, s, f, feat, K + k, bin0, 1, C, rh);
        double pg[CH], ph[CH], pw[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int b = min(bin0 + j, B - 1);
            pw[j] = sub ? __ldg(hp + (size_t)(C - 1) * B + b) : 0.0;
            pg[j] = sub ? __ldg(hp + (size_t)k * B + b) : 0.0;
            ph[j] = sub && !elide ? __ldg(hp + (size_t)(K + k) * B + b) : 0.0;
        }
        if (n > 1) { sg = a.nsum[(size_t)n * C + k]; sh = a.nsum[(size_t)n * C + K + k]; w_p = a.nsum[(size_t)n * C + C - 1]; }
        else {
            sg = chan_total<CH>(a, cg, s, feat, low, bin0, 1, rg);
            w_p = chan_total<CH>(a, cw, s, feat, low, bin0, 1, rw);
            sh = elide ? 2.0 * w_p : chan_total<CH>(a, chs, s, feat, low, bin0, 1, rh);
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            wl[j] = chan_value(a, cw, rw[j]);
            gl[j] = chan_value(a, cg, rg[j]);
            hl[j] = elide ? 0.0 : chan_value(a, chs, rh[j]);
        }
        if (low) {
            long long lw[CH], lg[CH], lh[CH];
            chan_load_low<CH>(a, cw, s, feat, bin0, 1, lw);
            chan_load_low<CH>(a, cg, s, feat, bin0, 1, lg);
            chan_load_low<CH>(a, chs, s, feat, bin0, 1, lh);
            chan_add_low<CH>(a, cw, lw, wl);
            chan_add_low<CH>(a, cg, lg, gl);
            if (!elide) chan_add_low<CH>(a, chs, lh, hl);
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int b = bin0 + j;
            if (sub) { wl[j] = pw[j] - wl[j]; gl[j] = pg[j] - gl[j]; }
            if (elide) hl[j] = 2.0 * wl[j];
            else if (sub) hl[j] = ph[j] - hl[j];
            if (b >= B) { wl[j] = 0.0; gl[j] = 0.0; hl[j] = 0.0; }
            else if (keep) {
                hn[(size_t)k * B + b] = gl[j];
                hn[(size_t)(K + k) * B + b] = hl[j];
                if (k == 0) hn[(size_t)(C - 1) * B + b] = wl[j];
            }
        }
    }
    if (n == 1 && f == 0 && lane == 0) { a.nsum[C + k] = sg; a.nsum[C + K + k] = sh; if (k == 0) a.nsum[2 * C - 1] = w_p; }
    if (lane == 0) {
        s_sum[k] = sg; s_sum[K + k] = sh;
        if (k == 0) s_sum[C - 1] = w_p;
        s_gp[k] = term_gh(sg, sh, w_p, a.lambda, a.L2);
    }
    if (numeric) { // running sums over the bins: inside the lane, then over the lanes' totals
#pragma unroll
        for (int j = 1; j < CH; ++j) { gl[j] += gl[j - 1]; hl[j] += hl[j - 1]; wl[j] += wl[j - 1]; }
        double ig = gl[CH - 1], ih = hl[CH - 1], iw = wl[CH - 1];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double tg = __shfl_up_sync(FULL, ig, d), th = __shfl_up_sync(FULL, ih, d), tw = __shfl_up_sync(FULL, iw, d);
            if (lane >= d) { ig += tg; ih += th; iw += tw; }
        }
        ig = __shfl_up_sync(FULL, ig, 1); ih = __shfl_up_sync(FULL, ih, 1); iw = __shfl_up_sync(FULL, iw, 1);
        if (lane > 0) {
#pragma unroll
            for (int j = 0; j < CH; ++j) { gl[j] += ig; hl[j] += ih; wl[j] += iw; }
        }
    }
#pragma unroll
    for (int j = 0; j < CH; ++j) {
        const double w_l = wl[j], w_r = w_p - w_l;
        double g = terms_gh(gl[j], hl[j], w_l, sg - gl[j], sh - hl[j], w_r, a.lambda, a.L2);
        bool ok = bin0 + j < b_max && w_l > a.min_weight && w_r > a.min_weight;
        if (constraint != 0) { // pred_scalar on left / right sums (src/predict.jl:205-208, 235-238)
            const double pl = a.neb * gl[j] / fmax(DBL_EPSILON, hl[j] + a.lambda * w_l + a.L2);
            const double pr = a.neb * (sg - gl[j]) / fmax(DBL_EPSILON, (sh - hl[j]) + a.lambda * w_r + a.L2);
            ok = ok && ((constraint == -1 && pl > pr) || (constraint == 1 && pl < pr));
        }
        s_gain[k][j * 32 + lane] = k > 0 || ok ? g : -DBL_MAX; // not a candidate: no sum exceeds gamma (gains are not negative)
    }
    __syncthreads();
    if (k == 0) {
        double gain_p = s_gp[0], lg = a.gamma; // get_best_split starts at gamma and takes strict improvements (fit-utils.jl:444-450)
        int lb = 0x7fffffff;
        for (int q = 1; q < K; ++q) gain_p += s_gp[q];
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const double first = s_gain[0][j * 32 + lane];
            double g = first;
            for (int q = 1; q < K; ++q) g += s_gain[q][j * 32 + lane];
            g -= gain_p;
            if (first != -DBL_MAX && g > lg && a.level < a.D) { lg = g; lb = bin0 + j; }
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            const double og = __shfl_xor_sync(FULL, lg, d);
            const int ob = __shfl_xor_sync(FULL, lb, d);
            if (og > lg || (og == lg && ob < lb)) { lg = og; lb = ob; }
        }
        if (lane == 0) {
            a.fbest_gain[(size_t)i * F + f] = lg;
            a.fbest_bin[(size_t)i * F + f] = lb == 0x7fffffff ? -1 : lb;
            s_bin = lb;
        }
    }
    __syncthreads();
    const int bin = s_bin;
    if (bin != 0x7fffffff) {
        double *l = a.fbest_left + ((size_t)i * F + f) * C;
#pragma unroll
        for (int j = 0; j < CH; ++j)
            if (bin0 + j == bin) { l[k] = gl[j]; l[K + k] = hl[j]; if (k == 0) l[C - 1] = wl[j]; }
    }
    __syncthreads();
    if (k != 0) return;
    if (lane == 0) s_last = arrive(a.ticket + n) == (unsigned)(F - 1);
    __syncwarp();
    if (!s_last) return;
    node_decide<false>(a, n, s_sum, s_left, s_right, lane);
}

// Stage 3 (sharded with peer access only): every rank picks, for every node, the best of the ranks' candidates
// (ties: lowest feature slot, as in the single-GPU order) and applies it.  All ranks read identical tables.
__global__ void __launch_bounds__(256) k_scan_final(ScanArgs a) {
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int C = a.C;
    const int m = 1 << (a.level - 1);
    const int i = blockIdx.x * (blockDim.x >> 5) + wid;
    __shared__ double s_sum_all[8][72], s_left_all[8][72], s_right_all[8][72];
    double *s_sum = s_sum_all[wid], *s_left = s_left_all[wid], *s_right = s_right_all[wid];
    if (i >= m) return;
    const int n = m + i;
    if (a.kind[n] == EVB_KIND_NONE) return;
    for (int c = lane; c < C; c += 32) s_sum[c] = a.nsum[(size_t)n * C + c];
    const int RC = 3 + C;
    double bg = a.gamma;
    int bs = 0x7fffffff, bb = -1, bq = -1;
    if (lane < a.world) {
        const double *rec = a.cand_local + ((size_t)i * a.world + lane) * RC;
        const double g = __ldcv(rec), sl = __ldcv(rec + 1), bn = __ldcv(rec + 2);
        if (sl >= 0.0 && g > bg) { bg = g; bs = (int)sl; bb = (int)bn; bq = lane; }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const double og = __shfl_xor_sync(FULL, bg, d);
        const int os = __shfl_xor_sync(FULL, bs, d), ob = __shfl_xor_sync(FULL, bb, d), oq = __shfl_xor_sync(FULL, bq, d);
        if (os != 0x7fffffff && (og > bg || (og == bg && os < bs))) { bg = og; bs = os; bb = ob; bq = oq; }
    }
    const bool has = bs != 0x7fffffff;
    if (has) {
        const double *rec = a.cand_local + ((size_t)i * a.world + bq) * RC;
        for (int c = lane; c < C; c += 32) s_left[c] = __ldcv(rec + 3 + c);
    }
    __syncwarp();
    apply_split(a, n, has, bg, bs, bb, s_sum, s_left, s_right, lane);
    if (has && lane == 0) { const int s0 = a.seg_start[n]; a.cur_l[n] = s0; a.cur_r[n] = s0 + a.seg_cnt[n]; }
}

// Cross-GPU barrier for the peer-access path: every rank writes the sequence number into its slot of every
// rank's flag array and waits (bounded, ~2 s) until all slots of its own array have reached it.
struct BarrierArgs {
    int *peer_flags[EVB_MAX_PEERS];
    int *flags_local;
    int *err;
    int world, rank;
    int *seq_dev; // barriers passed so far: kept on the device so that a replayed CUDA graph keeps counting
    unsigned max_polls; // polls of ~100 ns before the wait gives up with EVB_DERR_PEER (20 M: about two seconds)
};
__global__ void k_peer_barrier(BarrierArgs a) {
    const int t = threadIdx.x;
    int seq = 0;
    if (t == 0) { seq = *a.seq_dev + 1; *a.seq_dev = seq; } // one warp, launched alone on the stream: no race
    seq = __shfl_sync(FULL, seq, 0);
    if (t >= a.world) return;
    __threadfence_system();
    *(volatile int *)(a.peer_flags[t] + a.rank) = seq;
    __threadfence_system();
    volatile int *mine = a.flags_local + t;
    for (unsigned it = 0; it < a.max_polls; ++it) {
        if (*mine - seq >= 0) { __threadfence_system(); return; }
        if ((it & 1023u) == 1023u && *(volatile int *)a.err != 0) return;
        __nanosleep(100);
    }
    atomicCAS(a.err, 0, EVB_DERR_PEER);
}

// ------------------------------------------------------------------------------------------ partition
struct PartArgs {
    const uint8_t *xC; // feature-major bins [nfeats][n]: the rows of a node ascend, so its reads of one feature are
                       // as dense as the node is (whole sectors near the root, one sector per row deep down)
    long long n;
    const uint32_t *rows_in;
    uint32_t *rows_out;
    const uint8_t *t_split;
    const uint32_t *t_packed;
    int32_t *seg_start, *seg_cnt, *bslot, *cum, *slot_node, *rbase;
    int32_t *cur_l, *cur_r;     // next free place for left rows (upwards) / past the last free one for right rows (downwards)
    // sibling pairs of the level: {first child's id (the root alone at level 1), rows of the pairs before, rows up to the second
    // child, position -> place in the row list}; the entry after the last one holds the sum of all rows
    const int4 *pl;
    int4 *pl_next;
    uint8_t *kind;
    LevelPlan *plan;
    uint32_t *done;             // CTAs that have finished; the last one plans the next level
    const double *nsum; // node sums [id][C]; channel C-1 is the sum of weights
    unsigned long long *hsum;   // accumulators of the level's build slots, cleared here (the scan has read them)
    unsigned long long *hlow;
    const uint32_t *low_any;
    uint32_t *hcnt;
    size_t acc_sums, acc_cnts;  // words per build slot
    int C, by_weight;   // by_weight: sharded run, pick the build child by weight sum instead of row count
    int level, D;
};

// Children segments / counts, build-or-subtract choice (src/fit.jl:123-129: the child with fewer rows is built, ties build
// the left child), build slots and the histogram plan of the next level.  One CTA of 256 threads; a level of at most 32
// nodes is one warp's work (no barriers: 2.1 -> 1 us).
template <bool WARP>
__device__ __forceinline__ void plan_level(const PartArgs &a, int *sm) {
    const int lo = 1 << (a.level - 1), m = lo;
    const bool scan_children = a.level + 1 < a.D;
    const int step = WARP ? 32 : (int)blockDim.x;
    auto excl = [&](int v, int &total) -> int {
        if constexpr (WARP) {
            const int incl = warp_incl_scan_i(v, threadIdx.x);
            total = __shfl_sync(FULL, incl, 31);
            return incl - v;
        } else {
            return block_excl_scan(v, sm, &total);
        }
    };
    int carry_slot = 0, carry_rows = 0, carry_all = 0;
    for (int base = 0; base < m; base += step) {
        const int i = base + threadIdx.x;
        const int n = lo + i;
        int sp = 0, cnt_build = 0, cnt_all = 0, build_child = 0;
        const int nq = min(n, 2 * m - 1); // all loads at once, needed or not
        const int split = a.t_split[nq - 1], s0 = a.seg_start[nq], c0 = a.seg_cnt[nq], nl = __ldcg(a.cur_l + nq) - s0;
        if (i < m && split) {
            sp = 1;
            const int L = n << 1, Rn = L + 1;
            a.seg_start[L] = s0; a.seg_cnt[L] = nl;
            a.seg_start[Rn] = s0 + nl; a.seg_cnt[Rn] = c0 - nl;
            cnt_all = c0;
            if (scan_children) {
                // With rows sharded over GPUs the global row counts would cost one more collective per level, so there the
                // child with the smaller weight sum is built: every rank knows the sums from the split scan, and with unit
                // weights it is the same rule.
                const bool build_left = a.by_weight ? a.nsum[(size_t)Rn * a.C + a.C - 1] >= a.nsum[(size_t)L * a.C + a.C - 1] : c0 - nl >= nl;
                a.kind[L] = build_left ? EVB_KIND_BUILD : EVB_KIND_SUB;
                a.kind[Rn] = build_left ? EVB_KIND_SUB : EVB_KIND_BUILD;
                build_child = build_left ? L : Rn;
                cnt_build = build_left ? nl : c0 - nl;
            }
        }
        int tot_s, tot_r, tot_a;
        const int slot = carry_slot + excl(sp, tot_s), cpre = carry_rows + excl(cnt_build, tot_r), apre = carry_all + excl(cnt_all, tot_a);
        if (sp && scan_children) {
            a.bslot[n << 1] = slot; a.bslot[(n << 1) + 1] = slot;
            a.slot_node[slot] = build_child;
            a.cum[slot] = cpre;
            a.rbase[slot] = s0 - cpre + (build_child & 1 ? nl : 0);
            a.pl_next[slot] = make_int4(n << 1, apre, apre + nl, s0 - apre);
        }
        carry_slot += tot_s; carry_rows += tot_r; carry_all += tot_a;
    }
    if (threadIdx.x == 0 && scan_children) {
        a.cum[carry_slot] = carry_rows;
        a.pl_next[carry_slot] = make_int4(0, carry_all, 0, 0);
        a.plan[a.level + 1].nbuild = carry_slot;
        a.plan[a.level + 1].npl = carry_slot;
        a.plan[a.level + 1].total = carry_all;
        a.plan[a.level + 1].R = carry_rows;
    }
}

// Stable within a chunk, chunks in any order: left rows fill a node's segment from its start, right rows from its end, and a
// chunk reserves its places with one atomic per side.  Histogram sums are integers, so the order of the rows of a node means
// nothing to them; what it is good for is the density of the reads, which a chunk of adjacent rows keeps.  One pass over the
// row list instead of two, no list of work items, no bit vectors, and the CTA that finishes last plans the next level: three
// launches and the prefix sums between them less per level.
// A chunk is NI rows per thread.  A chunk inside one node (nearly all of them while nodes are large) takes the block-wide
// path, else every warp looks its rows' nodes up and the lanes of the same node and side share an atomic.
// Every CTA takes a range of adjacent chunks: the node of the next one is known without a search unless it ends, and its row ids are
// on their way while this one's bins arrive and its places are reserved.  What bounds a chunk is that chain of trips to L2, so
// CTAs matter more than rows per thread: six CTAs of four rows a thread 0.640 ms per tree at 10M x 100, depth 11 (5M x 50 gaussian
// 0.153), four of eight 0.69 (0.163), eight of four (registers spill) 0.67 (0.167); chunks dealt out in turn and searched for
// one by one, four of eight, took 0.727 (0.192).
constexpr int PART_WARPS = EVB_PART_THREADS / 32, PART_CTAS = 6;
template <int NI>
__device__ __forceinline__ void partition_chunks(const PartArgs &a, int b, int G, int npl, int total, uint32_t *s_bits, int *s_pref, int *s_misc) {
    constexpr int CHUNK = NI * EVB_PART_THREADS;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nchunks = (total + CHUNK - 1) / CHUNK;
    // node of position p of the level's row order, its bounds [n0, n1)
    auto locate = [&](int p, int &node, int &n0, int &n1, int &off) {
        int l = 0, r = npl - 1; // largest pair with pl_cum <= p
        while (l < r) { const int mid = (l + r + 1) >> 1; if (a.pl[mid].y <= p) l = mid; else r = mid - 1; }
        const int4 pr = a.pl[l];
        off = pr.w; // the pair's segments are adjacent
        if (p < pr.z) { node = pr.x; n0 = pr.y; n1 = pr.z; }
        else { node = pr.x + 1; n0 = pr.z; n1 = a.pl[l + 1].y; }
    };
    const int first = (int)((long long)nchunks * b / G), last = (int)((long long)nchunks * (b + 1) / G);
    int node = 0, n0 = 0, n1 = 0, off = 0;
    bool ahead = false;
    uint32_t next[NI];
    for (int chunk = first; chunk < last; ++chunk) {
        const int p0 = chunk * CHUNK, p1 = min(total, p0 + CHUNK);
        if (p0 >= n1 || p0 < n0) { locate(p0, node, n0, n1, off); ahead = false; }
        uint32_t row[NI], x[NI];
        if (p1 <= n1) { // one node
            const uint32_t pk = a.t_packed[node - 1];
            if (!((pk >> 24) & 1u)) { ahead = false; continue; } // not split; uniform
            const uint8_t *xf = a.xC + (size_t)(pk & 0xffffu) * a.n;
            const uint32_t *in = a.rows_in + (p0 + off);
            const int cnt = p1 - p0;
            // all row ids first, then all gathers: NI independent loads in flight per thread in each phase
#pragma unroll
            for (int i = 0; i < NI; ++i) { const int q = i * EVB_PART_THREADS + threadIdx.x; row[i] = ahead ? next[i] : q < cnt ? __ldg(in + q) : 0xffffffffu; }
#pragma unroll
            for (int i = 0; i < NI; ++i) x[i] = row[i] != 0xffffffffu ? (uint32_t)__ldg(xf + row[i]) : 0xffffu;
            // the next chunk's row ids, if it lies in the same node
            const int more = min(total, p1 + CHUNK) - p1;
            ahead = chunk + 1 < last && p1 + more <= n1;
            if (ahead) {
#pragma unroll
                for (int i = 0; i < NI; ++i) { const int q = i * EVB_PART_THREADS + threadIdx.x; next[i] = q < more ? __ldg(in + CHUNK + q) : 0xffffffffu; }
            }
            unsigned left = 0;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const unsigned bal = __ballot_sync(FULL, x[i] != 0xffffu && goes_left(pk, x[i]));
                left |= ((bal >> lane) & 1u) << i;
                if (lane == 0) s_bits[i * PART_WARPS + wid] = bal;
            }
            __syncthreads();
            if (wid == 0) { // NI * 8 <= 32 words: one per lane
                const int c = lane < NI * PART_WARPS ? __popc(s_bits[lane]) : 0, incl = warp_incl_scan_i(c, lane);
                s_pref[lane] = incl - c;
                if (lane == 31) {
                    s_misc[0] = atomicAdd(a.cur_l + node, incl);
                    s_misc[1] = atomicSub(a.cur_r + node, cnt - incl) - (cnt - incl);
                }
            }
            __syncthreads();
            const int dl = s_misc[0], dr = s_misc[1];
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int q = i * EVB_PART_THREADS + threadIdx.x;
                if (q < cnt) {
                    const int before = s_pref[q >> 5] + __popc(s_bits[q >> 5] & ((1u << lane) - 1u));
                    a.rows_out[(left >> i) & 1u ? dl + before : dr + (q - before)] = row[i];
                }
            }
            __syncthreads();
        } else {
            ahead = false;
            // 2 * node + side of every row, 0: not a row of a split node
            uint32_t key[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int q = p0 + i * EVB_PART_THREADS + threadIdx.x;
                key[i] = 0u;
                if (q < p1) {
                    if (q >= n1 || q < n0) locate(q, node, n0, n1, off);
                    x[i] = a.t_packed[node - 1];
                    row[i] = __ldg(a.rows_in + (q + off));
                    if ((x[i] >> 24) & 1u) key[i] = (uint32_t)node << 1;
                }
            }
#pragma unroll
            for (int i = 0; i < NI; ++i)
                if (key[i] && goes_left(x[i], (uint32_t)__ldg(a.xC + (size_t)(x[i] & 0xffffu) * a.n + row[i]))) key[i] |= 1u;
            int base[NI];
            unsigned peers[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                peers[i] = __match_any_sync(FULL, key[i]);
                const int c = __popc(peers[i]);
                base[i] = 0;
                if (key[i] && (peers[i] & ((1u << lane) - 1u)) == 0u)
                    base[i] = (key[i] & 1u) ? atomicAdd(a.cur_l + (key[i] >> 1), c) : atomicSub(a.cur_r + (key[i] >> 1), c) - c;
            }
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int at = __shfl_sync(FULL, base[i], __ffs(peers[i]) - 1);
                if (key[i]) a.rows_out[at + __popc(peers[i] & ((1u << lane) - 1u))] = row[i];
            }
        }
    }
}
__global__ void __launch_bounds__(EVB_PART_THREADS, PART_CTAS) k_partition(PartArgs a) {
    __shared__ uint32_t s_bits[EVB_PART_CHUNK / 32];
    __shared__ int s_pref[EVB_PART_CHUNK / 32], s_misc[34];
    const LevelPlan *plan = a.plan + a.level; // all of it at once
    const int npl = load_now(&plan->npl), total = load_now(&plan->total), nbuild = load_now(&plan->nbuild);
    const int low = a.hlow ? load_now(reinterpret_cast<const int32_t *>(a.low_any)) : 0;
    {
        const size_t nb = (size_t)nbuild, ns = nb * a.acc_sums, nc = nb * a.acc_cnts;
        const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, st = (size_t)gridDim.x * blockDim.x;
        for (size_t i = i0; i < ns; i += st) a.hsum[i] = 0ull;
        if (low) for (size_t i = i0; i < ns; i += st) a.hlow[i] = 0ull;
        for (size_t i = i0; i < nc; i += st) a.hcnt[i] = 0u;
    }
    // few rows: small chunks, so that they spread over the GPU (their chain of dependent loads is what takes the time)
    const int each = total / (int)gridDim.x;
    if (each > 2 * EVB_PART_THREADS) partition_chunks<4>(a, blockIdx.x, gridDim.x, npl, total, s_bits, s_pref, s_misc);
    else if (each > EVB_PART_THREADS) partition_chunks<2>(a, blockIdx.x, gridDim.x, npl, total, s_bits, s_pref, s_misc);
    else partition_chunks<1>(a, blockIdx.x, gridDim.x, npl, total, s_bits, s_pref, s_misc);
    __syncthreads();
    if (threadIdx.x == 0) s_misc[33] = arrive(a.done) == gridDim.x - 1;
    __syncthreads();
    if (!s_misc[33]) return;
    if (threadIdx.x == 0) *a.done = 0u;
    if (a.level > 6) plan_level<false>(a, s_misc);
    else if (threadIdx.x < 32) plan_level<true>(a, s_misc);
}

PartArgs make_part_args(evb_handle *h, int level) {
    PartArgs a;
    a.xC = h->xC; a.n = h->n; a.rows_in = h->rows[(level - 1) & 1]; a.rows_out = h->rows[level & 1];
    a.t_split = h->t_split; a.t_packed = h->t_packed;
    a.seg_start = h->seg_start; a.seg_cnt = h->seg_cnt;
    a.bslot = h->bslot; a.cum = h->cum; a.slot_node = h->slot_node; a.rbase = h->rbase; a.kind = h->kind; a.cur_l = h->cur_l; a.cur_r = h->cur_r;
    const size_t np = (size_t)h->maxslots + 1;
    a.pl = h->pl + ((level - 1) & 1 ? np : 0); a.pl_next = h->pl + (level & 1 ? np : 0);
    a.plan = h->plan; a.done = h->ticket; a.level = level; a.D = h->D; // entry 0 of the tickets belongs to no node
    a.nsum = h->nsum; a.C = h->C; a.by_weight = h->world > 1 ? 1 : 0;
    const bool clear = evb_acc_direct(h); // else the conversion to doubles has cleared them
    a.hsum = h->hsum_q; a.hcnt = h->hcnt_q; a.hlow = h->hlow_q; a.low_any = h->low + evb_low_any(level);
    a.acc_sums = clear ? (size_t)h->B * h->SC * h->nq : 0; a.acc_cnts = clear ? (size_t)h->B * h->SC : 0;
    return a;
}

} // namespace

static_assert(EVB_PART_CHUNK == 1024 && EVB_PART_THREADS == 256, "k_partition assumes 32 ballot words per chunk");

int32_t evb_launch_tree_begin(evb_handle *h, bool quantize, bool all_rows, const uint32_t *gen_js_host) {
    BeginArgs a;
    a.seg_start = h->seg_start; a.seg_cnt = h->seg_cnt; a.bslot = h->bslot; a.t_feat = h->t_feat; a.kind = h->kind; a.t_bin = h->t_bin;
    a.t_split = h->t_split; a.t_gain = h->t_gain; a.t_w = h->t_w; a.t_pred = h->t_pred; a.t_packed = h->t_packed; a.nsum = h->nsum;
    a.plan = h->plan; a.ticket = h->ticket; a.low = h->low; a.rows = h->rows[0]; a.cum = h->cum; a.slot_node = h->slot_node; a.rbase = h->rbase;
    a.pl = h->pl;
    a.nids = h->nn + 2; a.nn = h->nn; a.K = h->K; a.C = h->C; a.D = h->D; a.all_rows = all_rows ? 1 : 0;
    a.gen_js_host = gen_js_host; a.gen_js = reinterpret_cast<uint32_t *>(h->gen_d); a.ngen_js = EVB_GEN_WORDS + h->F;
    evb_hg_quant_args(h, &a.q);
    if (!quantize) a.q.grad = nullptr;
    const int64_t threads = std::max<int64_t>(quantize || all_rows ? h->n : 0, std::max(a.nids, a.ngen_js));
    evb_tic(h, EVB_T_ROWS_INIT);
    const cudaError_t e = evb_launch(k_tree_begin, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, h->st, a);
    evb_toc(h, EVB_T_ROWS_INIT);
    EVB_CUDA(e);
    return EVB_OK;
}

static int32_t launch_peer_barrier(evb_handle *h) {
    BarrierArgs b;
    for (int q = 0; q < EVB_MAX_PEERS; ++q) b.peer_flags[q] = q < h->world ? h->peer_flags[q] : nullptr;
    b.flags_local = h->peer_flags[h->rank]; b.err = h->d_err; b.world = h->world; b.rank = h->rank; b.seq_dev = h->d_barrier_seq;
    b.max_polls = 20000000u;
    k_peer_barrier<<<1, 32, 0, h->st>>>(b);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

// Diagnostic: one flag barrier of a two-rank world whose second rank does not exist, on the handle's own GPU: rank 1's
// flag is never written, so the wait runs out after `max_polls` polls and the kernel leaves EVB_DERR_PEER in the
// error word -- the path a sharded run takes when a peer stops answering, without a second GPU and without a hang.
int32_t evb_launch_lonely_barrier(evb_handle *h, int *flags, int *seq, unsigned max_polls) {
    BarrierArgs b;
    for (int q = 0; q < EVB_MAX_PEERS; ++q) b.peer_flags[q] = q < 2 ? flags : nullptr;
    b.flags_local = flags; b.err = h->d_err; b.world = 2; b.rank = 0; b.seq_dev = seq; b.max_polls = max_polls;
    k_peer_barrier<<<1, 32, 0, h->st>>>(b);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_scan(evb_handle *h, int level) {
    ScanArgs a;
    a.hcomp = h->hcomp; a.hist = h->hist; a.nsum = h->nsum; a.kind = h->kind; a.bslot = h->bslot; a.js0 = h->js_d;
    a.feattypes = h->feattypes_d; a.mono = h->mono_d; a.t_feat = h->t_feat; a.t_bin = h->t_bin; a.t_split = h->t_split;
    a.t_gain = h->t_gain; a.t_w = h->t_w; a.t_pred = h->t_pred; a.t_packed = h->t_packed;
    a.F = h->F; a.C = h->C; a.K = h->K; a.B = h->B; a.level = level; a.D = h->D; a.hist_nodes = h->hist_nodes;
    a.loss = h->p.loss; a.neb = -h->p.eta / (double)h->p.bagging_size;
    a.elide_h = h->Ce != h->C ? 1 : 0;
    const bool direct = evb_acc_direct(h);
    a.qsum = direct ? h->hsum_q : nullptr; a.qcnt = direct ? h->hcnt_q : nullptr; a.qinv = h->d_qinv; a.SC = h->SC;
    a.qlow = direct ? h->hlow_q : nullptr; a.low = h->low + evb_low_slot(level); a.low_unit = evb_hg_low_unit(h->hgeo.hb);
    a.nq = h->nq; a.unit_w = h->unit_w ? 1 : 0;
    const bool fused = h->world == 1 && !h->obl_gain;
    a.gmax = evb_gmax(h, false); a.ng = h->ng;
    a.ticket = fused ? h->ticket : nullptr; a.cur_l = h->cur_l; a.cur_r = h->cur_r; a.seg_start = h->seg_start; a.seg_cnt = h->seg_cnt;
    a.lambda = h->p.lambda; a.L2 = h->p.L2; a.gamma = h->p.gamma; a.min_weight = h->p.min_weight;
    a.fbest_gain = h->fbest_gain; a.fbest_bin = h->fbest_bin; a.fbest_left = h->fbest_left;
    a.obl_gain = h->obl_gain; a.obl_best = h->obl_best;
    a.plan = h->plan + level; a.slot_node = h->slot_node; a.slots = evb_level_slots(level);
    const bool p2p = h->p2p && h->world > 1;
    a.world = p2p ? h->world : 1; a.rank = p2p ? h->rank : 0;
    for (int q = 0; q < EVB_MAX_PEERS; ++q) a.peer_cand[q] = p2p && q < h->world ? h->peer_cand[q] : nullptr;
    a.cand_local = p2p ? h->peer_cand[h->rank] : nullptr;
    const int m = evb_level_nodes(level);
    const int slots = evb_level_slots(level);
    const int Fown = (h->F - a.rank + a.world - 1) / a.world;
    if (p2p) {
        // all ranks' histograms of this level are complete -> sum the owned feature slots from the peers' memory
        evb_tic(h, EVB_T_ALLREDUCE);
        int32_t rc = launch_peer_barrier(h);
        PeerReduceArgs r;
        for (int q = 0; q < EVB_MAX_PEERS; ++q) r.peer_hcomp[q] = q < h->world ? h->peer_hcomp[q] : nullptr;
        r.hsum = h->hsum; r.plan = h->plan + level; r.world = h->world; r.rank = h->rank; r.F = h->F; r.CB = h->C * h->B; r.level = level;
        r.K = h->K; r.elided = h->Ce != h->C ? 1 : 0;
        if (rc == EVB_OK) k_peer_reduce<<<slots * (Fown + 1), 256, 0, h->st>>>(r);
        evb_toc(h, EVB_T_ALLREDUCE);
        EVB_CHECK(rc);
        a.hcomp = h->hsum;
    }
    const long long warps = (long long)slots * Fown * (level > 1 ? 2 : 1);
    evb_tic(h, EVB_T_SCAN);
    if (fused && evb_scan_multi(h)) {
#define EVB_SCAN(M) EVB_CUDA(evb_launch(k_scan_multi<M>, dim3((unsigned)warps), dim3(32 * h->K), 0, h->st, a))
        if (h->B <= 32) EVB_SCAN(1); else if (h->B <= 64) EVB_SCAN(2); else if (h->B <= 128) EVB_SCAN(4); else EVB_SCAN(8);
#undef EVB_SCAN
    } else if (warps > 0) {
        const unsigned grid = (unsigned)((warps + 7) / 8), few = (unsigned)((warps + 3) / 4);
        const bool own = h->p.loss >= EVB_MAE;
        const bool obl = h->obl_gain != nullptr;
#define EVB_SCAN(M) do { \
            if (own && obl) EVB_CUDA(evb_launch(k_scan_feat<M, true, true, false, true>, dim3(grid), dim3(256), 0, h->st, a)); \
            else if (own) EVB_CUDA(evb_launch(k_scan_feat<M, true, false, false, true>, dim3(grid), dim3(256), 0, h->st, a)); \
            else if (obl) EVB_CUDA(evb_launch(k_scan_feat<M, false, true, false, true>, dim3(grid), dim3(256), 0, h->st, a)); \
            else if (h->K == 1 && h->C == 3 && !a.qlow) EVB_CUDA(evb_launch(k_scan_feat<M, false, false, true, false>, dim3(grid), dim3(256), 0, h->st, a)); \
            else if (h->K == 1 && h->C == 3) EVB_CUDA(evb_launch(k_scan_feat<M, false, false, true, true>, dim3(scan_threads(M, true, true) == 128 ? few : grid), dim3(scan_threads(M, true, true)), 0, h->st, a)); \
            else EVB_CUDA(evb_launch(k_scan_feat<M, false, false, false, true>, dim3(grid), dim3(256), 0, h->st, a)); } while (0)
        if (h->B <= 32) EVB_SCAN(1); else if (h->B <= 64) EVB_SCAN(2); else if (h->B <= 128) EVB_SCAN(4); else EVB_SCAN(8);
#undef EVB_SCAN
    }
    evb_toc(h, EVB_T_SCAN);
    EVB_CUDA(cudaGetLastError());
    if (h->obl_gain && level < h->D) {
        evb_tic(h, EVB_T_SCAN);
        k_obl_sum<<<(h->F * h->B + 127) / 128, 128, 0, h->st>>>(a);
        k_obl_pick<<<1, 1024, 0, h->st>>>(a);
        evb_toc(h, EVB_T_SCAN);
    }
    if (fused) return EVB_OK;
    evb_tic(h, EVB_T_SCAN);
    if (h->K == 1 && h->C == 3 && h->p.loss < EVB_MAE) k_scan_node<true><<<(m + 7) / 8, 256, 0, h->st>>>(a);
    else k_scan_node<false><<<(m + 7) / 8, 256, 0, h->st>>>(a);
    evb_toc(h, EVB_T_SCAN);
    if (p2p) {
        evb_tic(h, EVB_T_ALLREDUCE); int32_t rc = launch_peer_barrier(h); evb_toc(h, EVB_T_ALLREDUCE); EVB_CHECK(rc);
        evb_tic(h, EVB_T_SCAN);
        k_scan_final<<<(m + 7) / 8, 256, 0, h->st>>>(a);
        evb_toc(h, EVB_T_SCAN);
    }
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}

int32_t evb_launch_partition(evb_handle *h, int level) {
    PartArgs a = make_part_args(h, level);
    const int64_t chunks = (h->n + EVB_PART_THREADS - 1) / EVB_PART_THREADS; // the smallest ones
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(h->num_sms * PART_CTAS, chunks));
    evb_tic(h, EVB_T_PARTITION);
    const cudaError_t e = evb_launch(k_partition, dim3(grid), dim3(EVB_PART_THREADS), 0, h->st, a);
    evb_toc(h, EVB_T_PARTITION);
    EVB_CUDA(e);
    return EVB_OK;
}
