// A whole tree in one launch (`grow_tree!`, src/fit.jl:62-137; GPU counterpart ext/EvoTreesKernelAbstractionsExt/fit.jl:23-77), for one
// output and tables whose rows fit the shared memory of the GPU: gradients to fixed point, histograms, split scan, decisions, rows to the
// children, and, without a row sample, predictions, the next round's gradients, the evaluation rows and the finished tree.
//
// What bounds these tables is the chain of dependent steps of a level, each a launch of its own before: 25 us a level, of which the
// work was a few.  Here a CTA keeps its share for the whole tree in shared memory: one group of features (a word of bins for four of
// them) of one range of rows, the words of their gradients, and its own lists of the rows of every node.  Per level:
//   histograms   lane = row of a tile, cells and banks as in evb_histg.cuh, an image per build slot; sums of all row ranges meet in L2
//   (barrier)    the grid has at most one CTA per SM and is launched cooperatively
//   scan         a warp per (node, feature), the arithmetic of k_scan_feat
//   (barrier)
//   decisions    every CTA takes all of them, so that nothing has to be handed around; the children's weights say which one is built
//   rows         every CTA moves its own rows, looking up the split feature's bin (other groups' CTAs do the same for theirs)
// With one range of rows a CTA scans its own features' sums and the first barrier falls away.
// Where at most 16 CTAs hold the rows they are one cluster: sums, histograms and best splits lie in their shared memory, added to and handed
// out by remote accesses, and its barriers are the hardware's (0.4 us with the wait for the slowest CTA, 1.3 through L2).
// ms per tree of level kernels and this one: 1503 x 7 logloss, depth 5 0.085 and 0.041; 100k x 10, 32 bins, depth 6 0.095 and 0.060; 60k x 77
// poisson (54 columns), depth 6 0.124 and 0.095; 6.4k x 80, 128 bins, depth 7 0.169 and 0.119. At 100k x 10 a level takes 8 us: histograms 1.4,
// barriers 1.7 and 1.3, scan 1.2, decisions 1.1, rows 1.5 to 2.8.
#include "evb_histg.cuh"
#include "evb_device.cuh"
#include <string.h>
#include <algorithm>

namespace {

using namespace evb_hg;

constexpr int T = 512, NW = T / 32;
constexpr int MAX_D = 10;

struct GrowArgs {
    const uint8_t *xC;          // [nfeats][n]
    float *grad;                // [n][NQ] gradient records
    const uint8_t *mask;        // rows with mask <= cond are sampled; null: all
    const uint32_t *js0;        // column sample of this tree: null: all columns, or
    int js_inline;              // (no launch before this one to bring them: the CTAs of a launch reading pinned memory cost 250 us) js
    uint16_t js[EVB_GROW_JS];
    const uint8_t *feattypes;
    const int32_t *mono;
    unsigned long long *sum, *low; // [2][slots][F][nq][B]: sums of a level's build slots, second set of sums
    uint32_t *cnt;              // [2][slots][F][B]
    size_t sum_set, cnt_set;    // words of one of the two
    uint32_t *lowflag;          // evb_handle::low
    double *hist, *nsum;
    double2 *best;              // [2][M][F][3] {gain, bin or -1}, {g, h}, {w, -}: best split of a feature and its left sums
    double *qinv;
    unsigned *signs;
    const unsigned *gmax;       // [NQ] bits of max |g| of this tree's gradients
    unsigned *gmax_next;        // of the next tree's
    int32_t *t_feat;
    uint8_t *t_bin, *t_split;
    float *t_gain, *t_w, *t_pred;
    uint32_t *t_packed;
    LevelPlan *plan;
    uint32_t *bar;              // arrivals at the grid's barriers; CTAs that are done (the last one clears both)
    int *err;
    long long n;
    int cond, F, B, D, hist_nodes, loss, elide, hb, ng, round_bits, nn;
    int NG, NR, rpc, lw, M;
    uint8_t lc[MAX_D];          // [level] log2 of the columns of an image
    int o_x, o_q, o_idx, o_node;
    int o_sum, o_cnt, o_best, o_hist, fo; // one cluster only: sums of the features a CTA scans, fo at most; o_hist == 0: their histograms are in `hist`
    unsigned max_polls;
    double low_unit, neb, lambda, L2, gamma, min_weight;
    // no row sample: the kernel also clears the tree before and brings it to every row afterwards
    int whole, next_grads;
    float *pred;
    const void *y;
    uint32_t *nidx;
    AlphaSet alpha;
    const uint4 *pub_src;
    uint4 *pub_dst;
    int pub_n, pub_err;         // 16-byte words of the finished tree; word of the error code
    const uint8_t *ev_xT;       // evaluation rows (ev_n == 0: none), as in EvalArgs
    const void *ev_y;
    const float *ev_w;
    float *ev_pred;
    double *ev_part, *ev_sum;
    long long ev_n;
    int ev_RS, ev_metric;
};

// Shared memory.  Addresses are sums of launch constants: pointers kept in a struct that is indexed, or registers that spill, live in
// local memory, which every barrier of the grid empties from L1 -- a step that reads them then waits for L2 again and again.
struct Pairs { // state of a level: slot = parent's number in its level (at level 1 the root alone); slots of parents that did not split are empty
    unsigned char *b;
    int M;
    __device__ __forceinline__ double *sum() const { return reinterpret_cast<double *>(b); }          // [2 slots][3]
    __device__ __forceinline__ int *build() const { return reinterpret_cast<int *>(b + 24 * M); }     // 0: the left child is built, 1: the right one
    __device__ __forceinline__ int *st() const { return reinterpret_cast<int *>(b + 28 * M); }        // its rows in the list: left [st, mid), right [mid, en); ascending
    __device__ __forceinline__ int *mid() const { return reinterpret_cast<int *>(b + 32 * M); }
    __device__ __forceinline__ int *en() const { return reinterpret_cast<int *>(b + 36 * M); }
    __device__ __forceinline__ uint32_t *dec() const { return reinterpret_cast<uint32_t *>(b + 40 * M); } // the parents' splits (packed as in t_packed); 0: none
};
constexpr int PAIR_BYTES = 48, NODE_BYTES = 2 * PAIR_BYTES + 8 + 32, MISC_BYTES = 512; // (8: the cursors of right rows, and room)
extern __shared__ __align__(128) unsigned char s_raw[];
// image(s), bins [word][row], words of gradients [channel][row], row lists, then per node of a level
#define S_IMG (reinterpret_cast<uint32_t *>(s_raw))
#define S_X (reinterpret_cast<uint32_t *>(s_raw + a.o_x))
#define S_Q (reinterpret_cast<int32_t *>(s_raw + a.o_q))
#define S_IDX(cur) (reinterpret_cast<uint16_t *>(s_raw + a.o_idx + (cur) * 2 * a.rpc))
#define S_PAIRS(cur) (Pairs{s_raw + a.o_node + (cur) * PAIR_BYTES * a.M, a.M})
#define S_CR (reinterpret_cast<int *>(s_raw + a.o_node + 2 * PAIR_BYTES * a.M))                                    /* where a node's right rows begin so far */
#define S_OUT (reinterpret_cast<double4 *>(s_raw + a.o_node + (2 * PAIR_BYTES + 8) * a.M))                          /* [node] left sums, gain */
#define S_MISC (reinterpret_cast<int *>(s_raw + a.o_node + NODE_BYTES * a.M))
#define S_UNIT (reinterpret_cast<double *>(s_raw + a.o_node + NODE_BYTES * a.M + 64))                              /* units of the channels' sums */
#define S_ROOT (reinterpret_cast<double *>(s_raw + a.o_node + NODE_BYTES * a.M + 96))                               /* sums of the root (one cluster) */
#define S_INF (S_MISC + 8)                                                                                          /* [NQ] the channel has an infinity */
#define S_RED (reinterpret_cast<double *>(s_raw + a.o_node + NODE_BYTES * a.M + 128))                              /* [2 NW] */
#define S_QUANT (reinterpret_cast<Quant *>(s_raw + a.o_node + NODE_BYTES * a.M + 128))                             /* [NQ], while the rows are loaded */
#define S_TREE (reinterpret_cast<uint32_t *>(s_raw + a.o_node + NODE_BYTES * a.M + MISC_BYTES))                    /* [nn] packed nodes */
#define S_VALUE (reinterpret_cast<float *>(S_TREE + a.nn))                                                         /* [nn] leaf values */
#define S_FEAT (S_TREE + 2 * a.nn)                                                                                 /* [F] feature | numeric << 16 | (constraint + 1) << 17 */
#define S_LEAF (reinterpret_cast<uint16_t *>(S_FEAT + a.F))                                                        /* leaf of every row this CTA updates */
// one cluster only
#define S_SUM (reinterpret_cast<unsigned long long *>(s_raw + a.o_sum))  /* [slot][fo][NQ][B] */
#define S_CNTS (reinterpret_cast<uint32_t *>(s_raw + a.o_cnt))           /* [slot][fo][B], then [slot] nonzero: the slot has something in `low` */
#define S_LOW (S_CNTS + (a.M / 2) * a.fo * a.B)
#define S_BEST (reinterpret_cast<double2 *>(s_raw + a.o_best))           /* [node][F][3], of all features */
enum { M_LEFT = 0, M_OK = 1, M_CNT = 2, M_MAX = 4 }; // M_MAX: two words

// shared memory of CTA `rank` of the cluster
__device__ __forceinline__ uint32_t remote(const void *p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void remote_add(uint32_t at, unsigned long long v) { asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(at), "l"(v) : "memory"); }
__device__ __forceinline__ void remote_add(uint32_t at, uint32_t v) { asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
__device__ __forceinline__ void remote_put(uint32_t at, double x, double y) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void remote_put(uint32_t at, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
template <typename F>
__device__ __forceinline__ void cluster_barrier(F meanwhile) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    meanwhile();
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_barrier() { cluster_barrier([] {}); }

// All CTAs have arrived `k` times.  The launch is cooperative, so all of them run; the wait is bounded all the same: a CTA whose
// wait runs out (or that sees another's has) leaves an error word and the kernel ends.
template <typename F>
__device__ __forceinline__ bool grid_barrier(const GrowArgs &a, int *ok, unsigned k, F meanwhile) {
    __syncthreads();
    if (threadIdx.x == T - 1) {
        const uint32_t target = k * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        bool good = false;
        for (unsigned i = 0; i < a.max_polls; ++i) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
            if (v >= target) { good = true; break; }
            if ((i & 1023u) == 1023u && *(volatile int *)a.err != 0) break;
        }
        if (!good) {
            atomicCAS(a.err, 0, EVB_DERR_GRID);
            if (a.pub_dst) reinterpret_cast<volatile int *>(a.pub_dst)[a.pub_err] = EVB_DERR_GRID;
        }
        *ok = good;
    } else meanwhile();
    __syncthreads();
    return *ok != 0;
}

// First maximum over the lanes: v the largest, id the smallest of those that have it (ids are not negative).  Doubles are compared as
// whole numbers, so that three reductions of the warp do it instead of five exchanges of three words.
__device__ __forceinline__ void warp_first_max(double &v, int &id) {
    const long long b = __double_as_longlong(v + 0.0); // -0 = 0
    const unsigned long long k = (unsigned long long)b ^ (b < 0 ? ~0ull : 1ull << 63);
    const uint32_t hi = __reduce_max_sync(FULL, (uint32_t)(k >> 32)), lo = __reduce_max_sync(FULL, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0u);
    const bool top = (uint32_t)(k >> 32) == hi && (uint32_t)k == lo;
    id = (int)__reduce_min_sync(FULL, top ? (uint32_t)id : 0x7fffffffu);
    const unsigned long long m = (unsigned long long)hi << 32 | lo;
    v = __longlong_as_double((long long)(m >> 63 ? m ^ (1ull << 63) : ~m));
}

// ---------------------------------------------------------------------------------------------- histograms of a level
// Rows of the build nodes of slots [s0, s1), a tile of 32 rows of one node per warp; lanes and banks as in evb_histg.cuh
// LC == 5: 32 columns, 8 / W replicas of W words, a bank for every lane.  With fewer columns 32 / columns lanes share one (their bins decide
// whether they meet), but an image is emptied faster and more of them fit: what small nodes want (level_columns).
template <int NQ, bool CNT, bool PACK, int PB, int C = 0>
__device__ __forceinline__ void add_cell(uint32_t addr, const uint32_t (&hi)[NQ], const uint32_t (&lo)[NQ]) {
    if constexpr (C < NQ) {
        red_at<2 * PB * C>(addr, hi[C]);
        red_at<2 * PB * C + PB>(addr, lo[C]);
        add_cell<NQ, CNT, PACK, PB, C + 1>(addr, hi, lo);
    } else if constexpr (CNT && !PACK) {
        red_at<2 * PB * NQ>(addr, 1u);
    }
}
template <int NQ, bool CNT, bool PACK, int LW, int LC>
__device__ __forceinline__ void add_rows(const GrowArgs &a, const Pairs &pr, const uint16_t *idx, int s0, int s1, bool second) {
    constexpr int P = planes(NQ, CNT, PACK), W = 1 << LW, PB = 4 << LC, R = 1 << (LC - 2 - LW);
    constexpr uint32_t STRIDE = P * PB;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float two_lb = __int_as_float((128 + a.hb) << 23); // 2^(hb + 1)
    Lane ln;
    ln.init(S_IMG, lane);
    const uint32_t rep = 16u * (uint32_t)(lane & (R * W - 1) & ~(W - 1)), slot_bytes = (uint32_t)(a.B + 1) * STRIDE;
    int base = 0;
    for (int s = s0; s < s1; ++s) {
        const int b = pr.build()[s], r0 = b ? pr.mid()[s] : pr.st()[s], cnt = (b ? pr.en()[s] : pr.mid()[s]) - r0, nt = (cnt + 31) >> 5;
        const uint32_t img = (uint32_t)(s - s0) * slot_bytes + rep;
        for (int t = (wid - base) & (NW - 1); t < nt; t += NW) {
            const int p = t * 32 + lane;
            const bool act = p < cnt;
            const int r = idx[r0 + (act ? p : 0)];
            uint32_t qh[NQ], ql[NQ];
            if constexpr (PACK) {
                const int32_t v = S_Q[r];
                qh[0] = (uint32_t)(v >> 6); ql[0] = ((uint32_t)v & 63u) | (1u << 19);
            } else {
                uint32_t some = 0u; // nonzero: something is left of the row
#pragma unroll
                for (int c = 0; c < NQ; ++c) {
                    const float left = take_apart(__int_as_float(S_Q[c * a.rpc + r]), two_lb, qh[c], ql[c]);
                    some |= __float_as_uint(left);
                    if (second) take_apart(left * two_lb, two_lb, qh[c], ql[c]);
                }
                if (!act) some = 0u;
                const bool any = __any_sync(FULL, some != 0u);
                if (second && !any) continue;
                if (!second && any && lane == 0) S_MISC[M_LEFT] = 1;
            }
            if (act) {
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const int word = (lane + w) & (W - 1);
                    const uint32_t v = S_X[word * a.rpc + r], at = img + 16u * (uint32_t)word;
#pragma unroll
                    for (int k = 0; k < 4; ++k) add_cell<NQ, CNT, PACK, PB>(__byte_perm(v, 0u, ln.sel[k]) * STRIDE + (ln.col[k] + at), qh, ql);
                }
            }
        }
        base += nt;
    }
}

// The images of slots [s0, s1) -> sums of the level; clears them.  A warp takes BO adjacent bins of FB features at a time, so that the
// lanes of a reduction fill whole sectors of [feature][channel][bin]; replicas are read in an order that differs from bin to bin
// (they sit 4 W columns apart: one bank for all bins).
template <int NQ, bool CNT, bool PACK, int LW, int LC, bool CL>
__device__ __forceinline__ void flush(const GrowArgs &a, const Pairs &pr, int set, int s0, int s1, int g, bool second) {
    constexpr int P = planes(NQ, CNT, PACK), W = 1 << LW, COLS = 1 << LC, R = 1 << (LC - 2 - LW), FB = LW == 0 ? 4 : 8, BO = 32 / FB, NC = 4 * W / FB;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, bo = lane % BO, f0 = g * 4 * W;
    const int nbb = (a.B + BO - 1) / BO, slot_words = (a.B + 1) * P * COLS;
    const bool own = a.NR == 1; // no other CTA adds to these cells
    int base = 0;
    for (int i = threadIdx.x; i < (s1 - s0) * (P * COLS); i += T) S_IMG[(i / (P * COLS)) * slot_words + i % (P * COLS)] = 0u; // the guard rows: other levels cut images elsewhere
    for (int slot = s0; slot < s1; ++slot) {
        if (!pr.dec()[slot] || (!own && pr.st()[slot] == pr.en()[slot])) continue;
#pragma unroll
    for (int ch = 0; ch < NC; ++ch, base += nbb)
    for (int bb = (wid - base) & (NW - 1); bb < nbb; bb += NW) {
        const int bin = bb * BO + bo, f = ch * FB + lane / BO;
        if (bin >= a.B) continue;
        uint32_t *p = S_IMG + (slot - s0) * slot_words + (bin + 1) * (P * COLS) + f;
        const bool out = f0 + f < a.F;
        // where the sums go: this CTA's share of the features (CL), CTA f % NR of the group's, or global memory
        const int lf = CL ? own ? f : f / a.NR : 0, rank = CL ? (f - lf * a.NR) * a.NG + g : 0;
        const size_t cell = CL && !second ? (size_t)slot * a.fo + lf : (size_t)slot * a.F + (f0 + f);
        auto put = [&](int c, unsigned long long v) {
            const size_t at = (cell * NQ + c) * a.B + bin;
            if (CL && !second) {
                if (own) S_SUM[at] = v;
                else if (v != 0ull) remote_add(remote(S_SUM + at, rank), v);
            } else {
                unsigned long long *d = (second ? a.low : a.sum) + (size_t)set * a.sum_set + at;
                if (own) *d = v;
                else if (v != 0ull) asm volatile("red.global.add.u64 [%0], %1;" ::"l"(d), "l"(v) : "memory");
            }
        };
        auto put_count = [&](uint32_t v) {
            const size_t at = cell * a.B + bin;
            if (CL) {
                if (own) S_CNTS[at] = v;
                else if (v != 0u) remote_add(remote(S_CNTS + at, rank), v);
            } else {
                uint32_t *d = a.cnt + (size_t)set * a.cnt_set + at;
                if (own) *d = v;
                else if (v != 0u) asm volatile("red.global.add.u32 [%0], %1;" ::"l"(d), "r"(v) : "memory");
            }
        };
        if constexpr (PACK) {
            long long v = 0;
            uint32_t c = 0;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                uint32_t *w = p + ((i + bo) & (R - 1)) * (4 * W);
                const uint32_t hi = w[0], lo = w[COLS];
                w[0] = 0u; w[COLS] = 0u;
                v += ((long long)(int32_t)hi << 6) + (long long)(lo & 0x7ffffu);
                c += lo >> 19;
            }
            if (out && (own || c != 0u)) { put(0, (unsigned long long)v); put_count(c); }
        } else {
            if constexpr (CNT) {
                uint32_t c = 0;
#pragma unroll
                for (int i = 0; i < R; ++i) { uint32_t *w = p + ((i + bo) & (R - 1)) * (4 * W) + 2 * COLS * NQ; c += *w; *w = 0u; }
                if (!own && c == 0u) continue; // no row: all words are zero
                if (out && !second) put_count(c);
            }
#pragma unroll
            for (int c = 0; c < NQ; ++c) {
                long long hi = 0, lo = 0;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    uint32_t *w = p + ((i + bo) & (R - 1)) * (4 * W) + 2 * COLS * c;
                    hi += (long long)(int32_t)w[0]; lo += (long long)(int32_t)w[COLS];
                    w[0] = 0u; w[COLS] = 0u;
                }
                if (out) put(c, (unsigned long long)((hi << (a.hb + 1)) + lo));
            }
        }
    }
    }
}

// Nodes of so few rows in this range that most cells of an image would stay empty or hold one row: every row straight to the sums, one
// reduction per feature and channel (and one for the count), no image, no barrier.
template <int NQ, bool CNT, bool PACK, bool CL>
__device__ __forceinline__ void add_direct(const GrowArgs &a, const Pairs &pr, const uint16_t *idx, int np, int set, int g, int level, bool second) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, f0 = g * (4 << a.lw), nf = min(4 << a.lw, a.F - f0);
    const float two_lb = __int_as_float((128 + a.hb) << 23);
    int base = 0;
    for (int s = 0; s < np; ++s) {
        const int b = pr.build()[s], r0 = b ? pr.mid()[s] : pr.st()[s], cnt = (b ? pr.en()[s] : pr.mid()[s]) - r0, nt = (cnt + 31) >> 5;
        bool left_any = false;
        for (int t = (wid - base) & (NW - 1); t < nt; t += NW) {
            const bool act = t * 32 + lane < cnt;
            const int r = idx[r0 + (act ? t * 32 + lane : 0)];
            unsigned long long v[NQ];
            uint32_t some = 0u;
#pragma unroll
            for (int c = 0; c < NQ; ++c) {
                if constexpr (PACK) v[c] = (unsigned long long)(long long)S_Q[r];
                else {
                    uint32_t hi, lo;
                    const float left = take_apart(__int_as_float(S_Q[c * a.rpc + r]), two_lb, hi, lo);
                    some |= __float_as_uint(left);
                    if (second) take_apart(left * two_lb, two_lb, hi, lo);
                    v[c] = (unsigned long long)(((long long)(int32_t)hi << (a.hb + 1)) + (long long)(int32_t)lo);
                }
            }
            if (!act) some = 0u;
            left_any = left_any || some != 0u;
            if (!act || (second && some == 0u)) continue;
            for (int f = 0; f < nf; ++f) {
                const uint32_t bin = (S_X[(f >> 2) * a.rpc + r] >> (8 * (f & 3)) & 0xffu) - 1u;
                if (CL && !second) {
                    const int lf = f / a.NR, rank = (f - lf * a.NR) * a.NG + g, cell = s * a.fo + lf;
                    const uint32_t at = remote(S_SUM + cell * NQ * a.B, rank) + 8u * bin;
#pragma unroll
                    for (int c = 0; c < NQ; ++c) if (v[c] != 0ull) remote_add(at + 8u * (uint32_t)(c * a.B), v[c]);
                    if (CNT || PACK) remote_add(remote(S_CNTS + cell * a.B, rank) + 4u * bin, 1u);
                } else {
                    const size_t cell = (size_t)s * a.F + f0 + f;
                    unsigned long long *d = (second ? a.low : a.sum) + (size_t)set * a.sum_set + cell * NQ * a.B + bin;
#pragma unroll
                    for (int c = 0; c < NQ; ++c) if (v[c] != 0ull) asm volatile("red.global.add.u64 [%0], %1;" ::"l"(d + c * a.B), "l"(v[c]) : "memory");
                    if ((CNT || PACK) && !second) asm volatile("red.global.add.u32 [%0], 1;" ::"l"(a.cnt + (size_t)set * a.cnt_set + cell * a.B + bin) : "memory");
                }
            }
        }
        base += nt;
        if constexpr (!PACK) {
            if (!second && __any_sync(FULL, left_any)) { // all slots are looked through again (rows that leave nothing are skipped)
                if (lane == 0) S_MISC[M_LEFT] = 1;
                if constexpr (CL) { if (lane < (int)gridDim.x) remote_put(remote(S_LOW + s, lane), 1u); }
                else if (lane == 0) a.lowflag[evb_low_slot(level) + s] = 1u;
            }
        }
    }
}
template <int NQ, bool CNT, bool PACK, bool CL>
__device__ __forceinline__ void direct_level(const GrowArgs &a, const Pairs &pr, const uint16_t *idx, int np, int set, int g, int level) {
    add_direct<NQ, CNT, PACK, CL>(a, pr, idx, np, set, g, level, false);
    if constexpr (!PACK) {
        __syncthreads();
        if (S_MISC[M_LEFT] == 0) return;
        add_direct<NQ, CNT, PACK, CL>(a, pr, idx, np, set, g, level, true);
        __syncthreads();
        if (threadIdx.x == 0) S_MISC[M_LEFT] = 0;
    }
}
template <int NQ, bool CNT, bool PACK, int LW, int LC, bool CL>
__device__ __forceinline__ void hist_level(const GrowArgs &a, const Pairs &pr, const uint16_t *idx, int np, int set, int g, int level) {
    const int fit = a.o_x / ((a.B + 1) * planes(NQ, CNT, PACK) * (4 << LC)); // images come first in shared memory
    for (int s0 = 0; s0 < np; s0 += fit) {
        const int s1 = min(np, s0 + fit);
        for (bool second = false;; second = true) {
            add_rows<NQ, CNT, PACK, LW, LC>(a, pr, idx, s0, s1, second);
            __syncthreads();
            const bool again = !PACK && !second && S_MISC[M_LEFT] != 0;
            flush<NQ, CNT, PACK, LW, LC, CL>(a, pr, set, s0, s1, g, second);
            if (second) {
                if constexpr (CL) {
                    for (int e = threadIdx.x; e < (s1 - s0) * (int)gridDim.x; e += T) remote_put(remote(S_LOW + s0 + e / gridDim.x, e % gridDim.x), 1u);
                } else for (int s = s0 + (int)threadIdx.x; s < s1; s += T) a.lowflag[evb_low_slot(level) + s] = 1u;
            }
            __syncthreads();
            if (!again) break;
            if (threadIdx.x == 0) S_MISC[M_LEFT] = 0; // (read again behind the next barrier)
        }
    }
}

// ---------------------------------------------------------------------------------------------- split scan
// One warp: node n (of pair `slot`, number j of the level) and feature slot f.  The same sums, in the same order, as k_scan_feat.
template <int NQ, bool CNT, bool PACK, int CH, bool CL>
__device__ __forceinline__ void scan(const GrowArgs &a, int level, int set, int slot, int f, int lf, int n, int j, bool sub, const double *node_sum) {
    const int lane = threadIdx.x & 31, B = a.B, F = a.F, bin0 = lane * CH;
    const bool counted = CNT || PACK, keep = n < a.hist_nodes, elide = a.elide != 0;
    const size_t cell = (size_t)slot * F + f, own = (size_t)slot * a.fo + lf;
    const unsigned long long *ps = CL ? S_SUM + own * NQ * B : a.sum + (size_t)set * a.sum_set + cell * NQ * B;
    const uint32_t *pc = CL ? S_CNTS + own * B : a.cnt + (size_t)set * a.cnt_set + cell * B;
    const double *hp = a.hist + ((size_t)(n >> 1) * F + f) * 3 * B;
    double *hn = a.hist + ((size_t)n * F + f) * 3 * B;
    // one cluster: histograms of this level and the one before also in shared memory, the larger half for the levels that are an even
    // number of levels above the last one kept
    const bool near = CL && a.o_hist != 0;
    const int hs = elide ? 2 : 3, up = a.D - 2 - level;
    auto near_at = [&](int node, int above) {
        return reinterpret_cast<double *>(s_raw + a.o_hist) + ((size_t)((above & 1) ? max(1, a.M >> 1) : 0) + node) * a.fo * hs * B + (size_t)lf * hs * B;
    };
    double *kn = near ? near_at(j, up) : nullptr;
    if (near) hp = near_at(j >> 1, up + 1);
    const int wo = near ? hs - 1 : 2;
    auto ldu = [](const unsigned long long *p) { if constexpr (CL) return *p; else return __ldcg(p); };
    auto ldc = [](const uint32_t *p) { if constexpr (CL) return *p; else return __ldcg(p); };
    long long rg[CH], rh[CH], rw[CH];
    double pg[CH], ph[CH], pw[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const int b = min(bin0 + i, B - 1);
        rg[i] = (long long)ldu(ps + b);
        rh[i] = elide ? 0ll : (long long)ldu(ps + B + b);
        rw[i] = counted ? (long long)ldc(pc + b) : (long long)ldu(ps + (NQ - 1) * B + b);
        pg[i] = ph[i] = pw[i] = 0.0;
        if (sub) { pg[i] = CL ? hp[b] : __ldcg(hp + b); if (!elide) ph[i] = CL ? hp[B + b] : __ldcg(hp + B + b); pw[i] = CL ? hp[wo * B + b] : __ldcg(hp + wo * B + b); }
    }
    const uint32_t feat = S_FEAT[f];
    const double ig = S_UNIT[0], ih = elide ? 0.0 : S_UNIT[NQ > 1 ? 1 : 0], iw = counted ? 1.0 : S_UNIT[NQ - 1];
    const bool numeric = (feat >> 16) & 1u, low = !PACK && (CL ? S_LOW[slot] : __ldcg(a.lowflag + evb_low_slot(level) + slot)) != 0u;
    const int constraint = (int)((feat >> 17) & 3u) - 1;
    double g[CH], h[CH], w[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) { g[i] = (double)rg[i] * ig; h[i] = (double)rh[i] * ih; w[i] = (double)rw[i] * iw; }
    double sg, sh, sw;
    if (n == 1) {
        long long tg = 0, th = 0, tw = 0;
#pragma unroll
        for (int i = 0; i < CH; ++i) if (bin0 + i < B) { tg += rg[i]; th += rh[i]; tw += rw[i]; }
        sg = (double)warp_sum(tg) * ig; sh = (double)warp_sum(th) * ih; sw = (double)warp_sum(tw) * iw;
    } else { sg = node_sum[0]; sh = node_sum[1]; sw = node_sum[2]; }
    if (low) {
        const unsigned long long *pl = a.low + (size_t)set * a.sum_set + cell * NQ * B;
        long long tg = 0, th = 0, tw = 0;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int b = min(bin0 + i, B - 1);
            const long long lg = (long long)__ldcg(pl + b), lh = elide ? 0ll : (long long)__ldcg(pl + B + b), lw = counted ? 0ll : (long long)__ldcg(pl + (NQ - 1) * B + b);
            g[i] += (double)lg * (ig * a.low_unit); h[i] += (double)lh * (ih * a.low_unit); w[i] += (double)lw * (counted ? 0.0 : iw * a.low_unit);
            if (bin0 + i < B) { tg += lg; th += lh; tw += lw; }
        }
        if (n == 1) {
            sg += (double)warp_sum(tg) * (ig * a.low_unit); sh += (double)warp_sum(th) * (ih * a.low_unit);
            if (!counted) sw += (double)warp_sum(tw) * (iw * a.low_unit);
        }
    }
    if (n == 1) {
        if (elide) sh = 2.0 * sw; // h = 2w (src/loss.jl:52)
        if (f == 0 && lane == 0) { a.nsum[3] = sg; a.nsum[4] = sh; a.nsum[5] = sw; }
        if (CL && f == 0 && lane < (int)gridDim.x) { remote_put(remote(S_ROOT, lane), sg, sh); remote_put(remote(S_ROOT + 2, lane), sw, 0.0); }
    }
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const int b = bin0 + i;
        if (sub) { g[i] = pg[i] - g[i]; h[i] = ph[i] - h[i]; w[i] = pw[i] - w[i]; }
        if (elide) h[i] = 2.0 * w[i];
        if (b >= B) g[i] = h[i] = w[i] = 0.0;
        else if (keep) {
            hn[b] = g[i]; hn[B + b] = h[i]; hn[2 * B + b] = w[i];
            if (near && up >= 0) { kn[b] = g[i]; kn[wo * B + b] = w[i]; if (!elide) kn[B + b] = h[i]; }
        }
    }
    if (numeric) { // running sums over the bins: inside the lane, then over the lanes' totals
#pragma unroll
        for (int i = 1; i < CH; ++i) { g[i] += g[i - 1]; h[i] += h[i - 1]; w[i] += w[i - 1]; }
        double tg = g[CH - 1], th = h[CH - 1], tw = w[CH - 1];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double ug = __shfl_up_sync(FULL, tg, d), uw = __shfl_up_sync(FULL, tw, d), uh = elide ? 0.0 : __shfl_up_sync(FULL, th, d);
            if (lane >= d) { tg += ug; th += uh; tw += uw; }
        }
        tg = __shfl_up_sync(FULL, tg, 1); tw = __shfl_up_sync(FULL, tw, 1); if (!elide) th = __shfl_up_sync(FULL, th, 1);
        if (lane > 0) {
#pragma unroll
            for (int i = 0; i < CH; ++i) { g[i] += tg; h[i] += th; w[i] += tw; }
        }
        if (elide) {
#pragma unroll
            for (int i = 0; i < CH; ++i) h[i] = 2.0 * w[i];
        }
    }
    const double gain_p = term_gh(sg, sh, sw, a.lambda, a.L2);
    const int b_max = numeric ? B - 1 : B;
    double lg = a.gamma, bg = 0.0, bh = 0.0, bw = 0.0;
    int lb = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        const double w_l = w[i], w_r = sw - w_l;
        double v = terms_gh(g[i], h[i], w_l, sg - g[i], sh - h[i], w_r, a.lambda, a.L2);
        bool ok = bin0 + i < b_max && w_l > a.min_weight && w_r > a.min_weight;
        if (constraint != 0) { // pred_scalar on left / right sums (src/predict.jl:205-208, 235-238)
            const double pl = a.neb * g[i] / fmax(DBL_EPSILON, h[i] + a.lambda * w_l + a.L2);
            const double pr = a.neb * (sg - g[i]) / fmax(DBL_EPSILON, (sh - h[i]) + a.lambda * w_r + a.L2);
            ok = ok && ((constraint == -1 && pl > pr) || (constraint == 1 && pl < pr));
        }
        v -= gain_p;
        if (ok && v > lg) { lg = v; lb = bin0 + i; bg = g[i]; bh = h[i]; bw = w_l; }
    }
    const int mine = lb;
    warp_first_max(lg, lb);
    if constexpr (CL) { // to every CTA
        const int src = min(lb / CH, 31);
        bg = __shfl_sync(FULL, bg, src); bh = __shfl_sync(FULL, bh, src); bw = __shfl_sync(FULL, bw, src);
        if (lane < (int)gridDim.x) {
            const uint32_t rec = remote(S_BEST + ((size_t)j * F + f) * 3, lane);
            remote_put(rec, lg, lb == 0x7fffffff ? -1.0 : (double)lb);
            remote_put(rec + 16, bg, bh);
            remote_put(rec + 32, bw, 0.0);
        }
    } else {
        double2 *rec = a.best + (((size_t)set * a.M + j) * F + f) * 3;
        if (lane == 0) rec[0] = make_double2(lg, lb == 0x7fffffff ? -1.0 : (double)lb);
        if (mine == lb && lb != 0x7fffffff) { rec[1] = make_double2(bg, bh); rec[2] = make_double2(bw, 0.0); }
    }
}

template <int NQ, bool CNT, bool PACK, int CH, bool CL>
__device__ __forceinline__ void scan_level(const GrowArgs &a, const Pairs &pr, int level, int set, int np, int g) {
    const int both = level > 1 ? 1 : 0, wid = threadIdx.x >> 5;
    const bool own = CL || a.NR == 1; // the CTA's own features; else all (pair, feature, child) over all CTAs
    // one cluster: features r, r + NR, r + 2 NR .. of the group
    const int r = CL ? (int)blockIdx.x / a.NG : 0, stride = CL ? a.NR : 1, in_group = min(4 << a.lw, a.F - g * (4 << a.lw));
    const int f0 = own ? g * (4 << a.lw) + r : 0, nf = CL ? (in_group - r + stride - 1) / stride : own ? in_group : a.F;
    if (nf <= 0) return;
    const int total = (np * nf) << both, step = own ? NW : NW * (int)gridDim.x;
    const float per_nf = 1.0f / (float)nf;
    for (int t = own ? wid : wid * (int)gridDim.x + (int)blockIdx.x; t < total; t += step) {
        const int which = t & both, e = t >> both, s = (int)(((float)e + 0.5f) * per_nf), lf = e - s * nf, f = f0 + lf * stride; // (e / nf: fewer than 2^20 of them)
        if (!pr.dec()[s]) continue;
        const int c = pr.build()[s] ^ which, j = 2 * s + c;
        scan<NQ, CNT, PACK, CH, CL>(a, level, set, s, f, lf, (1 << (level - 1)) + j, j, which != 0, pr.sum() + 3 * j);
    }
}

// ---------------------------------------------------------------------------------------------- decisions
__device__ __forceinline__ float leaf_of(const GrowArgs &a, double g, double h, double w) { return (float)(a.neb * g / fmax(DBL_EPSILON, h + a.lambda * w + a.L2)); }

// Every CTA decides every node, a warp per node, and so knows the slots of the next level.  The child with the smaller weight is built, the left one when they are equal (with unit weights the reference's rule on
// row counts, src/fit.jl:123-129).  Returns whether the thread's warp has split a node.
template <bool CL>
__device__ __forceinline__ bool decide(const GrowArgs &a, const Pairs &pr, const Pairs &nx, int level, int set) {
    const int lane = threadIdx.x & 31, F = a.F, nodes = 1 << (level - 1);
    bool any = false;
    auto records = [&](int j) { return CL ? S_BEST + (size_t)j * F * 3 : a.best + ((size_t)set * a.M + j) * F * 3; };
    auto ld = [](const double2 *p) { if constexpr (CL) return *p; else return __ldcg(p); };
    double2 q0, q1, q2; // the first 32 features' records of the warp's next node are on their way while it decides one
    auto ahead = [&](int j) {
        q0 = make_double2(0.0, -1.0);
        if (j < nodes && lane < F && pr.dec()[j >> 1]) { const double2 *r = records(j) + 3 * lane; q0 = ld(r); q1 = ld(r + 1); q2 = ld(r + 2); }
    };
    ahead(threadIdx.x >> 5);
    for (int j = threadIdx.x >> 5; j < nodes; j += NW) {
        const int n = nodes + j, s = j >> 1;
        if (!pr.dec()[s]) {
            if (lane == 0) { nx.dec()[j] = 0u; nx.st()[j] = nx.mid()[j] = nx.en()[j] = pr.en()[s]; }
            ahead(j + NW);
            continue;
        }
        const double2 *rec = records(j);
        double2 l1 = make_double2(0.0, 0.0), l2 = l1; // left sums of the lane's best feature
        double s0, s1, s2;
        if (level == 1) { s0 = CL ? S_ROOT[0] : __ldcg(a.nsum + 3); s1 = CL ? S_ROOT[1] : __ldcg(a.nsum + 4); s2 = CL ? S_ROOT[2] : __ldcg(a.nsum + 5); }
        else { s0 = pr.sum()[3 * j]; s1 = pr.sum()[3 * j + 1]; s2 = pr.sum()[3 * j + 2]; }
        double bg = a.gamma;
        int bs = 0x7fffffff, bb = -1;
        if (q0.y >= 0.0 && q0.x > bg) { bg = q0.x; bs = lane; bb = (int)q0.y; l1 = q1; l2 = q2; }
        ahead(j + NW);
#pragma unroll 2
        for (int f = lane + 32; f < F; f += 32) {
            const double2 r = ld(rec + 3 * f), r1 = ld(rec + 3 * f + 1), r2 = ld(rec + 3 * f + 2);
            if (r.y >= 0.0 && r.x > bg) { bg = r.x; bs = f; bb = (int)r.y; l1 = r1; l2 = r2; }
        }
        warp_first_max(bg, bs);
        const bool has = bs != 0x7fffffff;
        const uint32_t feat = has ? S_FEAT[bs] : 0u;
        const int src = bs & 31;
        bb = __shfl_sync(FULL, bb, src);
        l1.x = __shfl_sync(FULL, l1.x, src); l1.y = __shfl_sync(FULL, l1.y, src); l2.x = __shfl_sync(FULL, l2.x, src);
        any = any || has;
        if (lane != 0) continue;
        const uint32_t packed = has ? (feat & 0xffffu) | ((uint32_t)(bb + 1) << 16) | (1u << 24) | (((feat >> 16) & 1u) << 25) : 0u;
        const double r0 = s0 - l1.x, r1 = s1 - l1.y, r2 = s2 - l2.x;
        nx.dec()[j] = packed;
        S_TREE[n - 1] = packed;
        if (!has) S_VALUE[n - 1] = leaf_of(a, s0, s1, s2);
        if (level + 1 == a.D) { // children at max depth are leaves (src/fit.jl:74-82)
            if (has) { S_TREE[2 * n - 1] = S_TREE[2 * n] = 0u; S_VALUE[2 * n - 1] = leaf_of(a, l1.x, l1.y, l2.x); S_VALUE[2 * n] = leaf_of(a, r0, r1, r2); }
        } else {
            const int c = level == 1 ? 0 : j & 1, st = c ? pr.mid()[s] : pr.st()[s], en = c ? pr.en()[s] : pr.mid()[s];
            double *ns = nx.sum() + 6 * j;
            ns[0] = l1.x; ns[1] = l1.y; ns[2] = l2.x; ns[3] = r0; ns[4] = r1; ns[5] = r2;
            nx.build()[j] = r2 >= l2.x ? 0 : 1;
            nx.st()[j] = has ? st : en; nx.mid()[j] = has ? st : en; nx.en()[j] = en; // mid: grows while the rows are placed
            S_CR[j] = en;
        }
        if (level == 1) { pr.sum()[0] = s0; pr.sum()[1] = s1; pr.sum()[2] = s2; }
        S_OUT[j] = make_double4(l1.x, l1.y, l2.x, bg);
    }
    return any;
}
// What a level has decided goes to the tree in global memory while the CTA waits for others
__device__ __forceinline__ void record(const GrowArgs &a, const Pairs &pr, int level) {
    const int nodes = 1 << (level - 1), j = (int)(blockIdx.x + gridDim.x * threadIdx.x);
    if (j >= nodes || !pr.dec()[j >> 1]) return; // CTA j % gridDim.x writes what belongs to node j (the grid has no fewer than 2^9 threads)
    const int n = nodes + j;
    const uint32_t packed = S_TREE[n - 1];
    const double s0 = pr.sum()[3 * j], s1 = pr.sum()[3 * j + 1], s2 = pr.sum()[3 * j + 2];
    a.t_w[n - 1] = (float)s2;
    if (!packed) { a.t_pred[n - 1] = S_VALUE[n - 1]; return; }
    const double4 l = S_OUT[j];
    double *c = a.nsum + (size_t)6 * n;
    c[0] = l.x; c[1] = l.y; c[2] = l.z; c[3] = s0 - l.x; c[4] = s1 - l.y; c[5] = s2 - l.z;
    a.t_gain[n - 1] = (float)l.w; a.t_bin[n - 1] = (uint8_t)((packed >> 16) & 0xffu); a.t_feat[n - 1] = (int32_t)(packed & 0xffffu) + 1; a.t_split[n - 1] = 1; a.t_packed[n - 1] = packed;
    if (level + 1 == a.D) {
        a.t_pred[2 * n - 1] = S_VALUE[2 * n - 1]; a.t_pred[2 * n] = S_VALUE[2 * n];
        a.t_w[2 * n - 1] = (float)l.z; a.t_w[2 * n] = (float)(s2 - l.z);
    } else atomicAdd(&a.plan[level + 1].nbuild, 1);
}

// The CTA's rows to the children of the nodes that split: left rows from the start of the node's places, right rows from its end.  Every
// warp takes a stretch of adjacent places, up to U tiles of one node at a time: one reservation per side for all of them.  Rows whose
// way ends here -- nodes that did not split, `last`: children of the last level -- have their leaf noted if they are among the rows
// [u0, u1) that this CTA updates.
__device__ __forceinline__ void place(const GrowArgs &a, const Pairs &pr, const Pairs &nx, const uint16_t *in, uint16_t *out, int level, int cnt, const uint8_t *xrows, bool last, int u0,
                                      int u1) {
    constexpr int U = 8;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, each = ((cnt + 32 * NW - 1) / (32 * NW)) * 32, nodes = 1 << (level - 1);
    const unsigned below = (1u << lane) - 1u;
    int p = wid * each, j = 0;
    const int pend = min(cnt, p + each);
    if (p >= pend) return;
    for (; j < nodes; j += 32) { // first node that ends behind p
        const int i = j + lane, s = i >> 1;
        const unsigned m = __ballot_sync(FULL, i < nodes && ((i & 1) ? pr.en()[s] : pr.mid()[s]) > p);
        if (m) { j += __ffs(m) - 1; break; }
    }
    auto end_of = [&](int i) { return (i & 1) ? pr.en()[i >> 1] : pr.mid()[i >> 1]; };
    auto start_of = [&](int i) { return (i & 1) ? pr.mid()[i >> 1] : pr.st()[i >> 1]; };
    const uint32_t n_up = (uint32_t)(u1 - u0);
    while (p < pend) {
        while (j < nodes && end_of(j) <= p) ++j;
        if (j >= nodes) break;
        p = max(p, start_of(j));
        if (p >= pend) break;
        const int lim = min(pend, end_of(j));
        if (p >= lim) continue; // nothing of the node is left, and what lies before it belongs to nodes that have ended
        if (lim - p >= 64 || lim == pend) { // one node
            const uint32_t dec = nx.dec()[j], bin = (dec >> 16) & 0xffu, lo = (dec >> 25) & 1u ? 0u : bin, span = bin - lo; // left: lo <= x <= bin
            const uint8_t *xf = xrows + (size_t)(dec & 0xffffu) * a.n;
            if (dec && !last) {
                for (; p < lim; p += 32 * U) {
                    uint32_t row[U], x[U];
                    unsigned l[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) { const int q = p + 32 * u + lane; row[u] = q < lim ? in[q] : 0xffffu; }
#pragma unroll
                    for (int u = 0; u < U; ++u) x[u] = row[u] != 0xffffu ? (uint32_t)__ldg(xf + row[u]) : 0u;
                    int nl = 0;
#pragma unroll
                    for (int u = 0; u < U; ++u) { l[u] = __ballot_sync(FULL, row[u] != 0xffffu && x[u] - lo <= span); nl += __popc(l[u]); }
                    const int nr = min(lim - p, 32 * U) - nl;
                    int at = 0;
                    if (lane == 0) at = atomicAdd(nx.mid() + j, nl);
                    if (lane == 1) at = atomicSub(S_CR + j, nr) - nr;
                    int dl = __shfl_sync(FULL, at, 0), dr = __shfl_sync(FULL, at, 1);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int b = __popc(l[u] & below);
                        if (row[u] != 0xffffu) out[(l[u] >> lane) & 1u ? dl + b : dr + lane - b] = (uint16_t)row[u];
                        dl += __popc(l[u]); dr += 32 - __popc(l[u]);
                    }
                }
            } else if (a.whole) {
                const uint32_t id = dec ? 2u * (uint32_t)(nodes + j) : (uint32_t)(nodes + j);
                for (; p < lim; p += 32 * U) {
                    uint32_t row[U], x[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) { const int q = p + 32 * u + lane; row[u] = q < lim ? (uint32_t)in[q] - (uint32_t)u0 : 0xffffffffu; }
#pragma unroll
                    for (int u = 0; u < U; ++u) x[u] = dec && row[u] < n_up ? (uint32_t)__ldg(xf + u0 + row[u]) : 0u;
#pragma unroll
                    for (int u = 0; u < U; ++u) if (row[u] < n_up) S_LEAF[row[u]] = (uint16_t)(id + (dec && x[u] - lo > span ? 1u : 0u));
                }
            }
            p = lim;
        } else { // several small ones: every lane finds its row's node, lanes of one child share a reservation
            uint32_t key[2], row[2], dec[2], x[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int q = p + 32 * u + lane;
                int l = j, r = nodes - 1; // first node that ends behind q
                while (l < r) { const int m = (l + r) >> 1; if (end_of(m) > q) r = m; else l = m + 1; }
                const bool act = q < pend && q < end_of(l) && q >= start_of(l);
                row[u] = act ? (uint32_t)in[q] : 0xffffu;
                dec[u] = act ? nx.dec()[l] : 0u;
                key[u] = act ? (uint32_t)l + 1u : 0u;
                const bool look = dec[u] && (!last || row[u] - (uint32_t)u0 < n_up);
                x[u] = look ? (uint32_t)__ldg(xrows + (size_t)(dec[u] & 0xffffu) * a.n + row[u]) : 0u;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t bin = (dec[u] >> 16) & 0xffu, lo = (dec[u] >> 25) & 1u ? 0u : bin, child = x[u] - lo <= bin - lo ? 0u : 1u;
                const bool moves = dec[u] && !last;
                if (key[u] && !moves && a.whole && row[u] - (uint32_t)u0 < n_up) {
                    const uint32_t n = (uint32_t)nodes + key[u] - 1u;
                    S_LEAF[row[u] - u0] = (uint16_t)(dec[u] ? 2u * n + child : n);
                }
                if (last) continue;
                const unsigned peers = __match_any_sync(FULL, moves ? 2u * key[u] + child : 0u);
                const int c = __popc(peers);
                int at = 0;
                if (moves && (peers & below) == 0u) at = child ? atomicSub(S_CR + (key[u] - 1u), c) - c : atomicAdd(nx.mid() + (key[u] - 1u), c);
                at = __shfl_sync(FULL, at, __ffs(peers) - 1);
                if (moves) out[at + __popc(peers & below)] = (uint16_t)row[u];
            }
            p += 64;
        }
    }
}

// Predictions of the CTA's share of its rows and the gradients of the next round (`predict!`, src/predict.jl:1-62; `update_grads!`)
template <int NQ>
__device__ __forceinline__ void update_rows(const GrowArgs &a, long long row0, int u0, int u1, bool unit_w) {
    unsigned m0 = 0u, m1 = 0u; // bits of the largest |g|, |h| of this thread's rows (a NaN is larger than all numbers)
    for (int r = u0 + (int)threadIdx.x; r < u1; r += T) {
        const long long i = row0 + r;
        const uint32_t id = S_LEAF[r - u0];
        float p = a.pred[i], g[2];
        pred_add(a.loss, 1, &p, S_VALUE + (id - 1));
        a.pred[i] = p;
        a.nidx[i] = id;
        if (!a.next_grads) continue;
        float *rec = a.grad + (size_t)i * NQ;
        const float w = unit_w ? 1.0f : rec[NQ - 1];
        switch (a.loss) { // one loss at a time: grad_row folds to its formula
        case EVB_MSE: grad_row(EVB_MSE, 1, a.elide != 0, &p, a.y, 1, i, w, g, a.alpha); break;
        case EVB_LOGLOSS: grad_row(EVB_LOGLOSS, 1, false, &p, a.y, 1, i, w, g, a.alpha); break;
        case EVB_POISSON: grad_row(EVB_POISSON, 1, false, &p, a.y, 1, i, w, g, a.alpha); break;
        case EVB_GAMMA: grad_row(EVB_GAMMA, 1, false, &p, a.y, 1, i, w, g, a.alpha); break;
        default: grad_row(EVB_TWEEDIE, 1, false, &p, a.y, 1, i, w, g, a.alpha);
        }
        rec[0] = g[0];
        m0 = max(m0, __float_as_uint(fabsf(g[0])));
        if (NQ > 1 && a.ng > 1) { rec[1] = g[1]; m1 = max(m1, __float_as_uint(fabsf(g[1]))); }
    }
    if (!a.next_grads) return;
    unsigned *s = reinterpret_cast<unsigned *>(S_MISC + M_MAX);
    m0 = __reduce_max_sync(FULL, m0); m1 = __reduce_max_sync(FULL, m1);
    if ((threadIdx.x & 31) == 0) { atomicMax(s, m0); atomicMax(s + 1, m1); }
    __syncthreads();
    if (threadIdx.x < a.ng && s[threadIdx.x] > *(volatile unsigned *)(a.gmax_next + threadIdx.x)) atomicMax(a.gmax_next + threadIdx.x, s[threadIdx.x]);
}

// The CTA's share of the evaluation rows: their predictions and its part of the metric's sums (k_eval_tree)
__device__ __forceinline__ void evaluate(const GrowArgs &a) {
    const int rw = a.ev_RS >> 2, pitch = rw + 1, room = a.o_x / (4 * pitch); // rows that fit where the images were
    const long long e0 = a.ev_n * blockIdx.x / gridDim.x, e1 = a.ev_n * (blockIdx.x + 1) / gridDim.x;
    double sv = 0.0, sw = 0.0;
    const bool staged = room >= 32;
    for (long long b0 = e0; b0 < e1; b0 += staged ? room : e1 - e0) {
        const long long b1 = staged ? min(e1, b0 + room) : e1;
        if (staged) {
            __syncthreads();
            const uint4 *src = reinterpret_cast<const uint4 *>(a.ev_xT + (size_t)b0 * a.ev_RS);
            const int cpr = rw >> 2, chunks = (int)(b1 - b0) * cpr;
#pragma unroll 4
            for (int c = threadIdx.x; c < chunks; c += T) {
                const uint4 v = __ldg(src + c);
                const int r = c / cpr;
                uint32_t *d = S_IMG + r * pitch + (c - r * cpr) * 4;
                d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
            }
            __syncthreads();
        }
        for (long long i = b0 + threadIdx.x; i < b1; i += T) {
            const uint8_t *x = staged ? reinterpret_cast<const uint8_t *>(S_IMG + (int)(i - b0) * pitch) : a.ev_xT + (size_t)i * a.ev_RS;
            float p = a.ev_pred[i];
            pred_add(a.loss, 1, &p, S_VALUE + (traverse(S_TREE, x) - 1));
            a.ev_pred[i] = p;
            const float w = a.ev_w ? a.ev_w[i] : 1.0f;
            sv += (double)metric_row(a.ev_metric, 1, &p, a.ev_y, 1, i, w, a.alpha);
            sw += (double)w;
        }
    }
    sv = warp_sum(sv); sw = warp_sum(sw);
    if ((threadIdx.x & 31) == 0) { S_RED[threadIdx.x >> 5] = sv; S_RED[NW + (threadIdx.x >> 5)] = sw; }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int w = 0; w < NW; ++w) t += S_RED[threadIdx.x * NW + w];
        a.ev_part[2 * blockIdx.x + threadIdx.x] = t;
    }
}

// bins of the CTA's features, a 32-bit word for four of them: [word][row]
__device__ __forceinline__ uint32_t column(const GrowArgs &a, int f) { return a.js_inline ? a.js[f] : a.js0 ? a.js0[f] : (uint32_t)f; }
__device__ __forceinline__ void load_bins(const GrowArgs &a, uint32_t *x, int f0, long long row0, int nr) {
    const int quads = (nr + 3) >> 2;
    for (int w = 0; w < 1 << a.lw; ++w) {
        const uint8_t *col[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { const int f = f0 + 4 * w + k; col[k] = f < a.F ? a.xC + (size_t)column(a, f) * a.n + row0 : nullptr; }
#pragma unroll 4
        for (int e = threadIdx.x; e < quads; e += T) {
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = 0u;
                if (col[k]) { // four rows at any byte: two aligned words (the matrix ends with room for the second one)
                    const uintptr_t p = reinterpret_cast<uintptr_t>(col[k] + 4 * e);
                    const uint32_t *d = reinterpret_cast<const uint32_t *>(p & ~(uintptr_t)3);
                    v[k] = __funnelshift_r(__ldg(d), __ldg(d + 1), 8 * (uint32_t)(p & 3));
                }
            }
            const uint32_t a0 = __byte_perm(v[0], v[1], 0x5140), a1 = __byte_perm(v[2], v[3], 0x5140), b0 = __byte_perm(v[0], v[1], 0x7362), b1 = __byte_perm(v[2], v[3], 0x7362);
            *reinterpret_cast<uint4 *>(x + (size_t)w * a.rpc + 4 * e) =
                make_uint4(__byte_perm(a0, a1, 0x5410), __byte_perm(a0, a1, 0x7632), __byte_perm(b0, b1, 0x5410), __byte_perm(b0, b1, 0x7632));
        }
    }
}

__device__ __forceinline__ void clear_sums(const GrowArgs &a, int NQ, int set, int np, int level) {
    const size_t per = (size_t)a.F * a.B, i0 = (size_t)blockIdx.x * T + threadIdx.x, st = (size_t)gridDim.x * T;
    unsigned long long *s = a.sum + (size_t)set * a.sum_set;
    uint32_t *c = a.cnt + (size_t)set * a.cnt_set;
    for (size_t i = i0; i < np * per * NQ; i += st) s[i] = 0ull;
    for (size_t i = i0; i < np * per; i += st) c[i] = 0u;
    if (!a.low) return;
    unsigned long long *l = a.low + (size_t)set * a.sum_set;
    for (int k = 0; k < np; ++k)
        if (__ldcg(a.lowflag + evb_low_slot(level) + k) != 0u)
            for (size_t i = i0; i < per * NQ; i += st) l[k * per * NQ + i] = 0ull;
}

// one cluster, several ranges of rows: the sums that have been scanned
template <int NQ, bool PACK>
__device__ __forceinline__ void clear_own(const GrowArgs &a, int set, int np, int g) {
    for (int i = threadIdx.x; i < np * a.fo * NQ * a.B; i += T) S_SUM[i] = 0ull;
    for (int i = threadIdx.x; i < np * a.fo * a.B; i += T) S_CNTS[i] = 0u;
    if constexpr (!PACK) {
        const int r = (int)blockIdx.x / a.NG, end = min((g + 1) * (4 << a.lw), a.F);
        for (int s = 0; s < np; ++s) {
            if (!S_LOW[s]) continue;
            for (int f = g * (4 << a.lw) + r; f < end; f += a.NR)
                for (int i = threadIdx.x; i < NQ * a.B; i += T) a.low[(size_t)set * a.sum_set + ((size_t)s * a.F + f) * NQ * a.B + i] = 0ull;
        }
    }
}

// CL: the grid is one cluster; sums, histograms and best splits are exchanged through the CTAs' shared memory and the barriers are the cluster's
template <int NQ, bool CNT, bool PACK, int CH, bool CL>
__global__ void __launch_bounds__(T, 1) k_grow(GrowArgs a) {
    const int g = blockIdx.x % a.NG, f0 = g * (4 << a.lw);
    const long long row0 = (long long)(blockIdx.x / a.NG) * a.rpc;
    const int nr = (int)min((long long)a.rpc, a.n - row0), lane = threadIdx.x & 31;
    const int per_up = ((a.rpc >> 5) + a.NG - 1) / a.NG * 32, u0 = min(g * per_up, nr), u1 = min(u0 + per_up, nr); // rows this CTA updates
    if (blockIdx.x == 0 && threadIdx.x < NQ) a.gmax_next[threadIdx.x] = (int)threadIdx.x < a.ng ? 0u : a.gmax[threadIdx.x]; // (weights keep theirs)
    if (threadIdx.x == 0) {
        S_MISC[M_OK] = *(volatile int *)a.err == 0;
        S_MISC[M_LEFT] = 0; S_MISC[M_CNT] = 0; S_MISC[M_MAX] = 0; S_MISC[M_MAX + 1] = 0;
        const Pairs root = S_PAIRS(0);
        root.dec()[0] = 1u; root.build()[0] = 0; root.st()[0] = 0;
    }
    // (each warp has one trip to memory of these beside its rows: the last warps the features, warp 1 the scales)
    for (int f = T - 1 - (int)threadIdx.x; f < a.F; f += T) {
        const uint32_t feat = column(a, f);
        const int mono = a.mono[feat];
        S_FEAT[f] = feat | (a.feattypes[feat] != 0 ? 1u << 16 : 0u) | (mono >= -1 && mono <= 1 ? (uint32_t)(mono + 1) : 3u) << 17;
    }
    if (a.whole) { // a tree without nodes (k_tree_begin); what is written to it comes behind a barrier
        for (int i = (int)blockIdx.x * T + threadIdx.x; i < a.nn + 2; i += (int)gridDim.x * T) {
            for (int c = 0; c < 3; ++c) a.nsum[3 * i + c] = 0.0;
            if (i < a.nn) { a.t_feat[i] = 0; a.t_bin[i] = 0; a.t_split[i] = 0; a.t_gain[i] = 0.f; a.t_w[i] = 0.f; a.t_packed[i] = 0u; a.t_pred[i] = 0.f; }
            if (i >= 1 && i <= a.D) {
                const int root = i == 1 ? 1 : 0;
                a.plan[i].nbuild = root; a.plan[i].npl = root; a.plan[i].R = root ? a.n : 0; a.plan[i].total = root ? (int)a.n : 0; a.plan[i].n_sel = root ? (int)a.n : 0;
            }
        }
    }
    if (threadIdx.x >= 32 && threadIdx.x < 32 + NQ) {
        const int c = threadIdx.x - 32;
        double unit;
        const Quant k = quant_of(a.gmax[c], PACK, a.hb, a.round_bits, &unit);
        S_QUANT[c] = k;
        S_UNIT[c] = unit;
        S_INF[c] = k.kind == QK_INF;
    }
    // rows on their way to shared memory before anything waits: gradients as they are, scaled in place when the scale is known
    const float *rec = a.grad + (size_t)row0 * NQ;
#pragma unroll 4
    for (int i = threadIdx.x; i < nr >> 2; i += T) { // four records at a time
        float v[4 * NQ];
#pragma unroll
        for (int c = 0; c < NQ; ++c) {
            const float4 t = __ldcg(reinterpret_cast<const float4 *>(rec) + (size_t)i * NQ + c);
            v[4 * c] = t.x; v[4 * c + 1] = t.y; v[4 * c + 2] = t.z; v[4 * c + 3] = t.w;
        }
#pragma unroll
        for (int c = 0; c < NQ; ++c) *reinterpret_cast<float4 *>(S_Q + c * a.rpc + 4 * i) = make_float4(v[c], v[NQ + c], v[2 * NQ + c], v[3 * NQ + c]);
    }
    for (int i = (nr & ~3) + threadIdx.x; i < nr; i += T) {
#pragma unroll
        for (int c = 0; c < NQ; ++c) S_Q[c * a.rpc + i] = __float_as_int(__ldcg(rec + (size_t)i * NQ + c));
    }
    load_bins(a, S_X, f0, row0, nr);
    {
        uint4 *z = reinterpret_cast<uint4 *>(S_IMG);
        for (int i = threadIdx.x; i < a.o_x / 16; i += T) z[i] = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (CL) {
            const int slots = a.M / 2;
            for (int i = threadIdx.x; i < slots * a.fo * NQ * a.B; i += T) S_SUM[i] = 0ull;
            for (int i = threadIdx.x; i < slots * a.fo * a.B + slots; i += T) S_CNTS[i] = 0u;
        }
    }
    __syncthreads();
    if (!S_MISC[M_OK]) { // the tree before this one was given up: its barriers have counts and its sums rows left
        if (a.pub_dst && threadIdx.x == 0) reinterpret_cast<volatile int *>(a.pub_dst)[a.pub_err] = *(volatile int *)a.err;
        return;
    }
    {
        Quant k[NQ];
#pragma unroll
        for (int c = 0; c < NQ; ++c) k[c] = S_QUANT[c];
#pragma unroll 2
        for (int i = threadIdx.x; i < nr; i += T) {
#pragma unroll
            for (int c = 0; c < NQ; ++c) S_Q[c * a.rpc + i] = quant(k[c], __int_as_float(S_Q[c * a.rpc + i]), a.signs + c, a.qinv + c);
        }
    }
    if (!a.mask) for (int i = threadIdx.x; i < nr; i += T) S_IDX(0)[i] = (uint16_t)i;
    else
        for (int i0 = (int)threadIdx.x - lane; i0 < nr; i0 += T) {
            const int i = i0 + lane;
            const bool in = i < nr && (int)__ldg(a.mask + row0 + i) <= a.cond;
            const unsigned m = __ballot_sync(FULL, in);
            int at = 0;
            if (lane == 0) at = atomicAdd(S_MISC + M_CNT, __popc(m));
            at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (in) S_IDX(0)[at] = (uint16_t)i;
        }
    __syncthreads();
    if (threadIdx.x == 0) { const int c = a.mask ? S_MISC[M_CNT] : nr; const Pairs root = S_PAIRS(0); root.mid()[0] = c; root.en()[0] = c; }
    if constexpr (CL) cluster_barrier(); // the sums of all CTAs are empty
    else __syncthreads();

    const int cnt = S_PAIRS(0).en()[0];
    int np = 1, done_np = 0; // slots of the level and of the one before
    unsigned arrivals = 0;
    for (int level = 1; level < a.D; ++level) {
        const int cur = (level - 1) & 1, set = level & 1;
        const Pairs pr = S_PAIRS(cur), nx = S_PAIRS(cur ^ 1);
        const uint16_t *idx = S_IDX(cur);
        auto write_out = [&] {
            if (level == 1) return;
            record(a, nx, level - 1); // (nx: still the level before)
            if (g != 0) return;
            int rows = 0; // of this CTA's range that were added up, for the host's statistics
            for (int k = threadIdx.x; k < np; k += T) if (pr.dec()[k]) rows += pr.build()[k] ? pr.en()[k] - pr.mid()[k] : pr.mid()[k] - pr.st()[k];
            if (rows > 0) atomicAdd(reinterpret_cast<unsigned long long *>(&a.plan[level].R), (unsigned long long)rows);
        };
        auto hist = [&] {
            const int lc = a.lc[level];
            if (lc == 0) direct_level<NQ, CNT, PACK, CL>(a, pr, idx, np, set, g, level);
            else if (CL || a.lw == 0) {
                if (lc == 5) hist_level<NQ, CNT, PACK, 0, 5, CL>(a, pr, idx, np, set, g, level);
                else if (lc == 4) hist_level<NQ, CNT, PACK, 0, 4, CL>(a, pr, idx, np, set, g, level);
                else hist_level<NQ, CNT, PACK, 0, 3, CL>(a, pr, idx, np, set, g, level);
            } else if (a.lw == 1) {
                if (lc == 5) hist_level<NQ, CNT, PACK, 1, 5, CL>(a, pr, idx, np, set, g, level);
                else if (lc == 4) hist_level<NQ, CNT, PACK, 1, 4, CL>(a, pr, idx, np, set, g, level);
                else hist_level<NQ, CNT, PACK, 1, 3, CL>(a, pr, idx, np, set, g, level);
            } else {
                if (lc == 5) hist_level<NQ, CNT, PACK, 2, 5, CL>(a, pr, idx, np, set, g, level);
                else hist_level<NQ, CNT, PACK, 2, 4, CL>(a, pr, idx, np, set, g, level);
            }
        };
        if constexpr (CL) {
            hist();
            cluster_barrier();
        } else {
            hist();
            if (a.NR > 1) {
                if (!grid_barrier(a, S_MISC + M_OK, ++arrivals, [] {})) return;
                if (level > 1) clear_sums(a, NQ, set ^ 1, done_np, level - 1);
            }
        }
        if (level == 1 && (S_INF[0] | S_INF[NQ > 1 ? 1 : 0] | S_INF[NQ - 1])) { // infinities of both signs: no sum means anything
            if (threadIdx.x < NQ && *(volatile unsigned *)(a.signs + threadIdx.x) == 3u && a.gmax[threadIdx.x] >= 0x7f800000u) S_UNIT[threadIdx.x] = __longlong_as_double(0x7ff8000000000000ll);
            __syncthreads();
        }
        scan_level<NQ, CNT, PACK, CH, CL>(a, pr, level, set, np, g);
        if constexpr (CL) {
            if (a.NR > 1) {
                __syncthreads();
                clear_own<NQ, PACK>(a, set, np, g);
            }
            if constexpr (!PACK) { __syncthreads(); for (int s = threadIdx.x; s < np; s += T) S_LOW[s] = 0u; }
            cluster_barrier(write_out);
        } else if (gridDim.x > 1) { if (!grid_barrier(a, S_MISC + M_OK, ++arrivals, write_out)) return; }
        else { write_out(); __syncthreads(); }
        const bool split = __syncthreads_or(decide<CL>(a, pr, nx, level, set)) != 0;
        const bool last = level + 1 == a.D || !split;
        if (!last || a.whole) place(a, pr, nx, idx, S_IDX(cur ^ 1), level, cnt, a.xC + row0, last, u0, u1);
        if (last) { // these were the last sums
            record(a, pr, level);
            if (!CL && a.NR > 1) clear_sums(a, NQ, set, np, level);
            break;
        }
        done_np = np;
        np = 1 << (level - 1);
        __syncthreads();
    }
    if (a.whole) {
        __syncthreads();
        update_rows<NQ>(a, row0, u0, u1, CNT || PACK);
        if (a.ev_n > 0) evaluate(a);
    }
    if constexpr (CL) {
        cluster_barrier();
        if (blockIdx.x != 0) return;
    } else { // the CTA that is done last hands the tree over
        __syncthreads();
        if (threadIdx.x == 0) S_MISC[M_OK] = arrive(a.bar + 1) == gridDim.x - 1;
        __syncthreads();
        if (!S_MISC[M_OK]) return;
        if (threadIdx.x < 2) a.bar[threadIdx.x] = 0u;
        if (a.low) for (int i = threadIdx.x; i < a.nn + 2; i += T) a.lowflag[i] = 0u;
    }
    if (a.ev_n > 0 && threadIdx.x < 32) {
        double v = 0.0, w = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) { v += __ldcg(a.ev_part + 2 * b); w += __ldcg(a.ev_part + 2 * b + 1); }
        v = warp_sum(v); w = warp_sum(w);
        if (threadIdx.x == 0) { a.ev_sum[0] = v; a.ev_sum[1] = w; }
    }
    __syncthreads();
    publish(a.pub_src, a.pub_dst, a.pub_n);
}

constexpr int SMEM_MAX = 227 * 1024, MAX_CLUSTER = 16;
template <int NQ, bool CNT, bool PACK, int CH, bool CL>
cudaError_t launch(const GrowArgs *a, int grid, size_t smem, cudaStream_t st, int *clusters) {
    cudaError_t e = cudaFuncSetAttribute(k_grow<NQ, CNT, PACK, CH, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
    if (e == cudaSuccess && CL) e = cudaFuncSetAttribute(k_grow<NQ, CNT, PACK, CH, CL>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid); c.blockDim = dim3(T); c.dynamicSmemBytes = smem; c.stream = st;
    cudaLaunchAttribute at;
    if (CL) { at.id = cudaLaunchAttributeClusterDimension; at.val.clusterDim.x = (unsigned)grid; at.val.clusterDim.y = at.val.clusterDim.z = 1; }
    else { at.id = cudaLaunchAttributeCooperative; at.val.cooperative = 1; }
    c.attrs = &at; c.numAttrs = 1;
    if (clusters) return cudaOccupancyMaxActiveClusters(clusters, k_grow<NQ, CNT, PACK, CH, CL>, &c);
    return cudaLaunchKernelEx(&c, k_grow<NQ, CNT, PACK, CH, CL>, *a);
}
template <int NQ, bool CNT, bool PACK, int CH>
cudaError_t launch(const evb_handle *h, const GrowGeom &g, const GrowArgs *a, int *clusters) {
    return g.cluster ? launch<NQ, CNT, PACK, CH, true>(a, g.NG * g.NR, g.smem, h->st, clusters) : launch<NQ, CNT, PACK, CH, false>(a, g.NG * g.NR, g.smem, h->st, clusters);
}
template <int NQ, bool CNT, bool PACK>
cudaError_t launch(const evb_handle *h, const GrowGeom &g, const GrowArgs *a, int *clusters) {
    return h->B <= 32 ? launch<NQ, CNT, PACK, 1>(h, g, a, clusters) : h->B <= 64 ? launch<NQ, CNT, PACK, 2>(h, g, a, clusters)
         : h->B <= 128 ? launch<NQ, CNT, PACK, 4>(h, g, a, clusters) : launch<NQ, CNT, PACK, 8>(h, g, a, clusters);
}
// launches the kernel for the handle, or (a == null) finds out how many clusters of its size the GPU holds
cudaError_t launch(const evb_handle *h, const GrowGeom &g, const GrowArgs *a, int *clusters) {
    if (h->hgeo.pack) return launch<1, true, true>(h, g, a, clusters);
    if (h->hgeo.cnt) return launch<2, true, false>(h, g, a, clusters);
    return h->nq == 2 ? launch<2, false, false>(h, g, a, clusters) : launch<3, false, false>(h, g, a, clusters);
}

// Columns of the images of every level, from what a level's rows and images cost in clocks: a reduction of a warp a clock, as often as
// the most lanes meet in a bank; an image read and cleared; 1300 for every pass over as many slots as fit `room`.  Returns the bytes used.
size_t level_columns(const evb_handle *h, GrowGeom &g, size_t room, double *clocks) {
    static const double meet[6] = {0, 0, 0, 3.8, 2.0, 1.0}; // (of 4 and 2 lanes: features of few bins meet nearly always)
    static const int choice[3][3] = {{5, 4, 3}, {5, 4, 3}, {5, 4, 0}};
    const int P = planes(h->nq, h->hgeo.cnt, h->hgeo.pack);
    size_t used = 0;
    *clocks = 0.0;
    for (int level = 1; level < h->D; ++level) {
        const int slots = evb_level_slots(level);
        const double tiles = (double)g.rpc / (level == 1 ? 32.0 : 64.0) + 0.5 * slots;
        double least = 0.0;
        size_t bytes = 0;
        if (g.NR > 1 && level > 2 && g.rpc / 2 < slots * h->B / 2) { // few rows a cell: without images
            g.lc[level] = 0;
            *clocks += tiles * (4 << g.lw) * (h->nq + 1) * 4.0;
            continue;
        }
        for (int lc : choice[g.lw]) {
            const size_t img = (size_t)(h->B + 1) * P * 4 << lc;
            const long long share = 4ll << g.lw; // columns of one replica: rows of a cell = rows x share / columns
            if (!lc || img > room || (long long)g.rpc * share >> lc > (h->hgeo.pack ? 8100 : 8050)) continue; // (more than a cell can hold)
            const int fit = (int)std::min<size_t>(room / img, slots), passes = (slots + fit - 1) / fit;
            const double c = tiles * (4 << g.lw) * P * meet[lc] / 0.87 + slots * (double)img / 64.0 + passes * 1300.0;
            if (bytes && c >= least) continue;
            least = c; bytes = fit * img; g.lc[level] = (uint8_t)lc;
        }
        if (!bytes) return 0;
        used = std::max(used, bytes);
        *clocks += least;
    }
    return (used + 127) & ~(size_t)127;
}
// bits of the high words
int grow_bits(const evb_handle *h, const GrowGeom &g) {
    long long rows = 0;
    for (int level = 1; level < h->D; ++level) if (g.lc[level]) rows = std::max(rows, ((long long)g.rpc * (4ll << g.lw) >> g.lc[level]) + 32);
    int hb = 21, log_n = 0;
    while (hb > 18 && (1ll << (31 - hb)) - 64 < rows) --hb;
    while ((1ll << log_n) < h->n) ++log_n;
    return std::min(hb, (61 - log_n) / 2);
}

// Clocks of a tree: histograms, the steps whose length is a chain of trips (12000 a level over the grid, 9000 in a cluster), rounds of
// scans and decisions beyond the first, the rows of a CTA through a step, and over the grid what meets in L2: sums of all row ranges, a
// sector per row and feature group for the way to the children.  And of the level kernels.  Both from the sweeps that gave the other
// figures here (100 shapes of 1k to 600k rows, 4 to 128 features, depths 4 to 9).
double tree_clocks(const evb_handle *h, const GrowGeom &g, double hist) {
    const int ch = h->B <= 32 ? 0 : h->B <= 64 ? 1 : h->B <= 128 ? 2 : 3;
    static const double scan[4] = {2400, 3900, 7000, 13000};
    const int scanners = g.cluster ? std::min(g.NG * std::min(g.NR, 4 << g.lw), h->F) : g.NG * g.NR;
    double c = hist + 10000.0;
    for (int level = 1; level < h->D; ++level) {
        const double slots = evb_level_slots(level), cells = std::min(slots * h->B, g.rpc / (level > 1 ? 2.0 : 1.0));
        const int nodes = evb_level_nodes(level), scans = (nodes * h->F + scanners * NW - 1) / (scanners * NW);
        c += (g.cluster ? 9000.0 : 12000.0) + 0.5 * g.rpc + scans * scan[ch] - 3900.0 + (nodes + NW - 1) / NW * 1200.0 - 1200.0;
        if (!g.cluster) c += g.NR * cells * h->F * (h->nq + 1) / 300.0 + (double)g.NG * h->n * std::min(32, nodes) / 2500.0;
    }
    return c;
}
// The estimate runs at 0.65 of what is measured, this one at 0.95; the line between them (`worth`) lies where the measured ones cross: the points below, none
// held out.  From 0.67 to 0.83 neither kernel is ahead by a rule.
// Measured, level kernels / this kernel, at estimates of: 0.47 (50k x 50, depth 6) 1.49, 0.59 (60k x 54 poisson, depth 6) 1.30, 0.67 (130k x 108,
// 32 bins, depth 7) 0.99, 0.74 (353k x 11, depth 7) 1.16, 0.80 (250k x 33 weighted, depth 7) 1.01, 0.83 (407k x 14 weighted, depth 7) 0.92; from depth
// 8 on 0.48 (16.6k x 23) 1.33, 0.54 (290k x 4, depth 9) 1.28, 0.57 (28k x 30) 1.12, 0.64 (41k x 63) 0.94, 0.70 (200k x 20) 0.90, 0.86 (140k x 17, depth 9) 0.83.
double level_kernel_clocks(const evb_handle *h) {
    return (h->D - 1) * (38000.0 + 0.0015 * (double)h->n * h->nfeats) * (h->B <= 64 ? 1.0 : h->B <= 128 ? 1.3 : 1.7);
}
double worth(const evb_handle *h) { return (h->D <= 7 ? 0.81 : 0.6) * level_kernel_clocks(h); }

// One cluster of CTAs
bool cluster_geom(const evb_handle *h, GrowGeom &best, double least) {
    const int B = h->B, D = h->D, NQ = h->nq, M = 1 << std::max(1, D - 2), hs = h->Ce != h->C ? 2 : 3, NG = (h->F + 3) / 4;
    const size_t small = (size_t)NODE_BYTES * M + MISC_BYTES + (size_t)h->nn * 8 + (size_t)h->F * 4, room = 226 * 1024;
    if (NG > MAX_CLUSTER) return false;
    int NR = (int)std::min<long long>(MAX_CLUSTER / NG, (h->n + 127) / 128);
    const long long rpc = ((h->n + NR - 1) / NR + 31) & ~31ll;
    // More rows a CTA: the whole grid is faster (us per tree: 22k x 7, 2.8k rows a CTA 44 and 44; 26k x 5, 3.3k 40 and 38; 13k x 13, 3.3k, 128 bins 90 and 72; 100k x 10 81 and 60)
    if (rpc > 2816) return false;
    NR = (int)((h->n + rpc - 1) / rpc);
    GrowGeom g = {};
    g.on = g.cluster = true; g.NG = NG; g.NR = NR; g.rpc = (int)rpc; g.fo = (std::min(4, h->F) + NR - 1) / NR;
    const size_t slots = (size_t)M / 2, kept = (size_t)std::max(1, M / 2) + std::max(1, M / 4);
    size_t o = (size_t)rpc * (8 + 4 * NQ) + small + (((rpc >> 5) + NG - 1) / NG * 64);
    auto take = [&](size_t bytes) { const size_t at = (o + 15) & ~(size_t)15; o = at + bytes; return at; };
    const size_t sum = take(slots * g.fo * NQ * B * 8), cnt = take((slots * g.fo * B + slots) * 4), bst = take((size_t)M * h->F * 48);
    const size_t without = o;
    size_t hist = take(kept * g.fo * hs * B * 8), base = 0;
    double clocks = 0.0;
    if (o + 128 < room) base = level_columns(h, g, room - 128 - o, &clocks);
    if (!base) { // histograms of parents from L2
        o = without; hist = 0;
        if (o + 128 < room) base = level_columns(h, g, room - 128 - o, &clocks);
    }
    if (!base || tree_clocks(h, g, clocks) > least) return false;
    g.o_x = (int)base; // the images come first
    g.o_sum = (int)(base + sum); g.o_cnt = (int)(base + cnt); g.o_best = (int)(base + bst); g.o_hist = hist ? (int)(base + hist) : 0;
    g.smem = base + o;
    g.hb = grow_bits(h, g);
    int clusters = 0;
    if (launch(h, g, nullptr, &clusters) != cudaSuccess || clusters < 1) { cudaGetLastError(); return false; }
    best = g;
    return true;
}

} // namespace

// Words of features and rows of a CTA.  Called again when the number of sampled columns changes.
void evb_grow_configure(evb_handle *h) {
    GrowGeom &g = h->grow;
    g = GrowGeom{};
    const int loss = h->p.loss, D = h->D, B = h->B;
    const bool gh = loss == EVB_MSE || loss == EVB_LOGLOSS || loss == EVB_POISSON || loss == EVB_GAMMA || loss == EVB_TWEEDIE;
    if (!gh || h->K != 1 || h->use_q2 || h->p.tree_type == 1 || D < 2 || D > MAX_D || (h->p.flags & EVB_FLAG_FULL_PARTITION) || h->nfeats > 65535) return;
    const int NQ = h->nq, P = planes(NQ, h->hgeo.cnt, h->hgeo.pack), M = 1 << std::max(1, D - 2);
    const size_t small = (size_t)NODE_BYTES * M + MISC_BYTES + (size_t)h->nn * 8 + (size_t)h->F * 4, room = 226 * 1024;
    double least = worth(h);
    for (int lw = 0; lw <= 2; ++lw) {
        const int W = 1 << lw, NG = (h->F + 4 * W - 1) / (4 * W);
        if (NG > h->num_sms) continue;
        const long long pr = 4 + 4 * W + 4 * NQ; // bytes of a row: its two places, bins and words
        int NR = h->num_sms / NG;
        NR = (int)std::min<long long>(NR, std::max<long long>(1, h->n / 512));
        const long long rpc = ((h->n + NR - 1) / NR + 31) & ~31ll;
        NR = (int)((h->n + rpc - 1) / rpc);
        GrowGeom t = {};
        t.on = true; t.lw = lw; t.NG = NG; t.NR = NR; t.rpc = (int)rpc;
        const size_t rest = small + (size_t)(rpc * pr) + (size_t)(((rpc >> 5) + NG - 1) / NG * 64); // and the leaves of the rows it updates
        double clocks = 0.0;
        if (rpc > 65504 || rest >= room) continue;
        const size_t base = level_columns(h, t, room - rest, &clocks);
        if (!base) continue;
        clocks = tree_clocks(h, t, clocks);
        if (clocks > least) continue;
        least = clocks;
        t.o_x = (int)base; t.smem = base + rest; t.hb = grow_bits(h, t);
        g = t;
        break; // few features a CTA: fewer row ranges share a sum
    }
    cluster_geom(h, g, least);
}

// words of the sums and of the counts of one level; records of one level
size_t evb_grow_sums(const evb_handle *h) { return (size_t)h->maxslots * h->nfeats * h->nq * h->B; }
size_t evb_grow_cnts(const evb_handle *h) { return (size_t)h->maxslots * h->nfeats * h->B; }
size_t evb_grow_best(const evb_handle *h) { return (size_t)(1 << std::max(1, h->D - 2)) * h->nfeats * 3; }

// Evaluation rows inside the launch: up to this many a CTA.  Kernels of their own cost 10 us a tree, and have many times the threads of one
// cluster.  us per tree, inside and in launches of its own: 1503 x 7 (16 CTAs) with 5k rows 45.4 and 52.6, 20k 49.1 and 53.2, 60k 55.4 and 55.2, 300k 98.1 and 57.7;
// 5000 x 20 (15 CTAs) 10k 57.2 and 63.7, 40k 62.4 and 64.3, 300k 93.4 and 85.7; 100k x 10 (147 CTAs) 100k 63.5 and 73.5, 500k 71.8 and 80.8.
constexpr int EVAL_ROWS = 3072;
int32_t evb_launch_grow(evb_handle *h, bool masked, uint8_t mask_cond, int slot, bool next_grads) {
    const GrowGeom &g = h->grow;
    const bool eval_inside = h->ev_n <= (int64_t)EVAL_ROWS * g.NG * g.NR;
    GrowArgs a = {};
    a.xC = h->xC; a.grad = h->grad; a.mask = masked ? h->mask_d : nullptr; a.cond = mask_cond; a.feattypes = h->feattypes_d; a.mono = h->mono_d;
    if (h->F < h->nfeats) {
        if (masked || h->F > EVB_GROW_JS) a.js0 = h->js_d;
        else { a.js_inline = 1; for (int f = 0; f < h->F; ++f) a.js[f] = (uint16_t)h->h_js[slot][EVB_GEN_WORDS + f]; }
    }
    a.sum = h->g_sum; a.low = h->g_low; a.cnt = h->g_cnt; a.sum_set = evb_grow_sums(h); a.cnt_set = evb_grow_cnts(h); a.lowflag = h->low;
    a.hist = h->hist; a.nsum = h->nsum; a.best = h->g_best; a.qinv = h->d_qinv; a.signs = h->d_signs;
    a.gmax = evb_gmax(h, false); a.gmax_next = evb_gmax(h, true);
    a.t_feat = h->t_feat; a.t_bin = h->t_bin; a.t_split = h->t_split; a.t_gain = h->t_gain; a.t_w = h->t_w; a.t_pred = h->t_pred; a.t_packed = h->t_packed;
    a.plan = h->plan; a.bar = h->g_bar; a.err = h->d_err; a.n = h->n;
    a.F = h->F; a.B = h->B; a.D = h->D; a.hist_nodes = h->hist_nodes; a.loss = h->p.loss; a.elide = h->Ce != h->C; a.hb = g.hb; a.ng = h->ng; a.nn = h->nn;
    a.round_bits = evb_hg_round_bits(h);
    a.NG = g.NG; a.NR = g.NR; a.rpc = g.rpc; a.lw = g.lw; a.M = 1 << std::max(1, h->D - 2);
    static_assert(sizeof(a.lc) == sizeof(g.lc), "levels");
    memcpy(a.lc, g.lc, sizeof(a.lc));
    a.o_sum = g.o_sum; a.o_cnt = g.o_cnt; a.o_best = g.o_best; a.o_hist = g.o_hist; a.fo = g.fo;
    a.o_x = g.o_x; a.o_q = a.o_x + (g.rpc * 4 << g.lw); a.o_idx = a.o_q + g.rpc * 4 * h->nq; a.o_node = a.o_idx + g.rpc * 4;
    a.max_polls = h->grow_polls;
    a.low_unit = evb_hg_low_unit(g.hb); a.neb = -h->p.eta / (double)h->p.bagging_size;
    a.lambda = h->p.lambda; a.L2 = h->p.L2; a.gamma = h->p.gamma; a.min_weight = h->p.min_weight;
    a.alpha = evb_alpha_set(h);
    if (!masked) {
        a.whole = 1; a.next_grads = next_grads ? 1 : 0; a.pred = h->pred; a.y = h->y; a.nidx = h->nidx;
        if (h->ev_n == 0 || eval_inside) { // else the evaluation's own kernels hand the tree over
            a.pub_src = reinterpret_cast<const uint4 *>(h->plan); a.pub_dst = static_cast<uint4 *>(h->h_tree[slot]); a.pub_n = (int)(h->h_tree_bytes / 16);
            a.pub_err = (int)(h->d_err - reinterpret_cast<int *>(h->plan));
        }
        if (h->ev_n > 0 && eval_inside) {
            a.ev_xT = h->ev_xT; a.ev_y = h->ev_y; a.ev_w = h->ev_w; a.ev_pred = h->ev_pred; a.ev_part = h->ev_part; a.ev_sum = h->d_evsum; a.ev_n = h->ev_n;
            a.ev_RS = h->RS; a.ev_metric = h->ev_metric;
        }
    }
    evb_tic(h, EVB_T_HIST);
    const cudaError_t e = launch(h, g, &a, nullptr);
    evb_toc(h, EVB_T_HIST);
    EVB_CUDA(e);
    return masked || eval_inside || h->ev_n == 0 ? EVB_OK : evb_launch_eval(h, nullptr, h->h_tree[slot]);
}
