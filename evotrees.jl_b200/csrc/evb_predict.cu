// Inference over all trees: `_predict` and `_predict_leaf_indices` (src/predict.jl:118-136, 173-185; GPU counterpart
// ext/EvoTreesKernelAbstractionsExt/predict.jl:115-158), `binarize` of the rows (src/fit-utils.jl:66-72) included.
//
// A model is packed once (evb_model_create) and its trees stay on the device; a call then moves only rows and predictions.
// The kernels take raw features, turn them into bins in shared memory and walk the trees from there: the bins never reach
// global memory.  Predictions (and leaf ids) are stored straight into pinned host memory.
#include "evb_device.cuh"
#include <algorithm>
#include <atomic>
#include <mutex>
#include <new>
#include <vector>
#include <string.h>
#include <sys/mman.h>
#include <stdlib.h>

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Trees in device memory: tree t at word t * tw.  Every tree of a model is a complete one of `levels` tests: [ni] nodes in heap order, then the
// values of the 2^levels leaves, [leaf][K].  A node is feature | b << 16 | a << 24: a row whose bin is x goes left where (x ^ a) <= b -- numeric
// tests have a = 0 and b the bin, categories a the bin and b = 0.  A leaf above the last level is a node that sends every row left (STOP), and so
// on to the last level, where its value is.  A walk is the same number of steps for all lanes, about half the instructions of one
// that looks for the end of its path (25 a level), and the trees take half the room.  ni: 2^levels, at least four, so that every part starts on a
// 16-byte boundary.
constexpr uint32_t STOP = 0x00ff0000u;
struct PredArgs {
    const void *x;          // raw features (T = float / double) or bins (T = uint8_t)
    long long ld;           // row-major: elements between rows; column-major: between features
    int row_major;
    int vec;                // row-major float rows whose features can be read as float4 (16-byte aligned rows)
    const void *edges;      // [nfeats][nedges] ascending, same type as x
    int nedges, nfeats, FW; // FW: words of four bins per row
    const uint32_t *trees;
    int ni, tw, levels;     // levels: tests on the longest path of a tree
    bool early;             // most paths end above the last level (evb_model::early)
    float *out;             // column k of row i at k * out_ld + i
    long long out_ld;
    uint32_t *leaf_idx;     // null, or tree t of row i at t * out_ld + i
    int n, K, loss, ntrees, apply_link;
};

// bins 4 w .. 4 w + 3 of row i as one word: searchsortedfirst(edges[j], x) = 1 + number of edges below x.  Four searches
// side by side; lanes are adjacent rows.
template <typename T>
__device__ __forceinline__ uint32_t bin_word(const PredArgs &a, long long i, int w) {
    const T *x = static_cast<const T *>(a.x);
    const int j0 = 4 * w, nj = min(4, a.nfeats - j0);
    T v[4];
    if (sizeof(T) == 4 && a.vec && nj == 4) {
        const float4 q = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(a.x) + i * a.ld + j0);
        v[0] = (T)q.x; v[1] = (T)q.y; v[2] = (T)q.z; v[3] = (T)q.w;
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = (T)0;
            if (q < nj) v[q] = a.row_major ? x[i * a.ld + j0 + q] : x[(long long)(j0 + q) * a.ld + i];
        }
    }
    uint32_t word = 0;
    if constexpr (sizeof(T) == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) word |= (uint32_t)v[q] << (8 * q);
        return word;
    } else {
        const T *e = static_cast<const T *>(a.edges) + (size_t)j0 * a.nedges;
        int lo[4] = {0, 0, 0, 0};
        int len = a.nedges; // the answer lies in [lo, lo + len]: the four searches halve the same length
        while (len > 0) {
            const int half = (len + 1) >> 1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nj && __ldg(e + (size_t)q * a.nedges + lo[q] + half - 1) < v[q]) lo[q] += half;
            len -= half;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nj) word |= (uint32_t)(lo[q] + 1) << (8 * q);
        return word;
    }
}

template <int KMAX>
__device__ __forceinline__ void link_row(int loss, int K, float (&p)[KMAX]) { // apply_prediction_link! (src/predict.jl:105-116)
    constexpr int U = KMAX > 8 ? 1 : KMAX;
    if (loss == EVB_LOGLOSS) {
#pragma unroll U
        for (int k = 0; k < KMAX; ++k) if (k < K) p[k] = sigmoidf_(p[k]);
    } else if (loss == EVB_GAUSSIAN_MLE || loss == EVB_LOGISTIC_MLE) {
#pragma unroll U
        for (int k = 1; k < KMAX; k += 2) if (k < K) p[k] = softplusf_(p[k]);
    } else if (loss == EVB_POISSON || loss == EVB_GAMMA || loss == EVB_TWEEDIE) {
#pragma unroll U
        for (int k = 0; k < KMAX; ++k) if (k < K) p[k] = expf(p[k]);
    } else if (loss == EVB_MLOGLOSS) {
        float s = 0.0f;
#pragma unroll U
        for (int k = 0; k < KMAX; ++k) if (k < K) { p[k] = expf(p[k]); s += p[k]; }
#pragma unroll U
        for (int k = 0; k < KMAX; ++k) if (k < K) p[k] /= s;
    }
}

// pred_add (evb_device.cuh) for up to KMAX outputs in registers.  Loops over a K that only the launch knows index p, so it lived in local
// memory: adding a tree took 900 clocks at seven classes, most of the time of a call of some thousand rows.
template <int KMAX>
__device__ __forceinline__ void add_leaf(int loss, int K, float (&p)[KMAX], const float *leaf, int stride) {
    if constexpr (KMAX > 8) {
        float v[KMAX];
        for (int k = 0; k < K; ++k) v[k] = leaf[k * stride];
        pred_add(loss, K, p, v);
    } else {
#pragma unroll
        for (int k = 0; k < KMAX; ++k) if (k < K) p[k] += leaf[k * stride];
        if (loss == EVB_LOGLOSS) {
#pragma unroll
            for (int k = 0; k < KMAX; ++k) p[k] = fminf(fmaxf(p[k], -15.0f), 15.0f);
        } else if (loss == EVB_GAUSSIAN_MLE || loss == EVB_LOGISTIC_MLE) {
#pragma unroll
            for (int k = 1; k < KMAX; k += 2) p[k] = fmaxf(-15.0f, p[k]);
        } else if (loss == EVB_MLOGLOSS) {
            float q[KMAX];
#pragma unroll
            for (int k = 0; k < KMAX; ++k) q[k] = k < K ? p[k] : -INFINITY;
#pragma unroll
            for (int d = 1; d < KMAX; d <<= 1)
#pragma unroll
                for (int k = 0; k + d < KMAX; k += 2 * d) q[k] = fmaxf(q[k], q[k + d]);
#pragma unroll
            for (int k = 0; k < KMAX; ++k) p[k] = fmaxf(-15.0f, p[k] - q[0]);
        }
    }
}

// Leaf values of n trees, [tree][K] at `stride`, in order: the next tree's are on their way while one is added, the loss is told apart once
template <int KMAX, int LOSS>
__device__ __forceinline__ void add_trees_of(int K, float (&p)[KMAX], const float *leaf, int n, int stride) {
    float v[KMAX];
    auto fetch = [&](int t) {
#pragma unroll
        for (int k = 0; k < KMAX; ++k) v[k] = k < K ? leaf[(t * K + k) * stride] : 0.0f;
    };
    fetch(0);
    for (int t = 1; t <= n; ++t) {
        float w[KMAX];
#pragma unroll
        for (int k = 0; k < KMAX; ++k) w[k] = v[k];
        if (t < n) fetch(t);
        add_leaf<KMAX>(LOSS, K, p, w, 1);
    }
}
template <int KMAX>
__device__ __forceinline__ void add_trees(int loss, int K, float (&p)[KMAX], const float *leaf, int n, int stride) {
    if (n <= 0) return;
    if constexpr (KMAX > 8) { for (int t = 0; t < n; ++t) add_leaf<KMAX>(loss, K, p, leaf + t * K * stride, stride); }
    else if (loss == EVB_MLOGLOSS) add_trees_of<KMAX, EVB_MLOGLOSS>(K, p, leaf, n, stride);
    else if (loss == EVB_LOGLOSS) add_trees_of<KMAX, EVB_LOGLOSS>(K, p, leaf, n, stride);
    else if (loss == EVB_GAUSSIAN_MLE || loss == EVB_LOGISTIC_MLE) add_trees_of<KMAX, EVB_GAUSSIAN_MLE>(K, p, leaf, n, stride);
    else add_trees_of<KMAX, EVB_MSE>(K, p, leaf, n, stride);
}
template <int KMAX>
__device__ __forceinline__ void put_row(const PredArgs &a, long long i, const float (&p)[KMAX]) {
    constexpr int U = KMAX > 8 ? 1 : KMAX;
#pragma unroll U
    for (int k = 0; k < KMAX; ++k) if (k < a.K) a.out[(size_t)k * a.out_ld + i] = p[k];
}

// Leaf (0 .. 2^levels - 1) of a row in one tree; word(w): the row's bins 4 w .. 4 w + 3, node(i): the tree's node i.  early: a lane leaves the loop
// where its path ends (PredArgs::early)
template <typename N, typename X>
__device__ __forceinline__ int walk(int levels, bool early, N node, X word) {
    int i = 0, l = 0;
    if (early) {
        for (; l < levels; ++l) {
            const uint32_t pk = node(i);
            if (pk == STOP) break;
            const uint32_t x = __byte_perm(word((pk & 0xffffu) >> 2), 0u, 0x4440u | (pk & 3u));
            i = 2 * i + ((x ^ (pk >> 24)) <= ((pk >> 16) & 0xffu) ? 1 : 2);
        }
        return ((i + 1) << (levels - l)) - (1 << levels); // the leftmost leaf below
    }
    for (; l < levels; ++l) {
        const uint32_t pk = node(i);
        const uint32_t x = __byte_perm(word((pk & 0xffffu) >> 2), 0u, 0x4440u | (pk & 3u));
        i = 2 * i + ((x ^ (pk >> 24)) <= ((pk >> 16) & 0xffu) ? 1 : 2);
    }
    return i + 1 - (1 << levels);
}
// the same for the id of the node where the row's path ends (`predict_leaf_idx`): the first that stops, else the leaf itself
template <typename N, typename X>
__device__ __forceinline__ int walk_id(int levels, N node, X word, int &leaf) {
    int i = 0, l = 0;
    for (; l < levels; ++l) {
        const uint32_t pk = node(i);
        if (pk == STOP) break;
        const uint32_t x = __byte_perm(word((pk & 0xffffu) >> 2), 0u, 0x4440u | (pk & 3u));
        i = 2 * i + ((x ^ (pk >> 24)) <= ((pk >> 16) & 0xffu) ? 1 : 2);
    }
    leaf = ((i + 1) << (levels - l)) - (1 << levels);
    return i + 1;
}

// ---------------------------------------------------------------------------------- few rows
// One CTA per row, one thread per tree: what bounds a call with a handful of rows is latency, so the levels of all trees
// are walked at the same time and only the sum over the trees is serial (the clamps of `predict!` do not commute, so the
// trees are added in order).  Bins: one warp per feature counts the edges below the value, 32 edges per load.
// Measured (call of 1 row x 10 features, 101 trees of depth 6): 365 us with one thread walking all trees, every tree uploaded
// by the call and a stream and eight events made for it, 31 us like this.
constexpr int ONE_THREADS = 256;
template <int KMAX, typename T>
__global__ void __launch_bounds__(ONE_THREADS) k_predict_one(PredArgs a) {
    extern __shared__ uint32_t s_one[]; // [FW] bins of the row, then [ONE_THREADS][K] leaf values
    const int K = a.K, tid = threadIdx.x, lane = tid & 31;
    const long long i = blockIdx.x;
    uint8_t *s_bins = reinterpret_cast<uint8_t *>(s_one);
    float *s_leaf = reinterpret_cast<float *>(s_one + a.FW);
    for (int j = tid >> 5; j < a.nfeats; j += ONE_THREADS / 32) {
        const T v = a.row_major ? static_cast<const T *>(a.x)[i * a.ld + j] : static_cast<const T *>(a.x)[(long long)j * a.ld + i];
        int c = 0;
        if constexpr (sizeof(T) == 1) c = (int)v;
        else {
            const T *e = static_cast<const T *>(a.edges) + (size_t)j * a.nedges;
            for (int b = 0; b < a.nedges; b += 32) c += __popc(__ballot_sync(FULL, b + lane < a.nedges && __ldg(e + min(b + lane, a.nedges - 1)) < v));
            ++c;
        }
        if (lane == 0) s_bins[j] = (uint8_t)c;
    }
    float p[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) p[k] = 0.0f;
    for (int t0 = 0; t0 < a.ntrees; t0 += ONE_THREADS) {
        __syncthreads();
        const int t = t0 + tid;
        if (t < a.ntrees) {
            const uint32_t *tr = a.trees + (size_t)t * a.tw;
            auto node = [&](int n) { return __ldg(tr + n); };
            auto word = [&](uint32_t w) { return s_one[w]; };
            int leaf;
            if (a.leaf_idx) a.leaf_idx[(size_t)t * a.out_ld + i] = (uint32_t)walk_id(a.levels, node, word, leaf);
            else leaf = walk(a.levels, a.early, node, word);
            for (int k = 0; k < K; ++k) s_leaf[tid * K + k] = __uint_as_float(__ldg(tr + a.ni + leaf * K + k));
        }
        __syncthreads();
        if (tid == 0) {
            const int nt = min(ONE_THREADS, a.ntrees - t0);
            add_trees<KMAX>(a.loss, K, p, s_leaf, nt, 1);
        }
    }
    if (tid == 0) {
        if (a.apply_link) link_row<KMAX>(a.loss, K, p);
        put_row<KMAX>(a, i, p);
    }
}

// ---------------------------------------------------------------------------------- some thousand rows
// One CTA per 32 rows (lane = row).  Seven warps share the trees of a block of TB and leave the leaf values in shared
// memory, four trees at a time per lane so that four chains of loads overlap; the eighth warp adds the previous block's
// values in order meanwhile.  Nodes come through L1: 32 rows do not pay for copying a tree into shared memory.  Bins are
// word-major ([word of the row][row]): a lane only ever reads its own bank.
// Measured (call of 20 011 rows x 28, 201 trees of depth 8, five classes): 0.206 ms, with k_predict_tiles 0.175.  Used where two trees and
// 32 rows do not fit shared memory.
constexpr int MID_WARPS = 8, MID_ILP = 4;
template <int KMAX, typename T>
__global__ void __launch_bounds__(MID_WARPS * 32) k_predict_mid(PredArgs a, int TB) {
    extern __shared__ uint32_t s_mid[]; // [FW][32] bins, then [2][TB][K][32] leaf values
    const int K = a.K, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long row0 = (long long)blockIdx.x * 32, i = row0 + lane;
    const bool act = i < a.n;
    for (int w = wid; w < a.FW; w += MID_WARPS) s_mid[w * 32 + lane] = act ? bin_word<T>(a, i, w) : 0u;
    float *s_leaf = reinterpret_cast<float *>(s_mid + a.FW * 32);
    __syncthreads();
    float p[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) p[k] = 0.0f;
    int buf = 0;
    for (int t0 = 0;; t0 += TB, buf ^= 1) {
        const int nt = min(TB, a.ntrees - t0); // <= 0: only the last block's sum is left
        if (wid > 0) {
            for (int tb = wid - 1; tb < nt; tb += (MID_WARPS - 1) * MID_ILP) {
                const uint32_t *tr[MID_ILP];
                int at[MID_ILP], id[MID_ILP];
#pragma unroll
                for (int u = 0; u < MID_ILP; ++u) {
                    const int t = tb + u * (MID_WARPS - 1);
                    tr[u] = a.trees + (size_t)(t0 + (t < nt ? t : tb)) * a.tw;
                    at[u] = 0; id[u] = 0;
                }
                for (int l = 0; l < a.levels; ++l) {
                    uint32_t pk[MID_ILP];
#pragma unroll
                    for (int u = 0; u < MID_ILP; ++u) pk[u] = id[u] == 0 ? __ldg(tr[u] + at[u]) : STOP;
#pragma unroll
                    for (int u = 0; u < MID_ILP; ++u) {
                        if (id[u] == 0 && pk[u] == STOP) id[u] = at[u] + 1;
                        const uint32_t x = __byte_perm(s_mid[((pk[u] & 0xffffu) >> 2) * 32 + lane], 0u, 0x4440u | (pk[u] & 3u));
                        at[u] = 2 * at[u] + ((x ^ (pk[u] >> 24)) <= ((pk[u] >> 16) & 0xffu) ? 1 : 2);
                    }
                }
#pragma unroll
                for (int u = 0; u < MID_ILP; ++u) {
                    const int t = tb + u * (MID_WARPS - 1);
                    if (t < nt) {
                        const uint32_t *lf = tr[u] + a.ni + (at[u] + 1 - (1 << a.levels)) * K;
                        float *d = s_leaf + ((size_t)(buf * TB + t) * K) * 32 + lane;
                        for (int k = 0; k < K; ++k) d[k * 32] = __uint_as_float(__ldg(lf + k));
                        if (a.leaf_idx && act) a.leaf_idx[(size_t)(t0 + t) * a.out_ld + i] = (uint32_t)(id[u] ? id[u] : at[u] + 1);
                    }
                }
            }
        } else if (t0 > 0) {
            const int np = min(TB, a.ntrees - (t0 - TB));
            const float *s = s_leaf + ((size_t)(buf ^ 1) * TB * K) * 32 + lane;
            add_trees<KMAX>(a.loss, K, p, s, np, 32);
        }
        if (nt <= 0) break;
        __syncthreads();
    }
    if (wid == 0 && act) {
        if (a.apply_link) link_row<KMAX>(a.loss, K, p);
        put_row<KMAX>(a, i, p);
    }
}

// The same division of work with the trees in shared memory: a CTA of 32 warps takes RG groups of 32 rows, WARPS / RG warps each, one
// of which adds; blocks of TB trees arrive by cp.async while the block before is walked.  A node then is one bank conflict away
// instead of a line of L1 per lane, and so is a leaf: its K values cost k_predict_mid K loads of up to 32 lines each.  What bounds it is
// instructions, 13 a level, and with several outputs the chain of additions.  us of a call, before (k_predict_mid, nodes that say where a path
// ends, sums in local memory) and here: 20k x 28, 200 trees of depth 8, five classes 241 and 175; 900 x 12, 200 of depth 6, seven classes 128
// and 59; 90k x 12, the same model 616 and 346; 1.5k x 60, 100 of depth 9, two outputs 84 and 63; 6k x 30 doubles, 150 of depth 10 141 and 115.
constexpr int TILE_WARPS = 32;
template <int KMAX, typename T>
__global__ void __launch_bounds__(TILE_WARPS * 32, 1) k_predict_tiles(PredArgs a, int RG, int TB) {
    extern __shared__ __align__(16) uint32_t s_tl[]; // [2][TB][tw] trees, [2][TB][K][R] leaf values, [FW][R] bins; R = 32 RG rows
    const int K = KMAX > 8 ? a.K : KMAX, tw = a.tw, R = 32 * RG, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, grp = wid % RG, role = wid / RG, walkers = (TILE_WARPS - grp + RG - 1) / RG - 1;
    float *s_leaf = reinterpret_cast<float *>(s_tl + (size_t)2 * TB * tw);
    uint32_t *s_bins = reinterpret_cast<uint32_t *>(s_leaf + (size_t)2 * TB * K * R);
    auto load_block = [&](int t0, int buf) {
        const int nt = min(TB, a.ntrees - t0);
        if (nt > 0) {
            const uint4 *src = reinterpret_cast<const uint4 *>(a.trees + (size_t)t0 * tw);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_tl + (size_t)buf * TB * tw);
            for (int c = threadIdx.x; c < nt * (tw >> 2); c += TILE_WARPS * 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)c * 16u), "l"(src + c) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_block(0, 0);
    const long long row0 = (long long)blockIdx.x * R, i = row0 + grp * 32 + lane;
    const bool act = i < a.n;
    for (int e = wid; e < a.FW * RG; e += TILE_WARPS) {
        const int w = e / RG, g = e - w * RG;
        const long long r = row0 + g * 32 + lane;
        s_bins[w * R + g * 32 + lane] = r < a.n ? bin_word<T>(a, r, w) : 0u;
    }
    const uint32_t *xcol = s_bins + grp * 32 + lane;
    float p[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) p[k] = 0.0f;
    int buf = 0;
    for (int t0 = 0;; t0 += TB, buf ^= 1) {
        const int nt = min(TB, a.ntrees - t0); // <= 0: only the last block's sum is left
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads(); // this block's trees and the last one's leaf values are in place, the other buffers free
        load_block(t0 + TB, buf ^ 1);
        if (role > 0) {
            for (int t = role - 1; t < nt; t += walkers) {
                const uint32_t *tr = s_tl + ((size_t)buf * TB + t) * tw;
                auto node = [&](int n) { return tr[n]; };
                auto word = [&](uint32_t w) { return xcol[w * R]; };
                int leaf;
                if (a.leaf_idx) {
                    const uint32_t id = (uint32_t)walk_id(a.levels, node, word, leaf);
                    if (act) a.leaf_idx[(size_t)(t0 + t) * a.out_ld + i] = id;
                } else leaf = walk(a.levels, a.early, node, word);
                const float *lf = reinterpret_cast<const float *>(tr + a.ni) + leaf * K;
                float *d = s_leaf + ((size_t)(buf * TB + t) * K) * R + grp * 32 + lane;
                constexpr int U = KMAX > 8 ? 1 : KMAX;
#pragma unroll U
                for (int k = 0; k < KMAX; ++k) if (k < K) d[k * R] = lf[k];
            }
        } else if (t0 > 0) {
            const int np = min(TB, a.ntrees - (t0 - TB));
            const float *d = s_leaf + ((size_t)(buf ^ 1) * TB * K) * R + grp * 32 + lane;
            add_trees<KMAX>(a.loss, K, p, d, np, R);
        }
        if (nt <= 0) break;
    }
    if (role == 0 && act) {
        if (a.apply_link) link_row<KMAX>(a.loss, K, p);
        put_row<KMAX>(a, i, p);
    }
}

// ---------------------------------------------------------------------------------- many rows
// One thread = one row.  The CTA's bins sit in shared memory word-major, and the trees (nodes + leaf tables) stream through
// two shared-memory buffers of TB trees each: while the threads walk the trees of one buffer, `cp.async` fills the other,
// so a traversal step costs two shared-memory loads and the trip to L2 is off the critical path.
template <int KMAX, typename T>
__global__ void __launch_bounds__(1024) k_predict_staged(PredArgs a, int TB) {
    extern __shared__ __align__(16) uint32_t s_pr[]; // [FW][blockDim.x] bins, then 2 x TB x tw tree words
    const int K = a.K, rows = blockDim.x, tw = a.tw;
    uint32_t *s_rows = s_pr;
    uint32_t *s_trees = s_pr + (size_t)rows * a.FW; // rows is a multiple of 4: 16-byte aligned
    const long long row0 = (long long)blockIdx.x * rows;
    auto load_block = [&](int t0, int buf) { // trees t0 .. t0 + TB - 1 -> buffer `buf`, 16 bytes per copy
        const int nt = min(TB, a.ntrees - t0);
        const uint4 *src = reinterpret_cast<const uint4 *>(a.trees + (size_t)t0 * tw);
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_trees + (size_t)buf * TB * tw);
        for (int c = threadIdx.x; c < nt * (tw >> 2); c += rows)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)c * 16u), "l"(src + c) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_block(0, 0);
    const long long i = row0 + threadIdx.x;
    const bool act = i < a.n;
    uint32_t *xcol = s_rows + threadIdx.x;
    if (act)
        for (int w = 0; w < a.FW; ++w) xcol[w * rows] = bin_word<T>(a, i, w);
    float p[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) p[k] = 0.0f;
    int buf = 0;
    for (int t0 = 0; t0 < a.ntrees; t0 += TB, buf ^= 1) {
        const int nt = min(TB, a.ntrees - t0);
        if (t0 + TB < a.ntrees) load_block(t0 + TB, buf ^ 1); // the other buffer was consumed before the last barrier
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads(); // this block's trees are in place for everybody
        if (act) {
            for (int t = 0; t < nt; ++t) {
                const uint32_t *tr = s_trees + ((size_t)buf * TB + t) * tw;
                auto node = [&](int n) { return tr[n]; };
                auto word = [&](uint32_t w) { return xcol[w * rows]; };
                int leaf;
                if (a.leaf_idx) a.leaf_idx[(size_t)(t0 + t) * a.out_ld + i] = (uint32_t)walk_id(a.levels, node, word, leaf);
                else leaf = walk(a.levels, a.early, node, word);
                add_leaf<KMAX>(a.loss, K, p, reinterpret_cast<const float *>(tr + a.ni) + leaf * K, 1);
            }
        }
        __syncthreads(); // everybody is done with this buffer: the next iteration refills it
    }
    if (!act) return;
    if (a.apply_link) link_row<KMAX>(a.loss, K, p);
    put_row<KMAX>(a, i, p);
}

// rows of more bins than shared memory holds: bins in global memory ([row][FW] words), one thread per row
template <typename T>
__global__ void __launch_bounds__(256) k_bin_rows(PredArgs a, uint32_t *xw) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= a.n) return;
    for (int w = blockIdx.y; w < a.FW; w += gridDim.y) xw[(size_t)i * a.FW + w] = bin_word<T>(a, i, w);
}
template <int KMAX>
__global__ void __launch_bounds__(256) k_predict_wide(PredArgs a, const uint32_t *xw) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= a.n) return;
    const uint32_t *xr = xw + (size_t)i * a.FW;
    float p[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) p[k] = 0.0f;
    const int K = a.K;
    for (int t = 0; t < a.ntrees; ++t) {
        const uint32_t *tr = a.trees + (size_t)t * a.tw;
        auto node = [&](int n) { return __ldg(tr + n); };
        auto word = [&](uint32_t w) { return xr[w]; };
        int leaf;
        if (a.leaf_idx) a.leaf_idx[(size_t)t * a.out_ld + i] = (uint32_t)walk_id(a.levels, node, word, leaf);
        else leaf = walk(a.levels, a.early, node, word);
        add_leaf<KMAX>(a.loss, K, p, reinterpret_cast<const float *>(tr + a.ni) + leaf * K, 1);
    }
    if (a.apply_link) link_row<KMAX>(a.loss, K, p);
    put_row<KMAX>(a, i, p);
}

} // namespace

// ================================================================================================= models
static int32_t no_host_memory() {
    evb_set_error("out of host memory");
    return EVB_ERR_ARG;
}
struct evb_model {
    int device = 0, loss = 0, K = 1, ntrees = 0, ni = 4, tw = 8, levels = 0, nfeats = 0, nedges = 0;
    bool early = false;               // fewer than an eighth of the complete trees' inner nodes test anything
    void *block = nullptr;            // trees, then the edges as double and as float
    const uint32_t *d_trees = nullptr;
    const double *d_e64 = nullptr;
    const float *d_e32 = nullptr;
    // Where the trees and the edges came from and what they held when they were packed: a call compares them while the GPU
    // works, so a tree that was changed in place since is noticed.
    std::vector<const void *> src;    // [ntrees][4]: feat, cond_bin, split, leaf_pred
    std::vector<int32_t> nodes;       // nodes of every tree
    std::vector<size_t> at;           // offset of every tree's copy in `snap`, then its size
    unsigned char *snap = nullptr;
    const void *src_edges = nullptr, *src_ft = nullptr;
    std::vector<unsigned char> snap_edges, snap_ft;
    evb_model() = default;
    evb_model(const evb_model &) = delete;
    evb_model &operator=(const evb_model &) = delete;
    ~evb_model() { free(snap); }
};

namespace {

size_t tree_bytes(int nn, int K, int part) { return part == 0 ? (size_t)nn * 8 : part == 3 ? (size_t)nn * K * 4 : (size_t)nn; }

struct VerifyJob { const evb_model *m; std::atomic<int> bad; };
void verify_range(void *c, size_t b, size_t e) {
    VerifyJob &j = *static_cast<VerifyJob *>(c);
    for (size_t t = b; t < e && j.bad.load(std::memory_order_relaxed) == 0; ++t) {
        size_t o = j.m->at[t];
        for (int q = 0; q < 4; ++q) {
            const size_t n = tree_bytes(j.m->nodes[t], j.m->K, q);
            if (memcmp(j.m->src[t * 4 + q], j.m->snap + o, n) != 0) { j.bad.store(1); return; }
            o += n;
        }
    }
}
// the sources still hold what was packed
bool model_current(const evb_model *m) {
    VerifyJob j{m, {0}};
    const size_t per = m->ntrees > 0 ? m->at[m->ntrees] / m->ntrees : 0;
    const size_t slice = per ? std::max<size_t>(1, ((size_t)256 << 10) / per) : 1;
    evb_parallel(verify_range, &j, (size_t)m->ntrees, slice);
    return j.bad.load() == 0 && (m->snap_edges.empty() || memcmp(m->src_edges, m->snap_edges.data(), m->snap_edges.size()) == 0) &&
           (m->snap_ft.empty() || memcmp(m->src_ft, m->snap_ft.data(), m->snap_ft.size()) == 0);
}

// Large blocks of host memory that are about to be written by several threads: huge pages where the system has them (a page fault
// every 4 KB costs more than the copy).  Freed with free().
unsigned char *big_alloc(size_t bytes) {
    constexpr size_t HUGE_PAGE = (size_t)2 << 20;
    if (bytes < 2 * HUGE_PAGE) return static_cast<unsigned char *>(malloc(bytes ? bytes : 1));
    void *p = nullptr;
    if (posix_memalign(&p, HUGE_PAGE, bytes) != 0) return nullptr;
    madvise(p, bytes, MADV_HUGEPAGE);
    return static_cast<unsigned char *>(p);
}

// Trees -> packed trees.  With a snapshot a tree is copied there first and packed from the copy, so that the two agree.
struct PackJob {
    const evb_model *m;
    const void *const *src;
    const int32_t *nodes;
    const uint8_t *feattypes;
    bool categories;            // some feature is not numeric
    unsigned char *snap;
    std::atomic<long long> bad; // tree and node of a test that cannot be: (tree << 32 | node) + 1; -1: out of memory
    std::atomic<long long> tests; // nodes of all trees that paths come to and that test something
};
// last of the nodes [b, e) that has a test; -1: none
int deepest_split(const uint8_t *split, int b, int e) {
    while (e - b >= 8) {
        uint64_t v;
        memcpy(&v, split + e - 8, 8);
        if (v) break;
        e -= 8;
    }
    while (e > b && split[e - 1] == 0) --e;
    return e > b ? e - 1 : -1;
}
// A node of the complete tree is the tree's own node of the same number where a path comes there: `live` says whether one does.  Nothing branches on
// what a node holds (mispredicted ones cost more than the rest).  NUM: no categories.  Returns whether a test is of a feature that is none.
template <bool NUM>
bool pack_nodes(uint32_t *tr, int n, const unsigned char *feat, const uint8_t *bin, const uint8_t *split, const uint8_t *numeric, uint64_t nfeats, uint32_t *live, long long &tests) {
    uint32_t bad = 0u, n_tests = 0u;
    for (int i = 0; i < n; ++i) {
        int64_t f;
        memcpy(&f, feat + (size_t)i * 8, 8); // (at any address)
        const uint64_t g = (uint64_t)(f - 1);
        const uint32_t s = split[i] != 0 ? 1u : 0u, known = g < nfeats ? 1u : 0u, q = known ? (uint32_t)g : 0u;
        bad |= s & ~known;
        uint32_t w = q | (uint32_t)bin[i] << (NUM || numeric[q] ? 16 : 24);
        w |= (uint32_t)(w == STOP) << 24; // bin 255 of feature 0: all rows go left as well, but the path does not end
        const uint32_t l = live[i] & s;
        tr[i] = l ? w : STOP;
        live[2 * i + 1] = live[2 * i + 2] = l;
        n_tests += l;
    }
    tests += n_tests;
    return bad != 0u;
}
void pack_trees_of(PackJob &j, char *dst, size_t first, size_t count) {
    const evb_model &m = *j.m;
    uint32_t *tr = reinterpret_cast<uint32_t *>(dst);
    const int last = (1 << m.levels) - 1; // first node of the last level
    const size_t row = (size_t)m.K * 4;
    std::vector<uint32_t> live((size_t)2 * last + 1);
    std::vector<int> ends((size_t)last + 1);
    long long tests = 0;
    for (size_t t = first; t < first + count; ++t, tr += m.tw) {
        const void *part[4];
        const int nn = j.nodes[t];
        size_t o = j.snap ? m.at[t] : 0;
        for (int q = 0; q < 4; ++q) {
            part[q] = j.src[t * 4 + q];
            if (!j.snap) continue;
            const size_t n = tree_bytes(nn, m.K, q);
            memcpy(j.snap + o, part[q], n);
            part[q] = j.snap + o;
            o += n;
        }
        const unsigned char *feat = static_cast<const unsigned char *>(part[0]);
        const uint8_t *bin = static_cast<const uint8_t *>(part[1]), *split = static_cast<const uint8_t *>(part[2]);
        const char *pred = static_cast<const char *>(part[3]); // floats, at any address as well
        const int inner = std::min(last, std::max(0, (nn - 1) / 2));        // nodes that may test something: their children are nodes of the tree
        live[0] = nn > 0 ? 1u : 0u;
        bool bad = deepest_split(split, inner, nn) >= 0;
        bad |= j.categories ? pack_nodes<false>(tr, inner, feat, bin, split, j.feattypes, (uint64_t)m.nfeats, live.data(), tests)
                            : pack_nodes<true>(tr, inner, feat, bin, split, nullptr, (uint64_t)m.nfeats, live.data(), tests);
        if (bad) {
            int i = 0;
            for (; i < nn; ++i) {
                int64_t f;
                memcpy(&f, feat + (size_t)i * 8, 8);
                if (split[i] && (f < 1 || f > m.nfeats || i >= inner)) break;
            }
            long long none = 0;
            j.bad.compare_exchange_strong(none, ((long long)t << 32 | i) + 1);
            continue;
        }
        for (int i = inner; i < last; ++i) { tr[i] = STOP; live[2 * i + 1] = live[2 * i + 2] = 0u; } // (a tree of fewer levels)
        for (int i = last; i < m.ni; ++i) tr[i] = 0u;
        // Values of the last level lie together in the tree too; those of paths that end above it go to the leftmost leaf below.  (Leaves
        // that no path comes to hold anything.)
        char *leaf = reinterpret_cast<char *>(tr + m.ni);
        const size_t have = (size_t)std::max(0, std::min(nn - last, last + 1)) * row;
        memcpy(leaf, pred + (have ? (size_t)last * row : 0), have);
        memset(leaf + have, 0, (size_t)(m.tw - m.ni) * 4 - have);
        int full = 0;
        for (int i = last; i <= 2 * last; ++i) full += (int)live[i];
        if (full == last + 1) continue;
        int n = 0;
        for (int i = 0; i < last; ++i) { ends[n] = i; n += (int)(live[i] & (tr[i] == STOP ? 1u : 0u)); }
        for (int e = 0; e < n; ++e) {
            const int i = ends[e], at = ((i + 1) << (m.levels - (31 - __builtin_clz((unsigned)i + 1u)))) - (last + 1);
            memcpy(leaf + (size_t)at * row, pred + (size_t)i * row, row);
        }
    }
    j.tests.fetch_add(tests);
}

void pack_trees(void *ctx, char *dst, size_t first, size_t count) { // (on any thread)
    PackJob &j = *static_cast<PackJob *>(ctx);
    try { pack_trees_of(j, dst, first, count); }
    catch (const std::bad_alloc &) { j.bad.store(-1); }
}

// src: [ntrees][4] pointers; packs, uploads and keeps the snapshot.  edges may be null (binned input only).
// All staging threads pack, straight into pinned buffers that are copied meanwhile; one thread into a zeroed image, its upload from
// pageable memory and a second pass for the snapshot took 2.4 ms at 200 trees of depth 11 and 39 at 500 of depth 13.
int32_t model_fill(evb_model *m, int ntrees, const void *const *src, const int32_t *nodes, const void *edges, int e_dtype, int nedges,
                   int nfeats, const uint8_t *feattypes, bool snapshot) {
    const int K = m->K;
    // Levels: down to the last test of any tree, whatever room its arrays have.  200 trees of depth 11 whose paths end at depth 4 take 4 steps
    // a row, not 10.
    int deepest = -1;
    for (int t = 0; t < ntrees; ++t) {
        const int i = deepest_split(static_cast<const uint8_t *>(src[t * 4 + 2]), std::min((int)nodes[t], deepest + 1), std::max(0, (nodes[t] - 1) / 2));
        deepest = std::max(deepest, i);
    }
    m->ntrees = ntrees; m->nfeats = nfeats; m->nedges = edges ? nedges : 0;
    m->levels = 0;
    while ((1 << m->levels) <= deepest + 1) ++m->levels;
    m->ni = std::max(4, 1 << m->levels);
    m->tw = m->ni + (((K << m->levels) + 3) & ~3);
    const size_t unit = (size_t)m->tw * 4, tbytes = (size_t)ntrees * unit, ne = (size_t)m->nedges * nfeats;
    const size_t o64 = (tbytes + 15) & ~(size_t)15, o32 = o64 + ne * 8, total = o32 + ne * 4 + 16;
    const bool categories = feattypes && memchr(feattypes, 0, (size_t)nfeats) != nullptr;
    PackJob job{m, src, nodes, feattypes, categories, nullptr, {0}, {0}};
    if (snapshot) {
        m->src.assign(src, src + (size_t)ntrees * 4);
        m->nodes.assign(nodes, nodes + ntrees);
        m->at.resize((size_t)ntrees + 1);
        size_t o = 0;
        for (int t = 0; t < ntrees; ++t) { m->at[t] = o; for (int q = 0; q < 4; ++q) o += tree_bytes(nodes[t], K, q); }
        m->at[ntrees] = o;
        m->snap = job.snap = big_alloc(o);
        if (!m->snap) { evb_set_error("out of host memory"); return EVB_ERR_ARG; }
        if (edges) { m->src_edges = edges; m->snap_edges.assign((const unsigned char *)edges, (const unsigned char *)edges + ne * (e_dtype == EVB_F64 ? 8 : 4)); }
        if (feattypes) { m->src_ft = feattypes; m->snap_ft.assign(feattypes, feattypes + nfeats); }
    }
    // Below half a megabyte everything goes up in one copy of an ordinary buffer (so do trees that are larger than a pinned buffer).
    const bool piped = tbytes > ((size_t)512 << 10) && unit <= evb_stage_bytes();
    const size_t hosted = piped ? o64 : 0; // bytes of the block that are not in `host`
    std::vector<unsigned char> host(total - hosted);
    if (edges) {
        double *e64 = reinterpret_cast<double *>(host.data() + (o64 - hosted));
        float *e32 = reinterpret_cast<float *>(host.data() + (o32 - hosted));
        for (size_t i = 0; i < ne; ++i) {
            if (e_dtype == EVB_F64) { e64[i] = static_cast<const double *>(edges)[i]; e32[i] = (float)e64[i]; }
            else { e32[i] = static_cast<const float *>(edges)[i]; e64[i] = e32[i]; }
        }
    }
    EVB_CUDA(evb_dev_alloc(&m->block, total));
    cudaStream_t st = nullptr;
    EVB_CUDA(evb_stream_get(&st));
    int32_t rc = EVB_OK;
    // a thread's piece: trees of 128 KB in the caller's arrays, whatever is left of them when they are packed
    size_t nodes_all = 0;
    for (int t = 0; t < ntrees; ++t) nodes_all += (size_t)std::max(nodes[t], 1);
    const size_t piece = std::max<size_t>(1, ((size_t)128 << 10) * ntrees / std::max<size_t>(1, nodes_all * (10 + (size_t)K * 4)));
    if (piped) rc = evb_h2d_made(m->block, unit, (size_t)ntrees, piece, pack_trees, &job, st);
    else {
        struct Hosted { PackJob *job; char *to; size_t unit; } hj{&job, reinterpret_cast<char *>(host.data()), unit};
        evb_parallel([](void *c, size_t b, size_t e) { Hosted &q = *static_cast<Hosted *>(c); pack_trees(q.job, q.to + b * q.unit, b, e - b); }, &hj, (size_t)ntrees, piece);
    }
    if (rc == EVB_OK && job.bad.load() == -1) rc = no_host_memory();
    if (rc == EVB_OK && job.bad.load() > 0) {
        const long long at = job.bad.load() - 1;
        evb_set_error("evb_model: node %lld of tree %lld tests a feature that is not one of %d or has no children", (at & 0xffffffffll) + 1, (at >> 32) + 1, nfeats);
        rc = EVB_ERR_ARG;
    }
    if (rc == EVB_OK) rc = evb_h2d_staged(static_cast<char *>(m->block) + hosted, host.data(), host.size(), st);
    if (cudaStreamSynchronize(st) != cudaSuccess && rc == EVB_OK) { evb_set_error("CUDA error %s while a model was uploaded", cudaGetErrorString(cudaGetLastError())); rc = EVB_ERR_CUDA; }
    evb_stream_put(st);
    EVB_CHECK(rc);
    m->early = 8 * job.tests.load() < (long long)ntrees * ((1 << m->levels) - 1);
    m->d_trees = static_cast<const uint32_t *>(m->block);
    m->d_e64 = reinterpret_cast<const double *>(static_cast<char *>(m->block) + o64);
    m->d_e32 = reinterpret_cast<const float *>(static_cast<char *>(m->block) + o32);
    return EVB_OK;
}

} // namespace

extern "C" void evb_model_destroy(evb_model *m) {
    if (!m) return;
    int prev = 0;
    cudaGetDevice(&prev);
    if (cudaSetDevice(m->device) == cudaSuccess) evb_dev_free(m->block);
    cudaSetDevice(prev);
    delete m;
}

static int32_t model_args(int32_t loss, int32_t K, int32_t ntrees, int32_t nfeats) {
    if (nfeats < 1 || nfeats > 65535 || ntrees < 0 || K < 1 || K > 64 || loss < 0 || loss > EVB_LOSS_LAST) {
        evb_set_error("evb_predict: invalid argument");
        return EVB_ERR_ARG;
    }
    return EVB_OK;
}

extern "C" int32_t evb_model_create(evb_model **out, int32_t device, int32_t loss, int32_t K, int32_t ntrees, const void *const *src,
                                    const int32_t *nodes, const void *edges, int32_t edges_dtype, int32_t nedges, int32_t nfeats,
                                    const uint8_t *feattypes) {
    if (!out) { evb_set_error("evb_model_create: out is null"); return EVB_ERR_ARG; }
    *out = nullptr;
    EVB_CHECK(model_args(loss, K, ntrees, nfeats));
    if ((ntrees > 0 && (!src || !nodes)) || !edges || nedges < 1 || nedges > 254 || (edges_dtype != EVB_F32 && edges_dtype != EVB_F64)) {
        evb_set_error("evb_model_create: invalid argument");
        return EVB_ERR_ARG;
    }
    EVB_CHECK(evb_check_device(device));
    evb_model *m = new (std::nothrow) evb_model();
    if (!m) { evb_set_error("out of host memory"); return EVB_ERR_ARG; }
    m->device = device; m->loss = loss; m->K = K;
    int32_t rc;
    try { rc = model_fill(m, ntrees, src, nodes, edges, edges_dtype, nedges, nfeats, feattypes, true); }
    catch (const std::bad_alloc &) { rc = no_host_memory(); }
    if (rc != EVB_OK) { evb_model_destroy(m); return rc; }
    *out = m;
    return EVB_OK;
}

// ================================================================================================= calls
namespace {

// Work buffers of one call at a time: three sets of {stream, pinned input, device input, pinned output}, of the size of a chunk of
// rows (12 MB of input and output, or one row).  A call takes one from the device's pool and puts it back; the pool keeps at most
// KEEP of them (evb_trim_cache gives them back).
constexpr int PRED_SLOTS = 3;
struct PredWs {
    struct Slot {
        cudaStream_t st = nullptr;
        cudaEvent_t done = nullptr, t0 = nullptr, t1 = nullptr;
        char *pin_in = nullptr, *pin_out = nullptr;
        void *d_in = nullptr, *d_aux = nullptr;
        size_t cap_pin_in = 0, cap_pin_out = 0, cap_in = 0, cap_aux = 0;
    } s[PRED_SLOTS];
    cudaEvent_t start = nullptr; // of a timed call
    int dev = 0;
};
constexpr size_t KEEP = 4;
struct PredPool { std::mutex mu; std::vector<PredWs *> free_ws; };
PredPool g_pred_pool[64];

void ws_delete(PredWs *w) {
    for (auto &s : w->s) {
        if (s.st) { cudaStreamSynchronize(s.st); cudaStreamDestroy(s.st); }
        if (s.done) cudaEventDestroy(s.done);
        if (s.t0) cudaEventDestroy(s.t0);
        if (s.t1) cudaEventDestroy(s.t1);
        if (s.pin_in) cudaFreeHost(s.pin_in);
        if (s.pin_out) cudaFreeHost(s.pin_out);
        evb_dev_free(s.d_in);
        evb_dev_free(s.d_aux);
    }
    if (w->start) cudaEventDestroy(w->start);
    delete w;
}
struct WsGuard { // the device is current
    PredWs *w = nullptr;
    explicit WsGuard(int dev) {
        if (dev < 64) {
            std::lock_guard<std::mutex> g(g_pred_pool[dev].mu);
            if (!g_pred_pool[dev].free_ws.empty()) { w = g_pred_pool[dev].free_ws.back(); g_pred_pool[dev].free_ws.pop_back(); return; }
        }
        w = new PredWs();
        w->dev = dev;
    }
    ~WsGuard() {
        for (auto &s : w->s) if (s.st) cudaStreamSynchronize(s.st); // an error may have left work behind
        if (w->dev < 64) {
            std::lock_guard<std::mutex> g(g_pred_pool[w->dev].mu);
            if (g_pred_pool[w->dev].free_ws.size() < KEEP) { g_pred_pool[w->dev].free_ws.push_back(w); return; }
        }
        ws_delete(w);
    }
};
int32_t slot_streams(PredWs::Slot &s, bool timed) {
    if (!s.st) EVB_CUDA(cudaStreamCreateWithFlags(&s.st, cudaStreamNonBlocking));
    if (!s.done) EVB_CUDA(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
    if (timed && !s.t0) { EVB_CUDA(cudaEventCreate(&s.t0)); EVB_CUDA(cudaEventCreate(&s.t1)); }
    return EVB_OK;
}
int32_t pinned_reserve(char *&p, size_t &cap, size_t bytes) {
    if (cap >= bytes) return EVB_OK;
    if (p) { cudaFreeHost(p); p = nullptr; cap = 0; }
    const size_t want = (std::max<size_t>(bytes, 65536) + 65535) & ~(size_t)65535;
    EVB_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&p), want, cudaHostAllocDefault));
    cap = want;
    return EVB_OK;
}
int32_t device_reserve(void *&p, size_t &cap, size_t bytes) {
    if (cap >= bytes) return EVB_OK;
    evb_dev_free(p);
    p = nullptr; cap = 0;
    EVB_CUDA(evb_dev_alloc(&p, bytes));
    cap = bytes;
    return EVB_OK;
}

constexpr int MAX_SMEM = 227 * 1024;
template <typename K>
int32_t allow_smem(K kern, size_t bytes) { // more than the default 48 KB of dynamic shared memory
    if (bytes > 48 * 1024) EVB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
    return EVB_OK;
}

// which kernel takes a chunk of n rows (what one launch gets, not what the call has)
enum { PK_ONE, PK_MID, PK_TILES, PK_STAGED, PK_WIDE };
struct PredPlan { int kind, rows, TB; size_t smem; };
PredPlan plan_kernel(const evb_model &m, int n, bool more, int num_sms) { // more: another chunk's kernel will run beside this one
    PredPlan p{PK_WIDE, 256, 0, 0};
    const int FW = (m.nfeats + 3) / 4;
    const size_t tree = (size_t)m.tw * 4;
    // a CTA per row while the rows alone do not give every SM several of the 32-row CTAs of the next kernel
    const size_t one = (size_t)FW * 4 + (size_t)ONE_THREADS * m.K * 4;
    if (n <= 4 * num_sms && one <= 96 * 1024) return {PK_ONE, 1, 0, one};
    // Staged: the largest CTA that still gives every SM one, as long as two blocks of trees fit beside its rows.  One thread a row needs rows:
    // below `mid_rows` of a launch the next kernel is faster.  ms of kernels of a call, staged and tiles: 4M x 10, depth 6 (285k rows a
    // chunk) 3.10 and 3.65; 1M x 28 five classes, depth 8 (79k) 2.95 and 2.68; 300k x 6, depth 9 (50k) 0.52 and 0.43.
    const int mid_rows = 64 * 1024;
    if (n > mid_rows) {
        for (int rows = 1024; rows >= 128; rows >>= 1) {
            if (rows > 256 && (n + rows - 1) / rows < num_sms) continue;
            const size_t rb = (size_t)rows * FW * 4, room = (size_t)200 * 1024;
            if (rb + 2 * tree > room) continue;
            const int TB = (int)std::min<size_t>(8, (room - rb) / (2 * tree));
            return {PK_STAGED, rows, TB, rb + 2 * (size_t)TB * tree};
        }
    }
    {
        // The fewest groups of rows a CTA with which all CTAs have an SM at once (chunks overlap: twice their rows, but the last one's time shows): every CTA copies all trees.  us of a
        // call, 1, 2 and 4 groups: 900 x 12 seven classes 59, 63, 71; 9k x 12 seven classes 112, 99, 107; 20k x 28 five classes, in chunks (every one with two times its rows) 203, 180, 190;
        // 6k x 30, depth 10 115, 122, 132; 90k x 12 seven classes, in chunks 529, 383, 342.  k_predict_mid: 77, 122, 206, 127, 489.
        const int RG = std::max(1, std::min(4, (n * (more ? 2 : 1) + 32 * num_sms - 1) / (32 * num_sms)));
        const size_t R = 32 * RG, room = (size_t)216 * 1024, bins = FW * R * 4, per = 2 * (tree + m.K * R * 4);
        if (bins + per <= room) {
            const int most = (int)((room - bins) / per), walk = TILE_WARPS / RG - 1;
            int TB = std::min(most, 64);
            if (TB > walk) TB = TB / walk * walk;
            return {PK_TILES, RG, TB, bins + (size_t)TB * per};
        }
    }
    const size_t rb = (size_t)FW * 128;
    int TB = std::max(1, 96 / m.K); // 2 x TB x K x 128 bytes <= 24 KB
    if (TB > (MID_WARPS - 1) * MID_ILP) TB = TB / ((MID_WARPS - 1) * MID_ILP) * ((MID_WARPS - 1) * MID_ILP);
    const size_t mid = rb + (size_t)2 * TB * m.K * 128;
    if (mid <= MAX_SMEM - 1024) return {PK_MID, 32, TB, mid};
    return p;
}

template <int K, typename T>
int32_t launch_tiles(const PredPlan &p, const PredArgs &a, cudaStream_t st) {
    EVB_CHECK(allow_smem(k_predict_tiles<K, T>, p.smem));
    k_predict_tiles<K, T><<<(a.n + 32 * p.rows - 1) / (32 * p.rows), TILE_WARPS * 32, p.smem, st>>>(a, p.rows, p.TB);
    return EVB_OK;
}
template <int KMAX, typename T>
int32_t launch_t(const PredPlan &p, PredArgs &a, uint32_t *xw, cudaStream_t st) {
    if (p.kind == PK_ONE) {
        EVB_CHECK(allow_smem(k_predict_one<KMAX, T>, p.smem));
        k_predict_one<KMAX, T><<<a.n, ONE_THREADS, p.smem, st>>>(a);
    } else if (p.kind == PK_MID) {
        EVB_CHECK(allow_smem(k_predict_mid<KMAX, T>, p.smem));
        k_predict_mid<KMAX, T><<<(a.n + 31) / 32, MID_WARPS * 32, p.smem, st>>>(a, p.TB);
    } else if (p.kind == PK_TILES) {
        if constexpr (KMAX > 8) EVB_CHECK((launch_tiles<64, T>(p, a, st)));
        else switch (a.K) { // outputs known at compile time: adding a tree is a third shorter
            case 1: EVB_CHECK((launch_tiles<1, T>(p, a, st))); break;
            case 2: EVB_CHECK((launch_tiles<2, T>(p, a, st))); break;
            case 3: EVB_CHECK((launch_tiles<3, T>(p, a, st))); break;
            case 4: EVB_CHECK((launch_tiles<4, T>(p, a, st))); break;
            case 5: EVB_CHECK((launch_tiles<5, T>(p, a, st))); break;
            case 6: EVB_CHECK((launch_tiles<6, T>(p, a, st))); break;
            case 7: EVB_CHECK((launch_tiles<7, T>(p, a, st))); break;
            default: EVB_CHECK((launch_tiles<8, T>(p, a, st)));
        }
    } else if (p.kind == PK_STAGED) {
        EVB_CHECK(allow_smem(k_predict_staged<KMAX, T>, p.smem));
        k_predict_staged<KMAX, T><<<(a.n + p.rows - 1) / p.rows, p.rows, p.smem, st>>>(a, p.TB);
    } else {
        k_bin_rows<T><<<dim3((a.n + 255) / 256, std::min(a.FW, 64)), 256, 0, st>>>(a, xw);
        k_predict_wide<KMAX><<<(a.n + 255) / 256, 256, 0, st>>>(a, xw);
    }
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}
template <typename T>
int32_t launch_k(const PredPlan &p, PredArgs &a, uint32_t *xw, cudaStream_t st) {
    if (a.K <= 1) return launch_t<1, T>(p, a, xw, st);
    if (a.K <= 2) return launch_t<2, T>(p, a, xw, st);
    if (a.K <= 8) return launch_t<8, T>(p, a, xw, st);
    return launch_t<64, T>(p, a, xw, st);
}

// Models most of whose paths end early: a lane leaves the loop there.  That is two instructions more a level and lanes that wait for each other, so it pays
// where little is left of the complete trees, and not where a few warps an SM wait for their loads.  us of a call, to the last level and leaving, 200 trees of
// depth 11, one output, at shares of the inner nodes that test something: 500k rows 1.0 1938 and 2050, 0.37 1920 and 1931, 0.14 1908 and 1793, 0.11 1922 and 1471; 20k rows
// 0.14 174 and 177, 0.11 175 and 167; 2k rows 0.11 76 and 84; depth 8, 500k rows 0.26 1377 and 1298, 0.10 1369 and 1239.
constexpr int EARLY_ROWS = 8 * 1024;

// Rows of a chunk, of in_row bytes going up and out_row coming back each.
// Big enough that a chunk's fixed costs (about 15 us of launches) vanish in its transfer, small enough that the
// first transfer and the last kernel, which nothing overlaps with, do not show; three of them stay in the host's L3.  10M x 50
// floats, on a slow box: 4 MB 73 ms, 8 MB 56, 12 and 16 MB 47, 24 MB 46; 500k x 100: 6.5, 4.4, 4.05, 4.1, 4.8.
int64_t chunk_rows(int64_t nobs, size_t in_row, size_t out_row) {
    const size_t total = (size_t)nobs * (in_row + out_row);
    size_t cbytes = total / 6;
    cbytes = std::min<size_t>(std::max<size_t>(cbytes, (size_t)1 << 20), (size_t)12 << 20);
    // Whole CTAs of the kernels where that many rows fit; wide rows: as many as fit, so that no slot pins more than 12 MB (or one row).
    int64_t chunk = (int64_t)std::max<size_t>(1, cbytes / (in_row + out_row));
    if (chunk > 32) chunk -= chunk % (chunk >= 1024 ? 1024 : 32);
    return std::min<int64_t>(chunk, nobs);
}

// x: host rows (x_type 0 float, 2 double, -1 bins); out / leaf_idx: host.  `check`: compare the model's sources while the
// GPU works and return EVB_ERR_STALE when they changed.
int32_t predict_rows(const evb_model &m, int ntrees, const void *x, int x_type, int row_major, int64_t nobs, int apply_link, float *out,
                     uint32_t *leaf_idx, double *ms_out, bool check) {
    if (ms_out) *ms_out = 0.0;
    if (nobs == 0) return EVB_OK;
    WsGuard g(m.device);
    PredWs &w = *g.w;
    static int num_sms[64] = {};
    int sms = m.device < 64 ? num_sms[m.device] : 0;
    if (sms == 0) {
        EVB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device));
        if (m.device < 64) num_sms[m.device] = sms;
    }
    const size_t es = x_type < 0 ? 1 : x_type == EVB_F64 ? 8 : 4;
    const size_t in_row = es * m.nfeats, out_row = 4 * ((size_t)m.K + (leaf_idx ? ntrees : 0));
    const int64_t chunk = chunk_rows(nobs, in_row, out_row);
    // one row or a few: the kernel reads them from pinned memory itself
    const bool zero_copy = (size_t)nobs * in_row <= (size_t)16 * 1024;
    PredArgs a;
    a.row_major = row_major; a.nedges = m.nedges; a.nfeats = m.nfeats; a.FW = (m.nfeats + 3) / 4;
    a.edges = x_type == EVB_F64 ? (const void *)m.d_e64 : (const void *)m.d_e32;
    a.trees = m.d_trees; a.ni = m.ni; a.tw = m.tw; a.levels = m.levels; a.K = m.K; a.loss = m.loss; a.ntrees = ntrees; a.apply_link = apply_link;
    int64_t first[PRED_SLOTS] = {-1, -1, -1};
    int rows_in[PRED_SLOTS] = {};
    double ms = 0.0, until = 0.0; // ms during which kernels ran, up to `until` ms after the start (chunks overlap)
    auto collect = [&](int q) -> int32_t { // results of the chunk in slot q -> the caller's arrays
        PredWs::Slot &s = w.s[q];
        if (first[q] < 0) return EVB_OK;
        EVB_CUDA(cudaStreamSynchronize(s.st));
        const int64_t r0 = first[q], nr = rows_in[q];
        evb_copy_packed(s.pin_out, out + r0, (size_t)nr * 4, (size_t)nobs * 4, 0, (size_t)nr * 4 * m.K, false);
        if (leaf_idx) evb_copy_packed(s.pin_out + (size_t)nr * 4 * m.K, leaf_idx + r0, (size_t)nr * 4, (size_t)nobs * 4, 0, (size_t)nr * 4 * ntrees, false);
        float b = 0.f, e = 0.f;
        if (ms_out && cudaEventElapsedTime(&b, w.start, s.t0) == cudaSuccess && cudaEventElapsedTime(&e, w.start, s.t1) == cudaSuccess && e > until) {
            ms += e - std::max<double>(b, until);
            until = e;
        }
        first[q] = -1;
        return EVB_OK;
    };
    int q = 0;
    for (int64_t r0 = 0; r0 < nobs; r0 += chunk, q = (q + 1) % PRED_SLOTS) {
        PredWs::Slot &s = w.s[q];
        const int64_t nr = std::min<int64_t>(chunk, nobs - r0);
        EVB_CHECK(collect(q));
        EVB_CHECK(slot_streams(s, ms_out != nullptr));
        if (ms_out && r0 == 0) {
            if (!w.start) EVB_CUDA(cudaEventCreate(&w.start));
            EVB_CUDA(cudaEventRecord(w.start, s.st));
        }
        EVB_CHECK(pinned_reserve(s.pin_in, s.cap_pin_in, (size_t)chunk * in_row));
        EVB_CHECK(pinned_reserve(s.pin_out, s.cap_pin_out, (size_t)chunk * out_row));
        // rows r0 .. r0 + nr: one piece of a row-major matrix, one segment per feature of a column-major one
        const char *xs = static_cast<const char *>(x);
        if (row_major) evb_copy_packed(s.pin_in, xs + (size_t)r0 * in_row, (size_t)nr * in_row, 0, 0, (size_t)nr * in_row, true);
        else evb_copy_packed(s.pin_in, xs + (size_t)r0 * es, (size_t)nr * es, (size_t)nobs * es, 0, (size_t)nr * in_row, true);
        a.n = (int)nr; a.ld = row_major ? m.nfeats : nr;
        a.early = m.early && nr > EARLY_ROWS;
        a.vec = row_major && es == 4 && (m.nfeats & 3) == 0;
        a.x = s.pin_in;
        if (!zero_copy) {
            EVB_CHECK(device_reserve(s.d_in, s.cap_in, (size_t)chunk * in_row));
            EVB_CUDA(cudaMemcpyAsync(s.d_in, s.pin_in, (size_t)nr * in_row, cudaMemcpyHostToDevice, s.st));
            a.x = s.d_in;
        }
        a.out = reinterpret_cast<float *>(s.pin_out); a.out_ld = nr;
        a.leaf_idx = leaf_idx ? reinterpret_cast<uint32_t *>(s.pin_out + (size_t)nr * 4 * m.K) : nullptr;
        const PredPlan p = plan_kernel(m, (int)nr, r0 + nr < nobs, sms);
        if (p.kind == PK_WIDE) EVB_CHECK(device_reserve(s.d_aux, s.cap_aux, (size_t)chunk * a.FW * 4));
        if (ms_out) EVB_CUDA(cudaEventRecord(s.t0, s.st));
        uint32_t *xw = static_cast<uint32_t *>(s.d_aux);
        EVB_CHECK(x_type < 0 ? launch_k<uint8_t>(p, a, xw, s.st) : x_type == EVB_F64 ? launch_k<double>(p, a, xw, s.st) : launch_k<float>(p, a, xw, s.st));
        if (ms_out) EVB_CUDA(cudaEventRecord(s.t1, s.st));
        first[q] = r0; rows_in[q] = (int)nr;
    }
    if (check && !model_current(&m)) { evb_set_error("evb_model_predict: the model's trees changed since they were packed"); return EVB_ERR_STALE; }
    for (int k = 0; k < PRED_SLOTS; ++k, q = (q + 1) % PRED_SLOTS) EVB_CHECK(collect(q)); // oldest first
    if (ms_out) *ms_out = ms;
    return EVB_OK;
}

} // namespace

// gives the kept work buffers of a device back (the device is current)
void evb_predict_trim(int device) {
    std::vector<PredWs *> ws;
    { std::lock_guard<std::mutex> g(g_pred_pool[device].mu); ws.swap(g_pred_pool[device].free_ws); }
    for (PredWs *w : ws) ws_delete(w);
}

extern "C" int32_t evb_model_predict(const evb_model *m, int32_t ntrees, const void *x, int32_t x_dtype, int32_t x_row_major, int64_t nobs,
                                     int32_t apply_link, float *out, uint32_t *leaf_idx, double *kernel_ms) {
    if (!m || !x || !out || nobs < 0 || ntrees < 0 || ntrees > m->ntrees || (x_dtype != EVB_F32 && x_dtype != EVB_F64)) {
        evb_set_error("evb_model_predict: invalid argument");
        return EVB_ERR_ARG;
    }
    EVB_CUDA(cudaSetDevice(m->device));
    try { return predict_rows(*m, ntrees, x, x_dtype, x_row_major, nobs, apply_link, out, leaf_idx, kernel_ms, true); }
    catch (const std::bad_alloc &) { return no_host_memory(); }
}

extern "C" int32_t evb_test_predict_plan(const evb_model *m, int32_t x_dtype, int64_t nobs, int32_t leaf_trees, int64_t launches[5]) {
    if (!m || nobs < 1 || leaf_trees < 0 || leaf_trees > m->ntrees || !launches || (x_dtype != -1 && x_dtype != EVB_F32 && x_dtype != EVB_F64)) {
        evb_set_error("evb_test_predict_plan: invalid argument");
        return EVB_ERR_ARG;
    }
    int sms = 0;
    EVB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device));
    for (int k = 0; k < 5; ++k) launches[k] = 0;
    const int64_t chunk = chunk_rows(nobs, (size_t)(x_dtype < 0 ? 1 : x_dtype == EVB_F64 ? 8 : 4) * m->nfeats, 4 * ((size_t)m->K + leaf_trees));
    for (int64_t r0 = 0; r0 < nobs; r0 += chunk) launches[plan_kernel(*m, (int)std::min(chunk, nobs - r0), r0 + chunk < nobs, sms).kind] += 1;
    return EVB_OK;
}

// one call with trees that are packed for it: evb_predict (bins) and evb_predict_x (raw features)
static int32_t predict_once(int32_t device, int32_t loss, int32_t K, int32_t ntrees, int32_t nn, const int64_t *feat, const uint8_t *cond_bin,
                            const uint8_t *split, const float *leaf_pred, const void *x, int x_type, int32_t x_row_major, const void *edges,
                            int32_t nedges, int64_t nobs, int32_t nfeats, const uint8_t *feattypes, int32_t apply_link, float *out,
                            uint32_t *leaf_idx, double *ms_out) {
    if (!feat || !cond_bin || !split || !leaf_pred || !x || !out || nobs < 0 || nn < 1) { evb_set_error("evb_predict: invalid argument"); return EVB_ERR_ARG; }
    EVB_CHECK(model_args(loss, K, ntrees, nfeats));
    EVB_CHECK(evb_check_device(device));
    if (nobs == 0) return EVB_OK;
    evb_model m;
    m.device = device; m.loss = loss; m.K = K;
    int32_t rc;
    try {
        std::vector<const void *> src((size_t)ntrees * 4);
        std::vector<int32_t> nodes(ntrees, nn);
        for (int t = 0; t < ntrees; ++t) {
            const size_t o = (size_t)t * nn;
            src[4 * t] = feat + o; src[4 * t + 1] = cond_bin + o; src[4 * t + 2] = split + o; src[4 * t + 3] = leaf_pred + o * K;
        }
        rc = model_fill(&m, ntrees, src.data(), nodes.data(), edges, x_type < 0 ? EVB_F32 : x_type, nedges, nfeats, feattypes, false);
        if (rc == EVB_OK) rc = predict_rows(m, ntrees, x, x_type, x_row_major, nobs, apply_link, out, leaf_idx, ms_out, false);
    } catch (const std::bad_alloc &) { rc = no_host_memory(); }
    evb_dev_free(m.block);
    return rc;
}

extern "C" int32_t evb_predict(int32_t device, int32_t loss, int32_t K, int32_t ntrees, int32_t nn, const int64_t *feat,
                               const uint8_t *cond_bin, const uint8_t *split, const float *leaf_pred, const uint8_t *x_bin,
                               int64_t nobs, int32_t nfeats, const uint8_t *feattypes, int32_t apply_link, float *out,
                               uint32_t *leaf_idx) {
    if (!x_bin) { evb_set_error("evb_predict: x_bin is null"); return EVB_ERR_ARG; }
    return predict_once(device, loss, K, ntrees, nn, feat, cond_bin, split, leaf_pred, x_bin, -1, 0, nullptr, 0, nobs, nfeats, feattypes, apply_link,
                        out, leaf_idx, nullptr);
}

extern "C" int32_t evb_predict_x(int32_t device, int32_t loss, int32_t K, int32_t ntrees, int32_t nn, const int64_t *feat,
                                 const uint8_t *cond_bin, const uint8_t *split, const float *leaf_pred, const void *x, int32_t x_dtype,
                                 int32_t x_row_major, const void *edges, int32_t nedges, int64_t nobs, int32_t nfeats,
                                 const uint8_t *feattypes, int32_t apply_link, float *out, uint32_t *leaf_idx, double *kernel_ms) {
    if (!x) { evb_set_error("evb_predict_x: x is null"); return EVB_ERR_ARG; }
    if (!edges || nedges < 1 || nedges > 254 || (x_dtype != EVB_F32 && x_dtype != EVB_F64)) {
        evb_set_error("evb_predict_x: edges / dtype invalid");
        return EVB_ERR_ARG;
    }
    return predict_once(device, loss, K, ntrees, nn, feat, cond_bin, split, leaf_pred, x, x_dtype, x_row_major, edges, nedges, nobs, nfeats, feattypes,
                        apply_link, out, leaf_idx, kernel_ms);
}
