// Internal declarations shared by the translation units of libevotrees_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string>
#include <vector>
#include "../../include/evb.h"

#define EVB_VERSION 1

// ---- error plumbing -------------------------------------------------------------------------------
void evb_set_error(const char *fmt, ...);
#define EVB_CUDA(call)                                                                                \
    do {                                                                                              \
        cudaError_t _e = (call);                                                                      \
        if (_e != cudaSuccess) {                                                                      \
            evb_set_error("CUDA error %s at %s:%d (%s)", cudaGetErrorString(_e), __FILE__, __LINE__, #call); \
            return EVB_ERR_CUDA;                                                                      \
        }                                                                                             \
    } while (0)
#define EVB_CHECK(call)                    \
    do {                                   \
        int32_t _s = (call);               \
        if (_s != EVB_OK) return _s;       \
    } while (0)

// device-side error codes written to evb_handle::d_err
enum { EVB_DERR_NONE = 0, EVB_DERR_WAIT_FULL = 1, EVB_DERR_WAIT_EMPTY = 2, EVB_DERR_BIN_RANGE = 3, EVB_DERR_PEER = 5, EVB_DERR_NAN = 6, EVB_DERR_GRID = 7 };

// ---- geometry constants ---------------------------------------------------------------------------
constexpr int EVB_TILE_ROWS = 32;    // rows per staged tile (one per producer lane)
constexpr int EVB_PART_CHUNK = 1024; // rows of the largest partition chunk
constexpr int EVB_PART_THREADS = 256;
constexpr int EVB_MAX_DEPTH = 15;
constexpr int EVB_GEN_WORDS = 12;    // 32-bit words of a generator state

enum { EVB_MASK_NONE = 0, EVB_MASK_HOST = 1, EVB_MASK_PCG = 2 }; // rows: all, a mask from the host, a mask made on the device
enum { EVB_KIND_NONE = 0, EVB_KIND_BUILD = 1, EVB_KIND_SUB = 2 };

// Per-level plan, device resident.  Written by k_tree_begin / k_sel_scan (root) and the last CTA of k_partition.
struct LevelPlan {
    int32_t nbuild;   // build slots used at this level
    int32_t npl;      // sibling pairs at this level (1 at the root)
    int64_t R;        // rows (local) inside build nodes
    int32_t n_sel;    // rows selected by the row mask (root only)
    int32_t total;    // rows of all sibling pairs
};

// geometry of the register-direct fixed-point histogram kernel (evb_histq2.cu)
struct Q2Geom {
    int NC;        // 16-byte chunks (16 features) per CTA group
    int ngroups;   // CTA groups (grid.y); xH rows hold ngroups * NC chunks
    int ntail;     // features kept beside the gradient word in xE (nfeats % 16 when that is 1..4, else 0)
    int nmain;     // features kept in xH
    int RSH;       // bytes per row of xH
    int G;         // grid.x
    int min_rows;  // rows per CTA below which fewer CTAs take part
    size_t smem;
};

// geometry of the integer histogram kernel for any loss (evb_histg.cuh)
constexpr int EVB_MAX_Q = 72; // quantised channels: 2 K + 1, K <= 32
struct HGeom {
    int nq, per, ngc;   // channels; channels per CTA; channel groups (grid.z)
    int W, wper, ngf;   // words of a row; words per CTA; feature groups (grid.y)
    int pack, cnt;      // packed words of unit-weight least squares; a plane of row counts in channel group 0
    int hb, TE, min_rows, threads, G;
    int queue;          // 32-bit words of shared memory before the row queue
    size_t smem;
};

// geometry of the kernel that grows a whole tree (evb_grow.cu)
struct GrowGeom {
    bool on;
    int lw, NG, NR, rpc; // log2 of the words of four features a CTA takes; CTAs side by side: feature groups x row ranges; rows of a range
    int hb;              // bits of the high words (the level kernels have their own: HGeom)
    uint8_t lc[10];      // [level] log2 of the columns of an image
    bool cluster;        // the grid is one cluster; offsets of what its CTAs keep in shared memory for it (GrowArgs)
    int o_x, o_sum, o_cnt, o_best, o_hist, fo;
    size_t smem;
};

struct evb_handle {
    evb_params p;
    int K, C, B, D, nn;        // nn = 2^D-1
    int Ce;                    // channels of a record with its weight: C, or K+1 for mse where h = 2w is rebuilt from w
    int nfeats, RS;            // RS: bytes per row of xT (16, or a multiple of 32)
    int64_t n;                 // local rows
    int dev, num_sms;
    cudaStream_t st;
    int busy;

    // row data
    void *edges_d;     // edges of the raw matrix the handle was made from (evb_create_m), dtype edges_dtype
    int edges_dtype, nedges;
    uint8_t *xT;       // [n][RS]  observation-major bins (1..B), zero padded; null when xH / xE hold them
    uint8_t *xC;       // [nfeats][n] feature-major copy (the layout of the caller's x_bin) read by the row partition
    float *grad;       // [n][nq]  gradient records (grad_row, evb_rows.cu)
    float *pred;       // [n][K]
    void *y;           // float [n][ycols] or uint32 [n]
    int y_dtype, ycols;
    uint32_t *nidx;    // [n] leaf of each row from the training traversal
    uint32_t *rows[2]; // [n] ping-pong row lists, segments ordered by node
    uint8_t *mask_d;   // [n]
    uint8_t *feattypes_d; // [nfeats]
    int32_t *mono_d;      // [nfeats]
    uint64_t *gen_d;      // [6] generator of the row mask (see k_sel_pcg), followed by js_d in the same block: one copy per tree
    uint32_t *js_d;       // [nfeats] 0-based feature id per slot
    int F;                // njs of the current tree
    bool grads_fresh;     // gradients already computed for the next round (fused into finalize)
    int bag_idx;

    // node state, indexed by heap id 0..nn (0 unused); children of level D-1 nodes need ids < 2^D
    int32_t *seg_start, *seg_cnt; // local row segment of each node
    int32_t *cur_l, *cur_r;       // partition cursors of split nodes
    uint32_t *ticket;             // [nn+2] features of a node whose scan is done; entry 0: CTAs of k_partition that are done
    int4 *pl;                     // 2 x [maxslots+1] sibling pairs of a level (PartArgs::pl)
    uint8_t *kind;
    int32_t *bslot;
    double *nsum;                 // [nn+1][C]
    // tree arrays (device), heap id - 1
    int32_t *t_feat; uint8_t *t_bin; uint8_t *t_split; float *t_gain; float *t_w; float *t_pred;
    uint32_t *t_packed;           // per node: feat0 | bin<<16 | split<<24 | numeric<<25 (for traversal)

    // plans
    LevelPlan *plan;       // [D+1]
    int32_t *cum;          // [maxslots+1] exclusive prefix of build-node row counts (current level)
    int32_t *slot_node;    // [maxslots]
    int32_t *rbase;        // [maxslots] place in the row list of a slot's first row, minus cum[slot] (behind slot_node)
    int maxslots;
    int32_t *scan_tmp;     // block counts for the mask compaction
    double *fbest_gain;    // [nodes of a level][nfeats] per-feature best split of the scan
    int32_t *fbest_bin;
    double *fbest_left;    // [nodes of a level][nfeats][C] left sums of that split (one output, or evb_scan_multi)
    double *obl_gain;      // oblivious trees: [nodes of a level + 1][nfeats * B] gain of every candidate, last row = level totals
    double *obl_best;      // [2] gain and candidate index (-1: none) of the level's shared split
    int *d_err;            // device error word
    int *h_err;            // pinned mirror

    // evaluation shard (evb_eval_attach): every grown tree is applied to ev_pred and the metric sums go to d_evsum
    int64_t ev_n;      // 0 = none attached
    uint8_t *ev_xT;    // [ev_n][RS]
    void *ev_y; float *ev_w; float *ev_pred;
    double *ev_part;   // [ev_blocks][2] per-block partial sums
    double *d_evsum;   // [2] inside the tree block: sum w*value, sum w
    int ev_metric, ev_blocks;
    double last_eval[2]; // sums of the tree collected last

    // fixed-point gradients (evb_histg.cuh)
    bool unit_w;          // no weights were given: the w channel is a row count
    bool gradq_valid;     // the fixed-point words are those of the current gradients
    int nq, ng;           // quantised channels; those of them that change from round to round (all but the weight)
    HGeom hgeo;
    int32_t *gradq;       // words of all rows, channel group by channel group
    unsigned *d_gmax;     // [2][nq] bits of max |g| over the rows, filled by the gradient kernels
    int gmax_sel;         // which of the two belongs to the gradients in place (evb_gmax)
    double *d_qinv;       // [nq] unit of every channel's sums
    unsigned *d_signs;    // [nq] signs of the infinities a channel has had (QuantArgs::signs)
    int SC;               // feature columns per bin of the accumulators
    unsigned long long *hsum_q;   // [maxslots][B][nq][SC] sums of q per build slot
    uint32_t *hcnt_q;             // [maxslots][B][SC] row counts
    unsigned long long *hlow_q;   // [maxslots][SC][nq][B] sums of what the words of a row leave (null: packed words leave nothing)
    uint32_t *low;                // [nn+2] build slots of a level that have something in hlow_q (evb_low_slot, evb_low_any)

    // register-direct variant (mse, one target, unit weights, many rows): rows as 16-byte chunks + {q, tail bins} per row
    bool use_q2;
    Q2Geom q2;
    uint8_t *xH;                  // [n][q2.RSH]
    uint2 *xE;                    // [n] {fixed-point gradient, bins of the tail features}

    // quantile loss: work memory of the per-leaf order-statistic selection
    uint32_t *qs_cnt, *qs_prefix, *qs_rank; float *qs_gamma;

    // whole trees in one launch
    GrowGeom grow;
    unsigned long long *g_sum, *g_low; // [2][maxslots][nfeats][nq][B]
    uint32_t *g_cnt;                   // [2][maxslots][nfeats][B]
    double2 *g_best;
    uint32_t *g_bar;
    unsigned grow_polls;               // of a wait at the grid's barrier before the tree is given up
    bool failed;                       // a tree was given up: predictions, gradients and sums are in no defined state, calls are refused

    // histograms
    double *hist;     // [2^(D-2) nodes][F][C][B] retained for the subtraction trick
    int hist_nodes;   // nodes with id < hist_nodes are retained
    double *hcomp;    // [maxslots][F][C][B] freshly built histograms of the level (exchanged between ranks; null on one GPU)

    // pinned host staging, double buffered so that tree t+1 can be enqueued before tree t is collected
    void *h_tree[2]; size_t h_tree_bytes;
    uint32_t *h_js[2];              // EVB_GEN_WORDS words of generator state, then the column sample
    cudaEvent_t ev_done[2];
    int tree_seq, pending;          // trees started / started but not yet collected
    // one CUDA graph per variant of the per-tree launch sequence (mask, gradients first, gradients fused, slot)
    bool use_graphs;
    cudaGraphExec_t graph[128];
    int graph_calls[128];
    int64_t graph_launches[128][EVB_NTIMERS];
    int graph_mask_cond;

    // multi-GPU
    void *nccl_comm; int rank, world;
    uint8_t nccl_id[128]; bool nccl_pending; // id recorded by evb_comm_init; the communicator is created by the first collective
    // peer access between the ranks' processes (CUDA IPC): histograms are summed by peer loads inside the split scan
    bool p2p;
    double *peer_hcomp[8]; double *peer_cand[8]; int *peer_flags[8];
    double *hsum; // sums over the ranks of the owned feature slots of hcomp
    void *ipc_opened[24]; int n_ipc_opened;
    int *d_barrier_seq; // device counter of the peer barriers passed

    // timing
    bool timing;
    std::vector<cudaEvent_t> ev; // pairs
    cudaEvent_t ev_tot[2];       // bracket of one whole evb_grow_tree
    std::vector<int> ev_class;
    size_t ev_used;
    evb_timings tm;
};

// Plain launches: kernels that were launched before their predecessor's end (programmatic dependent launch) and waited for it cost time
// at every size but the smallest -- CTAs that wait take the places of others.  ms per tree, with and without it: 1503 x 7 logloss 0.087 and
// 0.088, 100k x 10 0.096 and 0.094, 60k x 77 poisson 0.150 and 0.129, 250k x 33 weighted 0.151 and 0.144, 200k x 50 gaussian 0.209 and 0.190,
// 1M x 100 (half of the rows) 0.232 and 0.236, 2M x 20 logloss 0.317 and 0.303.
#ifdef __CUDACC__
template <typename... P, typename... A>
inline cudaError_t evb_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = st;
    return cudaLaunchKernelEx(&c, kern, P(args)...);
}
#endif

// ---- launchers (each enqueues on h->st and returns a status) ---------------------------------------
// evb_rows.cu
int32_t evb_launch_transpose(evb_handle *h, const uint8_t *xcol_dev, int64_t ld, int64_t nrows, int j0, int nj, uint8_t *xT, int RS, cudaStream_t st);
int32_t evb_launch_grads(evb_handle *h);
int32_t evb_launch_rows_init(evb_handle *h, int use_mask, uint8_t mask_cond);
int32_t evb_pcg_tables(int dev);
void evb_pcg_advance(uint64_t gen[6], int64_t n);
int32_t evb_launch_finalize(evb_handle *h, bool compute_grads, int mode, void *publish_to); // pinned host memory for the finished tree or null; mode: see FinArgs in evb_rows.cu
int32_t evb_launch_quantile_leaves(evb_handle *h, bool use_mask, uint8_t mask_cond);
int32_t evb_launch_nidx_from_partition(evb_handle *h, uint32_t *out_dev);
int32_t evb_launch_eval(evb_handle *h, const float *fixed_leaf_dev, void *publish_to);
int32_t evb_upload_binarize(evb_handle *h, const void *x, int32_t dtype, const void *edges, int32_t nedges); // raw host matrix -> h->xC
// evb_hist.cu
int evb_hist_mode_env();
// evb_histg.cu
int32_t evb_hg_configure(evb_handle *h);
int evb_hg_round_bits(const evb_handle *h);
size_t evb_hg_q_words(const evb_handle *h);
int32_t evb_launch_histg(evb_handle *h, int level);
int32_t evb_launch_acc_clear(evb_handle *h, int level);
int32_t evb_launch_acc_to_hcomp(evb_handle *h, int level);
// Rows of a level are dealt out to the CTAs of a histogram kernel with this many more for every build node: a flush costs what a
// few hundred rows do, so a CTA with several small nodes gets fewer rows than one inside a large node.  Per tree, equal ranges
// and 512 rows at least, then padded ones and 256: 1503 x 7 0.096 -> 0.087 ms, 60k x 77 0.183 -> 0.150, 250k x 33 weighted
// 0.208 -> 0.190, 2M x 28 five classes 0.98 -> 0.94, 5M x 50 gaussian 1.51 -> 1.49.  Positions stay below 2^31.
static inline int evb_pad_rows(const evb_handle *h) {
    const long long room = (0x7fffffffll - h->n) / (h->maxslots > 0 ? h->maxslots : 1);
    return room < 512 ? (room < 0 ? 0 : (int)room) : 512;
}
// Several outputs scanned side by side (k_scan_multi).  Up to EVB_MULTI_K warps of a CTA, each with its output's sums in registers;
// more outputs, losses with a gain of their own and oblivious trees (every bin's gain is kept) take one warp per feature.
#define EVB_MULTI_K 8
static inline bool evb_scan_multi(const evb_handle *h) { return h->K >= 2 && h->K <= EVB_MULTI_K && h->C == 2 * h->K + 1 && h->p.loss < EVB_MAE && h->p.tree_type != 1; }
// The split scan reads the integer accumulators itself unless ranks exchange histograms as doubles.
static inline bool evb_acc_direct(const evb_handle *h) { return h->world == 1; }
// evb_handle::low, a stretch of 2^(level-1) words per level: its build slots (at most half of them below the root), and in its last
// word whether any slot has something (the root's only slot says so itself)
__host__ __device__ static inline size_t evb_low_slot(int level) { return (size_t)1 << (level - 1); }
__host__ __device__ static inline size_t evb_low_any(int level) { return ((size_t)1 << level) - 1; }
static inline double evb_hg_low_unit(int hb) { return 1.0 / (double)(1ull << (2 * hb + 2)); } // units of hlow_q (g_low) in those of hsum_q (g_sum)
// evb_histq2.cu
bool evb_q2_wanted(const evb_handle *h);
int32_t evb_q2_configure(evb_handle *h);
int32_t evb_q2_build_layout(evb_handle *h);
int32_t evb_q2_clear_layout(evb_handle *h);
int32_t evb_launch_histq2(evb_handle *h, int level);
// evb_grow.cu
void evb_grow_configure(evb_handle *h);
size_t evb_grow_sums(const evb_handle *h);
size_t evb_grow_cnts(const evb_handle *h);
size_t evb_grow_best(const evb_handle *h);
int32_t evb_launch_grow(evb_handle *h, bool masked, uint8_t mask_cond, int slot, bool next_grads);
constexpr int EVB_GROW_JS = 512;   // sampled columns that travel with a launch
static inline bool evb_grows_whole(const evb_handle *h) { return h->grow.on && h->world == 1; }
static inline bool evb_one_launch(const evb_handle *h, bool masked) { return evb_grows_whole(h) && !masked && (h->F == h->nfeats || h->F <= EVB_GROW_JS); }
// Maxima of |g| of the gradients in place and, when the tree kernel reads them while it makes the next ones, of those
static inline unsigned *evb_gmax(const evb_handle *h, bool next) { return h->d_gmax + (size_t)h->nq * (evb_grows_whole(h) && next ? h->gmax_sel ^ 1 : h->gmax_sel); }
// evb_tree.cu
int32_t evb_launch_tree_begin(evb_handle *h, bool quantize, bool all_rows, const uint32_t *gen_js_host);
int32_t evb_launch_scan(evb_handle *h, int level);
int32_t evb_launch_partition(evb_handle *h, int level); // rows of the level's split nodes, plan of the next level
int32_t evb_launch_lonely_barrier(evb_handle *h, int *flags, int *seq, unsigned max_polls);
int32_t evb_check_device(int device); // evb_rows.cu: makes `device` current
void evb_predict_trim(int device);       // evb_predict.cu: kept work buffers back to the block cache
// evb_matrix.cu
int64_t evb_matrix_rows(const evb_matrix *m);
int evb_matrix_feats(const evb_matrix *m);
int evb_matrix_dtype(const evb_matrix *m);
cudaError_t evb_matrix_join(const evb_matrix *m, cudaStream_t st);
int32_t evb_matrix_binarize(const evb_matrix *m, const void *edges_dev, int nedges, uint8_t *xC, uint8_t *xT, int RS, uint8_t *xH, int RSH, uint2 *xE, int nmain,
                            int *err, cudaStream_t st);
// evb_nccl.cpp
int32_t evb_nccl_unique_id(uint8_t id[128]);
int32_t evb_nccl_init(evb_handle *h, const uint8_t id[128], int rank, int world);
int32_t evb_nccl_allreduce_f64(evb_handle *h, double *buf, size_t count);
int32_t evb_nccl_allreduce_i32(evb_handle *h, const int32_t *src, int32_t *dst, size_t count);
void evb_nccl_destroy(evb_handle *h);

// evb_stage.cu: pageable host memory -> device through a ring of pinned buffers filled by several host threads
// device memory through the library's block cache (evb_alloc.cu)
cudaError_t evb_dev_alloc(void **p, size_t bytes);
void evb_dev_free(void *p, bool really = false);
template <typename T> inline cudaError_t evb_dev_alloc(T **p, size_t bytes) { return evb_dev_alloc(reinterpret_cast<void **>(p), bytes); }
size_t evb_cached_bytes(int dev); // bytes the cache holds for reuse
cudaError_t evb_host_alloc(void **p, size_t bytes);
void evb_host_free(void *p);
cudaError_t evb_stream_get(cudaStream_t *st);
void evb_stream_put(cudaStream_t st);
cudaError_t evb_event_get(cudaEvent_t *ev);
void evb_event_put(cudaEvent_t ev);

// fn(ctx, begin, end) over [0, n) in slices by all staging threads and the caller
void evb_parallel(void (*fn)(void *, size_t, size_t), void *ctx, size_t n, size_t slice);
// host copies between a packed buffer and nseg strided segments by all staging threads (`up`: strided -> packed)
void evb_copy_packed(void *packed, const void *strided, size_t seg, size_t stride, size_t off, size_t len, bool up);
int32_t evb_d2h_staged(void *dst_host, const void *src_dev, size_t bytes, cudaStream_t st);
int32_t evb_h2d_staged(void *dst_dev, const void *src_host, size_t bytes, cudaStream_t st, bool drain = true);
size_t evb_stage_bytes();
int32_t evb_h2d_made(void *dst_dev, size_t unit, size_t count, size_t piece, void (*fill)(void *, char *, size_t, size_t), void *ctx, cudaStream_t st);
int32_t evb_h2d_staged_strided(void *dst_dev, const void *src_host, size_t seg_bytes, size_t nseg, size_t stride, cudaStream_t st, bool drain = true);

// timing helpers (evb_api.cu)
void evb_tic(evb_handle *h, int cls);
void evb_toc(evb_handle *h, int cls);

static inline int evb_level_nodes(int level) { return 1 << (level - 1); }            // nodes at depth `level`
static inline int evb_level_slots(int level) { return level <= 1 ? 1 : 1 << (level - 2); } // max build slots
