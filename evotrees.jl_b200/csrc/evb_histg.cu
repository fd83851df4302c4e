// Integer histograms of any loss (device code and its reasons: evb_histg.cuh): geometry, quantisation, launches.
#include "evb_histg.cuh"
#include <stdlib.h>
#include <algorithm>

namespace {

using namespace evb_hg;

struct KArgs {
    Args a;
    HGeom g;
};

template <int NQ, bool CNT, bool PACK>
__device__ __forceinline__ void run(const Args &a, uint32_t *smem, uint32_t *queue) { accumulate<NQ, CNT, PACK>(a, smem, queue, blockIdx.x, gridDim.x); }

// grid (row ranges, feature groups, channel groups)
__global__ void __launch_bounds__(1024, 1) k_histg(KArgs k) {
    extern __shared__ __align__(128) uint32_t s_img[];
    Args &a = k.a;
    if ((long long)blockIdx.x * a.min_rows >= max(1ll, (long long)a.plan->R + (long long)a.plan->nbuild * a.pad_rows)) return;
    evb_hg_select(k.g, a, blockIdx.y, blockIdx.z);
    const int P = evb_hg_planes(k.g, blockIdx.z), words = nparts(a.nfull, a.tails) * (a.B + 1) * P * 8;
    for (int i = threadIdx.x; i < words; i += blockDim.x) reinterpret_cast<uint4 *>(s_img)[i] = make_uint4(0u, 0u, 0u, 0u);
    uint32_t *queue = s_img + k.g.queue;
    if (threadIdx.x == 0) queue[QUEUE] = 0u;
    __syncthreads();
    EVB_HG_DISPATCH(k.g, blockIdx.z, run, a, s_img, queue)
}

// clears the accumulators of the level's build slots (all feature columns, sampled or not)
__global__ void __launch_bounds__(256) k_hg_clear(unsigned long long *hsum, uint32_t *hcnt, unsigned long long *hlow, const uint32_t *low_any, const LevelPlan *plan, size_t per_slot, int nq) {
    const size_t n = (size_t)plan->nbuild * per_slot, ns = n * nq;
    const bool low = hlow && *low_any;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += (size_t)gridDim.x * blockDim.x) {
        hsum[i] = 0ull;
        if (i < n) hcnt[i] = 0u;
        if (low) hlow[i] = 0ull;
    }
}

// hcomp[slot][f][channel][bin] (doubles, what ranks exchange) from the integer accumulators.  One CTA per (build slot,
// 32 feature slots).
struct ConvArgs {
    const unsigned long long *hsum;
    const uint32_t *hcnt;
    double *hcomp;
    const LevelPlan *plan;
    const uint32_t *js0;
    const double *qinv;
    const unsigned long long *hlow;
    const uint32_t *low;
    double low_unit;
    int B, SC, F, C, K, nq, elide, unit_w;
};
__global__ void __launch_bounds__(256) k_hg_to_hcomp(ConvArgs a) {
    __shared__ double t[64][33];
    const int s = blockIdx.x, f0 = blockIdx.y * 32;
    if (s >= a.plan->nbuild) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, f = f0 + lane;
    const int col = f < a.F ? (int)a.js0[f] : -1;
    const bool low = a.hlow && a.low[s];
    for (int c = 0; c < a.C; ++c) {
        const bool is_h = a.elide && c >= a.K && c < 2 * a.K; // h = 2w (src/loss.jl:52)
        const bool is_w = c == a.C - 1 || is_h;
        const int ch = is_w ? a.nq - 1 : c;
        const double unit = is_w && a.unit_w ? 1.0 : a.qinv[ch];
        const double mul = is_h ? 2.0 : 1.0;
        for (int bin0 = 0; bin0 < a.B; bin0 += 64) {
            for (int bl = w; bl < 64; bl += 8) {
                const int bin = bin0 + bl;
                double v = 0.0;
                if (bin < a.B && col >= 0) {
                    const size_t cell = (size_t)s * a.B + bin;
                    if (is_w && a.unit_w) v = (double)a.hcnt[cell * a.SC + col];
                    else {
                        v = (double)(long long)a.hsum[(cell * a.nq + ch) * a.SC + col] * unit;
                        if (low) v += (double)(long long)a.hlow[(((size_t)s * a.SC + col) * a.nq + ch) * a.B + bin] * (unit * a.low_unit);
                    }
                }
                t[bl][lane] = mul * v;
            }
            __syncthreads();
            for (int e = threadIdx.x; e < 64 * 32; e += 256) {
                const int fl = e >> 6, bl = e & 63, ff = f0 + fl, bin = bin0 + bl;
                if (ff < a.F && bin < a.B) a.hcomp[(((size_t)s * a.F + ff) * a.C + c) * a.B + bin] = t[bl][fl];
            }
            __syncthreads();
        }
    }
}

constexpr size_t SMEM_TWO = 113 * 1024 - QUEUE_BYTES;  // image of one of two CTAs per SM: 228 KB less 1 KB per CTA
constexpr size_t SMEM_ONE = 227 * 1024 - QUEUE_BYTES;

} // namespace

// Cuts the channels and the words of a row over CTAs so that an image fits shared memory: as many channels per CTA as
// possible (at most MAX_NQ) with at least one part of eight words, then as many parts as fit.  Two CTAs of 512 threads share an
// SM when their images do, so that one accumulates while the other empties its image; else one CTA of 1024 threads.
int32_t evb_hg_configure(evb_handle *h) {
    HGeom &g = h->hgeo;
    g.nq = h->nq;
    g.pack = h->p.loss == EVB_MSE && h->nq == 1; // one target, unit weights, hessians left out
    g.cnt = h->unit_w && !g.pack;
    if (g.pack) { g.per = 1; g.ngc = 1; }
    else {
        int per = std::min(g.nq, MAX_NQ);
        while (per > 1 && part_bytes(h->B, planes(per, g.cnt, false)) > SMEM_ONE) --per;
        g.ngc = (g.nq + per - 1) / per;
        g.per = (g.nq + g.ngc - 1) / g.ngc;
    }
    const size_t part = part_bytes(h->B, planes(g.per, g.cnt, g.pack));
    if (part > SMEM_ONE) { evb_set_error("histogram image does not fit shared memory (nbins=%d)", h->B); return EVB_ERR_LIMIT; }
    const int W = (h->nfeats + 3) / 4, fit = (int)(SMEM_ONE / part);
    auto most_parts = [&](int wper) { // of a CTA when each takes wper words
        int most = 0, nf, tl;
        for (int w = 0; w < W; w += wper) { split_words(std::min(wper, W - w), nf, tl); most = std::max(most, nparts(nf, tl)); }
        return most;
    };
    // all words of a row, else as many whole parts as fit; a tail of 5 or 6 words is two parts, then four words at least
    g.wper = W;
    if (most_parts(g.wper) > fit) g.wper = (W - 1) & ~7;
    while (g.wper > 8 && most_parts(g.wper) > fit) g.wper -= 8;
    if (g.wper < 8 && W >= 8) g.wper = 8;
    if (g.wper < 1 || most_parts(g.wper) > fit) g.wper = 4;
    g.ngf = (W + g.wper - 1) / g.wper;
    g.wper = std::min(g.wper, g.wper <= 4 ? g.wper : ((W + g.ngf - 1) / g.ngf + 7) & ~7); // the same number of CTAs, evenly filled
    // Fewer rows below the root than the SMs can share (1024 each): a CTA takes one part only, its flush is shorter too.  ms per tree, all
    // parts and one: 10k x 77 poisson 0.139 and 0.119, 60k x 77 0.146 and 0.130, 200k x 77 0.166 and 0.157, 600k x 77 0.239 and 0.247;
    // 100k x 40 logloss 0.142 and 0.131, 200k x 40 0.156 and 0.144, 800k x 40 0.232 and 0.239; 200k x 50 gaussian 0.191 and 0.175, 800k x 50
    // 0.327 and 0.314; 250k x 100 least squares 0.169 and 0.153.  The lines cross between 300k and 600k rows; this one lies at 303k
    // where all words fit one CTA, at 152k where they take two.
    if (h->n / 2 / 1024 * g.ngf < h->num_sms && g.wper > 8) g.wper = 8;
    g.wper = std::min(g.wper, W);
    g.ngf = (W + g.wper - 1) / g.wper;
    g.W = W;
    const int most = most_parts(g.wper);
    g.queue = (int)(most * part / 4);
    g.smem = most * part + QUEUE_BYTES;
    g.threads = most * part <= SMEM_TWO ? 512 : 1024;
    // Up to four words a row is cheap and 256 rows are too few for a flush.  ms per tree with 256 and 512: 100k x 10 least squares 0.099 and
    // 0.096, 100k x 16 logloss 0.124 and 0.118, 30k x 7 poisson 0.112 and 0.112, but 100k x 12 five classes 0.146 and 0.151; with more
    // words 60k x 28 five classes 0.149 and 0.160, 100k x 100 0.125 and 0.128, 60k x 77 poisson 0.132 and 0.131, 100k x 28 poisson 0.128 and 0.124
    g.min_rows = g.wper <= 4 ? 512 : 256;
    EVB_CUDA(cudaFuncSetAttribute(k_histg, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    int occ = 0;
    EVB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_histg, g.threads, g.smem));
    if (occ < 1) { evb_set_error("histogram kernel cannot be resident (smem=%zu)", g.smem); return EVB_ERR_CUDA; }
    g.G = std::max(1, occ * h->num_sms / (g.ngf * g.ngc));
    // More bits leave fewer rows with something left over, but an image then holds fewer rows: as many as the rows of a CTA at the
    // root allow without an extra flush, 18 at least (8 160 rows).  ms of histograms per tree with 15, 16, 17, 18, 19: 2M x 28 five
    // classes 0.649, 0.636, 0.633, 0.638, 0.656 (31 bits without the rest 0.617), 5M x 50 gaussian 2.01, 1.19, 1.120, 1.120, 1.187 (1.057).
    // The sums of all rows have to fit 63 bits.
    g.hb = 21;
    while (g.hb > 18 && (1ll << (31 - g.hb)) - 32 < h->n / g.G + 512) --g.hb;
    int log_n = 0;
    while ((1ll << log_n) < h->n) ++log_n;
    g.hb = std::min(g.hb, (61 - log_n) / 2);
    g.TE = g.pack ? 255 : (1 << (26 - g.hb)) - 1;
    return EVB_OK;
}

size_t evb_hg_q_words(const evb_handle *h) { return evb_hg_qoff(h->hgeo, h->n, h->hgeo.ngc) + 8; }

void evb_hg_args(const evb_handle *h, int level, evb_hg::Args *a) {
    a->xT = h->xT; a->q = h->gradq; a->rows = h->rows[(level - 1) & 1]; a->plan = h->plan + level; a->cum = h->cum; a->rbase = h->rbase;
    a->hsum = h->hsum_q; a->hcnt = h->hcnt_q; a->hlow = h->hlow_q; a->low = h->low + evb_low_slot(level); a->low_any = h->low + evb_low_any(level);
    a->hb = h->hgeo.hb; a->RS = h->RS; a->B = h->B; a->SC = h->SC; a->nq = h->nq; a->F = h->nfeats;
    a->TE = h->hgeo.TE; a->min_rows = h->hgeo.min_rows; a->pad_rows = evb_pad_rows(h); a->n = h->n;
}

// the width that weighted least squares has always had where its fixed-point kernel ran
int evb_hg_round_bits(const evb_handle *h) { return h->p.loss == EVB_MSE && h->Ce == 2 && !h->unit_w && h->B <= 128 && h->F == h->nfeats ? 29 : 0; }

void evb_hg_quant_args(const evb_handle *h, evb_hg::QuantArgs *a) {
    a->grad = h->grad; a->q = h->use_q2 ? reinterpret_cast<int32_t *>(h->xE) : h->gradq; a->gmax = evb_gmax(h, false); a->qinv = h->d_qinv; a->n = h->n;
    a->q2 = h->use_q2 ? 1 : 0; a->g = h->hgeo; a->signs = h->d_signs;
    a->bits = evb_hg_round_bits(h);
}

int32_t evb_launch_histg(evb_handle *h, int level) {
    const HGeom &g = h->hgeo;
    KArgs k;
    k.g = g;
    evb_hg_args(h, level, &k.a);
    evb_tic(h, EVB_T_HIST);
    const cudaError_t e = evb_launch(k_histg, dim3(g.G, g.ngf, g.ngc), dim3(g.threads), g.smem, h->st, k);
    evb_toc(h, EVB_T_HIST);
    EVB_CUDA(e);
    return EVB_OK;
}

int32_t evb_launch_acc_clear(evb_handle *h, int level) {
    const size_t per_slot = (size_t)h->B * h->SC;
    const size_t blocks = std::min<size_t>(((size_t)evb_level_slots(level) * per_slot * h->nq + 255) / 256, (size_t)h->num_sms * 8);
    evb_tic(h, EVB_T_HIST_REDUCE);
    const cudaError_t e = evb_launch(k_hg_clear, dim3((unsigned)blocks), dim3(256), 0, h->st, h->hsum_q, h->hcnt_q, h->hlow_q, h->low + evb_low_any(level),
                                         h->plan + level, per_slot, h->nq);
    evb_toc(h, EVB_T_HIST_REDUCE);
    EVB_CUDA(e);
    return EVB_OK;
}

// integer accumulators -> hcomp (doubles), for runs that exchange histograms between ranks
int32_t evb_launch_acc_to_hcomp(evb_handle *h, int level) {
    ConvArgs a;
    a.hsum = h->hsum_q; a.hcnt = h->hcnt_q; a.hcomp = h->hcomp; a.plan = h->plan + level; a.js0 = h->js_d; a.qinv = h->d_qinv;
    a.hlow = h->hlow_q; a.low = h->low + evb_low_slot(level); a.low_unit = evb_hg_low_unit(h->hgeo.hb);
    a.B = h->B; a.SC = h->SC; a.F = h->F; a.C = h->C; a.K = h->K; a.nq = h->nq; a.elide = h->Ce != h->C; a.unit_w = h->unit_w;
    evb_tic(h, EVB_T_HIST_REDUCE);
    k_hg_to_hcomp<<<dim3(evb_level_slots(level), (h->F + 31) / 32), 256, 0, h->st>>>(a);
    evb_toc(h, EVB_T_HIST_REDUCE);
    EVB_CUDA(cudaGetLastError());
    return evb_launch_acc_clear(h, level);
}
