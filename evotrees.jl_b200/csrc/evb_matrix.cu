// The raw feature matrix of a fit on the device: upload, quantile edges (`get_edges`, src/fit-utils.jl:7-24) and `binarize`
// (src/fit-utils.jl:66-72) into the training layouts.  The matrix may be column-major (a Julia Matrix) or row-major (a
// numpy array): nothing on the host transposes it.
#include "evb_internal.cuh"
#include <algorithm>
#include <new>
#include <string.h>

struct evb_matrix {
    int device = 0, nfeats = 0, dtype = 0, row_major = 0;
    int64_t n = 0;
    void *x = nullptr;
    cudaStream_t st = nullptr;
};

namespace {

constexpr unsigned FULL = 0xffffffffu;

// unsigned keys in the order of the values (NaN last)
__device__ __forceinline__ uint32_t key_of(float v) { const uint32_t b = __float_as_uint(v); return (b >> 31) ? ~b : b | 0x80000000u; }
__device__ __forceinline__ uint64_t key_of(double v) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double value_of(uint32_t k) { return (double)__uint_as_float((k >> 31) ? k & 0x7fffffffu : ~k); }
__device__ __forceinline__ double value_of(uint64_t k) { return __longlong_as_double((long long)((k >> 63) ? k & 0x7fffffffffffffffull : ~k)); }

// keys[f][s] = value of feature f in sampled row idx[s] (all rows when idx is null)
template <typename T, typename U>
__global__ void __launch_bounds__(256) k_sample_keys(const T *x, long long n, int nfeats, int row_major, const uint32_t *idx, int ns, U *keys) {
    const int s = blockIdx.x * 256 + threadIdx.x;
    if (s >= ns) return;
    const long long i = idx ? idx[s] : s;
    for (int f = blockIdx.y; f < nfeats; f += gridDim.y) keys[(size_t)f * ns + s] = key_of(row_major ? x[i * nfeats + f] : x[(long long)f * n + i]);
}

// Sorts the ns keys of one feature per CTA (least significant digit first, 8 bits a pass; every warp owns a contiguous piece
// of the keys and keeps the order of equal digits) and takes the quantiles.  A digit that all keys share costs no pass.
// What bounds it is the latency of the passes of a single CTA; 64 000 keys of 4 / 8 bytes stay in L2 meanwhile.
constexpr int SORT_THREADS = 1024, SORT_WARPS = SORT_THREADS / 32;
struct QuantArgs {
    const int32_t *lo, *hi;   // [nq] 0-based ranks of the two order statistics
    const double *g;          // [nq] weight of the second one
    double rtol;
    int nq;
};
template <typename T, typename U>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_quantiles(U *keys_a, U *keys_b, int ns, QuantArgs q, T *edges) {
    __shared__ uint32_t s_cnt[SORT_WARPS][256];
    __shared__ uint32_t s_warp[8];
    __shared__ int s_skip;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, f = blockIdx.x;
    U *src = keys_a + (size_t)f * ns, *dst = keys_b + (size_t)f * ns;
    const int per = ((ns + SORT_WARPS - 1) / SORT_WARPS + 31) & ~31;
    const int b0 = min(ns, wid * per), b1 = min(ns, b0 + per);
    constexpr int B = 8; // loads in flight per lane
    for (int shift = 0; shift < (int)sizeof(U) * 8; shift += 8) {
        for (int d = lane; d < 256; d += 32) s_cnt[wid][d] = 0u;
        if (tid == 0) s_skip = 0;
        __syncwarp();
        for (int p = b0; p < b1; p += 32 * B) {
            uint32_t d[B];
#pragma unroll
            for (int u = 0; u < B; ++u) { const int i = p + u * 32 + lane; d[u] = i < b1 ? (uint32_t)(src[i] >> shift) & 255u : 256u; }
#pragma unroll
            for (int u = 0; u < B; ++u) if (d[u] < 256u) atomicAdd(&s_cnt[wid][d[u]], 1u);
        }
        __syncthreads();
        // offsets: digits ascending, warps ascending inside a digit; thread d < 256 owns digit d
        uint32_t tot = 0;
        if (tid < 256) {
            for (int w = 0; w < SORT_WARPS; ++w) { const uint32_t c = s_cnt[w][tid]; s_cnt[w][tid] = tot; tot += c; }
            if (tot == (uint32_t)ns) s_skip = 1;
            uint32_t incl = tot;
            for (int o = 1; o < 32; o <<= 1) { const uint32_t v = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += v; }
            if (lane == 31) s_warp[wid] = incl;
            tot = incl - tot; // exclusive within the warp
        }
        __syncthreads();
        const bool skip = s_skip != 0;
        __syncthreads();
        if (skip) continue;
        if (tid < 256) {
            for (int w = 0; w < wid; ++w) tot += s_warp[w];
            for (int w = 0; w < SORT_WARPS; ++w) s_cnt[w][tid] += tot;
        }
        __syncthreads();
        for (int p = b0; p < b1; p += 32 * B) {
            U k[B];
#pragma unroll
            for (int u = 0; u < B; ++u) { const int i = p + u * 32 + lane; k[u] = i < b1 ? src[i] : (U)0; }
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int i = p + u * 32 + lane;
                const uint32_t d = i < b1 ? (uint32_t)(k[u] >> shift) & 255u : 256u + lane;
                const unsigned peers = __match_any_sync(FULL, d);
                const int rank = __popc(peers & ((1u << lane) - 1u));
                uint32_t o = 0;
                if (d < 256u) o = s_cnt[wid][d];
                __syncwarp();
                if (d < 256u) {
                    if (rank == 0) s_cnt[wid][d] = o + __popc(peers);
                    dst[o + rank] = k[u];
                }
                __syncwarp();
            }
        }
        __syncthreads(); // a CTA's global stores are visible to the CTA after its barrier
        U *t = src; src = dst; dst = t;
    }
    // type-7 quantile in double, rounded to the type of x; each product and sum is rounded by itself, as on the host
    for (int e = tid; e < q.nq; e += SORT_THREADS) {
        const double a = value_of(src[q.lo[e]]), b = value_of(src[q.hi[e]]), g = q.g[e];
        const double d = fabs(__dsub_rn(a, b)), m = fmax(fabs(a), fabs(b));
        const bool close = isfinite(a) && isfinite(b) && d <= __dmul_rn(q.rtol, m);
        edges[(size_t)f * q.nq + e] = (T)(close ? __dadd_rn(a, __dmul_rn(g, __dsub_rn(b, a))) : __dadd_rn(__dmul_rn(__dsub_rn(1.0, g), a), __dmul_rn(g, b)));
    }
}

// Bins of 16 adjacent features of one row per thread, written into every layout that exists: xC [nfeats][n] bytes, xT [n][RS]
// and xH [n][RSH] chunks of 16, and the tail features of the row into xE[row].y.  searchsortedfirst(edges[j], x) = 1 + number
// of edges below x; four searches side by side hide the latency of the edge loads (L1).
struct BinArgs {
    const void *x, *edges;
    long long n;
    int nfeats, nedges, row_major;
    uint8_t *xC, *xT, *xH;
    uint2 *xE;
    int RS, RSH, nmain;
    int *err;
};
template <typename T>
__global__ void __launch_bounds__(256) k_bin_layouts(BinArgs a) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= a.n) return;
    const T *x = static_cast<const T *>(a.x);
    const int c0 = blockIdx.y * 16;
    uint32_t word[4];
    bool nan = false;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int j0 = c0 + 4 * w, nj = a.nfeats - j0;
        T v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = (T)0;
            if (q < nj) v[q] = a.row_major ? x[i * a.nfeats + j0 + q] : x[(long long)(j0 + q) * a.n + i];
            nan |= v[q] != v[q];
        }
        const T *e = static_cast<const T *>(a.edges) + (size_t)j0 * a.nedges;
        int lo[4] = {0, 0, 0, 0}, len = a.nedges;
        while (len > 0) {
            const int half = (len + 1) >> 1;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < nj && __ldg(e + (size_t)q * a.nedges + lo[q] + half - 1) < v[q]) lo[q] += half;
            len -= half;
        }
        word[w] = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (q < nj) {
                word[w] |= (uint32_t)(lo[q] + 1) << (8 * q);
                if (a.xC) a.xC[(size_t)(j0 + q) * a.n + i] = (uint8_t)(lo[q] + 1);
            }
    }
    if (nan && a.err) atomicCAS(a.err, 0, EVB_DERR_NAN); // missing values are not supported (test/missings.jl)
    const uint4 v4 = make_uint4(word[0], word[1], word[2], word[3]);
    if (a.xT && c0 < a.RS) *reinterpret_cast<uint4 *>(a.xT + (size_t)i * a.RS + c0) = v4;
    if (a.xH && c0 < a.RSH) *reinterpret_cast<uint4 *>(a.xH + (size_t)i * a.RSH + c0) = v4;
    if (a.xE && c0 >= a.nmain && a.nfeats > a.nmain) a.xE[i] = make_uint2(0u, word[0]); // the tail starts a chunk of its own
}

} // namespace

extern "C" void evb_matrix_destroy(evb_matrix *m) {
    if (!m) return;
    int prev = 0;
    cudaGetDevice(&prev);
    if (cudaSetDevice(m->device) == cudaSuccess) {
        if (m->st) { cudaStreamSynchronize(m->st); evb_stream_put(m->st); }
        evb_dev_free(m->x);
    }
    cudaSetDevice(prev);
    delete m;
}

extern "C" int32_t evb_matrix_create(evb_matrix **out, int32_t device, int64_t nobs, int32_t nfeats, const void *x, int32_t x_dtype,
                                     int32_t x_row_major) {
    if (!out) { evb_set_error("evb_matrix_create: out is null"); return EVB_ERR_ARG; }
    *out = nullptr;
    if (!x || nobs < 1 || nobs > 2000000000ll || nfeats < 1 || nfeats > 65535 || (x_dtype != EVB_F32 && x_dtype != EVB_F64)) {
        evb_set_error("evb_matrix_create: invalid argument");
        return EVB_ERR_ARG;
    }
    EVB_CHECK(evb_check_device(device));
    const size_t bytes = (size_t)nobs * nfeats * (x_dtype == EVB_F64 ? 8 : 4);
    if (bytes > ((size_t)4 << 30)) { // training needs about as much again: take no more than half of what is free
        size_t free_b = 0, total_b = 0;
        EVB_CUDA(cudaMemGetInfo(&free_b, &total_b));
        if (bytes > (free_b + evb_cached_bytes(device)) / 2) { evb_set_error("evb_matrix_create: %zu bytes do not fit beside the training state", bytes); return EVB_ERR_LIMIT; }
    }
    evb_matrix *m = new (std::nothrow) evb_matrix();
    if (!m) { evb_set_error("out of host memory"); return EVB_ERR_ARG; }
    m->device = device; m->n = nobs; m->nfeats = nfeats; m->dtype = x_dtype; m->row_major = x_row_major ? 1 : 0;
    auto body = [&]() -> int32_t {
        EVB_CUDA(evb_stream_get(&m->st));
        EVB_CUDA(evb_dev_alloc(&m->x, bytes));
        return evb_h2d_staged(m->x, x, bytes, m->st, false);
    };
    const int32_t rc = body();
    if (rc != EVB_OK) { evb_matrix_destroy(m); return rc; }
    *out = m;
    return EVB_OK;
}

template <typename T, typename U>
static int32_t edges_t(evb_matrix *m, const uint32_t *rows, int32_t ns, int32_t nq, const int32_t *lo, const int32_t *hi, const double *g, double rtol, T *edges) {
    struct Buf { void *p = nullptr; ~Buf() { evb_dev_free(p); } } keys, aux;
    const size_t nk = (size_t)ns * m->nfeats, o_g = 0, o_lo = (size_t)nq * 8, o_hi = o_lo + (size_t)nq * 4, o_idx = o_hi + (size_t)nq * 4,
                 o_e = (o_idx + (rows ? (size_t)ns * 4 : 0) + 15) & ~(size_t)15;
    EVB_CUDA(evb_dev_alloc(&keys.p, 2 * nk * sizeof(U)));
    EVB_CUDA(evb_dev_alloc(&aux.p, o_e + (size_t)nq * m->nfeats * sizeof(T)));
    std::vector<char> host(o_idx + (rows ? (size_t)ns * 4 : 0));
    memcpy(host.data() + o_g, g, (size_t)nq * 8);
    memcpy(host.data() + o_lo, lo, (size_t)nq * 4);
    memcpy(host.data() + o_hi, hi, (size_t)nq * 4);
    if (rows) memcpy(host.data() + o_idx, rows, (size_t)ns * 4);
    char *d = static_cast<char *>(aux.p);
    EVB_CUDA(cudaMemcpyAsync(d, host.data(), host.size(), cudaMemcpyHostToDevice, m->st));
    U *ka = static_cast<U *>(keys.p), *kb = ka + nk;
    const dim3 grid((ns + 255) / 256, std::min(m->nfeats, m->row_major ? 8 : 65535)); // row-major: a thread takes adjacent features of its row
    k_sample_keys<T, U><<<grid, 256, 0, m->st>>>(static_cast<const T *>(m->x), m->n, m->nfeats, m->row_major, rows ? reinterpret_cast<uint32_t *>(d + o_idx) : nullptr, ns, ka);
    EVB_CUDA(cudaGetLastError());
    QuantArgs q{reinterpret_cast<int32_t *>(d + o_lo), reinterpret_cast<int32_t *>(d + o_hi), reinterpret_cast<double *>(d + o_g), rtol, nq};
    k_sort_quantiles<T, U><<<m->nfeats, SORT_THREADS, 0, m->st>>>(ka, kb, ns, q, reinterpret_cast<T *>(d + o_e));
    EVB_CUDA(cudaGetLastError());
    EVB_CUDA(cudaMemcpyAsync(edges, d + o_e, (size_t)nq * m->nfeats * sizeof(T), cudaMemcpyDeviceToHost, m->st));
    EVB_CUDA(cudaStreamSynchronize(m->st));
    return EVB_OK;
}

extern "C" int32_t evb_matrix_edges(evb_matrix *m, const uint32_t *rows, int32_t nrows, int32_t nedges, const int32_t *lo, const int32_t *hi,
                                    const double *g, double rtol, void *edges) {
    if (!m || !lo || !hi || !g || !edges || nedges < 1 || nedges > 254 || nrows < 1 || nrows > m->n || (!rows && nrows != m->n)) {
        evb_set_error("evb_matrix_edges: invalid argument");
        return EVB_ERR_ARG;
    }
    for (int e = 0; e < nedges; ++e)
        if (lo[e] < 0 || hi[e] < 0 || lo[e] >= nrows || hi[e] >= nrows) { evb_set_error("evb_matrix_edges: rank outside the sample"); return EVB_ERR_ARG; }
    if (rows)
        for (int s = 0; s < nrows; ++s) if ((int64_t)rows[s] >= m->n) { evb_set_error("evb_matrix_edges: sampled row out of range"); return EVB_ERR_ARG; }
    EVB_CUDA(cudaSetDevice(m->device));
    return m->dtype == EVB_F64 ? edges_t<double, uint64_t>(m, rows, nrows, nedges, lo, hi, g, rtol, static_cast<double *>(edges))
                               : edges_t<float, uint32_t>(m, rows, nrows, nedges, lo, hi, g, rtol, static_cast<float *>(edges));
}

int64_t evb_matrix_rows(const evb_matrix *m) { return m->n; }
int evb_matrix_feats(const evb_matrix *m) { return m->nfeats; }
int evb_matrix_dtype(const evb_matrix *m) { return m->dtype; }
// a stream waits until the matrix has arrived
cudaError_t evb_matrix_join(const evb_matrix *m, cudaStream_t st) {
    cudaEvent_t ev;
    cudaError_t e = evb_event_get(&ev);
    if (e != cudaSuccess) return e;
    e = cudaEventRecord(ev, m->st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, ev, 0);
    evb_event_put(ev);
    return e;
}

// bins of n rows of x (device) into the layouts that are not null
int32_t evb_launch_bin_layouts(const void *x, int dtype, int row_major, int64_t n, int nfeats, const void *edges, int nedges, uint8_t *xC, uint8_t *xT, int RS,
                               uint8_t *xH, int RSH, uint2 *xE, int nmain, int *err, cudaStream_t st) {
    BinArgs a;
    a.x = x; a.edges = edges; a.n = n; a.nfeats = nfeats; a.nedges = nedges; a.row_major = row_major; a.xC = xC; a.xT = xT; a.xH = xH; a.xE = xE;
    a.RS = RS; a.RSH = RSH; a.nmain = nmain; a.err = err;
    const int chunks = std::max((nfeats + 15) / 16, std::max(xT ? RS / 16 : 0, xH ? RSH / 16 : 0)); // the padding chunks are written as zeros
    const dim3 grid((unsigned)((n + 255) / 256), (unsigned)chunks);
    if (dtype == EVB_F64) k_bin_layouts<double><<<grid, 256, 0, st>>>(a);
    else k_bin_layouts<float><<<grid, 256, 0, st>>>(a);
    EVB_CUDA(cudaGetLastError());
    return EVB_OK;
}
int32_t evb_matrix_binarize(const evb_matrix *m, const void *edges_dev, int nedges, uint8_t *xC, uint8_t *xT, int RS, uint8_t *xH, int RSH, uint2 *xE, int nmain,
                            int *err, cudaStream_t st) {
    return evb_launch_bin_layouts(m->x, m->dtype, m->row_major, m->n, m->nfeats, edges_dev, nedges, xC, xT, RS, xH, RSH, xE, nmain, err, st);
}
