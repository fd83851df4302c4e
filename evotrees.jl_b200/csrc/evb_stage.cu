// Host-to-device copies of ordinary (pageable) host memory at pinned-memory speed: the data goes through a small ring
// of pinned buffers that several host threads fill while the copy engine drains the previous one.  A plain
// cudaMemcpy from pageable memory does the same staging inside the driver with one thread, which caps a 4 GB feature
// matrix at a fraction of the PCIe rate.  The ring and the worker threads are created on first use and kept for the
// life of the process.
#include "evb_internal.cuh"
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <math.h>
#include <pthread.h>
#include <stdlib.h>
#include <string.h>
#include <thread>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif
#include <stdint.h>

namespace {

// The ring stays in the last-level cache: the copy engine reads what the gather threads have just written without a trip
// to memory.  4 GB of features, measured: 3 x 8 MB 78 ms (51 GB/s, the link's rate), 6 x 4 MB 81 ms, 8 x 2 MB 87 ms; with
// stores that bypass the cache 3 x 64 MB 82 ms, 4 x 8 MB 84 ms.
constexpr int STAGE_NB = 3;
constexpr size_t STAGE_BYTES = (size_t)8 << 20;

struct StageRing {
    void *buf[STAGE_NB] = {nullptr, nullptr, nullptr};
    cudaEvent_t ev[STAGE_NB] = {nullptr, nullptr, nullptr};
    bool used[STAGE_NB] = {false, false, false};
    int next = 0;
    bool ready = false;
    std::mutex mu;
};
StageRing g_rings[64]; // one ring per device (events belong to a device)

int stage_threads() {
    static const int n = [] {
        if (const char *e = getenv("EVB_STAGE_THREADS")) { const int v = atoi(e); if (v >= 1 && v <= 64) return v; }
        const unsigned hc = std::thread::hardware_concurrency();
        int v = hc ? (int)hc * 3 / 4 : 4;
        // Seven threads copy at the host memory's rate; more only delay the DMA that reads the buffers (16 cores, 10M x 50 floats predicted:
        // 4 threads 58.2 ms, 6 49.6, 7 46.5, 8 48.3, 9 48.8, 12 53.4, 16 60.1; uploads of training matrices do not care from 6 on).
        return v < 1 ? 1 : v > 7 ? 7 : v;
    }();
    return n;
}

inline void cpu_pause() {
#if defined(__x86_64__)
    _mm_pause();
#else
    std::this_thread::yield();
#endif
}

// Copies bytes [off, off + len) of the packed sequence of nseg segments of seg bytes (segment k at strided + k * stride):
// `packed` is the address of byte `off`.  up: strided -> packed, else packed -> strided.
struct CopyJob {
    char *packed, *strided;
    size_t seg, stride, off, len;
    bool up;
};
void copy_range(const CopyJob &j, size_t o, size_t n) {
    size_t p = j.off + o;
    const size_t end = p + n;
    char *pk = j.packed + o;
    while (p < end) {
        const size_t k = p / j.seg, within = p - k * j.seg;
        const size_t m = j.seg - within < end - p ? j.seg - within : end - p;
        char *st = j.strided + k * j.stride + within;
        if (j.up) memcpy(pk, st, m);
        else memcpy(st, pk, m);
        p += m; pk += m;
    }
}

// Worker threads that live as long as the process and take slices of a job in turn with the calling thread.  Waking a
// sleeping thread costs 20-50 us, as much as copying a megabyte, and a transfer is a sequence of such copies: a worker
// that ran out of slices therefore looks for the next job for SPIN_US before it goes to sleep.  The pool is never
// destroyed: its threads may still be waiting when the process exits.
constexpr int SPIN_US = 150;
struct HostPool {
    std::mutex one_job;                     // one job at a time
    std::mutex m;
    std::condition_variable cv;
    std::atomic<unsigned> gen{0};           // jobs started
    std::atomic<int> sleepers{0}, inside{0};
    std::atomic<bool> open{false};
    std::atomic<size_t> next{0};
    void (*fn)(void *, size_t, size_t) = nullptr;
    void *ctx = nullptr;
    size_t len = 0, slice = 1;
    int nworkers = 0;
    void slices() {
        for (;;) {
            const size_t o = next.fetch_add(slice, std::memory_order_relaxed);
            if (o >= len) return;
            fn(ctx, o, len - o < slice ? len : o + slice);
        }
    }
    void worker() {
        unsigned seen = 0;
        for (;;) {
            const auto t0 = std::chrono::steady_clock::now();
            while (gen.load() == seen) {
                for (int i = 0; i < 64 && gen.load(std::memory_order_relaxed) == seen; ++i) cpu_pause();
                if (std::chrono::steady_clock::now() - t0 > std::chrono::microseconds(SPIN_US)) {
                    std::unique_lock<std::mutex> lk(m);
                    sleepers.fetch_add(1);
                    cv.wait(lk, [&] { return gen.load() != seen; });
                    sleepers.fetch_sub(1);
                }
            }
            seen = gen.load();
            inside.fetch_add(1);
            // the job's fields are only read while the job is open, and a job is only replaced when nobody is inside
            if (open.load()) slices();
            inside.fetch_sub(1);
        }
    }
    void run(void (*f)(void *, size_t, size_t), void *c, size_t n, size_t sl) {
        std::lock_guard<std::mutex> g(one_job);
        if (nworkers == 0) {
            nworkers = stage_threads() - 1;
            for (int t = 0; t < nworkers; ++t) std::thread([this] { worker(); }).detach();
        }
        while (inside.load() != 0) cpu_pause(); // a late worker that found the last job closed
        fn = f; ctx = c; len = n; slice = sl;
        next.store(0);
        open.store(true);
        gen.fetch_add(1);
        if (sleepers.load() != 0) { std::lock_guard<std::mutex> lk(m); cv.notify_all(); }
        slices();
        open.store(false);
        while (inside.load() != 0) cpu_pause(); // the slices the workers have taken
    }
};
HostPool *g_pool = new HostPool; // rings of different devices share the pool
// a forked child has none of the parent's threads: it starts with a pool of its own
const int g_atfork = pthread_atfork(nullptr, nullptr, [] { g_pool = new HostPool; });

} // namespace

// fn(ctx, begin, end) over [0, n) in slices, by all staging threads and the caller; small jobs (one slice) by the caller alone
void evb_parallel(void (*fn)(void *, size_t, size_t), void *ctx, size_t n, size_t slice) {
    if (n == 0) return;
    if (n <= slice || stage_threads() == 1) fn(ctx, 0, n);
    else g_pool->run(fn, ctx, n, slice);
}

// Host copies by all staging threads.
void evb_copy_packed(void *packed, const void *strided, size_t seg, size_t stride, size_t off, size_t len, bool up) {
    CopyJob j{(char *)packed, (char *)const_cast<void *>(strided), seg, stride, off, len, up};
    evb_parallel([](void *c, size_t b, size_t e) { copy_range(*static_cast<const CopyJob *>(c), b, e - b); }, &j, len, (size_t)128 << 10);
}

static int32_t ring_ready(StageRing &r) {
    if (r.ready) return EVB_OK;
    for (int b = 0; b < STAGE_NB; ++b) {
        if (!r.buf[b]) EVB_CUDA(cudaHostAlloc(&r.buf[b], STAGE_BYTES, cudaHostAllocDefault));
        if (!r.ev[b]) EVB_CUDA(cudaEventCreateWithFlags(&r.ev[b], cudaEventDisableTiming));
    }
    r.ready = true;
    return EVB_OK;
}

// Copies nseg segments of seg_bytes (segment k at src_host + k * stride) of pageable host memory to the device, packed
// back to back at dst_dev, on stream `st`: a block of rows of a column-major matrix, or (nseg = 1) a plain range.
// Returns when the host memory has been read (the caller may reuse or free it); with `drain` also the copies have
// completed.  Without it the last chunks may still be on their way from the pinned ring (in stream order on `st`), and a
// later call continues with the next ring buffer: a sequence of calls then streams without a gap.  One copy at a time
// per device (the ring is shared); concurrent callers wait for each other.
int32_t evb_h2d_staged_strided(void *dst_dev, const void *src_host, size_t seg_bytes, size_t nseg, size_t stride, cudaStream_t st, bool drain) {
    const size_t bytes = seg_bytes * nseg;
    if (bytes == 0) return EVB_OK;
    int dev = 0;
    EVB_CUDA(cudaGetDevice(&dev));
    if (bytes < ((size_t)1 << 20) || getenv("EVB_STAGE_OFF") || dev < 0 || dev >= 64) { // small: the driver's own staging is as good
        if (nseg == 1) EVB_CUDA(cudaMemcpyAsync(dst_dev, src_host, bytes, cudaMemcpyHostToDevice, st));
        else EVB_CUDA(cudaMemcpy2DAsync(dst_dev, seg_bytes, src_host, stride, seg_bytes, nseg, cudaMemcpyHostToDevice, st));
        return EVB_OK;
    }
    StageRing &g_ring = g_rings[dev];
    std::lock_guard<std::mutex> lock(g_ring.mu);
    EVB_CHECK(ring_ready(g_ring));
    const char *src = static_cast<const char *>(src_host);
    char *dst = static_cast<char *>(dst_dev);
    for (size_t off = 0; off < bytes; off += STAGE_BYTES) {
        const int b = g_ring.next;
        g_ring.next = (b + 1) % STAGE_NB;
        const size_t len = bytes - off < STAGE_BYTES ? bytes - off : STAGE_BYTES;
        if (g_ring.used[b]) EVB_CUDA(cudaEventSynchronize(g_ring.ev[b])); // the copy that last used this buffer has left it
        evb_copy_packed(g_ring.buf[b], src, seg_bytes, stride, off, len, true);
        EVB_CUDA(cudaMemcpyAsync(dst + off, g_ring.buf[b], len, cudaMemcpyHostToDevice, st));
        EVB_CUDA(cudaEventRecord(g_ring.ev[b], st));
        g_ring.used[b] = true;
    }
    if (drain)
        for (int q = 0; q < STAGE_NB; ++q)
            if (g_ring.used[q]) { EVB_CUDA(cudaEventSynchronize(g_ring.ev[q])); g_ring.used[q] = false; }
    return EVB_OK;
}

// Memory that is made on the way: fill(ctx, buffer, first, count) writes units [first, first + count) of `unit` bytes each to a pinned
// buffer (all staging threads, `piece` units at a time), which is copied while the next one is filled.  Returns when everything has arrived.
// unit <= STAGE_BYTES.
size_t evb_stage_bytes() { return STAGE_BYTES; }
int32_t evb_h2d_made(void *dst_dev, size_t unit, size_t count, size_t piece, void (*fill)(void *, char *, size_t, size_t), void *ctx, cudaStream_t st) {
    int dev = 0;
    EVB_CUDA(cudaGetDevice(&dev));
    if (unit == 0 || unit > STAGE_BYTES || dev < 0 || dev >= 64) { evb_set_error("evb_h2d_made: invalid argument"); return EVB_ERR_ARG; }
    StageRing &r = g_rings[dev];
    std::lock_guard<std::mutex> lock(r.mu);
    EVB_CHECK(ring_ready(r));
    // a few chunks at least, so that the first copy starts early
    const size_t per = std::max<size_t>(1, std::min(STAGE_BYTES, std::max<size_t>(unit * count / 4, (size_t)1 << 20)) / unit);
    struct Job { void (*fill)(void *, char *, size_t, size_t); void *ctx; char *buf; size_t first, unit; } j{fill, ctx, nullptr, 0, unit};
    for (size_t u = 0; u < count; u += per) {
        const int b = r.next;
        r.next = (b + 1) % STAGE_NB;
        const size_t n = std::min(per, count - u);
        if (r.used[b]) EVB_CUDA(cudaEventSynchronize(r.ev[b]));
        j.buf = static_cast<char *>(r.buf[b]); j.first = u;
        evb_parallel([](void *c, size_t b0, size_t e0) { Job &q = *static_cast<Job *>(c); q.fill(q.ctx, q.buf + b0 * q.unit, q.first + b0, e0 - b0); }, &j, n, piece);
        EVB_CUDA(cudaMemcpyAsync(static_cast<char *>(dst_dev) + u * unit, r.buf[b], n * unit, cudaMemcpyHostToDevice, st));
        EVB_CUDA(cudaEventRecord(r.ev[b], st));
        r.used[b] = true;
    }
    for (int q = 0; q < STAGE_NB; ++q)
        if (r.used[q]) { EVB_CUDA(cudaEventSynchronize(r.ev[q])); r.used[q] = false; }
    return EVB_OK;
}

int32_t evb_h2d_staged(void *dst_dev, const void *src_host, size_t bytes, cudaStream_t st, bool drain) {
    return evb_h2d_staged_strided(dst_dev, src_host, bytes, 1, bytes, st, drain);
}

// Device memory to ordinary (pageable) host memory through the same ring: while one buffer is filled by the copy engine, all
// staging threads empty the one before it (a fresh host array costs a page fault every 4 KB, which they share).  Returns
// when the data is there.  40 MB of predictions: 8-10 ms with cudaMemcpyAsync, about 1.5 ms like this.
int32_t evb_d2h_staged(void *dst_host, const void *src_dev, size_t bytes, cudaStream_t st) {
    int dev = 0;
    EVB_CUDA(cudaGetDevice(&dev));
    if (bytes < ((size_t)64 << 10) || dev < 0 || dev >= 64) {
        EVB_CUDA(cudaMemcpyAsync(dst_host, src_dev, bytes, cudaMemcpyDeviceToHost, st));
        EVB_CUDA(cudaStreamSynchronize(st));
        return EVB_OK;
    }
    StageRing &r = g_rings[dev];
    std::lock_guard<std::mutex> lock(r.mu);
    EVB_CHECK(ring_ready(r));
    char *dst = static_cast<char *>(dst_host);
    const char *src = static_cast<const char *>(src_dev);
    const size_t piece = std::min<size_t>(STAGE_BYTES, std::max<size_t>((size_t)1 << 20, bytes / 4 / 4096 * 4096));
    size_t prev_off = 0, prev_len = 0;
    int prev = -1;
    for (size_t off = 0; off < bytes || prev >= 0; off += piece) {
        int b = -1;
        size_t len = 0;
        if (off < bytes) {
            b = r.next;
            r.next = (b + 1) % STAGE_NB;
            len = std::min(piece, bytes - off);
            if (r.used[b]) { EVB_CUDA(cudaEventSynchronize(r.ev[b])); r.used[b] = false; }
            EVB_CUDA(cudaMemcpyAsync(r.buf[b], src + off, len, cudaMemcpyDeviceToHost, st));
            EVB_CUDA(cudaEventRecord(r.ev[b], st));
            r.used[b] = true;
        }
        if (prev >= 0) {
            EVB_CUDA(cudaEventSynchronize(r.ev[prev]));
            r.used[prev] = false;
            evb_copy_packed(r.buf[prev], dst + prev_off, prev_len, 0, 0, prev_len, false);
        }
        prev = b; prev_off = off; prev_len = len;
    }
    return EVB_OK;
}

// ---- passes over a host target by all staging threads (`_init_target`, src/init.jl:10-146) ---------------------------
namespace {
constexpr size_t HOST_SLICE = (size_t)1 << 16; // rows
template <typename F>
void host_slices(size_t n, const F &f) { // f(begin, end) on slices that start at multiples of HOST_SLICE
    evb_parallel([](void *c, size_t b, size_t e) { (*static_cast<const F *>(c))(b, e); }, const_cast<F *>(&f), n, HOST_SLICE);
}
template <typename F>
int32_t with_ints(const void *y, int32_t kind, const F &f) { // kind: bytes per value, + 16 when unsigned
    switch (kind) {
    case 1: f(static_cast<const int8_t *>(y)); return EVB_OK;
    case 2: f(static_cast<const int16_t *>(y)); return EVB_OK;
    case 4: f(static_cast<const int32_t *>(y)); return EVB_OK;
    case 8: f(static_cast<const int64_t *>(y)); return EVB_OK;
    case 17: f(static_cast<const uint8_t *>(y)); return EVB_OK;
    case 18: f(static_cast<const uint16_t *>(y)); return EVB_OK;
    case 20: f(static_cast<const uint32_t *>(y)); return EVB_OK;
    default: evb_set_error("evb_host: unknown integer type"); return EVB_ERR_ARG;
    }
}
} // namespace

extern "C" int32_t evb_host_range(const void *y, int32_t kind, int64_t n, int64_t range[2]) {
    if (!y || !range || n < 1) { evb_set_error("evb_host_range: invalid argument"); return EVB_ERR_ARG; }
    return with_ints(y, kind, [&](auto *v) {
        std::mutex mu;
        int64_t lo = (int64_t)v[0], hi = lo;
        host_slices((size_t)n, [&](size_t b, size_t e) {
            auto l = v[b], h = v[b];
            for (size_t i = b; i < e; ++i) { l = v[i] < l ? v[i] : l; h = v[i] > h ? v[i] : h; }
            std::lock_guard<std::mutex> g(mu);
            if ((int64_t)l < lo) lo = (int64_t)l;
            if ((int64_t)h > hi) hi = (int64_t)h;
        });
        range[0] = lo; range[1] = hi;
    });
}

extern "C" int32_t evb_host_count(const void *y, int32_t kind, int64_t n, int64_t lo, int32_t nvalues, int64_t *counts) {
    if (!y || !counts || n < 1 || nvalues < 1) { evb_set_error("evb_host_count: invalid argument"); return EVB_ERR_ARG; }
    for (int32_t k = 0; k < nvalues; ++k) counts[k] = 0;
    return with_ints(y, kind, [&](auto *v) {
        std::mutex mu;
        host_slices((size_t)n, [&](size_t b, size_t e) {
            std::vector<uint32_t> c((size_t)nvalues, 0u);
            for (size_t i = b; i < e; ++i) ++c[(size_t)((int64_t)v[i] - lo)];
            std::lock_guard<std::mutex> g(mu);
            for (int32_t k = 0; k < nvalues; ++k) counts[k] += c[k];
        });
    });
}

extern "C" int32_t evb_host_codes(const void *y, int32_t kind, int64_t n, int64_t lo, const uint32_t *code_of, uint32_t *codes) {
    if (!y || !code_of || !codes || n < 1) { evb_set_error("evb_host_codes: invalid argument"); return EVB_ERR_ARG; }
    return with_ints(y, kind, [&](auto *v) {
        host_slices((size_t)n, [&](size_t b, size_t e) { for (size_t i = b; i < e; ++i) codes[i] = code_of[(int64_t)v[i] - lo]; });
    });
}

// sample standard deviation (n - 1): slices are summed by themselves and added in order, so the result does not depend on
// the number of threads
extern "C" int32_t evb_host_std(const float *y, int64_t n, double *out) {
    if (!y || !out || n < 2) { evb_set_error("evb_host_std: invalid argument"); return EVB_ERR_ARG; }
    std::vector<double> part((size_t)n / HOST_SLICE + 1, 0.0);
    auto total = [&](double shift, bool square) {
        host_slices((size_t)n, [&](size_t b, size_t e) {
            double s[8] = {};
            for (size_t i = b; i < e; ++i) { const double d = (double)y[i] - shift; s[i & 7] += square ? d * d : d; }
            part[b / HOST_SLICE] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
        });
        double t = 0.0;
        for (const double v : part) t += v;
        return t;
    };
    const double mean = total(0.0, false) / (double)n;
    *out = sqrt(total(mean, true) / (double)(n - 1));
    return EVB_OK;
}
