// dev_context.cu -- device context of the library: the CUDA stream, error
// state, memory helpers, dataset upload and kernel timing.
//
// Every host thread works in an execution context: its stream, its device
// status words, its error slot, its grow-only scratch buffers and its random
// generator. The main thread uses the default context (whose generator is
// libc rand(), as in the reference); the batch driver gives each worker
// thread a context of its own (irwls_ctx_create / irwls_ctx_bind) so that
// trainings run concurrently on separate streams. Device memory is allocated
// stream-ordered (cudaMallocAsync / cudaFreeAsync on the context's stream),
// so that no thread's free waits for the whole device.
#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "dev_common.cuh"

namespace {

constexpr int IRWLS_SCRATCH_SLOTS = 4;

// glibc's rand() generator (the additive feedback generator of degree 31 and
// separation 3 behind its random_r), restated so that a worker thread can
// reproduce exactly the numbers srand(seed) then rand() would give in a
// single-threaded run, without sharing libc's state.
struct Rand31 {
    int32_t r[31];
    int f, b;
    void seed(unsigned s) {
        int32_t w = (int32_t)(s == 0 ? 1u : s);
        r[0] = w;
        for (int i = 1; i < 31; ++i) {
            // 16807 * w mod (2^31 - 1) without overflow (Schrage's method)
            const int32_t hi = w / 127773, lo = w % 127773;
            w = 16807 * lo - 2836 * hi;
            if (w < 0) w += 2147483647;
            r[i] = w;
        }
        f = 3;
        b = 0;
        for (int i = 0; i < 310; ++i) next();
    }
    int next() {
        const uint32_t v = (uint32_t)r[f] + (uint32_t)r[b];
        r[f] = (int32_t)v;
        const int out = (int)(v >> 1);
        if (++f >= 31) f = 0;
        if (++b >= 31) b = 0;
        return out;
    }
};

struct Ctx {
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;  // of the device the context was made on
    int *flags = nullptr;  // device status words, see irwls_dev_flags()
    int err = 0;
    char msg[512] = "";
    void *scratch[IRWLS_SCRATCH_SLOTS] = {};
    size_t scratch_bytes[IRWLS_SCRATCH_SLOTS] = {};
    unsigned *post = nullptr;  // pinned words of irwls_ctx_post
    unsigned post_seq = 0;
    int own_rng = 0;
    Rand31 rng;
};

Ctx g_default;
thread_local Ctx *t_ctx = nullptr;
inline Ctx *cur() { return t_ctx ? t_ctx : &g_default; }

int g_inited = 0;
int g_num_sms = 0;
std::atomic<long long> g_launches{0};

}  // namespace

extern "C" void irwls_set_error(int code, const char *fmt, ...) {
    Ctx *c = cur();
    if (c->err < 0) return;  // keep the first error (an error replaces a warning)
    c->err = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(c->msg, sizeof c->msg, fmt, ap);
    va_end(ap);
}
// A warning (positive code): the call returns its result, and the condition
// is reported unless an error or an earlier warning is already recorded.
extern "C" void irwls_set_warning(int code, const char *fmt, ...) {
    Ctx *c = cur();
    if (c->err) return;
    c->err = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(c->msg, sizeof c->msg, fmt, ap);
    va_end(ap);
}
extern "C" int irwls_get_error(void) { return cur()->err; }
extern "C" const char *irwls_get_error_message(void) { return cur()->msg; }
extern "C" void irwls_clear_error(void) {
    cur()->err = 0;
    cur()->msg[0] = 0;
}

cudaStream_t irwls_stream() { return cur()->stream; }
int *irwls_dev_flags() { return cur()->flags; }
int irwls_num_sms() { return g_num_sms; }

extern "C" long long irwls_launch_count(void) { return g_launches.load(); }
extern "C" void irwls_count_launch(int n) { g_launches += n; }

static int cuda_fail(cudaError_t e, const char *what) {
    irwls_set_error(-2, "CUDA error in %s: %s", what, cudaGetErrorString(e));
    return -2;
}

int irwls_check_launch(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, what);
    return 0;
}

// The library's memory pool on the current device. The device's own pool gives
// idle memory back at every synchronisation, and the next call's first allocation
// then maps it again: 120 to 140 us (of a prediction of 64 rows that takes 30), and
// 80 for each later step up. This one keeps up to POOL_KEEP bytes idle;
// irwls_dev_release_workspace gives them back. It is created once per device, is
// safe for any threads and streams (stream-ordered, as before), and where it cannot
// be created the device's pool serves.
constexpr unsigned long long POOL_KEEP = 2ULL << 30;
static cudaMemPool_t device_pool() {
    constexpr int kDevices = 64;
    static std::mutex lock;
    static cudaMemPool_t pools[kDevices];
    static bool tried[kDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> hold(lock);
    if (!tried[dev]) {
        tried[dev] = true;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        unsigned long long keep = POOL_KEEP;
        if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) {
            cudaGetLastError();
            pools[dev] = nullptr;
        } else if (cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            cudaMemPoolDestroy(pools[dev]);
            pools[dev] = nullptr;
        }
    }
    return pools[dev];
}

static cudaError_t pool_malloc(void **p, size_t bytes, Ctx *c) {
    return c->pool ? cudaMallocFromPoolAsync(p, bytes, c->pool, c->stream) : cudaMallocAsync(p, bytes, c->stream);
}

static int ctx_open(Ctx *c) {
    cudaError_t e;
    c->pool = device_pool();
    if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess)
        return cuda_fail(e, "cudaStreamCreate");
    if ((e = cudaMalloc((void **)&c->flags, 8 * sizeof(int))) != cudaSuccess) return cuda_fail(e, "flags alloc");
    if ((e = cudaMemset(c->flags, 0, 8 * sizeof(int))) != cudaSuccess) return cuda_fail(e, "flags init");
    return 0;
}

extern "C" int irwls_dev_init(void) {
    if (g_inited) return 0;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        irwls_set_error(-1, "no CUDA device available (%s); this library has no CPU path",
                        e != cudaSuccess ? cudaGetErrorString(e) : "0 devices");
        return -1;
    }
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if ((e = cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return cuda_fail(e, "cudaDeviceGetAttribute");
    if (ctx_open(&g_default)) return -2;
    g_inited = 1;
    return 0;
}

// Execution contexts of worker threads (the library must be initialised).
extern "C" void *irwls_ctx_create(void) {
    if (irwls_dev_init()) return nullptr;
    Ctx *c = new Ctx();
    if (ctx_open(c)) {
        delete c;
        return nullptr;
    }
    c->own_rng = 1;
    c->rng.seed(1);
    return c;
}
extern "C" void irwls_ctx_bind(void *h) { t_ctx = (Ctx *)h; }
extern "C" void irwls_ctx_destroy(void *h) {
    Ctx *c = (Ctx *)h;
    if (!c) return;
    cudaStreamSynchronize(c->stream);
    for (int k = 0; k < IRWLS_SCRATCH_SLOTS; ++k)
        if (c->scratch[k]) cudaFreeAsync(c->scratch[k], c->stream);
    cudaStreamSynchronize(c->stream);
    cudaFree(c->flags);
    if (c->post) cudaFreeHost(c->post);
    cudaStreamDestroy(c->stream);
    delete c;
}
// Error of a context (for the thread that created it, after a worker ended).
extern "C" int irwls_ctx_error(void *h, char *msg, int cap) {
    Ctx *c = (Ctx *)h;
    if (msg && cap > 0) snprintf(msg, (size_t)cap, "%s", c->msg);
    return c->err;
}

// The current context's random numbers: libc rand() in the default context,
// the context's own glibc-equivalent generator in worker contexts.
extern "C" void irwls_srand(unsigned seed) {
    Ctx *c = cur();
    if (c->own_rng) c->rng.seed(seed);
    else srand(seed);
}
extern "C" int irwls_rand(void) {
    Ctx *c = cur();
    return c->own_rng ? c->rng.next() : rand();
}
// n numbers of a private generator seeded with `seed` (tests compare them
// with libc's srand/rand).
extern "C" void irwls_rand_sequence(unsigned seed, int n, int *out) {
    Rand31 g;
    g.seed(seed);
    for (int i = 0; i < n; ++i) out[i] = g.next();
}

// Allocation-failure injection for tests of the error paths: armed with
// n > 0, the n-th device or pinned-host allocation of the library from then
// on fails as if the runtime had refused it (nothing is allocated).
static std::atomic<long long> g_fail_alloc{0};
extern "C" void irwls_debug_fail_alloc(long long n) { g_fail_alloc.store(n > 0 ? n : 0); }
// Device allocations above this are refused, as where memory is short.
static std::atomic<size_t> g_alloc_limit{~(size_t)0};
extern "C" void irwls_debug_alloc_limit(size_t bytes) { g_alloc_limit.store(bytes ? bytes : ~(size_t)0); }
// Bytes of digit slices at a time where rows are taken in slabs: `normal`, or what a
// test has set.
static std::atomic<size_t> g_slab_bytes{0};
extern "C" void irwls_debug_slab_bytes(size_t bytes) { g_slab_bytes.store(bytes); }
extern "C" size_t irwls_slab_bytes(size_t normal) {
    const size_t b = g_slab_bytes.load();
    return b ? b : normal;
}
static bool injected_alloc_failure() {
    long long v = g_fail_alloc.load();
    while (v > 0)
        if (g_fail_alloc.compare_exchange_weak(v, v - 1)) return v == 1;
    return false;
}

// Grow-only scratch buffer `slot` of the current context (stream-ordered).
extern "C" void *irwls_ctx_scratch(int slot, size_t bytes) {
    Ctx *c = cur();
    if (bytes > c->scratch_bytes[slot]) {
        if (c->scratch[slot]) cudaFreeAsync(c->scratch[slot], c->stream);
        c->scratch[slot] = nullptr;
        c->scratch_bytes[slot] = 0;
        if (injected_alloc_failure()) {
            irwls_set_error(-3, "device scratch of %zu bytes failed (injected failure)", bytes);
            return nullptr;
        }
        if (pool_malloc(&c->scratch[slot], bytes, c) != cudaSuccess) {
            cudaGetLastError();
            irwls_set_error(-3, "device scratch of %zu bytes failed", bytes);
            return nullptr;
        }
        c->scratch_bytes[slot] = bytes;
    }
    return c->scratch[slot];
}

extern "C" int irwls_dev_host_alloc(void **p, size_t bytes);
// The same with zeros in new memory (the users leave zeros behind).
extern "C" void *irwls_ctx_scratch_zeroed(int slot, size_t bytes) {
    Ctx *c = cur();
    const bool fresh = bytes > c->scratch_bytes[slot];
    void *p = irwls_ctx_scratch(slot, bytes);
    if (p && fresh && cudaMemsetAsync(p, 0, bytes, c->stream) != cudaSuccess) {
        cudaGetLastError();
        cudaFreeAsync(c->scratch[slot], c->stream);
        c->scratch[slot] = nullptr;
        c->scratch_bytes[slot] = 0;
        irwls_set_error(-2, "clearing %zu bytes of device scratch failed", bytes);
        return nullptr;
    }
    return p;
}

// The context's pinned words for a kernel that posts one value (word 1) and its
// number (word 0), and the next number; NULL: no memory.
extern "C" unsigned *irwls_ctx_post(unsigned *seq) {
    Ctx *c = cur();
    if (!c->post) {
        if (irwls_dev_host_alloc((void **)&c->post, 2 * sizeof(unsigned))) return nullptr;
        c->post[0] = 0;
    }
    *seq = ++c->post_seq;
    return c->post;
}

extern "C" int irwls_dev_sync(void) {
    cudaError_t e = cudaStreamSynchronize(cur()->stream);
    if (e != cudaSuccess) return cuda_fail(e, "stream synchronize");
    return 0;
}

// Waits until a kernel has posted `v` to *seq (post_seq). The stream is asked now
// and then, so that a failed kernel ends the wait. bytes: what the host reads,
// for the transfer counters.
extern "C" void irwls_count_bytes(long long h2d, long long d2h);
extern "C" int irwls_dev_wait_post(const unsigned *seq, unsigned v, size_t bytes) {
    for (;;) {
        for (int k = 0; k < 2000; ++k)
            if (__atomic_load_n(seq, __ATOMIC_ACQUIRE) == v) {
                irwls_count_bytes(0, (long long)bytes);
                return 0;
            }
        const cudaError_t e = cudaStreamQuery(cur()->stream);
        if (e == cudaErrorNotReady) {
            std::this_thread::yield();
            continue;
        }
        if (e != cudaSuccess) return cuda_fail(e, "waiting for a kernel's result");
        if (__atomic_load_n(seq, __ATOMIC_ACQUIRE) == v) continue;
        irwls_set_error(-2, "a kernel ended without posting its result");
        return -2;
    }
}

// NULL, or why not.
static const char *try_malloc(void **p, size_t bytes) {
    *p = nullptr;
    if (injected_alloc_failure() || bytes > g_alloc_limit.load()) return "injected failure";
    const cudaError_t e = pool_malloc(p, bytes ? bytes : 16, cur());
    if (e == cudaSuccess) return nullptr;
    cudaGetLastError();
    *p = nullptr;
    return cudaGetErrorString(e);
}
extern "C" int irwls_dev_malloc(void **p, size_t bytes) {
    const char *why = try_malloc(p, bytes);
    if (!why) return 0;
    irwls_set_error(-3, "device allocation of %zu bytes failed: %s", bytes, why);
    return -3;
}
// For what a call can do without: a refusal is no error of the call.
extern "C" int irwls_dev_malloc_try(void **p, size_t bytes) { return try_malloc(p, bytes) ? -3 : 0; }
extern "C" int irwls_dev_free(void *p) {
    if (p) cudaFreeAsync(p, cur()->stream);
    return 0;
}
extern "C" void irwls_count_bytes(long long h2d, long long d2h);
extern "C" int irwls_dev_h2d(void *d, const void *h, size_t bytes) {
    if (!bytes) return 0;
    irwls_count_bytes((long long)bytes, 0);
    cudaError_t e = cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, cur()->stream);
    return e == cudaSuccess ? 0 : cuda_fail(e, "H2D copy");
}
extern "C" int irwls_dev_d2h(void *h, const void *d, size_t bytes) {
    if (!bytes) return 0;
    irwls_count_bytes(0, (long long)bytes);
    cudaError_t e = cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, cur()->stream);
    return e == cudaSuccess ? 0 : cuda_fail(e, "D2H copy");
}
extern "C" int irwls_dev_d2d(void *d, const void *s, size_t bytes) {
    if (!bytes) return 0;
    cudaError_t e = cudaMemcpyAsync(d, s, bytes, cudaMemcpyDeviceToDevice, cur()->stream);
    return e == cudaSuccess ? 0 : cuda_fail(e, "D2D copy");
}
extern "C" int irwls_dev_memset(void *d, int byte, size_t bytes) {
    if (!bytes) return 0;
    cudaError_t e = cudaMemsetAsync(d, byte, bytes, cur()->stream);
    return e == cudaSuccess ? 0 : cuda_fail(e, "memset");
}
extern "C" int irwls_dev_host_alloc(void **p, size_t bytes) {
    if (injected_alloc_failure()) {
        *p = nullptr;
        irwls_set_error(-3, "pinned host allocation of %zu bytes failed (injected failure)", bytes);
        return -3;
    }
    cudaError_t e = cudaMallocHost(p, bytes ? bytes : 16);
    if (e != cudaSuccess) {
        *p = nullptr;
        return cuda_fail(e, "cudaMallocHost");
    }
    return 0;
}
extern "C" void irwls_dev_host_free(void *p) {
    if (p) cudaFreeHost(p);
}

extern "C" int irwls_dev_workspace(size_t bytes, void **d_ws) {
    *d_ws = irwls_ctx_scratch(1, bytes);
    return *d_ws ? 0 : -3;
}
static void stages_release();
extern "C" void irwls_dev_release_workspace(void) {
    Ctx *c = cur();
    if (c->scratch[1]) cudaFreeAsync(c->scratch[1], c->stream);
    c->scratch[1] = nullptr;
    c->scratch_bytes[1] = 0;
    if (c->pool) {
        cudaStreamSynchronize(c->stream);
        cudaMemPoolTrimTo(c->pool, 0);
    }
    stages_release();
}

// ---------------------------------------------------------------------------
// Dataset upload. Rows are walked on the host exactly as the reference walks
// its svm_sample lists, by several threads where there are many; the device
// keeps a dense copy (raw values for the raw-RBF mode, values by feature index
// otherwise) plus CSR by feature index, all in one allocation. The CSR, norms
// and labels go over in one copy, and the dense copy by feature index is made
// from them on the device (written on the host and copied as well it was 50 of
// the 64 MB of 8000 rows of 784 features, and most of the 11 ms).
// ---------------------------------------------------------------------------
extern "C" int irwls_model_feature_width(const model *m) {
    int w = 1;
    for (int i = 0; i < m->nSVs; ++i)
        for (const svm_sample *p = m->x[i]; p->index != -1; ++p)
            if (p->index + 1 > w) w = p->index + 1;
    return w;
}

// Training needs finite labels (prediction does not read them, so its
// datasets are not checked).
extern "C" int irwls_check_labels(const svm_dataset *ds, int n_rows) {
    for (int i = 0; i < n_rows; ++i)
        if (!isfinite(ds->y[i])) {
            irwls_set_error(-4, "non-finite label %g in row %d", ds->y[i], i);
            return -4;
        }
    return 0;
}

namespace {

// Pinned staging buffers, kept for the next upload: at most kStageKeep of them,
// each at most kStageBytes, until irwls_dev_release_workspace. An upload has its buffer to itself, from any thread
// or context, and gives it back with an event behind its copy on its stream;
// the next user takes one whose event has passed (or waits for it), so an
// upload itself does not wait. (Copies of pageable memory will not do instead:
// on this machine they may read it after the call has returned.)
constexpr int kStageKeep = 4;
constexpr size_t kStageBytes = (size_t)64 << 20;
struct Stage {
    void *p;
    size_t bytes;
    cudaEvent_t done;
};
std::mutex g_stage_mutex;
std::vector<Stage> g_stages;

void stage_free(const Stage &s) {
    cudaEventDestroy(s.done);
    irwls_dev_host_free(s.p);
}

int stage_take(size_t bytes, Stage *out) {
    int wait = -1;
    {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        g_stages.reserve(kStageKeep + 1);  // (giving back then needs no memory)
        int full = 0;
        for (size_t k = 0; k < g_stages.size(); ++k) {
            if (g_stages[k].bytes < bytes) continue;
            const bool free = cudaEventQuery(g_stages[k].done) == cudaSuccess;
            ++full;
            if (free || full == kStageKeep) {  // all kept buffers are large enough and busy: wait for this one
                *out = g_stages[k];
                g_stages.erase(g_stages.begin() + k);
                wait = !free;
                break;
            }
        }
    }
    cudaGetLastError();  // (a query that was not ready is no error)
    if (wait == 1 && cudaEventSynchronize(out->done) != cudaSuccess) {
        const int rc = cuda_fail(cudaGetLastError(), "staging");
        stage_free(*out);
        *out = {nullptr, 0, nullptr};
        return rc;
    }
    if (wait >= 0) return 0;
    size_t cap = bytes;
    if (bytes <= kStageBytes)  // the next power of two, so that slightly larger sets reuse it
        for (cap = 1 << 20; cap < bytes;) cap <<= 1;
    out->bytes = cap;
    if (irwls_dev_host_alloc(&out->p, cap)) return -3;
    if (cudaEventCreateWithFlags(&out->done, cudaEventDisableTiming) != cudaSuccess) {
        irwls_dev_host_free(out->p);
        out->p = nullptr;
        return cuda_fail(cudaGetLastError(), "staging event");
    }
    return 0;
}
// The copies from s are on the current stream.
int stage_give(Stage s) {
    if (!s.p) return 0;
    Stage drop = {nullptr, 0, nullptr};
    int rc = cudaEventRecord(s.done, cur()->stream) == cudaSuccess ? 0 : -2;
    if (rc || s.bytes > kStageBytes) {
        drop = s;
    } else {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        g_stages.push_back(s);
        if (g_stages.size() > kStageKeep) {  // the smallest goes
            size_t m = 0;
            for (size_t k = 1; k < g_stages.size(); ++k)
                if (g_stages[k].bytes < g_stages[m].bytes) m = k;
            drop = g_stages[m];
            g_stages.erase(g_stages.begin() + m);
        }
    }
    if (drop.p) {
        if (cudaEventSynchronize(drop.done) != cudaSuccess) rc = -2;
        stage_free(drop);
    }
    return rc;
}
// A buffer in use: given back also where an exception ends the upload.
struct StageHold {
    Stage s = {nullptr, 0, nullptr};
    int give() {
        const Stage t = s;
        s.p = nullptr;
        return stage_give(t);
    }
    ~StageHold() { give(); }
};

// fn(first row, last row, chunk) over `n` rows in `chunks` contiguous chunks,
// taken in turn by the caller and helpers - 1 other threads. The caller waits for
// the chunks, not for the threads: one that the system starts late (behind
// another library's spinning threads that cost up to 6 ms) finds nothing left
// and ends by itself. fn does not throw.
struct RowTeam {
    std::atomic<int> next{0}, done{0};
    int n = 0, chunks = 0;
    std::function<void(int, int, int)> fn;
    void work() {
        for (int c; (c = next.fetch_add(1)) < chunks;) {
            fn((int)((long long)n * c / chunks), (int)((long long)n * (c + 1) / chunks), c);
            done.fetch_add(1);
        }
    }
};
void over_rows(int n, int chunks, int helpers, std::function<void(int, int, int)> fn) {
    auto team = std::make_shared<RowTeam>();
    team->n = n;
    team->chunks = chunks;
    team->fn = std::move(fn);
    try {
        for (int t = 1; t < helpers; ++t) std::thread([team] { team->work(); }).detach();
    } catch (...) {  // (no thread to be had: the caller does it all)
    }
    team->work();
    while (team->done.load() < chunks) std::this_thread::yield();
}

}  // namespace

// The kept buffers given back (those in use come back later and are kept then).
static void stages_release() {
    std::vector<Stage> all;
    {
        std::lock_guard<std::mutex> lock(g_stage_mutex);
        all.swap(g_stages);
    }
    for (const Stage &s : all) {
        cudaEventSynchronize(s.done);
        stage_free(s);
    }
}
extern "C" long long irwls_staging_bytes(void) {
    std::lock_guard<std::mutex> lock(g_stage_mutex);
    long long b = 0;
    for (const Stage &s : g_stages) b += (long long)s.bytes;
    return b;
}

namespace {

// The dense rows by feature index from the CSR: a warp per row writes its
// zeros, then its entries (a row whose indices do not increase may name one
// twice: its first lane writes it in order, so the last entry stays).
__global__ void __launch_bounds__(256) dense_rows_kernel(const int *__restrict__ rp, const int *__restrict__ ci,
                                                         const double *__restrict__ cv, int n, int ld,
                                                         double *__restrict__ X) {
    const int lane = threadIdx.x & 31;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        double *row = X + (size_t)i * ld;
        for (int t = lane; t < ld; t += 32) row[t] = 0.0;
        const int p0 = rp[i], p1 = rp[i + 1];
        bool bad = false;
        for (int p = p0 + 1 + lane; p < p1; p += 32) bad |= ci[p] <= ci[p - 1];
        bad = __any_sync(0xffffffffu, bad);
        __syncwarp();
        if (!bad)
            for (int p = p0 + lane; p < p1; p += 32) row[ci[p]] = cv[p];
        else if (lane == 0)
            for (int p = p0; p < p1; ++p) row[ci[p]] = cv[p];
        __syncwarp();
    }
}

struct RowScan {
    long long nnz = 0;
    int width = 1, bad_row = -1, bad_index = 0;
    double bad_value = 0.0;
};

inline size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

// csr_only: no dense copy X (for consumers that read the rows as CSR only).
static int upload_rows_(svm_sample *const *rows, const double *q, const double *y, int n_rows, int mode,
                        double gamma, int raw_width, int width_hint, irwls_dev_set *out, int csr_only) {
    out->n_rows = n_rows;
    out->mode = mode;
    out->neg_gamma = -gamma;
    // threads: one more per 250000 entries by the first row's length, one in
    // the batching form's workers. (From 40000 on the warm time fell by 0.3 ms
    // of 6.3 at 240000 entries, but where another library's threads still spin
    // after a call of its own, a helper in the middle of a chunk can lose its
    // core for 6 ms: not worth it below a walk of several milliseconds.)
    int helpers = 1;
    if (!t_ctx && n_rows >= 64) {
        long long len = 1;
        for (const svm_sample *p = rows[0]; p->index != -1; ++p) ++len;
        const int hw = (int)std::thread::hardware_concurrency();
        helpers = (int)std::min<long long>(std::min(8, hw > 0 ? hw : 1), 1 + len * n_rows / 250000);
    }
    const int chunks = helpers > 1 ? 4 * helpers : 1;
    std::vector<int> count((size_t)n_rows + 1);
    std::vector<RowScan> scan(chunks);
    over_rows(n_rows, chunks, helpers, [&, rows](int i0, int i1, int t) {
        RowScan r;
        for (int i = i0; i < i1; ++i) {
            const svm_sample *p = rows[i];
            for (; p->index != -1; ++p) {
                if (p->index < 0 || !isfinite(p->value)) {
                    r.bad_row = i;
                    r.bad_index = p->index;
                    r.bad_value = p->value;
                    scan[t] = r;
                    return;
                }
                if (p->index + 1 > r.width) r.width = p->index + 1;
            }
            count[i] = (int)(p - rows[i]);
            r.nnz += p - rows[i];
        }
        scan[t] = r;
    });
    long long nnz = 0;
    int width = 1;
    for (const RowScan &r : scan) {
        if (r.bad_row >= 0) {
            if (r.bad_index < 0)
                irwls_set_error(-4, "negative feature index %d in row %d", r.bad_index, r.bad_row);
            else
                irwls_set_error(-4, "non-finite value %g of feature %d in row %d", r.bad_value, r.bad_index, r.bad_row);
            return -4;
        }
        nnz += r.nnz;
        width = std::max(width, r.width);
    }
    if (width_hint > width) width = width_hint;
    if (mode == IRWLS_K_RAW_RBF) width = raw_width > 0 ? raw_width : 1;
    out->width = width;
    out->ld = (width + 1) & ~1;
    out->nnz = nnz;
    if (nnz > 2147483647LL) {
        irwls_set_error(-4, "dataset has %lld stored entries; the device layout indexes them with int32", nnz);
        return -4;
    }
    const bool raw = mode == IRWLS_K_RAW_RBF && !csr_only;
    const size_t n = (size_t)n_rows;
    const size_t xbytes = csr_only ? 0 : round256(n * out->ld * sizeof(double));
    const size_t qb = round256(n * sizeof(double)), vb = round256((size_t)nnz * sizeof(double)),
                 rb = round256((n + 1) * sizeof(int)), ib = round256((size_t)nnz * sizeof(int));
    const size_t pack = 2 * qb + vb + rb + ib;   // q, y, cv, rp, ci
    const size_t head = raw ? xbytes : 0;        // the raw rows go over as they are
    StageHold stage;
    if (stage_take(head + pack, &stage.s)) return -3;
    unsigned char *h = (unsigned char *)stage.s.p;
    double *hX = (double *)h, *hq = (double *)(h + head), *hy = (double *)(h + head + qb),
           *hcv = (double *)(h + head + 2 * qb);
    int *hrp = (int *)(h + head + 2 * qb + vb), *hci = (int *)(h + head + 2 * qb + vb + rb);
    hrp[0] = 0;
    for (int i = 0; i < n_rows; ++i) hrp[i + 1] = hrp[i] + count[i];
    const int ld = out->ld;
    over_rows(n_rows, chunks, helpers, [=](int i0, int i1, int) {
        if (i1 > i0) {
            if (q) memcpy(hq + i0, q + i0, (size_t)(i1 - i0) * sizeof(double));
            else memset(hq + i0, 0, (size_t)(i1 - i0) * sizeof(double));
            if (y) memcpy(hy + i0, y + i0, (size_t)(i1 - i0) * sizeof(double));
            else memset(hy + i0, 0, (size_t)(i1 - i0) * sizeof(double));
        }
        for (int i = i0; i < i1; ++i) {
            const svm_sample *p = rows[i];
            for (int k = hrp[i]; k < hrp[i + 1]; ++k, ++p) {
                hci[k] = p->index;
                hcv[k] = p->value;
            }
            if (raw) {
                // maxdim consecutive values from the row start, as src/kernels.c:93-97 reads them
                double *row = hX + (size_t)i * ld;
                for (int t = 0; t < raw_width; ++t) row[t] = rows[i][t].value;
                for (int t = raw_width > 0 ? raw_width : 0; t < ld; ++t) row[t] = 0.0;
            }
        }
    });
    int rc = irwls_dev_malloc(&out->block, xbytes + pack);
    if (!rc) {
        unsigned char *d = (unsigned char *)out->block;
        out->X = (double *)d;
        out->q = (double *)(d + xbytes);
        out->y = (double *)(d + xbytes + qb);
        out->cv = (double *)(d + xbytes + 2 * qb);
        out->rp = (int *)(d + xbytes + 2 * qb + vb);
        out->ci = (int *)(d + xbytes + 2 * qb + vb + rb);
        rc |= irwls_dev_h2d(raw ? (void *)out->X : (void *)out->q, h, head + pack);
        if (!rc && !raw && !csr_only && n_rows > 0) {
            dense_rows_kernel<<<std::min((n_rows + 7) / 8, 16 * g_num_sms), 256, 0, cur()->stream>>>(
                out->rp, out->ci, out->cv, n_rows, ld, out->X);
            irwls_count_launch(1);
            rc |= irwls_check_launch("dense_rows");
        }
    }
    rc |= stage.give();
    if (rc) {
        irwls_dev_release(out);
        return rc < 0 ? rc : -3;
    }
    return 0;
}

static int upload_rows(svm_sample *const *rows, const double *q, const double *y, int n_rows, int mode,
                       double gamma, int raw_width, int width_hint, irwls_dev_set *out, int csr_only = 0) {
    memset(out, 0, sizeof *out);
    if (irwls_dev_init()) return -1;
    try {
        return upload_rows_(rows, q, y, n_rows, mode, gamma, raw_width, width_hint, out, csr_only);
    } catch (...) {  // no exception crosses the C interface
        irwls_set_error(-3, "host memory for the upload of %d rows failed", n_rows);
        irwls_dev_release(out);
        return -3;
    }
}

// The rows of ds as CSR only (no dense copy): for the linear prediction path.
extern "C" int irwls_dev_upload_csr(const svm_dataset *ds, int n_rows, int kernelType, double gamma, int width_hint,
                                    irwls_dev_set *out) {
    const int mode = kernelType == 0 ? IRWLS_K_LINEAR : IRWLS_K_NORM_RBF;
    return upload_rows(ds->x, ds->quadratic_value, ds->y, n_rows, mode, gamma, ds->maxdim, width_hint, out, 1);
}

extern "C" int irwls_dev_upload(const svm_dataset *ds, int n_rows, int kernelType, double gamma, int force_norm,
                                int width_hint, irwls_dev_set *out) {
    int mode = kernelType == 0 ? IRWLS_K_LINEAR
                               : ((ds->sparse == 0 && !force_norm) ? IRWLS_K_RAW_RBF : IRWLS_K_NORM_RBF);
    return upload_rows(ds->x, ds->quadratic_value, ds->y, n_rows, mode, gamma, ds->maxdim, width_hint, out);
}

extern "C" int irwls_dev_upload_model(const model *m, int width_hint, irwls_dev_set *out) {
    int mode = m->kernelType == 0 ? IRWLS_K_LINEAR : IRWLS_K_NORM_RBF;
    return upload_rows(m->x, m->quadratic_value, nullptr, m->nSVs, mode, m->Kgamma, m->maxdim, width_hint, out);
}

extern "C" void irwls_dev_release(irwls_dev_set *s) {
    if (!s) return;
    void *b[] = {s->X, s->q, s->y, s->rp, s->ci, s->cv};
    if (s->block) irwls_dev_free(s->block);
    else
        for (void *p : b) irwls_dev_free(p);
    memset(s, 0, sizeof *s);
}

// ---------------------------------------------------------------------------
// Timing of selected kernels with CUDA events on the library stream.
// ---------------------------------------------------------------------------
struct ProfSlot {
    std::vector<cudaEvent_t> pending;  // begin/end pairs not yet read
    std::vector<cudaEvent_t> pool;
    double ms = 0.0;
    long long launches = 0;
};
static ProfSlot g_prof[IRWLS_PROF_SLOTS];
static int g_prof_on = 0;

static cudaEvent_t prof_event(ProfSlot &s) {
    if (!s.pool.empty()) {
        cudaEvent_t e = s.pool.back();
        s.pool.pop_back();
        return e;
    }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
}
// Kernel timing is recorded in the default context only.
extern "C" void irwls_prof_enable(int on) { g_prof_on = on; }
extern "C" int irwls_prof_on(void) { return g_prof_on && !t_ctx; }
extern "C" void irwls_prof_begin(int slot) {
    if (!irwls_prof_on()) return;
    ProfSlot &s = g_prof[slot];
    cudaEvent_t e = prof_event(s);
    cudaEventRecord(e, g_default.stream);
    s.pending.push_back(e);
}
extern "C" void irwls_prof_end(int slot) {
    if (!irwls_prof_on()) return;
    ProfSlot &s = g_prof[slot];
    cudaEvent_t e = prof_event(s);
    cudaEventRecord(e, g_default.stream);
    s.pending.push_back(e);
    if (s.pending.size() > 4096) irwls_prof_collect();
}
extern "C" int irwls_prof_collect(void) {
    cudaStreamSynchronize(g_default.stream);
    for (auto &s : g_prof) {
        for (size_t i = 0; i + 1 < s.pending.size(); i += 2) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, s.pending[i], s.pending[i + 1]);
            s.ms += ms;
            s.launches += 1;
            s.pool.push_back(s.pending[i]);
            s.pool.push_back(s.pending[i + 1]);
        }
        s.pending.clear();
    }
    return 0;
}
extern "C" void irwls_prof_read(int slot, double *ms, long long *launches) {
    *ms = g_prof[slot].ms;
    *launches = g_prof[slot].launches;
}
extern "C" void irwls_prof_reset(void) {
    irwls_prof_collect();
    for (auto &s : g_prof) {
        s.ms = 0.0;
        s.launches = 0;
    }
}

extern "C" int irwls_dev_chol_info(int *info) {
    int flags[8];
    cudaError_t e = cudaMemcpyAsync(flags, cur()->flags, sizeof flags, cudaMemcpyDeviceToHost, cur()->stream);
    if (e != cudaSuccess) return cuda_fail(e, "read flags");
    if (irwls_dev_sync()) return -2;
    *info = flags[0];
    return 0;
}

// ---------------------------------------------------------------------------
// Benchmark support: transfer counters, L2 flush, stream timers and a probe of
// the device's FP64 FMA throughput (the roofline denominator of the FP64
// kernels: chains of independent DFMAs, no memory traffic).
// ---------------------------------------------------------------------------
static std::atomic<long long> g_h2d{0}, g_d2h{0};
extern "C" void irwls_count_bytes(long long h2d, long long d2h) {
    g_h2d += h2d;
    g_d2h += d2h;
}
extern "C" void irwls_transfer_bytes(long long *h2d, long long *d2h) {
    *h2d = g_h2d.load();
    *d2h = g_d2h.load();
}

static void *g_flush = nullptr;
extern "C" int irwls_l2_flush(size_t bytes) {
    if (irwls_dev_init()) return -1;
    if (!g_flush && irwls_dev_malloc(&g_flush, bytes)) return -3;
    return irwls_dev_memset(g_flush, 0x5a, bytes);
}

static cudaEvent_t g_t0 = nullptr, g_t1 = nullptr;
extern "C" int irwls_timer_start(void) {
    if (irwls_dev_init()) return -1;
    if (!g_t0) {
        cudaEventCreate(&g_t0);
        cudaEventCreate(&g_t1);
    }
    cudaEventRecord(g_t0, cur()->stream);
    return 0;
}
extern "C" double irwls_timer_stop(void) {
    cudaEventRecord(g_t1, cur()->stream);
    cudaEventSynchronize(g_t1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g_t0, g_t1);
    return ms;
}

namespace {
__global__ void fp64_probe_kernel(double *out, int iters) {
    double a[8];
    for (int k = 0; k < 8; ++k) a[k] = threadIdx.x * 1e-3 + k;
    const double b = 0.999999, c = 1e-7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
    }
    double s = 0;
    for (int k = 0; k < 8; ++k) s += a[k];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
__global__ void fp32_probe_kernel(float *out, int iters) {
    float a[8];
    for (int k = 0; k < 8; ++k) a[k] = threadIdx.x * 1e-3f + k;
    const float b = 0.9999f, c = 1e-4f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = fmaf(a[k], b, c);
    }
    float s = 0;
    for (int k = 0; k < 8; ++k) s += a[k];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
}  // namespace

// FP32 FMA throughput in TFLOP/s (one FMA = 2 flops), best of `reps` timed
// launches: the FP32-issue ceiling reported beside the tensor-core kernels.
extern "C" double irwls_fp32_peak_tflops(int reps) {
    if (irwls_dev_init()) return 0.0;
    const int blocks = 4 * g_num_sms, threads = 256, iters = 100000;
    float *d = nullptr;
    if (irwls_dev_malloc((void **)&d, (size_t)blocks * threads * sizeof(float))) return 0.0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 0.0;
    fp32_probe_kernel<<<blocks, threads, 0, cur()->stream>>>(d, iters);
    for (int r = 0; r < reps; ++r) {
        cudaEventRecord(e0, cur()->stream);
        fp32_probe_kernel<<<blocks, threads, 0, cur()->stream>>>(d, iters);
        cudaEventRecord(e1, cur()->stream);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double tf = 2.0 * 8 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
        if (tf > best) best = tf;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    irwls_dev_free(d);
    irwls_dev_sync();
    return best;
}

// FP64 FMA throughput in TFLOP/s, best of `reps` timed launches.
extern "C" double irwls_fp64_peak_tflops(int reps) {
    if (irwls_dev_init()) return 0.0;
    const int blocks = 4 * g_num_sms, threads = 256, iters = 20000;
    double *d = nullptr;
    if (irwls_dev_malloc((void **)&d, (size_t)blocks * threads * sizeof(double))) return 0.0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 0.0;
    fp64_probe_kernel<<<blocks, threads, 0, cur()->stream>>>(d, iters);
    for (int r = 0; r < reps; ++r) {
        cudaEventRecord(e0, cur()->stream);
        fp64_probe_kernel<<<blocks, threads, 0, cur()->stream>>>(d, iters);
        cudaEventRecord(e1, cur()->stream);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double tf = 2.0 * 8 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
        if (tf > best) best = tf;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    irwls_dev_free(d);
    irwls_dev_sync();
    return best;
}
