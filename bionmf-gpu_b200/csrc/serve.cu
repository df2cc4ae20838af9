// serve.cu -- the serving API (nmfb_serve_*): requests queued on the device
// while a persistent kernel (serve_kernel.cu) runs.
#include "batch.cuh"

#include <float.h>
#include <math.h>
#include <stdarg.h>
#include <stdlib.h>
#include <algorithm>
#include <atomic>
#include <chrono>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

using namespace nmfb_batched;

// ---------------------------------------------------------------------------
// Serving: a persistent k_serve launch fed with requests as they arrive.
namespace {

constexpr uint32_t SERVE_WT = 16, SERVE_JT = 16;   // tile shapes that size the launch's shared memory

// Tile shapes of a served problem: within the staging buffer the launch
// reserves for (max_m, max_k), the tallest update_H tile (narrow problems
// get many rows per tile: their per-tile work is small next to the staging
// latency) and the widest update_W tile.
void serve_tiles(uint32_t max_m, uint32_t max_k, uint32_t m, uint32_t k, uint32_t *wt, uint32_t *jt)
{
    uint64_t const ldmax = ((uint64_t)max_m + 31) / 32 * 32, ld = ((uint64_t)m + 31) / 32 * 32;
    SmemLayout const Lmax = smem_layout(max_m, ks_of(max_k), SERVE_WT, SERVE_JT, ldmax);
    uint32_t const cap = Lmax.hbuf > Lmax.wbuf ? Lmax.hbuf : Lmax.wbuf;
    uint32_t const cs = ld < (uint64_t)NT ? (uint32_t)ld : (uint32_t)NT;
    uint32_t w = cap / (cs + ks_of(k));
    w = w > 512 ? 512 : (w & ~7u);
    *wt = w < 8 ? 8 : w;
    uint32_t j = 64;
    while (j > 4 && (uint32_t)NT * (j + 4) > cap) j >>= 1;
    *jt = j;
}

struct ServeSlot {
    uint32_t ticket;      // ticket + 1 while occupied, 0 when free
    uint32_t n, m, k;
    float *V, *W, *H;
    uint32_t *labels;
};

uint64_t serve_bytes(uint32_t n, uint32_t m, uint32_t k)
{
    uint64_t const ldv = ((uint64_t)m + 31) / 32 * 32, ks = ks_of(k);
    return ((uint64_t)n * ldv + (uint64_t)n * ks + (uint64_t)m * ks + m) * 4u + 4 * 256u;
}

}  // namespace

struct nmfb_serve {
    int device;
    uint32_t max_m, max_k, capacity, ctas, nclusters;
    unsigned long long idle_ns;
    size_t smem;
    cudaStream_t kstream, cstream, rstream;   // kernel, uploads, results
    cudaMemPool_t pool;
    Problem *dRing, *hRing;                   // descriptors (device) and their pinned host copies
    uint32_t *dCtl;                           // [0] taken, [32] published
    uint32_t *hPub;                           // pinned: published value per slot (ticket + 1)
    volatile uint32_t *hClosing;              // mapped: set by destroy
    volatile uint32_t *hDone;                 // mapped: completion records, 4 words per slot
    uint32_t *dClosingAlias, *dDoneAlias;
    cudaEvent_t kdone;
    bool running;
    uint32_t next_ticket, published;
    std::vector<ServeSlot> slots;
    std::mutex mu;
    char err[512];
};

static int sfail(nmfb_serve *s, int code, const char *fmt, ...)
{
    if (s) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(s->err, sizeof(s->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define STRY(s, call)                                                                                      \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return sfail((s), NMFB_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));     \
    } while (0)

// Launch k_serve if it is not running and published work is untaken (caller holds mu).
static int serve_ensure_running(nmfb_serve *s)
{
    if (s->running) {
        cudaError_t const q = cudaEventQuery(s->kdone);
        if (q == cudaErrorNotReady) return NMFB_OK;
        if (q != cudaSuccess) return sfail(s, NMFB_ECUDA, "serving kernel: %s", cudaGetErrorString(q));
        s->running = false;
    }
    uint32_t taken = 0;
    STRY(s, cudaMemcpyAsync(&taken, s->dCtl, sizeof(uint32_t), cudaMemcpyDeviceToHost, s->kstream));
    STRY(s, cudaStreamSynchronize(s->kstream));
    if (taken >= s->published) return NMFB_OK;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = s->ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s->nclusters * s->ctas, 1, 1);
    cfg.blockDim = dim3(NT, 1, 1);
    cfg.dynamicSmemBytes = s->smem;
    cfg.stream = s->kstream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    STRY(s, cudaLaunchKernelEx(&cfg, serve_kernel(), (const Problem *)s->dRing, s->capacity, s->dCtl,
                               (const volatile uint32_t *)(s->dCtl + 32), (const volatile uint32_t *)s->dClosingAlias,
                               (volatile uint32_t *)s->dDoneAlias, s->idle_ns));
    STRY(s, cudaEventRecord(s->kdone, s->kstream));
    s->running = true;
    return NMFB_OK;
}

extern "C" {

uint64_t nmfb_serve_request_bytes(uint32_t n, uint32_t m, uint32_t k) { return serve_bytes(n, m, k); }

int nmfb_serve_create(nmfb_serve **out, int device, uint32_t max_m, uint32_t max_k, uint32_t capacity,
                      uint32_t ctas, uint32_t idle_ms)
{
    if (!out) return NMFB_EINVAL;
    *out = nullptr;
    nmfb_serve *s = new (std::nothrow) nmfb_serve();
    if (!s) return NMFB_ENOMEM;
    *out = s;
    s->device = device;
    if (max_m < 2 || max_k < KMIN || max_k > KMAX || capacity == 0 || capacity > (1u << 20) ||
        (ctas != 1 && ctas != 2 && ctas != 4 && ctas != 8) || idle_ms == 0)
        return sfail(s, NMFB_EINVAL, "serve: max_m >= 2, max_k in [2, 20], capacity in [1, 2^20], ctas 1/2/4/8, idle > 0");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return sfail(s, NMFB_ENODEV, "no CUDA device %d", device);
    }
    int major = 0, sms = 0, optin = 0;
    STRY(s, cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    if (major != 10) return sfail(s, NMFB_ENODEV, "device %d is not sm_100a", device);
    STRY(s, cudaSetDevice(device));
    STRY(s, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    STRY(s, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    s->max_m = max_m;
    s->max_k = max_k;
    s->capacity = capacity;
    s->ctas = ctas;
    s->idle_ns = (unsigned long long)idle_ms * 1000000ull;
    s->smem = problem_smem_bytes(max_m, max_k, SERVE_WT, SERVE_JT);
    if (s->smem + 64 > (size_t)optin)
        return sfail(s, NMFB_EINVAL, "serve: max_m = %u with max_k = %u does not fit shared memory", max_m, max_k);
    ServeKernel const kern = serve_kernel();
    STRY(s, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s->smem));
    {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ctas * (uint32_t)sms, 1, 1);
        cfg.blockDim = dim3(NT, 1, 1);
        cfg.dynamicSmemBytes = s->smem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int ncl = 0;
        STRY(s, cudaOccupancyMaxActiveClusters(&ncl, kern, &cfg));
        if (ncl < 1) return sfail(s, NMFB_EINVAL, "serve: no cluster of %u CTAs fits", ctas);
        s->nclusters = (uint32_t)ncl;
    }
    STRY(s, cudaStreamCreateWithFlags(&s->kstream, cudaStreamNonBlocking));
    STRY(s, cudaStreamCreateWithFlags(&s->cstream, cudaStreamNonBlocking));
    STRY(s, cudaStreamCreateWithFlags(&s->rstream, cudaStreamNonBlocking));
    STRY(s, cudaEventCreateWithFlags(&s->kdone, cudaEventDisableTiming));
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    STRY(s, cudaMemPoolCreate(&s->pool, &props));
    uint64_t keep = UINT64_MAX;
    STRY(s, cudaMemPoolSetAttribute(s->pool, cudaMemPoolAttrReleaseThreshold, &keep));
    STRY(s, cudaMalloc(&s->dRing, (size_t)capacity * sizeof(Problem)));
    STRY(s, cudaMalloc(&s->dCtl, 64 * sizeof(uint32_t)));
    STRY(s, cudaMemset(s->dCtl, 0, 64 * sizeof(uint32_t)));
    STRY(s, cudaMallocHost(&s->hRing, (size_t)capacity * sizeof(Problem)));
    STRY(s, cudaMallocHost(&s->hPub, (size_t)capacity * sizeof(uint32_t)));
    void *p = nullptr;
    STRY(s, cudaHostAlloc(&p, sizeof(uint32_t), cudaHostAllocMapped));
    s->hClosing = (volatile uint32_t *)p;
    *s->hClosing = 0;
    STRY(s, cudaHostGetDevicePointer((void **)&s->dClosingAlias, p, 0));
    STRY(s, cudaHostAlloc(&p, (size_t)capacity * 4 * sizeof(uint32_t), cudaHostAllocMapped));
    memset(p, 0, (size_t)capacity * 4 * sizeof(uint32_t));
    s->hDone = (volatile uint32_t *)p;
    STRY(s, cudaHostGetDevicePointer((void **)&s->dDoneAlias, p, 0));
    s->slots.assign(capacity, ServeSlot{});
    return NMFB_OK;
}

int nmfb_serve_destroy(nmfb_serve *s)
{
    if (!s) return NMFB_OK;
    cudaSetDevice(s->device);
    if (s->hClosing) *s->hClosing = 1;
    if (s->kstream) cudaStreamSynchronize(s->kstream);
    if (s->cstream) cudaStreamSynchronize(s->cstream);
    if (s->rstream) cudaStreamSynchronize(s->rstream);
    for (ServeSlot &sl : s->slots)
        if (sl.ticket) {
            cudaFree(sl.V);
            cudaFree(sl.W);
            cudaFree(sl.H);
            cudaFree(sl.labels);
        }
    if (s->dRing) cudaFree(s->dRing);
    if (s->dCtl) cudaFree(s->dCtl);
    if (s->hRing) cudaFreeHost(s->hRing);
    if (s->hPub) cudaFreeHost(s->hPub);
    if (s->hClosing) cudaFreeHost((void *)s->hClosing);
    if (s->hDone) cudaFreeHost((void *)s->hDone);
    if (s->pool) cudaMemPoolDestroy(s->pool);
    if (s->kdone) cudaEventDestroy(s->kdone);
    if (s->kstream) cudaStreamDestroy(s->kstream);
    if (s->cstream) cudaStreamDestroy(s->cstream);
    if (s->rstream) cudaStreamDestroy(s->rstream);
    delete s;
    return NMFB_OK;
}

const char *nmfb_serve_last_error(const nmfb_serve *s) { return s ? s->err : "null server"; }

int nmfb_serve_submit(nmfb_serve *s, const float *V, size_t ldv, uint32_t n, uint32_t m, uint32_t k, uint32_t seed,
                      uint32_t n_iters, uint32_t niter_test_conv, uint32_t stop_threshold, uint32_t *ticket)
{
    if (!s || !V || !ticket) return sfail(s, NMFB_EINVAL, "nmfb_serve_submit: null argument");
    if (n < 2 || m < 2 || m > s->max_m || ldv < m || k < KMIN || k > s->max_k || k > (n < m ? n : m))
        return sfail(s, NMFB_EINVAL, "request %u x %u, k = %u outside the server's limits (m <= %u, 2 <= k <= min(%u, n, m))",
                     n, m, k, s->max_m, s->max_k);
    if (n_iters == 0 || niter_test_conv == 0 || stop_threshold == 0)
        return sfail(s, NMFB_EINVAL, "nIters, niter_test_conv and stop_threshold must be positive");
    {
        uint32_t wt, jt;
        serve_tiles(s->max_m, s->max_k, m, k, &wt, &jt);
        if (problem_smem_bytes(m, k, wt, jt) > s->smem)
            return sfail(s, NMFB_EINVAL, "request %u x %u, k = %u: tiles exceed the server's shared memory", n, m, k);
    }
    std::lock_guard<std::mutex> lock(s->mu);
    STRY(s, cudaSetDevice(s->device));
    uint32_t const t = s->next_ticket, slot = t % s->capacity;
    ServeSlot &sl = s->slots[slot];
    if (sl.ticket) return sfail(s, NMFB_ESTATE, "all %u request slots are in use (fetch finished requests first)", s->capacity);
    uint32_t const ks = ks_of(k);
    uint64_t const ldp = ((uint64_t)m + 31) / 32 * 32;
    // CPU_RANDOM initialisation (src/NMF_routines.c:299-307), as nmfb_init_random
    std::vector<float> W((size_t)n * ks), H((size_t)m * ks);
    {
        char rstate[128];
        struct random_data rd;
        memset(&rd, 0, sizeof(rd));
        initstate_r(seed, rstate, sizeof(rstate), &rd);
        auto next = [&]() -> float {
            int32_t r;
            random_r(&rd, &r);
            return ((float)r) / ((float)RAND_MAX) + FLT_MIN;
        };
        for (uint32_t i = 0; i < n; i++)
            for (uint32_t c = 0; c < ks; c++) W[(size_t)i * ks + c] = (c < k) ? next() : 0.0f;
        for (uint32_t j = 0; j < m; j++)
            for (uint32_t c = 0; c < ks; c++) H[(size_t)j * ks + c] = (c < k) ? next() : 0.0f;
    }
    ServeSlot ns{};
    cudaError_t e = cudaMallocFromPoolAsync((void **)&ns.V, (size_t)n * ldp * sizeof(float), s->pool, s->cstream);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void **)&ns.W, W.size() * sizeof(float), s->pool, s->cstream);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void **)&ns.H, H.size() * sizeof(float), s->pool, s->cstream);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void **)&ns.labels, (size_t)m * sizeof(uint32_t), s->pool, s->cstream);
    if (e != cudaSuccess) {
        if (ns.V) cudaFreeAsync(ns.V, s->cstream);
        if (ns.W) cudaFreeAsync(ns.W, s->cstream);
        if (ns.H) cudaFreeAsync(ns.H, s->cstream);
        cudaGetLastError();
        return sfail(s, NMFB_ENOMEM, "request memory: %s", cudaGetErrorString(e));
    }
    // The request's V, W and H into its device buffers.  From pageable host memory
    // V's rows are packed at the device pitch (padding zero) into one of the
    // library's page-locked staging buffers, W and H behind them, and copied with
    // one DMA each (a pitched copy from pageable memory moves one short row at a
    // time); device or page-locked V is copied directly.  The staging buffer is
    // handed back once the copies are done (end of this call).
    cudaPointerAttributes pa;
    bool const pageable = !(cudaPointerGetAttributes(&pa, V) == cudaSuccess &&
                            (pa.type == cudaMemoryTypeDevice || pa.type == cudaMemoryTypeHost ||
                             pa.type == cudaMemoryTypeManaged));
    cudaGetLastError();
    size_t const vfl = (size_t)n * ldp;
    struct StageGuard {
        float *p;
        cudaStream_t st;
        ~StageGuard()
        {
            if (p) {
                cudaStreamSynchronize(st);   // the copies reading it are done
                nmfb_stage_put(p);
            }
        }
    } stage{pageable ? (float *)nmfb_stage_get((vfl + W.size() + H.size()) * sizeof(float)) : nullptr, s->cstream};
    if (stage.p) {
        for (uint32_t i = 0; i < n; i++) {
            float *d = stage.p + (size_t)i * ldp;
            memcpy(d, V + (size_t)i * ldv, m * sizeof(float));
            memset(d + m, 0, (ldp - m) * sizeof(float));
        }
        memcpy(stage.p + vfl, W.data(), W.size() * sizeof(float));
        memcpy(stage.p + vfl + W.size(), H.data(), H.size() * sizeof(float));
        STRY(s, cudaMemcpyAsync(ns.V, stage.p, vfl * sizeof(float), cudaMemcpyHostToDevice, s->cstream));
        STRY(s, cudaMemcpyAsync(ns.W, stage.p + vfl, W.size() * sizeof(float), cudaMemcpyHostToDevice, s->cstream));
        STRY(s, cudaMemcpyAsync(ns.H, stage.p + vfl + W.size(), H.size() * sizeof(float), cudaMemcpyHostToDevice,
                                s->cstream));
    } else {
        STRY(s, cudaMemsetAsync(ns.V, 0, vfl * sizeof(float), s->cstream));
        STRY(s, cudaMemcpy2DAsync(ns.V, ldp * sizeof(float), V, ldv * sizeof(float), m * sizeof(float), n,
                                  cudaMemcpyDefault, s->cstream));
        STRY(s, cudaMemcpyAsync(ns.W, W.data(), W.size() * sizeof(float), cudaMemcpyHostToDevice, s->cstream));
        STRY(s, cudaMemcpyAsync(ns.H, H.data(), H.size() * sizeof(float), cudaMemcpyHostToDevice, s->cstream));
    }
    Problem &P = s->hRing[slot];
    memset(&P, 0, sizeof(P));
    P.V = ns.V;
    P.W = ns.W;
    P.H = ns.H;
    P.labels = ns.labels;
    P.ldv = ldp;
    P.n = n;
    P.m = m;
    P.k = k;
    P.ks = ks;
    serve_tiles(s->max_m, s->max_k, m, k, &P.wt, &P.jt);
    P.n_iters = n_iters;
    P.niter_test_conv = niter_test_conv;
    P.stop_threshold = stop_threshold;
    STRY(s, cudaMemcpyAsync(s->dRing + slot, &P, sizeof(Problem), cudaMemcpyHostToDevice, s->cstream));
    s->hDone[4 * (size_t)slot] = 0;
    // the new published count follows the request's data on the same stream
    s->hPub[slot] = t + 1u;
    STRY(s, cudaMemcpyAsync(s->dCtl + 32, &s->hPub[slot], sizeof(uint32_t), cudaMemcpyHostToDevice, s->cstream));
    // the W / H vectors have been copied (into the staging buffer, or by the
    // pageable copies, which return once staged) and may go
    ns.ticket = t + 1u;
    ns.n = n;
    ns.m = m;
    ns.k = k;
    sl = ns;
    s->next_ticket = t + 1u;
    s->published = t + 1u;
    *ticket = t;
    return serve_ensure_running(s);
}

int nmfb_serve_poll(nmfb_serve *s, uint32_t ticket, int *done)
{
    if (!s || !done) return NMFB_EINVAL;
    uint32_t const slot = ticket % s->capacity;
    // The slot is rewritten by submit and fetch under the lock; read it under
    // the lock too, so a poll from one host thread never races them.
    std::lock_guard<std::mutex> lock(s->mu);
    if (s->slots[slot].ticket != ticket + 1u) return sfail(s, NMFB_EINVAL, "ticket %u is not pending", ticket);
    *done = (s->hDone[4 * (size_t)slot] == ticket + 1u) ? 1 : 0;
    if (*done) {
        std::atomic_thread_fence(std::memory_order_acquire);
        return NMFB_OK;
    }
    STRY(s, cudaSetDevice(s->device));
    return serve_ensure_running(s);
}

int nmfb_serve_wait(nmfb_serve *s, uint32_t ticket, double timeout_s)
{
    auto const t0 = std::chrono::steady_clock::now();
    for (;;) {
        int done = 0;
        int const rc = nmfb_serve_poll(s, ticket, &done);
        if (rc != NMFB_OK || done) return rc;
        if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() > timeout_s)
            return sfail(s, NMFB_ETIMEOUT, "request %u not finished after %.1f s", ticket, timeout_s);
        std::this_thread::sleep_for(std::chrono::microseconds(100));
    }
}

int nmfb_serve_fetch(nmfb_serve *s, uint32_t ticket, float *W, size_t ldw, float *H, size_t ldh, uint32_t *labels,
                     uint32_t *iterations, int *converged)
{
    if (!s) return NMFB_EINVAL;
    int done = 0;
    int rc = nmfb_serve_poll(s, ticket, &done);
    if (rc) return rc;
    if (!done) return sfail(s, NMFB_ESTATE, "request %u has not finished", ticket);
    uint32_t const slot = ticket % s->capacity;
    std::lock_guard<std::mutex> lock(s->mu);
    STRY(s, cudaSetDevice(s->device));
    ServeSlot &sl = s->slots[slot];
    uint32_t const ks = ks_of(sl.k);
    if ((W && ldw < sl.k) || (H && ldh < sl.k)) return sfail(s, NMFB_EINVAL, "leading dimension below k");
    if (W)
        STRY(s, cudaMemcpy2DAsync(W, ldw * sizeof(float), sl.W, ks * sizeof(float), sl.k * sizeof(float), sl.n,
                                  cudaMemcpyDeviceToHost, s->rstream));
    if (H)
        STRY(s, cudaMemcpy2DAsync(H, ldh * sizeof(float), sl.H, ks * sizeof(float), sl.k * sizeof(float), sl.m,
                                  cudaMemcpyDeviceToHost, s->rstream));
    if (labels)
        STRY(s, cudaMemcpyAsync(labels, sl.labels, (size_t)sl.m * sizeof(uint32_t), cudaMemcpyDeviceToHost, s->rstream));
    STRY(s, cudaStreamSynchronize(s->rstream));
    if (iterations) *iterations = s->hDone[4 * (size_t)slot + 1];
    if (converged) *converged = (int)s->hDone[4 * (size_t)slot + 2];
    STRY(s, cudaFreeAsync(sl.V, s->rstream));
    STRY(s, cudaFreeAsync(sl.W, s->rstream));
    STRY(s, cudaFreeAsync(sl.H, s->rstream));
    STRY(s, cudaFreeAsync(sl.labels, s->rstream));
    sl = ServeSlot{};
    return NMFB_OK;
}

}  // extern "C"
