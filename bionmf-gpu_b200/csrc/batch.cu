// batch.cu -- many independent KL-NMF solves in one persistent launch
// (rank-selection and restart sweeps), with exact integer consensus matrices
// and the FP64 cophenetic correlation of each rank's restarts.
// The kernels: batch_run.cuh (one problem), batch_kernel*.cu, consensus.cu.
#include "batch.cuh"

#include <float.h>
#include <math.h>
#include <stdarg.h>
#include <stdlib.h>
#include <algorithm>
#include <mutex>
#include <new>
#include <vector>

using namespace nmfb_batched;

// ---------------------------------------------------------------------------
struct nmfb_batch {
    int device;
    cudaStream_t stream;
    uint32_t n, m, nprob;
    size_t ldv;
    int sm_count;
    size_t smem_optin;
    std::vector<uint32_t> ranks;
    std::vector<uint32_t> wt, jt;        // per-problem tile shapes
    uint32_t cluster;                     // CTAs per problem (0 = automatic)
    uint32_t last_cluster;                // the value the last run used
    float *dV;
    float *dW, *dH;                       // per-problem slices (n x ks, m x ks)
    std::vector<size_t> woff, hoff;       // float offsets of each problem's slices
    uint32_t *dLabels;                    // nprob x m
    Problem *dProbs;
    uint32_t *dOrder, *dQueue;
    uint32_t **dLabelPtrs;
    uint32_t *dCounts;                    // workspaces of nmfb_batch_consensus, held under summary_lock
    double *dSummary;
    std::mutex summary_lock;
    int v_set, wh_set;
    cudaEvent_t ev0, ev1;
    float last_ms;
    char err[512];
};

static int bfail(nmfb_batch *b, int code, const char *fmt, ...)
{
    if (b) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(b->err, sizeof(b->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define BTRY(b, call)                                                                                      \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return bfail((b), NMFB_ECUDA, "%s: %s", #call, cudaGetErrorString(e_));     \
    } while (0)

// Default tile shapes: wt rows of W per update_H tile, jt columns of V per update_W tile.
static void default_tiles(uint32_t k, uint32_t m, uint32_t *wt, uint32_t *jt)
{
    (void)k;
    *wt = 32;
    *jt = m >= 64 ? 32 : 16;
}

static Problem make_problem(const nmfb_batch *b, uint32_t p)
{
    Problem P;
    memset(&P, 0, sizeof(P));
    uint32_t const k = b->ranks[p];
    P.V = b->dV;
    P.W = b->dW + b->woff[p];
    P.H = b->dH + b->hoff[p];
    P.labels = b->dLabels + (size_t)p * b->m;
    P.ldv = b->ldv;
    P.n = b->n;
    P.m = b->m;
    P.k = k;
    P.ks = ks_of(k);
    P.wt = b->wt[p];
    P.jt = b->jt[p];
    return P;
}

extern "C" {

int nmfb_batch_create(nmfb_batch **out, int device, uint32_t n, uint32_t m, uint32_t nprob, const uint32_t *ranks)
{
    if (!out) return NMFB_EINVAL;
    *out = nullptr;
    nmfb_batch *b = new (std::nothrow) nmfb_batch();
    if (!b) return NMFB_ENOMEM;
    *out = b;
    b->device = device;
    if (n < 2 || m < 2 || nprob == 0 || !ranks) return bfail(b, NMFB_EINVAL, "invalid batch dimensions");
    for (uint32_t p = 0; p < nprob; p++)
        if (ranks[p] < KMIN || ranks[p] > KMAX || ranks[p] > (n < m ? n : m))
            return bfail(b, NMFB_EINVAL, "problem %u: factorization rank %u must be in [2, min(%u, n, m)]", p, ranks[p],
                         KMAX);
    b->n = n;
    b->m = m;
    b->nprob = nprob;
    b->ldv = ((size_t)m + 31) / 32 * 32;
    b->ranks.assign(ranks, ranks + nprob);
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return bfail(b, NMFB_ENODEV, "no CUDA device %d", device);
    }
    cudaDeviceProp prop;
    BTRY(b, cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10)
        return bfail(b, NMFB_ENODEV, "device %d is sm_%d%d; this engine is built for sm_100a", device, prop.major, prop.minor);
    BTRY(b, cudaSetDevice(device));
    b->sm_count = prop.multiProcessorCount;
    b->smem_optin = prop.sharedMemPerBlockOptin;
    b->wt.resize(nprob);
    b->jt.resize(nprob);
    b->woff.resize(nprob);
    b->hoff.resize(nprob);
    size_t wtot = 0, htot = 0;
    for (uint32_t p = 0; p < nprob; p++) {
        default_tiles(ranks[p], m, &b->wt[p], &b->jt[p]);
        if (problem_smem_bytes(m, ranks[p], b->wt[p], b->jt[p]) + 64 > b->smem_optin)
            return bfail(b, NMFB_EINVAL, "m = %u with k = %u does not fit the batched engine's shared memory", m, ranks[p]);
        b->woff[p] = wtot;
        b->hoff[p] = htot;
        wtot += (size_t)n * ks_of(ranks[p]);
        htot += (size_t)m * ks_of(ranks[p]);
    }
    BTRY(b, cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    BTRY(b, cudaEventCreate(&b->ev0));
    BTRY(b, cudaEventCreate(&b->ev1));
    if (cudaMalloc(&b->dV, (size_t)n * b->ldv * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&b->dW, wtot * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&b->dH, htot * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&b->dLabels, (size_t)nprob * m * sizeof(uint32_t)) != cudaSuccess ||
        cudaMalloc(&b->dProbs, nprob * sizeof(Problem)) != cudaSuccess ||
        cudaMalloc(&b->dOrder, nprob * sizeof(uint32_t)) != cudaSuccess ||
        cudaMalloc(&b->dQueue, sizeof(uint32_t)) != cudaSuccess ||
        cudaMalloc(&b->dLabelPtrs, nprob * sizeof(uint32_t *)) != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, NMFB_ENOMEM, "device allocation for the batch failed");
    }
    BTRY(b, cudaMemsetAsync(b->dV, 0, (size_t)n * b->ldv * sizeof(float), b->stream));
    BTRY(b, cudaMemsetAsync(b->dW, 0, wtot * sizeof(float), b->stream));
    BTRY(b, cudaMemsetAsync(b->dH, 0, htot * sizeof(float), b->stream));
    std::vector<uint32_t *> lp(nprob);
    for (uint32_t p = 0; p < nprob; p++) lp[p] = b->dLabels + (size_t)p * m;
    BTRY(b, cudaMemcpyAsync(b->dLabelPtrs, lp.data(), nprob * sizeof(uint32_t *), cudaMemcpyHostToDevice, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    return NMFB_OK;
}

int nmfb_batch_destroy(nmfb_batch *b)
{
    if (!b) return NMFB_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    void *bufs[] = {b->dV, b->dW, b->dH, b->dLabels, b->dProbs, b->dOrder, b->dQueue, b->dLabelPtrs, b->dCounts, b->dSummary};
    for (void *p : bufs)
        if (p) cudaFree(p);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return NMFB_OK;
}

const char *nmfb_batch_last_error(const nmfb_batch *b) { return b ? b->err : "null batch"; }

int nmfb_batch_set_V(nmfb_batch *b, const float *V, size_t ldv)
{
    if (!b || !V || ldv < b->m) return bfail(b, NMFB_EINVAL, "nmfb_batch_set_V: bad arguments");
    BTRY(b, cudaSetDevice(b->device));
    BTRY(b, cudaMemcpy2DAsync(b->dV, b->ldv * sizeof(float), V, ldv * sizeof(float), b->m * sizeof(float), b->n,
                              cudaMemcpyDefault, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    b->v_set = 1;
    return NMFB_OK;
}

int nmfb_batch_init_random(nmfb_batch *b, const uint32_t *seeds)
{
    if (!b || !seeds) return bfail(b, NMFB_EINVAL, "nmfb_batch_init_random: bad arguments");
    BTRY(b, cudaSetDevice(b->device));
    uint32_t const n = b->n, m = b->m;
    size_t wmax = 0, hmax = 0;
    for (uint32_t p = 0; p < b->nprob; p++) {
        wmax = std::max(wmax, (size_t)n * ks_of(b->ranks[p]));
        hmax = std::max(hmax, (size_t)m * ks_of(b->ranks[p]));
    }
    float *stage = nullptr;
    BTRY(b, cudaMallocHost(&stage, 2 * (wmax + hmax) * sizeof(float)));
    cudaError_t e = cudaSuccess;
    for (uint32_t p = 0; p < b->nprob && e == cudaSuccess; p++) {
        float *W = stage + (p & 1) * (wmax + hmax);
        float *H = W + wmax;
        uint32_t const k = b->ranks[p], ks = ks_of(k);
        if (p >= 2) e = cudaStreamSynchronize(b->stream);   // the staging half of problem p-2 is free again
        if (e != cudaSuccess) break;
        // CPU_RANDOM initialisation (src/NMF_routines.c:206-233, 299-307):
        // srandom(seed); W (n x k) then H (m x k), random()/RAND_MAX + FLT_MIN.
        // (the generator through a private state: initstate_r / random_r
        // reproduce srandom / random's sequence without the process-wide one)
        char rstate[128];
        struct random_data rd;
        memset(&rd, 0, sizeof(rd));
        initstate_r(seeds[p], rstate, sizeof(rstate), &rd);
        auto next = [&]() -> float {
            int32_t r;
            random_r(&rd, &r);
            return ((float)r) / ((float)RAND_MAX) + FLT_MIN;
        };
        for (uint32_t i = 0; i < n; i++)
            for (uint32_t c = 0; c < ks; c++) W[(size_t)i * ks + c] = (c < k) ? next() : 0.0f;
        for (uint32_t j = 0; j < m; j++)
            for (uint32_t c = 0; c < ks; c++) H[(size_t)j * ks + c] = (c < k) ? next() : 0.0f;
        e = cudaMemcpyAsync(b->dW + b->woff[p], W, (size_t)n * ks * sizeof(float), cudaMemcpyHostToDevice, b->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(b->dH + b->hoff[p], H, (size_t)m * ks * sizeof(float), cudaMemcpyHostToDevice, b->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    cudaFreeHost(stage);
    if (e != cudaSuccess) return bfail(b, NMFB_ECUDA, "init_random: %s", cudaGetErrorString(e));
    b->wh_set = 1;
    return NMFB_OK;
}

int nmfb_batch_set_WH(nmfb_batch *b, uint32_t p, const float *W, size_t ldw, const float *H, size_t ldh)
{
    if (!b || p >= b->nprob || !W || !H) return bfail(b, NMFB_EINVAL, "nmfb_batch_set_WH: bad arguments");
    uint32_t const k = b->ranks[p], ks = ks_of(k);
    if (ldw < k || ldh < k) return bfail(b, NMFB_EINVAL, "nmfb_batch_set_WH: leading dimension below k");
    BTRY(b, cudaSetDevice(b->device));
    BTRY(b, cudaMemcpy2DAsync(b->dW + b->woff[p], ks * sizeof(float), W, ldw * sizeof(float), k * sizeof(float), b->n,
                              cudaMemcpyHostToDevice, b->stream));
    BTRY(b, cudaMemcpy2DAsync(b->dH + b->hoff[p], ks * sizeof(float), H, ldh * sizeof(float), k * sizeof(float), b->m,
                              cudaMemcpyHostToDevice, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    b->wh_set = 1;
    return NMFB_OK;
}

int nmfb_batch_set_tiles(nmfb_batch *b, uint32_t p, uint32_t wt, uint32_t jt)
{
    if (!b || p >= b->nprob) return bfail(b, NMFB_EINVAL, "nmfb_batch_set_tiles: bad problem");
    if (wt < 8 || wt > 512 || (wt & 7) || jt < 4 || jt > 64 || (jt & (jt - 1)))
        return bfail(b, NMFB_EINVAL, "tile shape out of range (wt in [8, 512], multiple of 8; jt a power of two in [4, 64])");
    if (problem_smem_bytes(b->m, b->ranks[p], wt, jt) + 64 > b->smem_optin)
        return bfail(b, NMFB_EINVAL, "tile shape does not fit shared memory");
    b->wt[p] = wt;
    b->jt[p] = jt;
    return NMFB_OK;
}

int nmfb_batch_set_cluster(nmfb_batch *b, uint32_t ctas)
{
    if (!b) return NMFB_EINVAL;
    if (ctas != 0 && ctas != 1 && ctas != 2 && ctas != 4 && ctas != 8)
        return bfail(b, NMFB_EINVAL, "CTAs per problem must be 0 (automatic), 1, 2, 4 or 8");
    b->cluster = ctas;
    return NMFB_OK;
}

int nmfb_batch_get_cluster(const nmfb_batch *b, uint32_t *ctas)
{
    if (!b || !ctas) return NMFB_EINVAL;
    *ctas = b->last_cluster;
    return NMFB_OK;
}

int nmfb_batch_run(nmfb_batch *b, uint32_t n_iters, uint32_t niter_test_conv, uint32_t stop_threshold,
                   uint32_t *iterations, int *converged)
{
    if (!b) return NMFB_EINVAL;
    if (n_iters == 0 || niter_test_conv == 0 || stop_threshold == 0)
        return bfail(b, NMFB_EINVAL, "nIters, niter_test_conv and stop_threshold must be positive");
    if (!b->v_set || !b->wh_set) return bfail(b, NMFB_ESTATE, "set V and the initial factors first");
    BTRY(b, cudaSetDevice(b->device));
    std::vector<Problem> P(b->nprob);
    std::vector<uint32_t> order(b->nprob);
    size_t smem = 0;
    for (uint32_t p = 0; p < b->nprob; p++) {
        P[p] = make_problem(b, p);
        P[p].n_iters = n_iters;
        P[p].niter_test_conv = niter_test_conv;
        P[p].stop_threshold = stop_threshold;
        order[p] = p;
        smem = std::max(smem, problem_smem_bytes(b->m, b->ranks[p], b->wt[p], b->jt[p]));
    }
    // largest rank first (all problems of a sweep share n and m), stable on the index
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return b->ranks[x] > b->ranks[y]; });
    BTRY(b, cudaMemcpyAsync(b->dProbs, P.data(), b->nprob * sizeof(Problem), cudaMemcpyHostToDevice, b->stream));
    BTRY(b, cudaMemcpyAsync(b->dOrder, order.data(), b->nprob * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream));
    BTRY(b, cudaMemsetAsync(b->dQueue, 0, sizeof(uint32_t), b->stream));
    uint32_t kmax = 0;
    for (uint32_t p = 0; p < b->nprob; p++) kmax = std::max(kmax, b->ranks[p]);
    BatchKernel const kern = kmax <= 10 ? batch_kernel10() : batch_kernel20();
    BTRY(b, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    BTRY(b, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem));
    if (per_sm < 1) return bfail(b, NMFB_EINVAL, "batched kernel does not fit on an SM with %zu B shared memory", smem);
    // CTAs per problem: automatic = 8 when the batch leaves most CTA slots idle
    // at one problem per 8 CTAs, else 4 (a problem's time shrinks about C-fold,
    // so the few problems that run to the iteration cap no longer set the
    // launch time).
    uint32_t const slots = (uint32_t)per_sm * (uint32_t)b->sm_count;
    uint32_t C = b->cluster ? b->cluster : ((uint64_t)b->nprob * 8 <= slots ? 8u : 4u);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * (uint32_t)b->sm_count, 1, 1);
    cfg.blockDim = dim3(NT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = b->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    BTRY(b, cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg));
    if (nclusters < 1) return bfail(b, NMFB_EINVAL, "no cluster of %u batched CTAs fits on the device", C);
    uint32_t ncl = (uint32_t)nclusters < b->nprob ? (uint32_t)nclusters : b->nprob;
    cfg.gridDim = dim3(ncl * C, 1, 1);
    b->last_cluster = C;
    BTRY(b, cudaEventRecord(b->ev0, b->stream));
    BTRY(b, cudaLaunchKernelEx(&cfg, kern, b->dProbs, (const uint32_t *)b->dOrder, b->nprob, b->dQueue));
    BTRY(b, cudaEventRecord(b->ev1, b->stream));
    BTRY(b, cudaMemcpyAsync(P.data(), b->dProbs, b->nprob * sizeof(Problem), cudaMemcpyDeviceToHost, b->stream));
    BTRY(b, cudaStreamSynchronize(b->stream));
    BTRY(b, cudaEventElapsedTime(&b->last_ms, b->ev0, b->ev1));
    for (uint32_t p = 0; p < b->nprob; p++) {
        if (iterations) iterations[p] = P[p].iterations;
        if (converged) converged[p] = (int)P[p].converged;
    }
    return NMFB_OK;
}

int nmfb_batch_last_ms(const nmfb_batch *b, double *ms)
{
    if (!b || !ms) return NMFB_EINVAL;
    *ms = b->last_ms;
    return NMFB_OK;
}

int nmfb_batch_get_classification(nmfb_batch *b, uint32_t *labels)
{
    if (!b || !labels) return bfail(b, NMFB_EINVAL, "null labels");
    BTRY(b, cudaSetDevice(b->device));
    BTRY(b, cudaMemcpy(labels, b->dLabels, (size_t)b->nprob * b->m * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    return NMFB_OK;
}

int nmfb_batch_get_WH(nmfb_batch *b, uint32_t p, float *W, size_t ldw, float *H, size_t ldh)
{
    if (!b || p >= b->nprob) return bfail(b, NMFB_EINVAL, "bad problem index");
    uint32_t const k = b->ranks[p], ks = ks_of(k);
    if ((W && ldw < k) || (H && ldh < k)) return bfail(b, NMFB_EINVAL, "leading dimension below k");
    BTRY(b, cudaSetDevice(b->device));
    // Through page-locked staging buffers of at most 8 MB, one DMA each, the next while
    // this one's rows are copied out (a pitched copy into pageable memory moves one short
    // row at a time).
    auto const fetch = [&](float *dst, size_t ld, const float *src, uint32_t rows) -> cudaError_t {
        size_t const step = ks, row = step * sizeof(float), len = k * sizeof(float);
        uint32_t const most = (uint32_t)((8u << 20) / row), chunk = rows < most ? rows : most;
        float *stage[2] = {(float *)nmfb_stage_get(chunk * row), rows > chunk ? (float *)nmfb_stage_get(chunk * row) : nullptr};
        cudaError_t e = cudaSuccess;
        if (!stage[0] || (rows > chunk && !stage[1])) {
            e = cudaMemcpy2D(dst, ld * sizeof(float), src, row, k * sizeof(float), rows, cudaMemcpyDeviceToHost);
        } else {
            auto const copy = [&](uint32_t r0, float *to) {
                return cudaMemcpyAsync(to, src + (size_t)r0 * ks, std::min(chunk, rows - r0) * row, cudaMemcpyDeviceToHost, b->stream);
            };
            e = copy(0, stage[0]);
            for (uint32_t r0 = 0, c = 0; r0 < rows; r0 += chunk, c ^= 1) {
                cudaError_t const es = cudaStreamSynchronize(b->stream);   // this chunk is there, and no copy in flight
                if (e == cudaSuccess) e = es;
                if (e != cudaSuccess) break;
                uint32_t const nr = std::min(chunk, rows - r0);
                if (rows - r0 > nr) e = copy(r0 + nr, stage[c ^ 1]);
                float *to = dst + (size_t)r0 * ld;
                const float *from = stage[c];
                for (uint32_t r = 0; r < nr; r++, to += ld, from += step) memcpy(to, from, len);
            }
        }
        nmfb_stage_put(stage[0]);
        nmfb_stage_put(stage[1]);
        return e;
    };
    if (W) BTRY(b, fetch(W, ldw, b->dW + b->woff[p], b->n));
    if (H) BTRY(b, fetch(H, ldh, b->dH + b->hoff[p], b->m));
    return NMFB_OK;
}

int nmfb_batch_consensus(nmfb_batch *b, uint32_t k, uint32_t *counts, uint32_t *nruns, double *cophenetic)
{
    if (!b) return NMFB_EINVAL;
    std::vector<uint32_t> sel;
    for (uint32_t p = 0; p < b->nprob; p++)
        if (b->ranks[p] == k) sel.push_back(p);
    if (nruns) *nruns = (uint32_t)sel.size();
    if (sel.empty()) return bfail(b, NMFB_EINVAL, "no problem of rank %u in the batch", k);
    BTRY(b, cudaSetDevice(b->device));
    uint32_t const m = b->m;
    size_t const mm = (size_t)m * m;
    // Workspaces, allocated on the first call that needs them and kept: the counts with
    // the selection, and the linkage's.  One call at a time has them, until its results
    // are on the host.
    std::lock_guard<std::mutex> const held(b->summary_lock);
    cudaError_t e = cudaSuccess;
    if (!b->dCounts) e = cudaMalloc(&b->dCounts, (mm + b->nprob) * sizeof(uint32_t));
    if (e == cudaSuccess && cophenetic && !b->dSummary)
        e = cudaMalloc(&b->dSummary, nmfb_summary_doubles(m) * sizeof(double) + nmfb_summary_ints(m) * sizeof(uint32_t));
    if (e != cudaSuccess) {
        cudaGetLastError();
        return bfail(b, NMFB_ECUDA, "consensus: %s", cudaGetErrorString(e));
    }
    uint32_t *const dC = b->dCounts, *const dSel = dC + mm;
    double *dOut = nullptr;
    e = cudaMemcpyAsync(dSel, sel.data(), sel.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) e = nmfb_launch_consensus(b->dLabelPtrs, dSel, (uint32_t)sel.size(), m, dC, b->stream);
    if (e == cudaSuccess && cophenetic)
        e = nmfb_launch_cophenetic(dC, m, (uint32_t)sel.size(), b->dSummary,
                                   reinterpret_cast<uint32_t *>(b->dSummary + nmfb_summary_doubles(m)), &dOut, b->stream);
    if (e == cudaSuccess && counts) e = cudaMemcpyAsync(counts, dC, mm * sizeof(uint32_t), cudaMemcpyDeviceToHost, b->stream);
    if (e == cudaSuccess && cophenetic)
        e = cudaMemcpyAsync(cophenetic, dOut, sizeof(double), cudaMemcpyDeviceToHost, b->stream);
    cudaError_t const es = cudaStreamSynchronize(b->stream);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) return bfail(b, NMFB_ECUDA, "consensus: %s", cudaGetErrorString(e));
    return NMFB_OK;
}

}  // extern "C"

