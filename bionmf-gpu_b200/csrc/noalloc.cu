// noalloc.cu -- nmfb_update_H_noalloc: the update_H half-iteration for callers
// that must not allocate device memory.
//
// Who needs it: a host framework that owns the whole device-memory budget
// (a caching allocator that has already reserved the HBM, or a plugin host
// that hands out every device buffer itself) cannot let a library call
// cudaMalloc behind its back, and a latency-sensitive loop cannot afford the
// device-wide synchronisation that cudaFree implies.  Such a caller keeps V, W
// and H in its own device buffers and calls this one function; everything
// else the update needs lives in a fixed, file-scope device array.
//
// Scratch: g_noalloc_scratch, NMFB_NOALLOC_SCRATCH_BYTES (16 MiB) per device,
// part of the library's device image: every GPU that loads the library holds
// it until the process exits.  Layout (offsets in bytes from the 256-aligned
// base):
//   [0, 32 KiB)            colpart: nsplit x k doubles (at most 4096), per-split
//                          column sums of W
//   [32 KiB, 16 MiB)       part:    nsplit x m x k floats, per-split partial
//                          sums of Q^T W (Q = V ./ (W H^T)); behind them colpart,
//                          where it does not fit the first 32 KiB
// Every scratch word a call reads is written earlier in the same call (each
// (split, row, factor) slot by exactly one CTA), so nothing carries over from
// the previous call and nothing has to be cleared.  All calls share the one
// array: two calls whose work overlaps on the GPU (different streams, or
// different host threads) race on it and both results are undefined.
//
// Host code sees g_noalloc_scratch only as a host-side stand-in symbol; the
// device address comes from cudaGetSymbolAddress, taken on the first call made
// while a device is current and cached with that device's current context (a
// call under a different context -- after cudaDeviceReset, say -- takes it
// again).  Make the first call on a device before any stream capture.
//
// The arithmetic follows the reference's update_H (src/NMF_routines.c:704-1000
// with kernel_mul_div, src/GPU_kernels.cu:1886-2058): colsum(W) in FP64 summed in split order,
// Haux = Q^T W with Q = V ./ (W H^T), then H = (H .* Haux) ./ colsum(W),
// product first, then a correctly-rounded division.  It is an FP32 SIMT
// variant of the engine's own update_H; results agree with nmfb_update_H to
// FP32 rounding, not bit for bit.
#include "../../include/nmfb200.h"
#include "fused_common.cuh"

#include <cuda_runtime.h>
#include <stdint.h>
#include <mutex>

namespace {

constexpr size_t NA_SCRATCH_BYTES = (size_t)NMFB_NOALLOC_SCRATCH_BYTES;
constexpr uint32_t NA_KMAX = 64;
constexpr uint32_t NA_COLPARTS = 4096;
constexpr size_t NA_COLPART_BYTES = (size_t)NA_COLPARTS * sizeof(double);   // 32 KiB
constexpr size_t NA_PART_FLOATS = (NA_SCRATCH_BYTES - NA_COLPART_BYTES) / sizeof(float);
static_assert(NA_PART_FLOATS == (size_t)NMFB_NOALLOC_MAX_MK, "header limit and scratch layout disagree");

constexpr int NA_THREADS = 128;   // one column j of V (one sample) per thread
constexpr int NA_WT = 32;         // rows of W staged in shared memory per step
constexpr int NA_VG = 4;          // rows of V a thread has in flight ahead of the ones it works on
constexpr int NA_FIN = 256;       // threads of a k_na_finish CTA
constexpr int NA_MAX_DEV = 64;

__device__ __align__(256) unsigned char g_noalloc_scratch[NA_SCRATCH_BYTES];

// Two FP32 values in a register pair; fma.rn.f32x2 is two FMAs in one instruction.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pair_of(float lo, float hi)
{
    pair_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 halves(pair_t p)
{
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
    return f;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c)
{
    pair_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ pair_t add2(pair_t a, pair_t b)
{
    pair_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// CTA (x, s) covers samples j in [NT x, NT x + NT) and rows i of split s.
// part[s][j][c] = sum_{i in split s} V[i][j] / (W_i . H_j) * W[i][c];
// CTAs with x == 0 also write colpart[s][c] = sum_{i in split s} W[i][c] (FP64).
// Bound by FP32 issue: KB packed FMAs (KB = k rounded up to 4), a division and
// KB / 4 broadcast loads an element.  V's next rows and the next tile of W are
// loaded ahead (a thread that loaded each V where it was used, with k padded to
// 32, took 162 us for 20000 x 1000 at k = 20).
template <int KB>
__global__ void __launch_bounds__(NA_THREADS, KB <= 32 ? 4 : 2)
    k_na_partials(const float *__restrict__ V, size_t ldv, const float *__restrict__ W, size_t ldw,
                  const float *__restrict__ H, size_t ldh, uint32_t n, uint32_t m, uint32_t k, uint32_t rows_per_split,
                  float *__restrict__ part, double *__restrict__ colpart)
{
    static_assert(KB % 4 == 0, "rows of W as 16-byte vectors");
    constexpr bool TILE = KB <= 32;
    constexpr int K2 = KB / 2, PER = NA_WT * KB / NA_THREADS;   // floats of a W tile per thread
    constexpr int SEG = NA_THREADS / KB;                        // row lanes of the column sums
    __shared__ __align__(16) float sW[2][NA_WT][KB];
    __shared__ double sC[SEG][KB];
    uint32_t const tid = threadIdx.x;
    uint32_t const j = blockIdx.x * NA_THREADS + tid;
    uint32_t const s = blockIdx.y;
    bool const active = j < m;
    bool const colsum_cta = blockIdx.x == 0;
    uint64_t const r0_wide = (uint64_t)s * rows_per_split;
    uint32_t const r0 = r0_wide < n ? (uint32_t)r0_wide : n;
    uint32_t const r1 = (uint64_t)r0 + rows_per_split < n ? r0 + rows_per_split : n;

    pair_t h[K2], acc[K2];
#pragma unroll
    for (int c = 0; c < K2; c++) {
        h[c] = pair_of((active && 2u * c < k) ? H[(size_t)j * ldh + 2 * c] : 0.0f,
                       (active && 2u * c + 1 < k) ? H[(size_t)j * ldh + 2 * c + 1] : 0.0f);
        acc[c] = 0;
    }
    double cs = 0.0;
    uint32_t const cc = tid % KB, seg = tid / KB;
    float wreg[PER];
    auto const load_w = [&](uint32_t i0) {
#pragma unroll
        for (int e = 0; e < PER; e++) {
            uint32_t const r = (tid + e * NA_THREADS) / KB, c = (tid + e * NA_THREADS) % KB;
            wreg[e] = (i0 + r < r1 && c < k) ? W[(size_t)(i0 + r) * ldw + c] : 0.0f;
        }
    };
    auto const store_w = [&](uint32_t b) {
#pragma unroll
        for (int e = 0; e < PER; e++) (&sW[b][0][0])[tid + e * NA_THREADS] = wreg[e];
    };
    float v[NA_VG], vn[NA_VG];
    auto const load_v = [&](uint32_t i0) {
#pragma unroll
        for (int r = 0; r < NA_VG; r++) vn[r] = (active && i0 + r < r1) ? V[(size_t)(i0 + r) * ldv + j] : 0.0f;
    };
    load_w(r0);
    load_v(r0);
    uint32_t b = 0;
    for (uint32_t i0 = r0; i0 < r1; i0 += NA_WT, b ^= 1u) {
        uint32_t const rows = min((uint32_t)NA_WT, r1 - i0);
        store_w(b);
        __syncthreads();   // (a buffer is rewritten two tiles on: past this barrier of the next tile)
        if (i0 + NA_WT < r1) load_w(i0 + NA_WT);
        // up to rank 32 a tile is summed by itself first (shorter FP32 chains); above, the
        // sums fill the registers and the splits are shorter instead
        pair_t tl[TILE ? K2 : 1];
        if (TILE)
#pragma unroll
            for (int c = 0; c < K2; c++) tl[c] = 0;
        if (colsum_cta && seg < (uint32_t)SEG)
            for (uint32_t r = seg; r < rows; r += SEG) cs += (double)sW[b][r][cc];
        for (uint32_t g = 0; g < rows; g += NA_VG) {
#pragma unroll
            for (int r = 0; r < NA_VG; r++) v[r] = vn[r];
            load_v(i0 + g + NA_VG);
#pragma unroll
            for (int r = 0; r < NA_VG; r++) {
                if (g + r >= rows) break;   // (uniform)
                pair_t w[K2];
#pragma unroll
                for (int q = 0; q < KB / 4; q++) {
                    ulonglong2 const x = reinterpret_cast<const ulonglong2 *>(&sW[b][g + r][0])[q];
                    w[2 * q] = x.x;
                    w[2 * q + 1] = x.y;
                }
                pair_t sum = 0;
#pragma unroll
                for (int c = 0; c < K2; c++) sum = fma2(w[c], h[c], sum);
                float2 const wh = halves(sum);
                float const q = v[r] / (wh.x + wh.y);
                pair_t const q2 = pair_of(q, q);
#pragma unroll
                for (int c = 0; c < K2; c++) {
                    if (TILE)
                        tl[c] = fma2(q2, w[c], tl[c]);
                    else
                        acc[c] = fma2(q2, w[c], acc[c]);
                }
            }
        }
        if (TILE)
#pragma unroll
            for (int c = 0; c < K2; c++) acc[c] = add2(acc[c], tl[c]);
    }
    if (active) {
        float *dst = part + ((size_t)s * m + j) * k;
#pragma unroll
        for (int c = 0; c < K2; c++) {
            float2 const a = halves(acc[c]);
            if (2u * c < k) dst[2 * c] = a.x;
            if (2u * c + 1 < k) dst[2 * c + 1] = a.y;
        }
    }
    if (colsum_cta) {   // the row lanes in order
        if (seg < (uint32_t)SEG) sC[seg][cc] = cs;
        __syncthreads();
        if (tid < k) {
            double t = 0.0;
            for (int l = 0; l < SEG; l++) t += sC[l][tid];
            colpart[(size_t)s * k + tid] = t;
        }
    }
}

// H[j][c] = (H[j][c] * sum_s part[s][j][c]) / (float)sum_s colpart[s][c].  A CTA
// takes NA_FIN / lanes entries; group l of its threads adds an entry's splits l, l +
// lanes, ... eight loads at a time, then the groups are added in order.  Latency-
// bound: `lanes` (1, 2, 4 or 8) grows with the splits.  The column sums once per CTA,
// by eight lanes a column (splits l, l + 8, ... in order, then a shuffle tree).
__global__ void __launch_bounds__(NA_FIN) k_na_finish(float *__restrict__ H, size_t ldh, uint32_t m, uint32_t k,
                                                      uint32_t nsplit, uint32_t lanes, const float *part,
                                                      const double *colpart)
{
    nmfb_tc::chain_wait();
    __shared__ float sA[NA_KMAX];
    __shared__ float sS[NA_FIN];
    for (uint32_t c0 = 0; c0 < k; c0 += NA_FIN / 8) {
        uint32_t const c = c0 + threadIdx.x / 8;
        double a = 0.0;
        if (c < k)
            for (uint32_t q = threadIdx.x % 8; q < nsplit; q += 64) {
                double v[8];
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = q + 8 * i < nsplit ? __ldcg(colpart + (size_t)(q + 8 * i) * k + c) : 0.0;
#pragma unroll
                for (int i = 0; i < 8; i++) a += v[i];
            }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (c < k && threadIdx.x % 8 == 0) sA[c] = (float)a;
    }
    size_t const total = (size_t)m * k;
    uint32_t const per = NA_FIN / lanes, e = threadIdx.x % per, l = threadIdx.x / per;
    for (size_t i0 = (size_t)blockIdx.x * per; i0 < total; i0 += (size_t)gridDim.x * per) {
        size_t const idx = i0 + e;
        float s = 0.0f;
        if (idx < total)
            for (uint32_t q = l; q < nsplit; q += 8 * lanes) {
                float p[8];
#pragma unroll
                for (int i = 0; i < 8; i++) p[i] = q + i * lanes < nsplit ? __ldcg(part + (size_t)(q + i * lanes) * total + idx) : 0.0f;
                s += ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
            }
        __syncthreads();   // sA (first pass); the previous pass's readers of sS
        sS[threadIdx.x] = s;
        __syncthreads();
        if (l == 0 && idx < total) {
            for (uint32_t g = 1; g < lanes; g++) s += sS[g * per + e];
            uint32_t const j = (uint32_t)(idx / k), c = (uint32_t)(idx % k);
            float *hp = H + (size_t)j * ldh + c;
            *hp = __fdiv_rn(*hp * s, sA[c]);
        }
    }
}

struct DeviceSlot {
    bool ready;
    void *cu_ctx;             // CUDA context the address below belongs to
    unsigned char *scratch;   // device address of g_noalloc_scratch in that context
    int sm_count;
};

std::mutex g_slot_mutex;
DeviceSlot g_slots[NA_MAX_DEV];

// The calling thread's current CUDA context (driver cuCtxGetCurrent, found
// through the runtime's entry-point query so the library links only cudart).
void *current_cu_ctx()
{
    typedef int (*GetCurrent)(void **);
    static GetCurrent fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<GetCurrent>(p);
    }
    void *c = nullptr;
    if (!fn || fn(&c) != 0) return nullptr;
    return c;
}

// With the device current: resolve the scratch array's device address and the
// SM count, once per device and context.  The address is cached with the
// context it was taken in: after cudaDeviceReset, or under another context of
// the same device, the module is loaded anew at another address, so a changed
// context resolves it again.  Allocates nothing.
int device_slot(int dev, DeviceSlot *out)
{
    std::lock_guard<std::mutex> lock(g_slot_mutex);
    DeviceSlot &slot = g_slots[dev];
    void *const cu_ctx = current_cu_ctx();
    if (!slot.ready || slot.cu_ctx != cu_ctx) {
        slot.ready = false;
        int major = 0, sms = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            return NMFB_ECUDA;
        }
        if (major != 10) return NMFB_ENODEV;
        void *ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_noalloc_scratch) != cudaSuccess || ptr == nullptr) {
            cudaGetLastError();
            return NMFB_ECUDA;
        }
        slot.scratch = static_cast<unsigned char *>(ptr);
        slot.sm_count = sms;
        slot.cu_ctx = cu_ctx;
        slot.ready = true;
    }
    *out = slot;
    return NMFB_OK;
}

template <int KB>
cudaError_t launch_partials(dim3 grid, cudaStream_t st, const float *V, size_t ldv, const float *W, size_t ldw,
                            const float *H, size_t ldh, uint32_t n, uint32_t m, uint32_t k, uint32_t rps,
                            float *part, double *colpart)
{
    k_na_partials<KB><<<grid, NA_THREADS, 0, st>>>(V, ldv, W, ldw, H, ldh, n, m, k, rps, part, colpart);
    return cudaGetLastError();
}

}  // namespace

extern "C" int nmfb_update_H_noalloc(const float *V, size_t ldv, const float *W, size_t ldw, float *H, size_t ldh,
                                     uint32_t n, uint32_t m, uint32_t k, void *stream)
{
    if (!V || !W || !H || n == 0 || m == 0 || k == 0 || k > NA_KMAX || ldv < m || ldw < k || ldh < k)
        return NMFB_EINVAL;
    if ((uint64_t)m * k > (uint64_t)NA_PART_FLOATS) return NMFB_ETOOBIG;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return NMFB_ENODEV;
    }
    if (dev < 0 || dev >= NA_MAX_DEV) return NMFB_ENODEV;
    DeviceSlot slot;
    int const rc = device_slot(dev, &slot);
    if (rc != NMFB_OK) return rc;

    double *colpart = reinterpret_cast<double *>(slot.scratch);
    float *part = reinterpret_cast<float *>(slot.scratch + NA_COLPART_BYTES);
    cudaStream_t const st = static_cast<cudaStream_t>(stream);

    // Splits over the rows of V: four CTAs per SM in one wave (above rank 32, where two
    // fit, twice as many shorter ones), limited by the scratch (nsplit * m * k floats,
    // nsplit * k column sums) and by n.
    uint32_t const xblocks = (m + NA_THREADS - 1) / NA_THREADS;
    uint64_t want = (uint64_t)(k <= 32 ? 4 : 8) * slot.sm_count / xblocks;
    uint64_t const fit = (uint64_t)NA_PART_FLOATS / ((uint64_t)m * k);
    if (want > fit) want = fit;
    // Column sums that do not fit their own part go behind the partials: at most two CTAs
    // per SM then, and at least k rows to a split, or the partials cost more than V (of
    // 263 splits at 4209 x 415 k = 35: 68 us, of 120 41).
    uint64_t const own = NA_COLPARTS / k;
    if (want > own) {
        uint64_t more = (NA_PART_FLOATS * sizeof(float) - 8) / ((uint64_t)m * k * sizeof(float) + k * sizeof(double));
        if (more > 2u * slot.sm_count) more = 2u * slot.sm_count;
        if (more > n / k) more = n / k;
        if (want > more) want = more > own ? more : own;
    }
    if (want > n / 16) want = n / 16;   // (a split of fewer rows costs k_na_finish more than it saves here)
    // Whole waves where the last one is nearly empty (6182 x 812 k = 59: 609 CTAs 109 us, 588
    // 102), and as few as give a split 4 k rows: below that the partials' traffic and their
    // addition cost more than a wave's balance (one wave: 76 us; 585 x 1766 k = 62 71 -> 37).
    // Longer splits keep their part of a wave: 50000 x 2000 k = 40 742 us in 2.8 waves, 959 in 2.
    uint64_t const slots = (uint64_t)(k <= 32 ? 4 : 2) * slot.sm_count, ctas = want * xblocks;
    if (ctas > slots && (ctas % slots < slots / 4 || n / want < 4 * k)) {
        uint64_t waves = ctas / slots;
        while (waves > 1 && (uint64_t)n * xblocks < 4 * k * waves * slots) waves--;
        want = waves * slots / xblocks;
    }
    if (want > n) want = n;
    if (want < 1) want = 1;
    uint32_t const rps = (uint32_t)((n + want - 1) / want);
    uint32_t const nsplit = (uint32_t)((n + rps - 1) / rps);

    if ((uint64_t)nsplit * k > NA_COLPARTS)
        colpart = reinterpret_cast<double *>(part + ((size_t)nsplit * m * k + 1) / 2 * 2);

    dim3 const grid(xblocks, nsplit);
    cudaError_t e;
    switch ((k + 3) / 4) {
#define NA_CASE(Q) \
    case Q: e = launch_partials<4 * Q>(grid, st, V, ldv, W, ldw, H, ldh, n, m, k, rps, part, colpart); break;
        NA_CASE(1) NA_CASE(2) NA_CASE(3) NA_CASE(4) NA_CASE(5) NA_CASE(6) NA_CASE(7) NA_CASE(8)
        NA_CASE(9) NA_CASE(10) NA_CASE(11) NA_CASE(12) NA_CASE(13) NA_CASE(14) NA_CASE(15)
#undef NA_CASE
    default: e = launch_partials<64>(grid, st, V, ldv, W, ldw, H, ldh, n, m, k, rps, part, colpart); break;
    }
    if (e != cudaSuccess) return NMFB_ECUDA;

    uint64_t const total = (uint64_t)m * k;
    uint32_t const lanes = nsplit >= 48 ? 8u : nsplit >= 24 ? 4u : nsplit >= 12 ? 2u : 1u;
    uint64_t blocks = (total * lanes + NA_FIN - 1) / NA_FIN;
    uint64_t const cap = (uint64_t)8 * slot.sm_count;
    if (blocks > cap) blocks = cap;
    if (nmfb_tc::launch_chained(k_na_finish, dim3((unsigned)blocks), NA_FIN, 0, st, H, ldh, m, k, nsplit, lanes,
                                (const float *)part, (const double *)colpart) != cudaSuccess) {
        cudaGetLastError();
        return NMFB_ECUDA;
    }
    return NMFB_OK;
}
