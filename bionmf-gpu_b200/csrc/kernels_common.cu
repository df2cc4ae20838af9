// kernels_common.cu -- small kernels shared by every update arm:
//   * deterministic column sums of W / H            (reference: matrix_to_row)
//   * mul-div update with fused EPS adjust       (reference: matrix_mul_div + matrix_adjust)
//   * classification (argmax) + device-side connectivity test and stop rule
//                                                   (reference: get_classification + get_difference)
//   * FP64 objective reductions (||V||^2, ||V-WH||^2, KL divergence)
//
// All reductions use fixed-order trees so results do not depend on timing.
#include "nmfb_internal.cuh"

#include <float.h>
#include <stdarg.h>

using nmfb::ConvState;

int nmfb_fail(nmfb_ctx *ctx, int code, const char *fmt, ...)
{
    if (ctx) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(ctx->err, sizeof(ctx->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

namespace {

__device__ __forceinline__ bool halted(const ConvState *st) { return st && *(volatile const uint32_t *)&st->converged; }

// EPS adjust of the reference (src/GPU_kernels.cu:2338-2345): fmaxf(x, FLT_MIN),
// which also maps NaN to FLT_MIN.
__device__ __forceinline__ float adjust_value(float v) { return fmaxf(v, FLT_MIN); }

// ---------------------------------------------------------------------------
// Column sums: block b reduces rows [r0, r1) of X (rows x kp) into part[b][*];
// the last block to retire sums the block partials (FP64) in a fixed order:
// thread group g (of blockDim / kp) sums blocks g, g + groups, ... in order,
// then the groups are added in order.  Latency-bound: blocks of 1024 threads,
// so that few blocks (and with them a short last sum) cover the rows, and four
// rows in flight per thread (256-thread blocks of 32 rows: 20 us at 8000 x 128).
constexpr int CS_NT = 1024;
__global__ void __launch_bounds__(CS_NT) k_colsum(const float *__restrict__ X, uint32_t rows, uint32_t kp,
                                                  double *__restrict__ part, float *__restrict__ acc,
                                                  uint32_t *__restrict__ ticket, const ConvState *st)
{
    if (halted(st)) return;
    __shared__ double red[CS_NT];
    __shared__ bool is_last;
    uint32_t const lanes = CS_NT / kp;  // row lanes per block
    uint32_t const c = threadIdx.x % kp;
    uint32_t const rl = threadIdx.x / kp;
    uint32_t const per = (rows + gridDim.x - 1) / gridDim.x;
    uint32_t const r0 = min(rows, blockIdx.x * per);
    uint32_t const r1 = min(rows, r0 + per);
    double s = 0.0;
    if (rl < lanes) {
        for (uint32_t r = r0 + rl; r < r1; r += 4 * lanes) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = r + i * lanes < r1 ? X[(size_t)(r + i * lanes) * kp + c] : 0.0f;
#pragma unroll
            for (int i = 0; i < 4; i++) s += (double)v[i];
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < kp) {
        double t = 0.0;
        for (uint32_t l = 0; l < lanes; l++)
            t += red[l * kp + threadIdx.x];
        part[(size_t)blockIdx.x * kp + threadIdx.x] = t;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double t = 0.0;
    if (rl < lanes)
        for (uint32_t b = rl; b < gridDim.x; b += 8 * lanes) {
            double v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = b + i * lanes < gridDim.x ? __ldcg(&part[(size_t)(b + i * lanes) * kp + c]) : 0.0;
#pragma unroll
            for (int i = 0; i < 8; i++) t += v[i];
        }
    red[threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.x < kp) {
        double u = 0.0;
        for (uint32_t g = 0; g < lanes; g++) u += red[g * kp + threadIdx.x];
        acc[threadIdx.x] = (float)u;
    }
    if (threadIdx.x == 0) *ticket = 0u;
}

// ---------------------------------------------------------------------------
// Factor update, one thread per entry of X (rows x kp):
//   mode FU_MULDIV: v = (X[r][c] * sum_s part[s][r][c]) / acc[c]  (matrix_mul_div,
//                   src/GPU_kernels.cu:2013-2019: product first, then the division),
//                   followed by the EPS adjust when `adjust` is set;
//   mode FU_ADJUST: v = fmaxf(X[r][c], FLT_MIN)                   (matrix_adjust).
// Padding columns c >= k are kept at 0.  The split partials are summed in a
// fixed order (eight at a time), so the result does not depend on scheduling.
enum { FU_MULDIV = 1, FU_ADJUST = 2 };

__global__ void __launch_bounds__(256) k_factor(int mode, float *__restrict__ X, uint32_t rows, uint32_t kp, uint32_t k,
                                                const float *__restrict__ part, uint32_t nsplit, size_t split_stride,
                                                const float *__restrict__ acc, int adjust, const ConvState *st)
{
    if (halted(st)) return;
    size_t const total = (size_t)rows * kp;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        uint32_t const c = (uint32_t)(idx % kp);
        float v = 0.0f;
        if (c < k) {
            if (mode == FU_MULDIV) {
                float s = 0.0f;
                for (uint32_t q = 0; q < nsplit; q += 8) s += nmfb_add8(part + idx, split_stride, q, nsplit);
                v = __fdiv_rn(X[idx] * s, acc[c]);
                if (adjust) v = adjust_value(v);
            } else {
                v = adjust_value(X[idx]);
            }
        }
        X[idx] = v;
    }
}

// ---------------------------------------------------------------------------
// Classification with the reference's lane-exact tie rule (kernel_idx_max,
// src/GPU_kernels.cu:2508-2656, 2880-3110, 3177-3267):
//   group width bdx = 32 for k <= 96, else next_pow2(ceil(ceil32(k)/3));
//   thread t scans columns t, t+bdx, t+2*bdx (< k), keeping the first strict max;
//   idle threads hold (-1, 0); shared-memory tree for half = bdx/2 .. 32 and a
//   xor butterfly for half = 16 .. 1, each lane keeping its own value on ties;
//   lane 0 holds the result.
// Optionally applies the test's EPS adjust to H first (adjust(H) happens right
// before get_classification in the reference, src/NMF_GPU.c:611-655).
// Also records first[label] = min sample index per label (canonical partition).
__global__ void k_classify(float *__restrict__ H, uint32_t m, uint32_t kp, uint32_t k, uint32_t bdx,
                           int adjust, uint32_t *__restrict__ labels, uint32_t *__restrict__ first,
                           const ConvState *st)
{
    if (halted(st)) return;
    extern __shared__ unsigned char smem_raw[];
    float *sval = reinterpret_cast<float *>(smem_raw);
    uint32_t *sidx = reinterpret_cast<uint32_t *>(sval + blockDim.x);
    uint32_t const groups = blockDim.x / bdx;
    uint32_t const g = threadIdx.x / bdx;
    uint32_t const t = threadIdx.x % bdx;
    uint32_t const j = blockIdx.x * groups + g;
    bool const valid = j < m;
    float *row = H + (size_t)(valid ? j : 0) * kp;

    if (adjust && valid) {
        for (uint32_t c = t; c < kp; c += bdx) {
            if (c >= k) continue;
            row[c] = adjust_value(row[c]);
        }
        __syncwarp();
    }
    float v = -1.0f;
    uint32_t id = 0;
    if (valid && t < k) {
        v = row[t];
        id = t;
        for (uint32_t it = 1; it < 3; it++) {
            uint32_t const c = t + it * bdx;
            if (c < k) {
                float const x = row[c];
                if (x > v) { v = x; id = c; }
            }
        }
    }
    if (bdx > 32) {
        sval[threadIdx.x] = v;
        sidx[threadIdx.x] = id;
        for (uint32_t half = bdx / 2; half >= 32; half >>= 1) {
            __syncthreads();
            if (t < half) {
                float const ov = sval[threadIdx.x + half];
                uint32_t const oi = sidx[threadIdx.x + half];
                if (v < ov) { v = ov; id = oi; }
            }
            __syncthreads();
            if (t < half) { sval[threadIdx.x] = v; sidx[threadIdx.x] = id; }
        }
        __syncthreads();
    }
    if (t < 32) {
        unsigned const mask = 0xffffffffu;
        for (uint32_t half = 16; half > 0; half >>= 1) {
            float const ov = __shfl_xor_sync(mask, v, half);
            uint32_t const oi = __shfl_xor_sync(mask, id, half);
            if (v < ov) { v = ov; id = oi; }
        }
        if (t == 0 && valid) {
            labels[j] = id;
            atomicMin(&first[id], j);
        }
    }
}

// Connectivity comparison and stop rule.  Two classification vectors define
// the same partition (get_difference == 0, src/common.c:1195-1209) iff every
// sample maps to the same first-occurrence representative in both.  The last
// block applies the reference's counter rule (src/NMF_GPU.c:695-709).
__global__ void k_conv_compare(const uint32_t *__restrict__ labels, uint32_t *__restrict__ first,
                               uint32_t *__restrict__ lastrep, uint32_t m, uint32_t nfirst, ConvState *st)
{
    if (halted(st)) return;
    __shared__ bool is_last;
    uint32_t local_diff = 0;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        uint32_t const rep = first[labels[j]];
        if (rep != lastrep[j]) local_diff = 1;
        lastrep[j] = rep;
    }
    if (__syncthreads_or(local_diff) && threadIdx.x == 0)
        atomicOr(&st->diff, 1u);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        is_last = (atomicAdd(&st->ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (uint32_t c = threadIdx.x; c < nfirst; c += blockDim.x)
        first[c] = 0xffffffffu;
    if (threadIdx.x == 0) {
        uint32_t const diff = atomicAdd(&st->diff, 0u);
        st->tests_done += 1;
        if (diff)
            st->inc = 0;
        else if (st->inc < st->stop_threshold)
            st->inc += 1;
        else {
            st->converged = 1;
            st->conv_tests = st->tests_done;
        }
        st->diff = 0;
        st->ticket = 0;
    }
}

// ---------------------------------------------------------------------------
// FP64 objectives over V (n x m, ld ldv) and W (n x kp), H (m x kp):
// out[0] = ||V||^2, out[1] = ||V - WH||^2, out[2] = KL(V || WH).
//
// Bound by the FP64 pipe (64 FMA per cycle and SM): k multiply-adds an element
// for WH and, for the divergence, a division and a logarithm (about 45 more).
// A CTA takes tiles of V in turn (CX threads across, 256 / CX down); up to 32
// columns at a time of the tile's rows of W and H are converted to FP64 once, in shared
// memory, and each thread forms 4 x 4 elements of WH from them, so an element costs half
// a shared load per multiply-add and no conversion.  (One thread per element
// with both rows read and converted from global memory was bound by the
// conversions and by the division of the element index: 1344 us for
// 12007 x 1501 at k = 20.)  WHAT selects the
// sums: OBJ_DOTS leaves out the division and the logarithm.  Thread, CTA and
// grid sums have fixed orders.
enum { OBJ_DOTS = 1, OBJ_KL = 2 };
// Threads across a tile: 64 columns, or the 4 to 32 that a narrower V has.  Up to 16
// columns the few threads that share a row of W read it themselves (H stays in shared
// memory, k <= m <= 16).  With 64-column tiles 1000000 x 2 k = 2 took 269 us (divergence)
// and 126 (dots), 200000 x 5 k = 3 109 and 49; now 59 and 50, 48 and 35 (a call).
__host__ __device__ constexpr int obj_cx(uint32_t m) { return m <= 4 ? 1 : m <= 8 ? 2 : m <= 16 ? 4 : m <= 32 ? 8 : 16; }
constexpr int obj_cols(int cx) { return 4 * cx; }
constexpr int obj_rows(int cx) { return 4 * (256 / cx); }
constexpr int OBJ_KC = 32;   // rank columns per shared-memory chunk

template <int WHAT, int CX>
__global__ void __launch_bounds__(256) k_objective(const float *__restrict__ V, size_t ldv, const float *__restrict__ W,
                                                   const float *__restrict__ H, uint32_t n, uint32_t m, uint32_t kp,
                                                   uint32_t k, double *__restrict__ part, double *__restrict__ out,
                                                   uint32_t *__restrict__ ticket)
{
    constexpr int TR = obj_rows(CX), TC = obj_cols(CX);
    constexpr bool NARROW = CX <= 4;
    __shared__ __align__(16) double sW[NARROW ? 1 : OBJ_KC][NARROW ? 2 : TR + 2];   // [column][row]; 16-byte rows for the paired loads
    __shared__ __align__(16) double sH[NARROW ? TC : OBJ_KC][TC + 2];
    __shared__ double red[3][8];
    __shared__ bool is_last;
    uint32_t const tid = threadIdx.x, tx = tid % CX, ty = tid / CX;
    uint32_t const tcols = (m + TC - 1) / TC, trows = (n + TR - 1) / TR;
    uint64_t const tiles = (uint64_t)tcols * trows;
    double sv = 0.0, sd = 0.0, kl = 0.0;
    if (NARROW) {
        for (uint32_t e = tid; e < TC * TC; e += 256) {
            uint32_t const r = e / TC, c = e % TC;
            sH[c][r] = r < m && c < k ? (double)H[(size_t)r * kp + c] : 0.0;
        }
        __syncthreads();
    }
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint32_t const i0 = (uint32_t)(t / tcols) * TR, j0 = (uint32_t)(t % tcols) * TC;
        // this thread's 4 x 4 elements of V; the leading dimension is a multiple of 32, so a
        // float4 starting below m lies in its row
        float4 v[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            uint32_t const i = i0 + ty * 4 + p, j = j0 + tx * 4;
            v[p] = (i < n && j < m) ? __ldcs(reinterpret_cast<const float4 *>(V + (size_t)i * ldv + j))
                                    : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        double wh[4][4] = {};
        if constexpr (NARROW) {   // (W's padding columns are 0)
            for (uint32_t c0 = 0; c0 < k; c0 += 4) {
                float4 w[4];
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    uint32_t const i = min(i0 + ty * 4 + p, n - 1);
                    w[p] = *reinterpret_cast<const float4 *>(W + (size_t)i * kp + c0);
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    double h[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) h[q] = sH[c0 + c][tx * 4 + q];
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        double const x = c == 0 ? w[p].x : c == 1 ? w[p].y : c == 2 ? w[p].z : w[p].w;
#pragma unroll
                        for (int q = 0; q < 4; q++) wh[p][q] += x * h[q];
                    }
                }
            }
        }
        for (uint32_t c0 = 0; !NARROW && c0 < k; c0 += OBJ_KC) {
            uint32_t const kc = min((uint32_t)OBJ_KC, k - c0);
            __syncthreads();   // the previous chunk's readers are done
            for (uint32_t e = tid; e < TR * kc; e += 256) {
                uint32_t const r = e / kc, c = e % kc;
                sW[c][r] = i0 + r < n ? (double)W[(size_t)(i0 + r) * kp + c0 + c] : 0.0;
                if (TC >= TR || r < TC) sH[c][r] = j0 + r < m ? (double)H[(size_t)(j0 + r) * kp + c0 + c] : 0.0;
            }
            __syncthreads();
#pragma unroll 4
            for (uint32_t c = 0; c < kc; c++) {
                double2 const wa = *reinterpret_cast<const double2 *>(&sW[c][ty * 4]);
                double2 const wb = *reinterpret_cast<const double2 *>(&sW[c][ty * 4 + 2]);
                double2 const ha = *reinterpret_cast<const double2 *>(&sH[c][tx * 4]);
                double2 const hb = *reinterpret_cast<const double2 *>(&sH[c][tx * 4 + 2]);
                double const w[4] = {wa.x, wa.y, wb.x, wb.y}, h[4] = {ha.x, ha.y, hb.x, hb.y};
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int q = 0; q < 4; q++) wh[p][q] += w[p] * h[q];
            }
        }
#pragma unroll
        for (int p = 0; p < 4; p++) {
            if (i0 + ty * 4 + p >= n) continue;
            float const vs[4] = {v[p].x, v[p].y, v[p].z, v[p].w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (j0 + tx * 4 + q >= m) continue;
                double const x = (double)vs[q], y = wh[p][q];
                if (WHAT & OBJ_DOTS) {
                    sv += x * x;
                    sd += (x - y) * (x - y);
                }
                if (WHAT & OBJ_KL) kl += (x > 0.0 ? x * log(x / y) : 0.0) - x + y;
            }
        }
    }
    double s[3] = {sv, sd, kl};
#pragma unroll
    for (int q = 0; q < 3; q++) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], off);
        if (tid % 32 == 0) red[q][tid / 32] = s[q];
    }
    __syncthreads();
    if (tid < 3) {
        double u = 0.0;
        for (int w = 0; w < 8; w++) u += red[tid][w];
        part[(size_t)blockIdx.x * 3 + tid] = u;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    // the CTAs' sums: warp q adds sum q, lane l the CTAs l, l + 32, ... in order, then a shuffle tree
    if (tid < 96) {
        double u = 0.0;
        for (uint32_t b = tid % 32; b < gridDim.x; b += 32) u += __ldcg(&part[(size_t)b * 3 + tid / 32]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) u += __shfl_xor_sync(0xffffffffu, u, off);
        if (tid % 32 == 0) out[tid / 32] = u;
    }
    if (tid == 0) *ticket = 0u;
}

inline unsigned grid_for(size_t items, unsigned block, unsigned cap)
{
    size_t g = (items + block - 1) / block;
    if (g > cap) g = cap;
    if (g == 0) g = 1;
    return (unsigned)g;
}

}  // namespace

// ---------------------------------------------------------------------------
int nmfb_colsum(nmfb_ctx *ctx, const float *X, uint32_t rows, float *acc, int which)
{
    // four rows per thread where that leaves at most a block per SM (1024 partials fit)
    unsigned const rows_per = 4 * (CS_NT / ctx->kp);
    unsigned grid = (rows + rows_per - 1) / rows_per;
    if (grid > (unsigned)ctx->sm_count) grid = (unsigned)ctx->sm_count;
    if (grid > 1024u) grid = 1024u;
    k_colsum<<<grid, CS_NT, 0, ctx->stream>>>(X, rows, ctx->kp, ctx->dColPart + (size_t)which * 1024 * ctx->kp, acc,
                                             ctx->dTickets + which, ctx->dState);
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

static int launch_factor(nmfb_ctx *ctx, int mode, float *X, uint32_t rows, const float *part, uint32_t nsplit,
                         size_t split_stride, const float *acc, int adjust, const ConvState *st)
{
    size_t const total = (size_t)rows * ctx->kp;
    unsigned const grid = grid_for(total, 256, 8u * (unsigned)ctx->sm_count);
    k_factor<<<grid, 256, 0, ctx->stream>>>(mode, X, rows, ctx->kp, ctx->k, part, nsplit, split_stride, acc, adjust, st);
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

int nmfb_muldiv(nmfb_ctx *ctx, float *X, uint32_t rows, const float *part, uint32_t nsplit, size_t split_stride,
                const float *acc, int adjust)
{
    return launch_factor(ctx, FU_MULDIV, X, rows, part, nsplit, split_stride, acc, adjust, ctx->dState);
}

int nmfb_adjust_rows(nmfb_ctx *ctx, float *X, uint32_t rows)
{
    return launch_factor(ctx, FU_ADJUST, X, rows, nullptr, 0, 0, nullptr, 0, nullptr);
}

static uint32_t classify_width(uint32_t k)
{
    uint32_t const kp32 = ((k + 31u) / 32u) * 32u;
    if (kp32 <= 96u) return 32u;
    uint32_t b = (kp32 + 2u) / 3u, p = 1;
    while (p < b) p <<= 1;
    return p > 1024u ? 1024u : p;
}

static int launch_classify(nmfb_ctx *ctx, int adjust, const ConvState *st)
{
    uint32_t const bdx = classify_width(ctx->k);
    uint32_t const block = bdx >= 256 ? bdx : 256;
    uint32_t const groups = block / bdx;
    uint32_t const grid = (ctx->m + groups - 1) / groups;
    size_t const smem = (size_t)block * (sizeof(float) + sizeof(uint32_t));
    k_classify<<<grid, block, smem, ctx->stream>>>(ctx->dH, ctx->m, ctx->kp, ctx->k, bdx, adjust, ctx->dLabels,
                                                  ctx->dFirst, st);
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

int nmfb_classify_and_test(nmfb_ctx *ctx, uint32_t niter_test_conv)
{
    (void)niter_test_conv;
    int rc = launch_classify(ctx, 1, ctx->dState);
    if (rc) return rc;
    unsigned const grid = grid_for(ctx->m, 256, 2u * (unsigned)ctx->sm_count);
    k_conv_compare<<<grid, 256, 0, ctx->stream>>>(ctx->dLabels, ctx->dFirst, ctx->dLastRep, ctx->m, ctx->kp,
                                                 ctx->dState);
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

int nmfb_classify_only(nmfb_ctx *ctx)
{
    int rc = launch_classify(ctx, 0, nullptr);
    if (rc) return rc;
    // first[] was consumed only as scratch here; restore it for the next test.
    NMFB_CUDA_TRY(ctx, cudaMemsetAsync(ctx->dFirst, 0xff, ctx->kp * sizeof(uint32_t), ctx->stream));
    return NMFB_OK;
}

int nmfb_reset_conv(nmfb_ctx *ctx, uint32_t stop_threshold)
{
    ConvState s;
    memset(&s, 0, sizeof(s));
    s.stop_threshold = stop_threshold;
    *ctx->hState = s;
    NMFB_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->dState, ctx->hState, sizeof(ConvState), cudaMemcpyHostToDevice,
                                       ctx->stream));
    NMFB_CUDA_TRY(ctx, cudaMemsetAsync(ctx->dLastRep, 0, ctx->m * sizeof(uint32_t), ctx->stream));
    NMFB_CUDA_TRY(ctx, cudaMemsetAsync(ctx->dFirst, 0xff, ctx->kp * sizeof(uint32_t), ctx->stream));
    // The host mirror is overwritten by the copy above only after it executes;
    // wait so that a later read of hState cannot see a stale value.
    NMFB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return NMFB_OK;
}

template <int CX>
static auto objective_kernel(int what)
{
    return what == OBJ_DOTS ? k_objective<OBJ_DOTS, CX> : what == OBJ_KL ? k_objective<OBJ_KL, CX>
                                                                         : k_objective<OBJ_DOTS | OBJ_KL, CX>;
}

static int objectives_rows(nmfb_ctx *ctx, const float *V, const float *W, uint32_t rows, int what, double out[3])
{
    // two CTAs per SM by registers (82 to 126 a thread), in two waves; dObj holds the partials of 1024
    int const cx = obj_cx(ctx->m);
    uint64_t const tr = obj_rows(cx), tc = obj_cols(cx), tiles = ((ctx->m + tc - 1) / tc) * ((rows + tr - 1) / tr);
    uint64_t grid = 4u * (uint64_t)ctx->sm_count;
    if (grid > tiles) grid = tiles;
    if (grid > 1024) grid = 1024;
    auto const kern = cx == 1   ? objective_kernel<1>(what)
                      : cx == 2 ? objective_kernel<2>(what)
                      : cx == 4 ? objective_kernel<4>(what)
                      : cx == 8 ? objective_kernel<8>(what)
                                : objective_kernel<16>(what);
    kern<<<(unsigned)grid, 256, 0, ctx->stream>>>(V, ctx->ldv, W, ctx->dH, rows, ctx->m, ctx->kp, ctx->k, ctx->dObj,
                                                 ctx->dObj + 3 * 1024, ctx->dObjTicket);
    NMFB_LAUNCH_CHECK(ctx);
    NMFB_CUDA_TRY(ctx, cudaMemcpyAsync(out, ctx->dObj + 3 * 1024, 3 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    NMFB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return NMFB_OK;
}

int nmfb_objectives_rows(nmfb_ctx *ctx, const float *V, const float *W, uint32_t rows, double out[3])
{
    return objectives_rows(ctx, V, W, rows, OBJ_DOTS | OBJ_KL, out);
}

int nmfb_objectives(nmfb_ctx *ctx, double *dot_V, double *dot_VWH, double *kl)
{
    double host[3];
    int const what = (dot_V || dot_VWH ? OBJ_DOTS : 0) | (kl ? OBJ_KL : 0);
    int const rc = ctx->splan ? nmfb_stream_objectives(ctx, host)
                              : objectives_rows(ctx, ctx->dV, ctx->dW, ctx->n, what ? what : OBJ_DOTS | OBJ_KL, host);
    if (rc) return rc;
    if (dot_V) *dot_V = host[0];
    if (dot_VWH) *dot_VWH = host[1];
    if (kl) *kl = host[2];
    return NMFB_OK;
}
