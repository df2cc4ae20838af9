// small.cu -- half-iterations of small matrices (the FP32 fused arm): two launches an iteration.
//
// A small problem's iteration is a chain of latencies, not work: the fused arm's four
// launches (two tensor-core halves, each with its k_finish) take 5 us each at 5000 x 38
// -- prologue, tensor-memory round trips, split partials, stores -- for 0.1 us of traffic.
// Here each CTA keeps a slab of rows of V and of W in shared memory, and
//   k_small_rows    updates its rows of W (no split: a row's sum is the CTA's own) and,
//                   while they are there, sums the next update_H's terms over its rows;
//   k_small_finish  adds the CTAs' sums and writes the new H.
// Inside a run both chain by programmatic dependent launch: k_small_rows loads V while
// k_small_finish runs.  update_H alone is k_small_rows (sums only) + k_small_finish,
// update_W alone k_small_rows (update only): the same operations in the same order, so
// a run gives what single steps give, bit for bit.
// FP32 SIMT like the batched engine (FMAs, one approximate reciprocal an element),
// FP64 column sums; formulas and EPS adjust as the general path.  All sums have
// fixed orders that depend on the sizes and the SM count only.
//
// (One cooperative launch for a whole run was faster alone, 9 us an iteration at
// 5000 x 38, but such launches follow one another: twelve contexts at once ran 1837
// runs/s of 60 iterations at 2000 x 100 against 3285 with the fused kernels.)
#include "nmfb_internal.cuh"
#include "fused_common.cuh"

#include <float.h>

using namespace nmfb_tc;
using nmfb::ConvState;

namespace {

constexpr int SNT = 512, SNW = SNT / 32;
constexpr int FNT = 128;          // threads of a k_small_finish CTA
constexpr uint32_t SM_KMAX = 24;
constexpr uint32_t MAXG = 32;     // thread groups whose sums one thread adds up
constexpr uint32_t DO_W = 1, DO_SUMS = 2, DO_ADJUST = 4;

struct SmallArgs {
    const float *V;
    size_t ldv;
    float *W, *H;          // n x kp, m x kp
    float *part;           // [CTA][m][KS]: sums of update_H
    double *cs;            // [CTA][KS]: column sums of W
    const ConvState *st;
    uint32_t n, m, k, kp;
    uint32_t nr, pitch;    // rows per CTA, row pitch of V in shared memory (odd)
    uint32_t grid, what;
};

// Row pitch of W, H and the group sums in shared memory: an odd number of 16-byte
// pieces, so that rows read side by side hit different banks (with the pitch ks,
// ranks 13..16 and 29..32 ran at half the speed of their neighbours).
__host__ __device__ constexpr uint32_t pitch_of(uint32_t ks) { return ((ks / 4u) | 1u) * 4u; }

struct SmallLayout {       // shared memory, offsets in floats
    uint32_t v, w, h, red, acch, total;
};
__host__ __device__ inline SmallLayout small_layout(uint32_t nr, uint32_t pitch, uint32_t m, uint32_t ks)
{
    SmallLayout L;
    uint32_t const rs = pitch_of(ks);
    L.red = 0;                                   // SNT rows
    L.w = L.red + SNT * rs;
    L.h = L.w + nr * rs;
    L.acch = L.h + m * rs;
    L.v = L.acch + ks;
    L.total = L.v + nr * pitch;
    return L;
}

// Copies to shared memory that nobody waits for one by one (a slab's loads are all in flight).
__device__ __forceinline__ void copy4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(float *dst, const float *src)   // through L2
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int KS>
__device__ __forceinline__ void row4(const float *p, float (&x)[KS])
{
#pragma unroll
    for (int q = 0; q < KS / 4; q++) {
        float4 const f = reinterpret_cast<const float4 *>(p)[q];
        x[4 * q] = f.x;
        x[4 * q + 1] = f.y;
        x[4 * q + 2] = f.z;
        x[4 * q + 3] = f.w;
    }
}

template <int KS>
__device__ __forceinline__ void put4(float *p, const float (&x)[KS])
{
#pragma unroll
    for (int q = 0; q < KS / 4; q++)
        reinterpret_cast<float4 *>(p)[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
}

// One element: wh = a . b, acc += (v / wh) b.  (Padding columns of a and b are 0.)
template <int KS>
__device__ __forceinline__ void element(float v, const float (&a)[KS], const float (&b)[KS], float (&acc)[KS])
{
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
    for (int c = 0; c < KS; c += 2) {
        s0 = fmaf(a[c], b[c], s0);
        s1 = fmaf(a[c + 1], b[c + 1], s1);
    }
    float const q = v * rcp_approx(s0 + s1);
#pragma unroll
    for (int c = 0; c < KS; c++) acc[c] = fmaf(q, b[c], acc[c]);
}

// FP64 column sums of a rows x KS matrix in shared memory, a warp per column (rows
// lane, lane + 32, ... in order, then a shuffle tree): put(c, sum) in lane 0.
template <int KS, class F>
__device__ __forceinline__ void column_sums(const float *X, uint32_t rows, F put)
{
    for (uint32_t c = threadIdx.x / 32; c < (uint32_t)KS; c += SNW) {
        double t = 0.0;
        for (uint32_t r = threadIdx.x % 32; r < rows; r += 32) t += (double)X[r * pitch_of(KS) + c];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        if (threadIdx.x % 32 == 0) put(c, t);
    }
}

// (Two to an SM where the registers allow it without spills: one context's CTAs meet
// another's, and its own next launch starts while the last one ends -- 5000 x 38 14.2 -> 10.2 us.)
template <int KS>
__global__ void __launch_bounds__(SNT, KS <= 16 ? 2 : 1) k_small_rows(const SmallArgs a)
{
    extern __shared__ __align__(16) float sm[];
    SmallLayout const L = small_layout(a.nr, a.pitch, a.m, KS);
    float *const sV = sm + L.v, *const sW = sm + L.w, *const sH = sm + L.h, *const red = sm + L.red;
    float *const acch = sm + L.acch;
    uint32_t const tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    uint32_t const blk = blockIdx.x, m = a.m, k = a.k;
    uint32_t const r0 = min(a.n, blk * a.nr), nrows = min(a.n, r0 + a.nr) - r0;
    constexpr uint32_t K4 = KS / 4, RS = pitch_of(KS);

    chain_next();
    // V before the wait: where this launch is chained, V was complete before the chain began
    for (uint32_t i = warp; i < nrows; i += SNW)
        for (uint32_t j = lane; j < m; j += 32) copy4(sV + i * a.pitch + j, a.V + (size_t)(r0 + i) * a.ldv + j);
    chain_wait();
    auto const load_factor = [&](float *dst, const float *src, uint32_t rows) {
        for (uint32_t e = tid; e < rows * K4; e += SNT) copy16(dst + e / K4 * RS + e % K4 * 4, src + (size_t)(e / K4) * a.kp + e % K4 * 4);
    };
    load_factor(sW, a.W + (size_t)r0 * a.kp, nrows);
    load_factor(sH, a.H, m);
    bool const over = __ldcg(&a.st->converged) != 0;
    copies_done();
    if (over) return;
    __syncthreads();
    if (a.what & DO_W) {
        column_sums<KS>(sH, m, [&](uint32_t c, double s) { acch[c] = (float)s; });
        // (the first barrier below comes before anything divides by them)
        // ---- update_W: thread group g of a pass takes columns g, g + groups, ... of its row
        for (uint32_t i0 = 0; i0 < nrows; i0 += SNT) {
            uint32_t const rows = min((uint32_t)SNT, nrows - i0), groups = min(min(SNT / rows, m), MAXG);
            uint32_t const ii = tid % rows, g = tid / rows;
            float w[KS], acc[KS];
#pragma unroll
            for (int c = 0; c < KS; c++) acc[c] = 0.0f;
            if (g < groups) {
                row4<KS>(sW + (i0 + ii) * RS, w);
                const float *v = sV + (i0 + ii) * a.pitch;
#pragma unroll 2
                for (uint32_t j = g; j < m; j += groups) {
                    float h[KS];
                    row4<KS>(sH + j * RS, h);
                    element<KS>(v[j], w, h, acc);
                }
                put4<KS>(red + tid * RS, acc);
            }
            __syncthreads();
            for (uint32_t e = tid; e < rows * KS; e += SNT) {
                uint32_t const r = e / KS, c = e % KS;
                float s = red[r * RS + c];
                for (uint32_t q = 1; q < groups; q++) s += red[(q * rows + r) * RS + c];
                float *const w = sW + (i0 + r) * RS + c;
                float v = 0.0f;
                if (c < k) {
                    v = __fdiv_rn(*w * s, acch[c]);
                    if (a.what & DO_ADJUST) v = fmaxf(v, FLT_MIN);
                    a.W[(size_t)(r0 + i0 + r) * a.kp + c] = v;
                }
                *w = v;
            }
            __syncthreads();
        }
    }
    if (a.what & DO_SUMS) {
        // ---- update_H, this CTA's rows: thread group g of a pass takes rows g, g + groups, ...
        for (uint32_t j0 = 0; j0 < m; j0 += SNT) {
            uint32_t const cols = min((uint32_t)SNT, m - j0), groups = min(min(SNT / cols, nrows), MAXG);
            uint32_t const jj = tid % cols, g = tid / cols;
            float h[KS], acc[KS];
#pragma unroll
            for (int c = 0; c < KS; c++) acc[c] = 0.0f;
            if (g < groups) {
                row4<KS>(sH + (j0 + jj) * RS, h);
#pragma unroll 2
                for (uint32_t i = g; i < nrows; i += groups) {
                    float w[KS];
                    row4<KS>(sW + i * RS, w);
                    element<KS>(sV[i * a.pitch + j0 + jj], h, w, acc);
                }
            }
            float *const dst = a.part + ((size_t)blk * m + j0) * KS;
            if (groups == 1) {
                if (g == 0) put4<KS>(dst + (size_t)jj * KS, acc);
            } else {
                __syncthreads();
                if (g < groups) put4<KS>(red + tid * RS, acc);
                __syncthreads();
                for (uint32_t e = tid; e < cols * K4; e += SNT) {
                    const float *p = red + e / K4 * RS + e % K4 * 4;
                    float4 s = *reinterpret_cast<const float4 *>(p);
                    for (uint32_t q = 1; q < groups; q++) {
                        float4 const x = *reinterpret_cast<const float4 *>(p + q * cols * RS);
                        s.x += x.x;
                        s.y += x.y;
                        s.z += x.z;
                        s.w += x.w;
                    }
                    reinterpret_cast<float4 *>(dst)[e] = s;
                }
            }
        }
        column_sums<KS>(sW, nrows, [&](uint32_t c, double s) { a.cs[(size_t)blk * KS + c] = s; });
    }
}

// The new H: a warp adds the CTAs' sums of four entries of a row (lane l: CTAs l, l + 32,
// ... in order, then a shuffle tree) and the column sums of W that they are divided by.
template <int KS>
__global__ void __launch_bounds__(FNT) k_small_finish(const SmallArgs a)
{
    constexpr uint32_t K4 = KS / 4;
    chain_wait();
    chain_next();
    if (__ldcg(&a.st->converged)) return;
    uint32_t const lane = threadIdx.x % 32, warp = threadIdx.x / 32, chunks = a.m * K4;
    uint32_t e = blockIdx.x + warp * gridDim.x;
    bool const mine = e < chunks;
    if (!mine && warp > 0) return;   // (whole warps)
    e %= chunks;                     // (a CTA without entries of its own repeats one, see the launch)
    float s[4] = {};
    double t[4] = {};
    for (uint32_t q = lane; q < a.grid; q += 160) {   // (one round trip up to 160 CTAs)
        float4 x[5];
        double2 y[5], z[5];
#pragma unroll
        for (int u = 0; u < 5; u++) {
            uint32_t const b = min(q + 32 * u, a.grid - 1);   // (loads without a branch: all in flight at once)
            const double2 *const cs = reinterpret_cast<const double2 *>(a.cs + (size_t)b * KS + e % K4 * 4);
            x[u] = __ldcg(reinterpret_cast<const float4 *>(a.part) + (size_t)b * chunks + e);
            y[u] = __ldcg(cs);
            z[u] = __ldcg(cs + 1);
        }
#pragma unroll
        for (int u = 0; u < 5; u++) {
            if (q + 32 * u >= a.grid) continue;
            s[0] += x[u].x;
            s[1] += x[u].y;
            s[2] += x[u].z;
            s[3] += x[u].w;
            t[0] += y[u].x;
            t[1] += y[u].y;
            t[2] += z[u].x;
            t[3] += z[u].y;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            s[c] += __shfl_xor_sync(0xffffffffu, s[c], off);
            t[c] += __shfl_xor_sync(0xffffffffu, t[c], off);
        }
    uint32_t const c = e % K4 * 4 + lane;
    if (mine && lane < 4 && c < a.k) {
        float const tot = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
        float const col = (float)(lane == 0 ? t[0] : lane == 1 ? t[1] : lane == 2 ? t[2] : t[3]);
        float *const h = a.H + (size_t)(e / K4) * a.kp + c;
        float v = __fdiv_rn(__ldcg(h) * tot, col);
        if (a.what & DO_ADJUST) v = fmaxf(v, FLT_MIN);
        *h = v;
    }
}

struct SmallKernels {
    void (*rows)(const SmallArgs);
    void (*finish)(const SmallArgs);
};
SmallKernels small_kernels(uint32_t ks)
{
    switch (ks) {
    case 4: return {k_small_rows<4>, k_small_finish<4>};
    case 8: return {k_small_rows<8>, k_small_finish<8>};
    case 12: return {k_small_rows<12>, k_small_finish<12>};
    case 16: return {k_small_rows<16>, k_small_finish<16>};
    case 20: return {k_small_rows<20>, k_small_finish<20>};
    default: return {k_small_rows<24>, k_small_finish<24>};
    }
}

// The launch for a context's sizes: CTAs, rows per CTA, shared memory.
struct SmallPlan {
    uint32_t ks, grid, nr, pitch;
    size_t smem;
};
SmallPlan small_plan(const nmfb_ctx *ctx)
{
    SmallPlan p;
    p.ks = (ctx->k + 3u) & ~3u;
    p.nr = (ctx->n + (uint32_t)ctx->sm_count - 1) / (uint32_t)ctx->sm_count;
    p.grid = (ctx->n + p.nr - 1) / p.nr;
    p.pitch = ctx->m | 1u;
    p.smem = (size_t)small_layout(p.nr, p.pitch, ctx->m, p.ks).total * sizeof(float);
    return p;
}

SmallArgs small_args(const nmfb_ctx *ctx, const SmallPlan &p, uint32_t what)
{
    SmallArgs a;
    a.V = ctx->dV;
    a.ldv = ctx->ldv;
    a.W = ctx->dW;
    a.H = ctx->dH;
    a.part = ctx->dPart;
    a.cs = ctx->dColPart;
    a.st = ctx->dState;
    a.n = ctx->n;
    a.m = ctx->m;
    a.k = ctx->k;
    a.kp = ctx->kp;
    a.nr = p.nr;
    a.pitch = p.pitch;
    a.grid = p.grid;
    a.what = what;
    return a;
}

constexpr size_t SMALL_SMEM = SMEM_LIMIT - 1024;   // every launch's attribute: contexts share the kernels

int launch_rows(nmfb_ctx *ctx, uint32_t what, bool chained)
{
    SmallPlan const p = small_plan(ctx);
    SmallKernels const kern = small_kernels(p.ks);
    SmallArgs const a = small_args(ctx, p, what);
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(kern.rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMALL_SMEM));
    if (chained)
        NMFB_CUDA_TRY(ctx, launch_chained(kern.rows, dim3(p.grid), SNT, p.smem, ctx->stream, a));
    else
        kern.rows<<<p.grid, SNT, p.smem, ctx->stream>>>(a);
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

}  // namespace

// Whether a context's updates take this path: the FP32 fused arm's problems of rank <= 24
// with at most 8 KB of H (every CTA reads it, and k_small_finish adds as much from each
// CTA: at 300 x 1000 k = 12 an iteration took 31 us, 18 with the fused kernels) and a slab
// of V that CTAs get through in a few us (342000 lane operations / 512 lanes). Measured us
// an iteration, fused kernels / here: 5000 x 38 k = 3 22.8 / 10.2, 9973 x 127 k = 7 27.2 /
// 17.0, 10000 x 250 k = 8 26.6 / 18.2, 20000 x 60 k = 16 30.7 / 18.3, 20000 x 150 k = 8
// 33.3 / 19.8. The line on the slab is drawn for several contexts at once, whose work no
// longer hides in the others' latencies; runs/s of 60 iterations by four threads: 5000 x 38
// k = 3 2630 / 5425, 9973 x 127 k = 7 1915 / 2665, 20000 x 100 k = 8 1436 / 1809, left to the
// fused kernels 40000 x 150 k = 8 796 / 663, 30000 x 128 k = 16 1262 / 750.
bool nmfb_small_fits(const nmfb_ctx *ctx)
{
    if (ctx->arm != NMFB_ARM_FUSED || ctx->k > SM_KMAX || ctx->splan) return false;
    SmallPlan const p = small_plan(ctx);
    if ((uint64_t)ctx->m * p.ks > 2048 || (uint64_t)p.nr * ctx->m * (p.ks + 6) > 342000 || p.smem > SMALL_SMEM) return false;
    return (size_t)p.grid * ctx->m * p.ks <= ctx->part_items && (size_t)p.grid * p.ks <= (size_t)2 * 1024 * ctx->kp;
}

// fz_ok[0] here: the sums of the coming update_H are there (the W and H they were
// formed with are unchanged).
int nmfb_small_update_H(nmfb_ctx *ctx, int adjust)
{
    int rc = nmfb_prof_begin(ctx, 2);
    if (rc) return rc;
    if ((rc = nmfb_prof_begin(ctx, 0))) return rc;
    if (!ctx->fz_ok[0] && (rc = launch_rows(ctx, DO_SUMS, false))) return rc;
    if ((rc = nmfb_prof_end(ctx, 0))) return rc;
    SmallPlan const p = small_plan(ctx);
    // At least a CTA per SM, all as long: the next k_small_rows is placed while they run, and on
    // SMs without one it got two CTAs (10000 x 250 k = 8: 24.6 us an iteration, now 18.2)
    uint32_t const need = (ctx->m * (p.ks / 4) + FNT / 32 - 1) / (FNT / 32), sms = (uint32_t)ctx->sm_count;
    NMFB_CUDA_TRY(ctx, launch_chained(small_kernels(p.ks).finish, dim3(need > sms ? need : sms), FNT, 0, ctx->stream,
                                      small_args(ctx, p, adjust ? DO_ADJUST : 0u)));
    NMFB_LAUNCH_CHECK(ctx);
    ctx->fz_ok[0] = ctx->fz_ok[1] = 0;
    return nmfb_prof_end(ctx, 2);
}

// Inside a run an update_W that no test follows forms the next update_H's sums (not
// under profiling, which times the halves apart).
int nmfb_small_update_W(nmfb_ctx *ctx, int adjust)
{
    bool const ahead = ctx->in_run && !ctx->prof_on && !adjust;
    int rc = nmfb_prof_begin(ctx, 3);
    if (rc) return rc;
    if ((rc = nmfb_prof_begin(ctx, 1))) return rc;
    rc = launch_rows(ctx, DO_W | (ahead ? DO_SUMS : 0u) | (adjust ? DO_ADJUST : 0u), ctx->in_run != 0);
    if (rc || (rc = nmfb_prof_end(ctx, 1))) return rc;
    ctx->fz_ok[0] = ahead;
    ctx->fz_ok[1] = 0;
    return nmfb_prof_end(ctx, 3);
}
