// kernels_plain.cu -- the unfused FP32 SIMT arm (NMFB_ARM_PLAIN), the arm of
// ranks above 64 and of the blockwise mode.
//
// It keeps the structure of the reference's half-iteration
// (src/NMF_routines.c:376-525 / 1014-1164), with the n x m quotient
// materialised in HBM, but with hand-written kernels instead of cuBLAS:
//   1. acc  = colsum(W or H)                 (k_colsum, kernels_common.cu)
//   2. Q    = V ./ (W * H^T)    -> n x m      (k_quot)
//   3. Xaux = reduce(Q, other factor)         (k_red, split over the reduction)
//   4. X    = X .* Xaux ./ acc                (k_factor, kernels_common.cu)
// Both contractions are bound by FP32 issue: 2 n m k flops each, 72 TFLOP/s.
#include "nmfb_internal.cuh"
#include "fused_common.cuh"

using nmfb::ConvState;
using nmfb_tc::chain_next;
using nmfb_tc::chain_wait;
using nmfb_tc::launch_chained;

namespace {

__device__ __forceinline__ bool halted(const ConvState *st) { return st && *(volatile const uint32_t *)&st->converged; }

// Both kernels: a 128 x 64 output tile per CTA of 128 threads, 8 x 8 outputs per
// thread (rows 4 ty + {0..3} and 64 + 4 ty + .., columns 4 tx + .. and 32 + 4 tx +
// ..: every shared load is 16 bytes wide, conflict-free or broadcast, and feeds 16
// FMAs), 16 steps of the reduction staged at a time, the next 16 in registers
// meanwhile.
constexpr int TM = 128, TN = 64, TK = 16;
constexpr uint32_t RED_CHAIN = 512;   // longest FP32 chain of k_red, in steps of the reduction

struct Tile {
    float a[2][TK][TM + 4];
    float b[2][TK][TN + 4];
};

__device__ __forceinline__ void tile_fma(const float (&a)[TK][TM + 4], const float (&b)[TK][TN + 4], uint32_t tx,
                                         uint32_t ty, float (&acc)[8][8])
{
#pragma unroll
    for (int kk = 0; kk < TK; kk++) {
        float4 const a0 = *reinterpret_cast<const float4 *>(&a[kk][4 * ty]);
        float4 const a1 = *reinterpret_cast<const float4 *>(&a[kk][64 + 4 * ty]);
        float4 const b0 = *reinterpret_cast<const float4 *>(&b[kk][4 * tx]);
        float4 const b1 = *reinterpret_cast<const float4 *>(&b[kk][32 + 4 * tx]);
        float const av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        float const bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int p = 0; p < 8; p++)
#pragma unroll
            for (int q = 0; q < 8; q++) acc[p][q] = fmaf(av[p], bv[q], acc[p][q]);
    }
}

// Q = V ./ (W H^T) over n x m (matrix_div_sub in division mode; the reference uses
// fdividef, src/GPU_kernels.cu:1687-1695), the quotient in the epilogue of the
// product: no pass over V and W H^T of its own.  W: n x kp, H: m x kp (padding
// columns zero), V and Q: leading dimension ld, a multiple of 32; padding columns
// are neither used nor written.
__global__ void __launch_bounds__(128, 4) k_quot(const float *__restrict__ V, const float *W, const float *H, float *Q,
                                                 uint32_t n, uint32_t m, uint32_t kp, uint32_t k, size_t ld,
                                                 const ConvState *st)
{
    chain_next();
    chain_wait();
    if (halted(st)) return;
    __shared__ __align__(16) Tile s;
    uint32_t const tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
    uint32_t const i0 = blockIdx.y * TM, j0 = blockIdx.x * TN;
    // staging: thread t holds row t of W (16 columns) and half of row t % 64 of H
    bool const ina = i0 + tid < n, inb = j0 + tid % TN < m;
    const float *pa = W + (size_t)(i0 + tid) * kp;
    const float *pb = H + (size_t)(j0 + tid % TN) * kp + tid / TN * 8;
    float4 ra[4], rb[2];
    float4 const zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto const load = [&](uint32_t c0) {
#pragma unroll
        for (int q = 0; q < 4; q++) ra[q] = ina ? __ldcg(reinterpret_cast<const float4 *>(pa + c0) + q) : zero;
#pragma unroll
        for (int q = 0; q < 2; q++) rb[q] = inb ? __ldcg(reinterpret_cast<const float4 *>(pb + c0) + q) : zero;
    };
    auto const store = [&](uint32_t buf) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            s.a[buf][4 * q + 0][tid] = ra[q].x;
            s.a[buf][4 * q + 1][tid] = ra[q].y;
            s.a[buf][4 * q + 2][tid] = ra[q].z;
            s.a[buf][4 * q + 3][tid] = ra[q].w;
        }
        uint32_t const r = tid % TN, c = tid / TN * 8;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            s.b[buf][c + 4 * q + 0][r] = rb[q].x;
            s.b[buf][c + 4 * q + 1][r] = rb[q].y;
            s.b[buf][c + 4 * q + 2][r] = rb[q].z;
            s.b[buf][c + 4 * q + 3][r] = rb[q].w;
        }
    };
    float acc[8][8] = {};
    uint32_t const steps = (k + TK - 1) / TK;   // (kp is a multiple of 16)
    load(0);
    // V's tile into L2 while the product runs: each line once, by one of its eight threads
    if (tx == 0)
#pragma unroll
        for (int p = 0; p < 8; p++) {
            uint32_t const i = i0 + (p < 4 ? 0u : 64u) + 4 * ty + (p & 3);
#pragma unroll
            for (uint32_t j = j0; j < j0 + TN; j += 32)
                if (i < n && j < m) asm volatile("prefetch.global.L2 [%0];" ::"l"(V + (size_t)i * ld + j));
        }
    store(0);
    __syncthreads();
    for (uint32_t t = 0; t < steps; t++) {
        if (t + 1 < steps) load((t + 1) * TK);
        tile_fma(s.a[t & 1], s.b[t & 1], tx, ty, acc);
        if (t + 1 < steps) store((t + 1) & 1);
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 8; p++) {
        uint32_t const i = i0 + (p < 4 ? 0u : 64u) + 4 * ty + (p & 3);
        if (i >= n) continue;
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
            uint32_t const j = j0 + (q < 4 ? 0u : 32u) + 4 * tx;
            if (j >= m) continue;
            size_t const o = (size_t)i * ld + j;
            float4 const v = __ldcs(reinterpret_cast<const float4 *>(V + o));   // (a float4 from below m lies in the row)
            float4 const r = make_float4(__fdividef(v.x, acc[p][q]), __fdividef(v.y, acc[p][q + 1]),
                                         __fdividef(v.z, acc[p][q + 2]), __fdividef(v.w, acc[p][q + 3]));
            if (j + 4 <= m) {
                *reinterpret_cast<float4 *>(Q + o) = r;
            } else {
                Q[o] = r.x;
                if (j + 1 < m) Q[o + 1] = r.y;
                if (j + 2 < m) Q[o + 2] = r.z;
            }
        }
    }
}

// Out[o][c] = sum_r Q(o, r) * F[r][c] for r in this CTA's reduction chunk.
// Q(o, r) = Qm[o][r] when !TRANS, Qm[r][o] when TRANS (Qm has leading dim ldq, a
// multiple of 32).  F: nred x kp.  Partial results go to part[chunk][o][c] (o <
// nout, c < kp).  grid: row tiles x chunks x column tiles.
// A chunk longer than `piece` (LONG) is summed piece by piece, each added to the CTA's
// own partial (the registers are full, and the partial lies in L2): FP32 chains of at most
// RED_CHAIN terms.  In one chain, update_W at 60000 x 5000 k = 256 (5000 terms) was off by
// 17 * 2^-24 rms, now 2; the run takes 164 ms for 10 iterations, with half the splits and
// long chains 172.
template <bool TRANS, bool LONG>
__global__ void __launch_bounds__(128, 4) k_red(const float *Qm, size_t ldq, const float *F, uint32_t nout, uint32_t nred,
                                                uint32_t kp, uint32_t chunk, uint32_t piece, float *part, const ConvState *st)
{
    chain_next();
    chain_wait();
    if (halted(st)) return;
    __shared__ __align__(16) Tile s;
    uint32_t const tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
    uint32_t const o0 = blockIdx.x * TM, c0 = blockIdx.z * TN;
    uint32_t const r_begin = blockIdx.y * chunk, r_end = min(nred, r_begin + chunk);
    float4 ra[4], rb[2];
    float4 const zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // staging: TRANS: thread t holds row t / 8 of the 16, outputs 16 (t % 8) ..; else the 16
    // steps of output t.  F: row t / 8, columns 8 (t % 8) ...
    auto const load = [&](uint32_t r0) {
        if (TRANS) {
            uint32_t const r = r0 + tid / 8, o = o0 + tid % 8 * 16;
#pragma unroll
            for (int q = 0; q < 4; q++)   // (a float4 from below nout lies in the row; outputs past nout are not kept)
                ra[q] = r < r_end && o + 4 * q < nout ? __ldcg(reinterpret_cast<const float4 *>(Qm + (size_t)r * ldq + o) + q)
                                                      : zero;
        } else {
            uint32_t const o = o0 + tid;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t const r = r0 + 4 * q;
                float4 v = o < nout && r < r_end ? __ldcg(reinterpret_cast<const float4 *>(Qm + (size_t)o * ldq + r)) : zero;
                if (r + 1 >= r_end) v.y = 0.0f;   // past the reduction: the row's padding holds anything
                if (r + 2 >= r_end) v.z = 0.0f;
                if (r + 3 >= r_end) v.w = 0.0f;
                ra[q] = v;
            }
        }
        uint32_t const r = r0 + tid / 8, c = c0 + tid % 8 * 8;
#pragma unroll
        for (int q = 0; q < 2; q++)
            rb[q] = r < r_end && c + 4 * q < kp ? __ldcg(reinterpret_cast<const float4 *>(F + (size_t)r * kp + c) + q) : zero;
    };
    auto const store = [&](uint32_t buf) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (TRANS) {
                *reinterpret_cast<float4 *>(&s.a[buf][tid / 8][tid % 8 * 16 + 4 * q]) = ra[q];
            } else {
                s.a[buf][4 * q + 0][tid] = ra[q].x;
                s.a[buf][4 * q + 1][tid] = ra[q].y;
                s.a[buf][4 * q + 2][tid] = ra[q].z;
                s.a[buf][4 * q + 3][tid] = ra[q].w;
            }
        }
#pragma unroll
        for (int q = 0; q < 2; q++) *reinterpret_cast<float4 *>(&s.b[buf][tid / 8][tid % 8 * 8 + 4 * q]) = rb[q];
    };
    float acc[8][8] = {};
    uint32_t const steps = r_end > r_begin ? (r_end - r_begin + TK - 1) / TK : 0;
    if (steps) {
        load(r_begin);
        store(0);
    }
    __syncthreads();
    float *const outp = part + (size_t)blockIdx.y * nout * kp;
    auto const put = [&](bool add) {   // acc to the partial, or added to it
#pragma unroll
        for (int p = 0; p < 8; p++) {
            uint32_t const o = o0 + (p < 4 ? 0u : 64u) + 4 * ty + (p & 3);
            if (o >= nout) continue;
#pragma unroll
            for (int q = 0; q < 8; q += 4) {
                uint32_t const c = c0 + (q < 4 ? 0u : 32u) + 4 * tx;
                if (c >= kp) continue;
                float4 *const d = reinterpret_cast<float4 *>(outp + (size_t)o * kp + c);
                float4 x = make_float4(acc[p][q], acc[p][q + 1], acc[p][q + 2], acc[p][q + 3]);
                if (add) {
                    float4 const y = *d;
                    x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
                }
                *d = x;
            }
        }
    };
    uint32_t done = 0;   // steps already in the partial (LONG)
    for (uint32_t t = 0; t < steps; t++) {
        if (LONG && t - done == piece / TK) {
            put(done > 0);
            done = t;
#pragma unroll
            for (int p = 0; p < 8; p++)
#pragma unroll
                for (int q = 0; q < 8; q++) acc[p][q] = 0.0f;
        }
        if (t + 1 < steps) load(r_begin + (t + 1) * TK);
        tile_fma(s.a[t & 1], s.b[t & 1], tx, ty, acc);
        if (t + 1 < steps) store((t + 1) & 1);
        __syncthreads();
    }
    put(LONG && done > 0);
}

struct RedPlan {
    uint32_t nsplit, chunk, piece;
};

// Splits of the reduction: about eight CTAs per SM (above rank 128 more, or the chains of
// additions get longer with the rank), none longer than RED_CHAIN where the partials
// have room, in chunks of whole staging steps.
RedPlan plan_split(nmfb_ctx *ctx, uint32_t nout, uint32_t nred)
{
    uint32_t const ctiles = (ctx->k + TN - 1) / TN, tiles = (nout + TM - 1) / TM * (ctiles < 2 ? ctiles : 2);
    uint32_t want = (8u * (uint32_t)ctx->sm_count + tiles - 1) / tiles;
    if (want < (nred + RED_CHAIN - 1) / RED_CHAIN) want = (nred + RED_CHAIN - 1) / RED_CHAIN;
    if (want < 1) want = 1;
    if (want > NMFB_MAX_SPLIT) want = NMFB_MAX_SPLIT;
    // (the partials of all splits fit the context's buffer)
    size_t const fit = ctx->part_items / ((size_t)nout * ctx->kp);
    if (want > fit) want = fit > 0 ? (uint32_t)fit : 1u;
    uint32_t chunk = (nred + want - 1) / want;
    chunk = (chunk + TK - 1) / TK * TK;
    if (chunk == 0) chunk = TK;
    uint32_t const nsplit = (nred + chunk - 1) / chunk;
    uint32_t const pieces = (chunk + RED_CHAIN - 1) / RED_CHAIN;   // of equal length
    uint32_t const piece = ((chunk + pieces - 1) / pieces + TK - 1) / TK * TK;
    return {nsplit, chunk, piece};
}

int launch_red(nmfb_ctx *ctx, const float *Q, bool trans, const float *F, uint32_t nout, uint32_t nred, uint32_t *nsplit)
{
    RedPlan const p = plan_split(ctx, nout, nred);
    if ((size_t)p.nsplit * nout * ctx->kp > ctx->part_items)
        return nmfb_fail(ctx, NMFB_EINVAL, "partial buffer too small (%u splits of %u rows)", p.nsplit, nout);
    dim3 const g((nout + TM - 1) / TM, p.nsplit, (ctx->k + TN - 1) / TN);
    auto const kern = p.chunk > p.piece ? (trans ? k_red<true, true> : k_red<false, true>)
                                        : (trans ? k_red<true, false> : k_red<false, false>);
    NMFB_CUDA_TRY(ctx, launch_chained(kern, g, 128, 0, ctx->stream, Q, ctx->ldv, F, nout, nred, ctx->kp, p.chunk, p.piece,
                                      ctx->dPart, ctx->dState));
    NMFB_LAUNCH_CHECK(ctx);
    *nsplit = p.nsplit;
    return NMFB_OK;
}

int plain_half(nmfb_ctx *ctx, bool is_H, int adjust)
{
    // 1. column sums of the factor that is NOT being updated.
    float *X = is_H ? ctx->dH : ctx->dW;           // updated factor
    const float *Y = is_H ? ctx->dW : ctx->dH;     // other factor
    uint32_t const xrows = is_H ? ctx->m : ctx->n;
    uint32_t const yrows = is_H ? ctx->n : ctx->m;
    float *acc = is_H ? ctx->dAccW : ctx->dAccH;
    int const whole = is_H ? 2 : 3, main = is_H ? 0 : 1;
    int rc = nmfb_prof_begin(ctx, whole);
    if (rc) return rc;
    if ((rc = nmfb_colsum(ctx, Y, yrows, acc, is_H ? 0 : 1))) return rc;
    // 2. Q = V ./ (W * H^T) (n x m)
    if ((rc = nmfb_plain_quot(ctx, ctx->dV, ctx->dW, ctx->n, ctx->dWH))) return rc;
    // 3. Xaux = Q^T Y (update_H) or Q Y (update_W), split over the reduction.
    if ((rc = nmfb_prof_begin(ctx, main))) return rc;
    uint32_t nsplit = 0;
    if ((rc = launch_red(ctx, ctx->dWH, is_H, Y, xrows, yrows, &nsplit))) return rc;
    if ((rc = nmfb_prof_end(ctx, main))) return rc;
    // 4. X = X .* Xaux ./ acc  (+ EPS adjust on test iterations)
    rc = nmfb_muldiv(ctx, X, xrows, ctx->dPart, nsplit, (size_t)xrows * ctx->kp, acc, adjust);
    if (rc) return rc;
    return nmfb_prof_end(ctx, whole);
}

}  // namespace

// Building blocks, also of the streamed mode (stream.cu): the same kernels on
// `rows` rows of W and a rows x ldv block of V.
int nmfb_plain_quot(nmfb_ctx *ctx, const float *V, const float *W, uint32_t rows, float *Q)
{
    dim3 const g((ctx->m + TN - 1) / TN, (rows + TM - 1) / TM);
    NMFB_CUDA_TRY(ctx, launch_chained(k_quot, g, 128, 0, ctx->stream, V, W, ctx->dH, Q, rows, ctx->m, ctx->kp, ctx->k,
                                      ctx->ldv, ctx->dState));
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

int nmfb_plain_red(nmfb_ctx *ctx, const float *Q, int transQ, const float *F, uint32_t nout, uint32_t nred,
                   uint32_t *nsplit)
{
    return launch_red(ctx, Q, transQ != 0, F, nout, nred, nsplit);
}

int nmfb_plain_update_H(nmfb_ctx *ctx, int adjust) { return plain_half(ctx, true, adjust); }
int nmfb_plain_update_W(nmfb_ctx *ctx, int adjust) { return plain_half(ctx, false, adjust); }
