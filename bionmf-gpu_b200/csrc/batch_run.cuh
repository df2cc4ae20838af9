// batch_run.cuh -- one problem of the batched engine, run to its end by a
// thread-block cluster (device code of batch_kernel*.cu and serve_kernel.cu).
//
// Every problem runs the reference's complete loop (src/NMF_GPU.c:522-795):
// update_H, update_W; after every niter_test_conv iterations the EPS adjust of
// W (fused into the block's last update_W) and of H (fused into the
// classification), the argmax classification with the reference's lane-exact
// tie rule (src/GPU_kernels.cu:2508-2656, 3177-3267) and the connectivity test
// (src/common.c:1195-1209) with the stop rule of src/NMF_GPU.c:695-709; the
// remaining n_iters % niter_test_conv iterations run without adjust.
//
// Work distribution: persistent thread-block clusters of C CTAs (C = 1, 2, 4
// or 8; as many clusters as fit on the GPU, at most one per problem) take
// problems from an atomic work queue in the order the host gives (largest rank
// first), and one cluster runs one problem to its end.  Within a cluster, CTA r
// owns a contiguous slice of W's rows and every CTA holds the whole of H: the
// update_H partial sums over W's rows and the partial column sums of W are
// added across the cluster in rank order through distributed shared memory, so
// every CTA computes the same H, the same classification and the same stop
// decision.  Convergence iteration counts are data dependent (a sweep's
// problems stop after 430 to 2000 iterations), so with one CTA per problem the
// few longest problems set the launch time; splitting each problem over C SMs
// divides that tail by about C.  C = 1 keeps the single-CTA summation order.
//
// Per problem, in one CTA of NT = 256 threads:
//   shared memory: H (m x ks, ks = k rounded up to 4), a staging tile (rows of
//                  W for update_H, or an NT x (jt+1) tile of V for update_W),
//                  colsum vectors, labels and the previous partition;
//   global memory: V (n x ldv, shared by all problems of a sweep, L2-resident
//                  at sweep sizes) and W (n x ks, padding columns zero).
//   update_H: thread j owns sample j: h_j in registers, WH_ij = W_i . h_j with
//             W_i broadcast from the staged tile, Haux_j += (V_ij / WH_ij) W_i,
//             summed per tile of wt rows and then across tiles;
//             H_j = (H_j .* Haux_j) ./ colsum(W)   (product first, then a
//             correctly-rounded division, as kernel_mul_div);
//   update_W: thread i owns row i: W_i in registers, V staged through shared
//             memory in NT x jt tiles (coalesced loads, conflict-free reads),
//             H_j broadcast from shared memory; same formulas mirrored.
//   colsum(W) and colsum(H) are reduced from the rows each thread just wrote,
//   in a fixed order (warp shuffles, then warps in order).
// Ranks 2..20 are compiled as exact-rank instantiations (no padded flops).
// Problem inputs (V, W, H) are read through L2 only (cp.async.cg, ld.global.cg):
// the serving kernel outlives the requests whose buffers the host frees and
// reuses, and an SM's L1 is not coherent with copies the host makes meanwhile.
// Tile shapes (wt, jt) are per-problem values (nmfb_batch_set_tiles; the
// Python layer's autotuner picks them per (k, m) bucket).
#pragma once

#include "batch.cuh"

#include <float.h>

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

using namespace nmfb_batched;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    uint32_t const s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// 1/x with rcp.approx.ftz.f32 (PTX: at most 1 ulp of error); the quotient is
// v * (1/wh).  Every element the loops visit is a real one (no zero padding),
// so a zero denominator behaves as in the reference's division (v / 0 = inf,
// 0 / 0 = NaN).
__device__ __forceinline__ float quotient(float v, float wh)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(wh));
    return v * r;
}

// Load the first K of a 16-byte aligned row of KS floats with float4 loads.
template <int K>
__device__ __forceinline__ void load_row(const float *p, float (&x)[K])
{
    constexpr int KS = (int)ks_of(K);
#pragma unroll
    for (int q = 0; q < KS / 4; q++) {
        float4 const f = reinterpret_cast<const float4 *>(p)[q];
        if (4 * q + 0 < K) x[4 * q + 0] = f.x;
        if (4 * q + 1 < K) x[4 * q + 1] = f.y;
        if (4 * q + 2 < K) x[4 * q + 2] = f.z;
        if (4 * q + 3 < K) x[4 * q + 3] = f.w;
    }
}

// One element of a contraction: wh = a . b, q = v / wh, acc += q * b.
template <int K>
__device__ __forceinline__ void element(float v, const float (&a)[K], const float (&b)[K], float (&acc)[K])
{
    float wh = 0.0f;
#pragma unroll
    for (int c = 0; c < K; c++) wh = fmaf(a[c], b[c], wh);
    float const q = quotient(v, wh);
#pragma unroll
    for (int c = 0; c < K; c++) acc[c] = fmaf(q, b[c], acc[c]);
}

// Sum v[0..K) over the CTA in a fixed order; thread c < K writes out[c].
template <int K>
__device__ __forceinline__ void block_sum(float (&v)[K], float *red, float *out, uint32_t ks)
{
    uint32_t const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < K; c++)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], off);
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < K; c++) red[warp * ks + c] = v[c];
    __syncthreads();
    if (threadIdx.x < (uint32_t)K) {
        float s = 0.0f;
        for (int w = 0; w < NW; w++) s += red[w * ks + threadIdx.x];
        out[threadIdx.x] = s;
    }
    __syncthreads();
}

// This CTA's place in its problem's cluster: rank, cluster size and the rows
// [r0, r1) of W it owns.
struct Slice {
    uint32_t rank, size, r0, r1;
};

// Sum over the cluster, in rank order, of the float at offset `off` of every
// CTA's shared memory (this CTA's own included).
__device__ __forceinline__ float cluster_sum(float *sm, uint32_t off, uint32_t csize)
{
    cg::cluster_group cl = cg::this_cluster();
    float s = 0.0f;
    for (uint32_t q = 0; q < csize; q++) s += cl.map_shared_rank(sm, q)[off];
    return s;
}

// colsum(W) into accw: this CTA's rows (wsum, per thread), then for a cluster
// the partials of every CTA added in rank order.
template <int K>
__device__ void colsum_W(float (&wsum)[K], float *sm, const SmemLayout &L, const Slice &X)
{
    constexpr uint32_t KS = ks_of(K);
    if (X.size == 1) {
        block_sum<K>(wsum, sm + L.red, sm + L.accw, KS);
        return;
    }
    block_sum<K>(wsum, sm + L.red, sm + L.partw, KS);
    cg::this_cluster().sync();   // every CTA's partial column sums are written
    if (threadIdx.x < (uint32_t)K) sm[L.accw + threadIdx.x] = cluster_sum(sm, L.partw + threadIdx.x, X.size);
    __syncthreads();
}

// update_H: stage tile t (rows of V for columns [j0, j0+cs) and rows of W) into buffer b.
template <uint32_t KS>
__device__ __forceinline__ void stage_H(const Problem &P, float *buf, const SmemLayout &L, uint32_t j0, uint32_t i0,
                                        uint32_t rows)
{
    uint32_t const q4 = L.cs / 4;
    float *sV = buf, *sW = buf + P.wt * L.cs;
    // chunk e = r * q4 + q walks in steps of NT without a division per chunk
    uint32_t const dr = NT / q4, dq = NT - dr * q4;
    uint32_t r = threadIdx.x / q4, q = threadIdx.x - r * q4;
    const float *src_v = P.V + (size_t)i0 * P.ldv + j0;
    while (r < rows) {
        if (j0 + 4 * q < P.ldv) cp_async16(sV + r * L.cs + 4 * q, src_v + (size_t)r * P.ldv + 4 * q);
        r += dr;
        q += dq;
        if (q >= q4) {
            q -= q4;
            r += 1;
        }
    }
    const float *src = P.W + (size_t)i0 * KS;
    for (uint32_t e = threadIdx.x; e < rows * (KS / 4); e += NT) cp_async16(sW + 4 * e, src + 4 * e);
}

// With a cluster, each CTA sums over its own rows of W into `part`; after a
// cluster barrier every CTA adds the partials of all CTAs in rank order and
// updates its copy of H (the same values in every CTA).  The next write of
// `part` comes after the cluster barrier of the following colsum_W, so no CTA
// overwrites partials that another may still read.
template <int K>
__device__ void update_H(const Problem &P, float *sm, const SmemLayout &L, const Slice &X)
{
    constexpr uint32_t KS = ks_of(K);
    float *sH = sm + L.h;
    float *stage = sm + L.stage;
    uint32_t const half = (L.hbuf > L.wbuf ? L.hbuf : L.wbuf);
    const float *accW = sm + L.accw;
    uint32_t const tid = threadIdx.x, m = P.m, wt = P.wt;
    uint32_t const ntiles = (X.r1 - X.r0 + wt - 1) / wt;
    float hsum[K];
#pragma unroll
    for (int c = 0; c < K; c++) hsum[c] = 0.0f;
    for (uint32_t j0 = 0; j0 < m; j0 += NT) {
        uint32_t const j = j0 + tid;
        bool const active = j < m;
        float h[K], acc[K];
#pragma unroll
        for (int c = 0; c < K; c++) {
            h[c] = active ? sH[j * KS + c] : 0.0f;
            acc[c] = 0.0f;
        }
        __syncthreads();   // the staging region may still be read by the previous phase
        if (ntiles) stage_H<KS>(P, stage, L, j0, X.r0, min(wt, X.r1 - X.r0));
        cp_async_commit();
        for (uint32_t t = 0; t < ntiles; t++) {
            uint32_t const i0 = X.r0 + t * wt;
            uint32_t const rows = min(wt, X.r1 - i0);
            if (t + 1 < ntiles) stage_H<KS>(P, stage + ((t + 1) & 1) * half, L, j0, i0 + wt, min(wt, X.r1 - i0 - wt));
            cp_async_commit();
            cp_async_wait1();
            __syncthreads();
            const float *sV = stage + (t & 1) * half;
            const float *sW = sV + wt * L.cs;
            if (active) {
                float tl[K];
#pragma unroll
                for (int c = 0; c < K; c++) tl[c] = 0.0f;
#pragma unroll 4
                for (uint32_t r = 0; r < rows; r++) {
                    float w[K];
                    load_row<K>(sW + r * KS, w);
                    element<K>(sV[r * L.cs + tid], h, w, tl);
                }
#pragma unroll
                for (int c = 0; c < K; c++) acc[c] += tl[c];
            }
            __syncthreads();
        }
        if (active) {
            if (X.size == 1) {
#pragma unroll
                for (int c = 0; c < K; c++) {
                    float const hn = __fdiv_rn(h[c] * acc[c], accW[c]);
                    sH[j * KS + c] = hn;
                    hsum[c] += hn;
                }
            } else {
#pragma unroll
                for (int c = 0; c < K; c++) sm[L.part + j * KS + c] = acc[c];
            }
        }
    }
    if (X.size > 1) {
        cg::this_cluster().sync();   // every CTA's partials are written
        for (uint32_t j = tid; j < m; j += NT)
#pragma unroll
            for (int c = 0; c < K; c++) {
                float const tot = cluster_sum(sm, L.part + j * KS + c, X.size);
                float const hn = __fdiv_rn(sH[j * KS + c] * tot, accW[c]);
                sH[j * KS + c] = hn;
                hsum[c] += hn;
            }
    }
    block_sum<K>(hsum, sm + L.red, sm + L.acch, KS);
}

// update_W: stage V rows [i0, i0+rows) x columns [j0, j0+jt) into buffer b (row stride vst).
__device__ __forceinline__ void stage_W(const Problem &P, float *buf, const SmemLayout &L, uint32_t i0, uint32_t rows,
                                        uint32_t j0)
{
    // jt is a power of two (4..64), so q4 = jt / 4 divides NT: every thread keeps
    // one chunk column q and walks the rows in steps of NT / q4.
    uint32_t const q4 = P.jt / 4, dr = NT / q4;
    uint32_t const q = threadIdx.x & (q4 - 1);
    const float *src = P.V + (size_t)i0 * P.ldv + j0 + 4 * q;
    if (j0 + 4 * q < P.ldv)
        for (uint32_t r = threadIdx.x / q4; r < rows; r += dr) cp_async16(buf + r * L.vst + 4 * q, src + (size_t)r * P.ldv);
}

template <int K>
__device__ void update_W(const Problem &P, float *sm, const SmemLayout &L, bool adjust, const Slice &X)
{
    constexpr uint32_t KS = ks_of(K);
    const float *sH = sm + L.h;
    float *stage = sm + L.stage;
    uint32_t const half = (L.hbuf > L.wbuf ? L.hbuf : L.wbuf);
    const float *accH = sm + L.acch;
    uint32_t const tid = threadIdx.x, m = P.m, jt = P.jt;
    uint32_t const ntiles = (m + jt - 1) / jt;
    float wsum[K];
#pragma unroll
    for (int c = 0; c < K; c++) wsum[c] = 0.0f;
    for (uint32_t i0 = X.r0; i0 < X.r1; i0 += NT) {
        uint32_t const i = i0 + tid;
        bool const active = i < X.r1;
        uint32_t const rows = min((uint32_t)NT, X.r1 - i0);
        float w[K], aux[K];
#pragma unroll
        for (int c = 0; c < K; c++) {
            w[c] = active ? __ldcg(P.W + (size_t)i * KS + c) : 0.0f;
            aux[c] = 0.0f;
        }
        __syncthreads();   // the staging region may still be read by the previous phase
        stage_W(P, stage, L, i0, rows, 0);
        cp_async_commit();
        for (uint32_t t = 0; t < ntiles; t++) {
            uint32_t const j0 = t * jt;
            uint32_t const cols = min(jt, m - j0);
            if (t + 1 < ntiles) stage_W(P, stage + ((t + 1) & 1) * half, L, i0, rows, j0 + jt);
            cp_async_commit();
            cp_async_wait1();
            __syncthreads();
            if (active) {
                const float *vrow = stage + (t & 1) * half + tid * L.vst;
                float tl[K];
#pragma unroll
                for (int c = 0; c < K; c++) tl[c] = 0.0f;
                uint32_t const cols4 = cols & ~3u;
                const float *hrow = sH + j0 * KS;
                for (uint32_t jj = 0; jj < cols4; jj += 4) {
                    float4 const v4 = *reinterpret_cast<const float4 *>(vrow + jj);
                    float hj[K];
                    load_row<K>(hrow + (jj + 0) * KS, hj);
                    element<K>(v4.x, w, hj, tl);
                    load_row<K>(hrow + (jj + 1) * KS, hj);
                    element<K>(v4.y, w, hj, tl);
                    load_row<K>(hrow + (jj + 2) * KS, hj);
                    element<K>(v4.z, w, hj, tl);
                    load_row<K>(hrow + (jj + 3) * KS, hj);
                    element<K>(v4.w, w, hj, tl);
                }
                for (uint32_t jj = cols4; jj < cols; jj++) {
                    float hj[K];
                    load_row<K>(hrow + jj * KS, hj);
                    element<K>(vrow[jj], w, hj, tl);
                }
#pragma unroll
                for (int c = 0; c < K; c++) aux[c] += tl[c];
            }
            __syncthreads();
        }
        if (active) {
#pragma unroll
            for (int c = 0; c < K; c++) {
                float wn = __fdiv_rn(w[c] * aux[c], accH[c]);
                if (adjust) wn = fmaxf(wn, FLT_MIN);
                P.W[(size_t)i * KS + c] = wn;
                wsum[c] += wn;
            }
        }
    }
    colsum_W<K>(wsum, sm, L, X);
}

// Warp-per-sample classification of H with the reference's tie rule (k <= 32:
// lane t holds column t, idle lanes hold (-1, 0); xor butterfly 16..1, a lane
// takes the other value only if it is strictly larger).  With `adjust`, H is
// first clamped to FLT_MIN (the test's matrix_adjust).  Records first[label].
template <int K>
__device__ void classify(float *sm, const SmemLayout &L, uint32_t m, bool adjust)
{
    constexpr uint32_t KS = ks_of(K);
    float *sH = sm + L.h;
    uint32_t *lab = reinterpret_cast<uint32_t *>(sm + L.lab);
    uint32_t *first = reinterpret_cast<uint32_t *>(sm + L.first);
    uint32_t const lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t j = warp; j < m; j += NW) {
        float v = -1.0f;
        uint32_t id = 0;
        if (lane < (uint32_t)K) {
            float x = sH[j * KS + lane];
            if (adjust) {
                x = fmaxf(x, FLT_MIN);
                sH[j * KS + lane] = x;
            }
            v = x;
            id = lane;
        }
#pragma unroll
        for (uint32_t half = 16; half > 0; half >>= 1) {
            float const ov = __shfl_xor_sync(0xffffffffu, v, half);
            uint32_t const oi = __shfl_xor_sync(0xffffffffu, id, half);
            if (v < ov) {
                v = ov;
                id = oi;
            }
        }
        if (lane == 0) {
            lab[j] = id;
            atomicMin(&first[id], j);
        }
    }
    __syncthreads();
}

template <int K>
__device__ void run_problem(Problem &P, float *sm, uint32_t *s_ctl, const Slice &X)
{
    constexpr uint32_t KS = ks_of(K);
    SmemLayout const L = smem_layout(P.m, KS, P.wt, P.jt, P.ldv);
    uint32_t const tid = threadIdx.x, m = P.m;
    uint32_t *lab = reinterpret_cast<uint32_t *>(sm + L.lab);
    uint32_t *rep = reinterpret_cast<uint32_t *>(sm + L.rep);
    uint32_t *first = reinterpret_cast<uint32_t *>(sm + L.first);
    // s_ctl[0] = inc, [1] = converged, [2] = tests

    {
        const float4 *src = reinterpret_cast<const float4 *>(P.H);
        float4 *dst = reinterpret_cast<float4 *>(sm + L.h);
        for (uint32_t e = tid; e < m * KS / 4; e += NT) dst[e] = __ldcg(src + e);
    }
    for (uint32_t j = tid; j < m; j += NT) rep[j] = 0u;   // the first test compares with an all-zero vector
    if (tid < 32) first[tid] = 0xffffffffu;
    if (tid == 0) {
        s_ctl[0] = 0;
        s_ctl[1] = 0;
        s_ctl[2] = 0;
    }
    {   // colsum(W) of the initial W
        float ws[K];
#pragma unroll
        for (int c = 0; c < K; c++) ws[c] = 0.0f;
        for (uint32_t i = X.r0 + tid; i < X.r1; i += NT)
#pragma unroll
            for (int c = 0; c < K; c++) ws[c] += __ldcg(P.W + (size_t)i * KS + c);
        __syncthreads();
        colsum_W<K>(ws, sm, L, X);
    }

    uint32_t const J = P.niter_test_conv;
    uint32_t const nblocks = P.n_iters / J, rem = P.n_iters % J;
    for (uint32_t b = 0; b < nblocks; b++) {
        for (uint32_t it = 0; it < J; it++) {
            update_H<K>(P, sm, L, X);
            update_W<K>(P, sm, L, it + 1 == J, X);
        }
        classify<K>(sm, L, m, true);
        uint32_t local = 0;
        for (uint32_t j = tid; j < m; j += NT) {
            uint32_t const r = first[lab[j]];
            local |= (r != rep[j]) ? 1u : 0u;
            rep[j] = r;
        }
        int const any = __syncthreads_or((int)local);
        if (tid < 32) first[tid] = 0xffffffffu;
        if (tid == 0) {
            s_ctl[2] += 1;
            if (any)
                s_ctl[0] = 0;
            else if (s_ctl[0] < P.stop_threshold)
                s_ctl[0] += 1;
            else
                s_ctl[1] = 1;
        }
        __syncthreads();
        if (X.size > 1) {
            // Every CTA of the cluster holds the same H and labels, so their stop
            // decisions agree; still, take rank 0's, so that the cluster barriers
            // of the next iteration are reached by all CTAs or by none.  The
            // second barrier keeps rank 0 from changing s_ctl before the others
            // have read it.
            cg::cluster_group const cl = cg::this_cluster();
            cl.sync();
            uint32_t const stop0 = *cl.map_shared_rank(&s_ctl[1], 0u);
            cl.sync();
            if (tid == 0) s_ctl[1] = stop0;
            __syncthreads();
        }
        if (s_ctl[1]) break;
    }
    if (!s_ctl[1])
        for (uint32_t it = 0; it < rem; it++) {
            update_H<K>(P, sm, L, X);
            update_W<K>(P, sm, L, false, X);
        }
    // final classification (no adjust) and write-back (every CTA of a cluster
    // holds the same H and labels; rank 0 writes them)
    classify<K>(sm, L, m, false);
    if (X.rank == 0) {
        for (uint32_t j = tid; j < m; j += NT) P.labels[j] = lab[j];
        const float4 *src = reinterpret_cast<const float4 *>(sm + L.h);
        float4 *dst = reinterpret_cast<float4 *>(P.H);
        for (uint32_t e = tid; e < m * KS / 4; e += NT) dst[e] = src[e];
    }
    if (tid == 0) {
        P.converged = s_ctl[1];
        P.tests = s_ctl[2];
        P.iterations = s_ctl[1] ? s_ctl[2] * J : P.n_iters;
    }
    __syncthreads();
}

}  // namespace
