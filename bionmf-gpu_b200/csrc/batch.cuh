// batch.cuh -- descriptors and shared-memory layout of the batched engine
// (batch.cu, batch_kernel*.cu, serve.cu).
#pragma once

#include "nmfb_internal.cuh"

namespace nmfb_batched {

constexpr int NT = 256;
constexpr int NW = NT / 32;
constexpr uint32_t KMIN = 2, KMAX = 20;

struct Problem {
    const float *V;      // n x ldv
    float *W;            // n x ks
    float *H;            // m x ks
    uint32_t *labels;    // m: classification of the final H
    uint64_t ldv;
    uint32_t n, m, k, ks;
    uint32_t wt, jt;     // tile shapes
    uint32_t n_iters, niter_test_conv, stop_threshold;   // the problem's -i, -j, -t
    uint32_t iterations; // out
    uint32_t converged;  // out
    uint32_t tests;      // out: convergence tests performed
};

__host__ __device__ constexpr uint32_t ks_of(uint32_t k) { return (k + 3u) & ~3u; }

// Shared-memory layout of one problem (offsets in floats).  The staging region
// holds two buffers (double buffering) of either phase:
//   update_H: V rows [i0, i0+wt) x columns [j0, j0+cs) (cs = min(NT, ldv)) and
//             W rows [i0, i0+wt) (wt x ks);
//   update_W: V rows [i0, i0+NT) x columns [j0, j0+jt), row stride jt + 4
//             (16-byte aligned rows; float4 reads of 8 consecutive rows hit
//             8 distinct bank groups).
struct SmemLayout {
    uint32_t h, stage, red, accw, acch, lab, rep, first, part, partw, total;
    uint32_t cs, hbuf, wbuf, vst;   // update_H column span and buffer sizes; update_W row stride
};
__host__ __device__ inline SmemLayout smem_layout(uint32_t m, uint32_t ks, uint32_t wt, uint32_t jt, uint64_t ldv)
{
    SmemLayout L;
    L.cs = ldv < (uint64_t)NT ? (uint32_t)ldv : (uint32_t)NT;
    L.hbuf = wt * (L.cs + ks);
    L.vst = jt + 4;
    L.wbuf = NT * L.vst;
    uint32_t const stage = 2u * (L.hbuf > L.wbuf ? L.hbuf : L.wbuf);
    L.h = 0;
    L.stage = (m * ks + 3u) & ~3u;
    L.red = L.stage + stage;
    L.accw = L.red + NW * ks;
    L.acch = L.accw + ks;
    L.lab = L.acch + ks;
    L.rep = L.lab + m;
    L.first = L.rep + m;
    L.part = L.first + 32;                 // this CTA's update_H partials (m x ks), read by the cluster
    L.partw = L.part + ((m * ks + 3u) & ~3u);   // this CTA's partial column sums of W (ks)
    L.total = L.partw + ks;
    return L;
}

using BatchKernel = void (*)(Problem *, const uint32_t *, uint32_t, uint32_t *);
using ServeKernel = void (*)(const Problem *, uint32_t, uint32_t *, const volatile uint32_t *, const volatile uint32_t *,
                             volatile uint32_t *, unsigned long long);
BatchKernel batch_kernel10();   // batch_kernel10.cu: ranks 2..10
BatchKernel batch_kernel20();   // batch_kernel20.cu: ranks 2..20
ServeKernel serve_kernel();     // serve_kernel.cu

// Dynamic shared memory of a problem.
inline size_t problem_smem_bytes(uint32_t m, uint32_t k, uint32_t wt, uint32_t jt)
{
    uint64_t const ldv = ((uint64_t)m + 31) / 32 * 32;
    return (size_t)smem_layout(m, ks_of(k), wt, jt, ldv).total * sizeof(float);
}

}  // namespace nmfb_batched
