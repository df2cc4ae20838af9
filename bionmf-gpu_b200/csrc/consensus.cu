// consensus.cu -- exact integer consensus matrices and the FP64 cophenetic
// correlation of each rank's restarts (nmfb_batch_consensus).
#include "nmfb_internal.cuh"

#include <math.h>

namespace {

// ---------------------------------------------------------------------------
// Consensus: C[a][b] = number of runs r in `sel` with labels_r[a] == labels_r[b]
// (exact integer co-clustering counts).  One CTA per row a.
__global__ void k_consensus(const uint32_t *const *__restrict__ labels, const uint32_t *__restrict__ sel, uint32_t nsel,
                            uint32_t m, uint32_t *__restrict__ C)
{
    uint32_t const a = blockIdx.x;
    for (uint32_t b = threadIdx.x; b < m; b += blockDim.x) {
        uint32_t cnt = 0;
        for (uint32_t s = 0; s < nsel; s++) {
            const uint32_t *l = labels[sel[s]];
            cnt += (l[a] == l[b]) ? 1u : 0u;
        }
        C[(size_t)a * m + b] = cnt;
    }
}

__device__ __forceinline__ double consensus_distance(uint32_t c, double runs)
{
    return __dsub_rn(1.0, __ddiv_rn((double)c, runs));
}

// Cophenetic correlation (Brunet et al., PNAS 2004) of the consensus C over
// nruns runs, in FP64, one CTA of 1024 threads:
//   D = 1 - C / nruns (zero diagonal);
//   average-linkage (UPGMA) agglomeration: repeatedly merge the two active
//   clusters at the smallest distance, the lowest (a, b) slot pair first on
//   ties; the merged cluster keeps slot a and its distance to x becomes
//   (|a| D[a][x] + |b| D[b][x]) / (|a| + |b|); the cophenetic distance of two
//   samples is the height at which their clusters merge;
//   result = Pearson correlation of D and the cophenetic distances over all
//   pairs a < b (means first, then centred sums).
// Work buffers (global): Dw (m*m), coph (m*m), nnd and height (m each); csize,
// nnb, into, when (m each).
//
// Bound by its chain of m - 1 merges, each a few block-wide steps.  Every active
// slot a keeps its nearest slot b > a (the lowest b on ties), so a merge finds the
// smallest pair among m entries; afterwards only the rows whose nearest slot was
// one of the merged two are scanned again, a warp each.  Where two samples' slots
// meet is read off the merge steps at the end.  (Scanning all pairs twice in every
// merge, for the minimum and for the cophenetic distances, took 5.0 ms at m = 200.)
__global__ void __launch_bounds__(1024) k_cophenetic(const uint32_t *__restrict__ C, uint32_t m, uint32_t nruns,
                                                     double *__restrict__ Dw, double *__restrict__ coph, double *nnd,
                                                     double *height, uint32_t *csize, uint32_t *nnb, uint32_t *into,
                                                     uint32_t *when, double *__restrict__ out)
{
    __shared__ double s_d[32];
    __shared__ uint32_t s_a[32];
    __shared__ uint32_t s_scan[1024], s_nscan;
    __shared__ double s_r[3][1024];
    uint32_t const tid = threadIdx.x, nt = blockDim.x, lane = tid % 32, warp = tid / 32;
    double const runs = (double)nruns;
    size_t const mm = (size_t)m * m;
    for (size_t e = tid; e < mm; e += nt) {
        uint32_t const a = (uint32_t)(e / m), b = (uint32_t)(e % m);
        Dw[e] = (a == b) ? 0.0 : consensus_distance(C[e], runs);
    }
    for (uint32_t a = tid; a < m; a += nt) {
        csize[a] = 1;
        when[a] = 0xffffffffu;
    }
    __syncthreads();
    // nearest active slot b > a (lowest on ties) of row a, by one warp
    auto const scan = [&](uint32_t a) {
        double best = INFINITY;
        uint32_t bb = 0xffffffffu;
        for (uint32_t b = a + 1 + lane; b < m; b += 32)
            if (csize[b]) {
                double const d = Dw[(size_t)a * m + b];
                if (d < best) {
                    best = d;
                    bb = b;
                }
            }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            double const od = __shfl_xor_sync(0xffffffffu, best, off);
            uint32_t const ob = __shfl_xor_sync(0xffffffffu, bb, off);
            if (od < best || (od == best && ob < bb)) {
                best = od;
                bb = ob;
            }
        }
        if (lane == 0) {
            nnd[a] = best;
            nnb[a] = bb;
        }
    };
    for (uint32_t a = warp; a < m; a += nt / 32) scan(a);
    __syncthreads();
    for (uint32_t step = 0; step + 1 < m; step++) {
        // the smallest pair: over the active slots, the lowest slot on ties
        double best = INFINITY;
        uint32_t ba = 0xffffffffu;
        for (uint32_t a = tid; a < m; a += nt)
            if (csize[a] && nnd[a] < best) {
                best = nnd[a];
                ba = a;
            }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            double const od = __shfl_xor_sync(0xffffffffu, best, off);
            uint32_t const oa = __shfl_xor_sync(0xffffffffu, ba, off);
            if (od < best || (od == best && oa < ba)) {
                best = od;
                ba = oa;
            }
        }
        if (lane == 0) {
            s_d[warp] = best;
            s_a[warp] = ba;
        }
        if (tid == 0) s_nscan = 0;
        __syncthreads();
        best = s_d[lane];
        ba = s_a[lane];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            double const od = __shfl_xor_sync(0xffffffffu, best, off);
            uint32_t const oa = __shfl_xor_sync(0xffffffffu, ba, off);
            if (od < best || (od == best && oa < ba)) {
                best = od;
                ba = oa;
            }
        }
        uint32_t const A = ba, B = nnb[A];
        double const na = (double)csize[A], nb = (double)csize[B];
        __syncthreads();   // every thread has read the slots that change below
        if (tid == 0) {
            csize[A] += csize[B];
            csize[B] = 0;
            into[B] = A;
            when[B] = step;
            height[step] = best;
        }
        for (uint32_t x = tid; x < m; x += nt) {
            if (x == A) {
                uint32_t const q = atomicAdd(&s_nscan, 1u);
                if (q < 1024u) s_scan[q] = A;
            }
            if (x == A || x == B || !csize[x]) continue;
            double const d = __ddiv_rn(__dadd_rn(__dmul_rn(na, Dw[(size_t)A * m + x]), __dmul_rn(nb, Dw[(size_t)B * m + x])),
                                       __dadd_rn(na, nb));
            Dw[(size_t)A * m + x] = d;
            Dw[(size_t)x * m + A] = d;
            uint32_t const n = nnb[x];
            if (n == B || n == A) {   // (n == A only where x < A)
                uint32_t const q = atomicAdd(&s_nscan, 1u);
                if (q < 1024u) s_scan[q] = x;
            } else if (x < A && (d < nnd[x] || (d == nnd[x] && A < n))) {
                nnd[x] = d;
                nnb[x] = A;
            }
        }
        __syncthreads();
        if (s_nscan <= 1024u)
            for (uint32_t q = warp; q < s_nscan; q += nt / 32) scan(s_scan[q]);
        else   // more rows than the list holds: all of them
            for (uint32_t a = warp; a < m; a += nt / 32)
                if (csize[a]) scan(a);
        __syncthreads();
    }
    // Cophenetic distances: slot b was absorbed at step when[b] by slot into[b] (a
    // slot is its first sample); of two samples' slots the one absorbed first moves
    // on to its absorber until they meet.
    for (size_t e = tid; e < mm; e += nt) {
        uint32_t a = (uint32_t)(e / m), b = (uint32_t)(e % m), last = 0;
        double h = 0.0;
        if (a < b) {
            while (a != b) {
                bool const fa = when[a] < when[b];
                last = fa ? when[a] : when[b];
                if (fa)
                    a = into[a];
                else
                    b = into[b];
            }
            h = height[last];
        }
        coph[e] = h;   // (only a < b is read)
    }
    __syncthreads();
    // Pearson correlation over a < b: means, then centred sums.
    double const np = (double)m * (double)(m - 1) / 2.0;
    double sx = 0.0, sy = 0.0;
    for (size_t e = tid; e < mm; e += nt) {
        uint32_t const a = (uint32_t)(e / m), b = (uint32_t)(e % m);
        if (a < b) {
            sx += consensus_distance(C[e], runs);
            sy += coph[e];
        }
    }
    s_r[0][tid] = sx;
    s_r[1][tid] = sy;
    __syncthreads();
    for (uint32_t s = nt / 2; s > 0; s >>= 1) {
        if (tid < s) {
            s_r[0][tid] += s_r[0][tid + s];
            s_r[1][tid] += s_r[1][tid + s];
        }
        __syncthreads();
    }
    double const mx = s_r[0][0] / np, my = s_r[1][0] / np;
    __syncthreads();
    double cxy = 0.0, cxx = 0.0, cyy = 0.0;
    for (size_t e = tid; e < mm; e += nt) {
        uint32_t const a = (uint32_t)(e / m), b = (uint32_t)(e % m);
        if (a < b) {
            double const x = consensus_distance(C[e], runs) - mx;
            double const y = coph[e] - my;
            cxy += x * y;
            cxx += x * x;
            cyy += y * y;
        }
    }
    s_r[0][tid] = cxy;
    s_r[1][tid] = cxx;
    s_r[2][tid] = cyy;
    __syncthreads();
    for (uint32_t s = nt / 2; s > 0; s >>= 1) {
        if (tid < s)
            for (int q = 0; q < 3; q++) s_r[q][tid] += s_r[q][tid + s];
        __syncthreads();
    }
    if (tid == 0) out[0] = (s_r[1][0] > 0.0 && s_r[2][0] > 0.0) ? s_r[0][0] / sqrt(s_r[1][0] * s_r[2][0]) : 0.0;
}

}  // namespace

size_t nmfb_summary_doubles(uint32_t m) { return 2 * (size_t)m * m + 2 * (size_t)m + 1; }
size_t nmfb_summary_ints(uint32_t m) { return 4 * (size_t)m; }

cudaError_t nmfb_launch_consensus(const uint32_t *const *labels, const uint32_t *sel, uint32_t nsel, uint32_t m,
                                  uint32_t *C, cudaStream_t stream)
{
    k_consensus<<<m, 256, 0, stream>>>(labels, sel, nsel, m, C);
    return cudaGetLastError();
}

cudaError_t nmfb_launch_cophenetic(const uint32_t *C, uint32_t m, uint32_t nruns, double *dbl, uint32_t *ints,
                                   double **result, cudaStream_t stream)
{
    size_t const mm = (size_t)m * m;
    double *const out = dbl + 2 * mm + 2 * (size_t)m;
    k_cophenetic<<<1, 1024, 0, stream>>>(C, m, nruns, dbl, dbl + mm, dbl + 2 * mm, dbl + 2 * mm + m, ints, ints + m,
                                         ints + 2 * (size_t)m, ints + 3 * (size_t)m, out);
    *result = out;
    return cudaGetLastError();
}
