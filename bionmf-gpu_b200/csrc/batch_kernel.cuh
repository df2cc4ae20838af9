// batch_kernel.cuh -- k_batch; a file of its own per instantiation keeps the
// build parallel (each compiles a dozen ranks of run_problem).
#pragma once

namespace {

// KMAX: the largest rank the instantiation handles (10 or 20).  A batch whose
// ranks are all <= 10 (a rank sweep) runs the 10-rank variant: without the
// k = 11..20 paths in the kernel, its registers are allocated for k <= 10.
template <int KMAX>
__global__ void __launch_bounds__(NT, 2) k_batch(Problem *__restrict__ probs, const uint32_t *__restrict__ order,
                                                 uint32_t nprob, uint32_t *__restrict__ queue)
{
    extern __shared__ float4 smem4[];
    float *sm = reinterpret_cast<float *>(smem4);
    __shared__ uint32_t s_next;
    __shared__ uint32_t s_ctl[4];
    cg::cluster_group const cl = cg::this_cluster();
    uint32_t const crank = cl.block_rank(), csize = cl.num_blocks();
    for (;;) {
        __syncthreads();
        if (crank == 0 && threadIdx.x == 0) s_next = atomicAdd(queue, 1u);
        uint32_t q;
        if (csize > 1) {
            cl.sync();
            q = *cl.map_shared_rank(&s_next, 0u);
            // rank 0 rewrites s_next, and any CTA may leave the kernel, only after
            // every CTA has read it (and, earlier, every partial it needed)
            cl.sync();
        } else {
            __syncthreads();
            q = s_next;
        }
        if (q >= nprob) break;
        Problem P = probs[order[q]];
        uint32_t const chunk = (P.n + csize - 1) / csize;
        Slice const X{crank, csize, min(P.n, crank * chunk), min(P.n, crank * chunk + chunk)};
        switch (P.k) {
#define NMFB_BATCH_CASE(KK) \
    case KK: run_problem<KK>(P, sm, s_ctl, X); break;
            NMFB_BATCH_CASE(2) NMFB_BATCH_CASE(3) NMFB_BATCH_CASE(4) NMFB_BATCH_CASE(5) NMFB_BATCH_CASE(6)
            NMFB_BATCH_CASE(7) NMFB_BATCH_CASE(8) NMFB_BATCH_CASE(9) NMFB_BATCH_CASE(10)
#undef NMFB_BATCH_CASE
            default:
                if (KMAX > 10) {
                    switch (P.k) {
#define NMFB_BATCH_CASE(KK) \
    case KK: run_problem<(KMAX > 10 ? KK : 2)>(P, sm, s_ctl, X); break;
                        NMFB_BATCH_CASE(11) NMFB_BATCH_CASE(12) NMFB_BATCH_CASE(13) NMFB_BATCH_CASE(14)
                        NMFB_BATCH_CASE(15) NMFB_BATCH_CASE(16) NMFB_BATCH_CASE(17) NMFB_BATCH_CASE(18)
                        NMFB_BATCH_CASE(19) NMFB_BATCH_CASE(20)
#undef NMFB_BATCH_CASE
                        default: break;
                    }
                }
                break;
        }
        if (crank == 0 && threadIdx.x == 0) {
            Problem *dst = probs + order[q];
            dst->iterations = P.iterations;
            dst->converged = P.converged;
            dst->tests = P.tests;
        }
    }
}

}  // namespace
