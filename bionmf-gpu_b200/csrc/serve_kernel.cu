// serve_kernel.cu -- the device-side serving queue's persistent kernel.
#include "batch_run.cuh"

namespace {

__device__ __forceinline__ unsigned long long device_clock_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr uint32_t NO_TICKET = 0xffffffffu;

// Serving: requests are published one at a time into a ring of `capacity`
// descriptors while the kernel runs (the host copies a request's data and
// descriptor, then the new published count, in that order on one stream).
// A cluster's rank 0 claims the next published ticket with a compare-and-swap
// on `taken`, waiting at most idle_ns for one; after that, or once `closing`
// is set, the cluster leaves, and the host launches the kernel again when
// more work is published.  Every wait is bounded by idle_ns.  A finished
// problem's W, H and labels are in device memory before its completion record
// (host-mapped memory) is written: iterations, converged, tests, then the
// ticket + 1 after a system-scope fence.
__global__ void __launch_bounds__(NT, 2) k_serve(const Problem *__restrict__ ring, uint32_t capacity,
                                                 uint32_t *taken, const volatile uint32_t *published,
                                                 const volatile uint32_t *closing, volatile uint32_t *done,
                                                 unsigned long long idle_ns)
{
    extern __shared__ float4 smem4[];
    float *sm = reinterpret_cast<float *>(smem4);
    __shared__ uint32_t s_next;
    __shared__ uint32_t s_ctl[4];
    cg::cluster_group const cl = cg::this_cluster();
    uint32_t const crank = cl.block_rank(), csize = cl.num_blocks();
    for (;;) {
        __syncthreads();
        if (crank == 0 && threadIdx.x == 0) {
            uint32_t got = NO_TICKET;
            unsigned long long const t0 = device_clock_ns();
            for (;;) {
                uint32_t const t = *(volatile uint32_t *)taken;
                if (t < *published) {
                    if (atomicCAS(taken, t, t + 1u) == t) {
                        got = t;
                        break;
                    }
                    continue;
                }
                if (*closing || device_clock_ns() - t0 > idle_ns) break;
                __nanosleep(2000);
            }
            s_next = got;
        }
        uint32_t q;
        if (csize > 1) {
            cl.sync();
            q = *cl.map_shared_rank(&s_next, 0u);
            cl.sync();
        } else {
            __syncthreads();
            q = s_next;
        }
        if (q == NO_TICKET) break;
        uint32_t const slot = q % capacity;
        // the descriptor was written by a host copy: read it through L2
        Problem P;
        {
            const uint2 *src = reinterpret_cast<const uint2 *>(ring + slot);
            uint2 *dst = reinterpret_cast<uint2 *>(&P);
#pragma unroll
            for (uint32_t w = 0; w < sizeof(Problem) / sizeof(uint2); w++) dst[w] = __ldcg(src + w);
        }
        uint32_t const chunk = (P.n + csize - 1) / csize;
        Slice const X{crank, csize, min(P.n, crank * chunk), min(P.n, crank * chunk + chunk)};
        switch (P.k) {
#define NMFB_SERVE_CASE(KK) \
    case KK: run_problem<KK>(P, sm, s_ctl, X); break;
            NMFB_SERVE_CASE(2) NMFB_SERVE_CASE(3) NMFB_SERVE_CASE(4) NMFB_SERVE_CASE(5) NMFB_SERVE_CASE(6)
            NMFB_SERVE_CASE(7) NMFB_SERVE_CASE(8) NMFB_SERVE_CASE(9) NMFB_SERVE_CASE(10) NMFB_SERVE_CASE(11)
            NMFB_SERVE_CASE(12) NMFB_SERVE_CASE(13) NMFB_SERVE_CASE(14) NMFB_SERVE_CASE(15) NMFB_SERVE_CASE(16)
            NMFB_SERVE_CASE(17) NMFB_SERVE_CASE(18) NMFB_SERVE_CASE(19) NMFB_SERVE_CASE(20)
#undef NMFB_SERVE_CASE
            default: break;
        }
        // every CTA's stores of W (and rank 0's of H and the labels) are done
        __threadfence();
        if (csize > 1)
            cl.sync();
        else
            __syncthreads();
        if (crank == 0 && threadIdx.x == 0) {
            volatile uint32_t *rec = done + 4 * (size_t)slot;
            rec[1] = P.iterations;
            rec[2] = P.converged;
            rec[3] = P.tests;
            __threadfence_system();
            rec[0] = q + 1u;
        }
    }
}

}  // namespace

nmfb_batched::ServeKernel nmfb_batched::serve_kernel() { return k_serve; }
