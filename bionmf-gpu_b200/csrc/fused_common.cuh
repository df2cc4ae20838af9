// fused_common.cuh -- tcgen05 / TMA / mbarrier helpers shared by the fused
// half-iteration kernels (FP32 3xTF32 arm in kernels_fused.cu, BF16 arms in
// kernels_bf16.cu).  Every wait is bounded (WAIT_LIMIT_NS of %globaltimer).
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace nmfb_tc {

constexpr int BO = 128;          // output rows per CTA = TMEM lanes
constexpr uint32_t TMEM_COLS = 512;
constexpr int SMEM_LIMIT = 232448; // max dynamic shared memory per block on sm_100
constexpr unsigned long long WAIT_LIMIT_NS = 1000000000ull;

// How a half-iteration's tiles are dealt out.  Tile g is reduction tile g % tb
// of row block g / tb (BO output rows); CTA b takes tiles [b tpc, (b + 1) tpc).
// A row block's sum is then spread over the CTAs first(ob) .. last(ob); each
// writes a partial at the end of its run and every `run` reduction tiles (a
// chain of FP32 additions no longer than that), and k_finish adds the partials
// in tile order: a fixed order for given sizes and SM count.
struct TileSplit {
    uint32_t tb, total, tpc;   // tiles per row block, of all row blocks, per CTA
    uint32_t run;              // longest sum of tiles in one partial
    uint32_t slots;            // most partials of a row block
    __host__ __device__ uint32_t ctas() const { return (total + tpc - 1) / tpc; }
    __host__ __device__ uint32_t first(uint32_t ob) const { return ob * tb / tpc; }
    __host__ __device__ uint32_t last(uint32_t ob) const { return (ob * tb + tb - 1) / tpc; }
    // Partial that CTA b's sum of row block ob up to reduction tile c goes to, and the
    // number of them.  A CTA's tiles that start on a multiple of `run` (not 0) leave
    // the slot before their first one unused; the CTA writes zeros there.
    __host__ __device__ uint32_t slot(uint32_t ob, uint32_t b, uint32_t c) const { return c / run + (b - first(ob)); }
    __host__ __device__ uint32_t nslot(uint32_t ob) const { return slot(ob, last(ob), tb - 1) + 1; }
};

// Equal runs of tiles for `sms` CTAs.  With few tiles per CTA the runs are made
// longer where that saves k_finish more than it costs here: k_finish reads the
// partials of a row eight at a time, about 0.8 tile times a batch (0.8 us).
// Sums of 128 tiles where the partials of all O rows fit `part_rows` rows,
// longer ones otherwise (one partial per CTA and row block always fits:
// slots <= sms / row blocks + 3).
inline TileSplit plan_tiles(uint32_t O, uint32_t R, uint32_t br, uint32_t sms, size_t part_rows)
{
    TileSplit s;
    uint32_t const oblocks = (O + BO - 1) / BO;
    s.tb = (R + br - 1) / br;
    s.total = oblocks * s.tb;
    auto const slots = [&](uint32_t tpc) {
        uint32_t const most = (s.tb - 1) / tpc + 2;   // CTAs of a row block that starts inside a run
        return (most < s.tb ? most : s.tb) + (s.tb - 1) / s.run;
    };
    s.run = 128;
    uint32_t const even = (s.total + sms - 1) / sms;
    s.tpc = even;
    uint32_t best = 0xffffffffu;
    for (uint32_t tpc = even; tpc <= even + 8 && tpc <= s.tb; tpc++) {
        uint32_t const cost = 10 * tpc + 8 * ((slots(tpc) + 7) / 8);   // tenths of a tile time
        if (cost < best) {
            best = cost;
            s.tpc = tpc;
        }
    }
    while ((size_t)slots(s.tpc) * O > part_rows && s.run < s.tb) s.run *= 2;
    s.slots = slots(s.tpc);
    return s;
}

// Programmatic dependent launch: a kernel launched by launch_chained starts as
// soon as every CTA of the kernel before it has called chain_next (or left),
// and runs up to its own chain_wait, which returns when that kernel -- and so,
// each kernel of the chain waiting for the one before, all earlier work -- has
// completed and its writes are visible.  Every thread that reads or writes
// global memory calls chain_wait first, and what the kernel just before wrote is
// read through L2.  It hides a launch and the prologue
// (barriers, tensor-memory allocation), about 2 us a launch.  Not for a launch behind
// a long kernel that calls chain_next early: while it waits, other streams' kernels do
// not start (see fin_launch).
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_chained(void (*kern)(P...), dim3 grid, uint32_t block, size_t smem, cudaStream_t stream, A &&...args)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

// Column sums of a factor.  k_finish leaves one FP64 partial per CTA and column
// (cs[block][KP]); the next half-iteration's main kernel, which runs long before
// anything divides by the sums, adds them with its V producer's warp: CTA b takes
// columns b, b + gridDim.x, ... once its V loads are issued; lane l adds blocks l, l + 32, ... in order, then
// a shuffle tree.
struct ColSum {
    const double *cs;
    uint32_t nblk;
    float *acc;   // [KP]
};
template <int KP>
__device__ __forceinline__ void column_sums(const ColSum &a)
{
    uint32_t const lane = threadIdx.x % 32;
    for (uint32_t c = blockIdx.x; c < (uint32_t)KP; c += gridDim.x) {
        double t = 0.0;
        for (uint32_t b = lane; b < a.nblk; b += 32 * 8) {   // eight loads in flight
            double v[8];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = b + 32 * i < a.nblk ? __ldcg(a.cs + (size_t)(b + 32 * i) * KP + c) : 0.0;
#pragma unroll
            for (int i = 0; i < 8; i++) t += v[i];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
        if (lane == 0) a.acc[c] = (float)t;
    }
}

// PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Non-blocking probe of a phase (mbarrier.test_wait never suspends the thread).
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// L2 eviction policies for TMA loads: the streamed V evict-first, the small
// factor operands (re-read by every output block) evict-last.
__device__ __forceinline__ uint64_t policy_evict_first()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ uint64_t policy_evict_last()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Bounded wait: false once `limit_ns` of %globaltimer pass (the wait then sets
// the CTA's abort flag and records `code` in the error word) or when another
// role already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag,
                                          uint32_t *err, uint32_t code, unsigned long long limit_ns)
{
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long const t0 = globaltimer();
    while (!mbar_try_wait(bar, parity)) {
        if (*abort_flag) return false;
        if (globaltimer() - t0 > limit_ns) {
            *abort_flag = 1;
            atomicExch(err, code);
            return false;
        }
    }
    return true;
}

// Time limit of a polling loop: expired() is called once per fruitless poll and
// reset() whenever the loop got on.  %globaltimer is read every 64th fruitless
// poll only (every one for limits below 10 us): in the MMA issuer's loop a read
// per tile costs as much as issuing MMAs.
struct PollLimit {
    unsigned long long limit, t0;
    uint32_t polls, mask;
    __device__ __forceinline__ explicit PollLimit(unsigned long long limit_ns)
        : limit(limit_ns), t0(0), polls(0), mask(limit_ns < 10000 ? 0u : 63u)
    {
    }
    __device__ __forceinline__ void reset() { polls = 0; }
    __device__ __forceinline__ bool expired()
    {
        if (++polls & mask) return false;
        unsigned long long const now = globaltimer();
        if (polls == mask + 1) t0 = now;
        return now - t0 > limit;
    }
};

// Drain wait, used after a role has stopped (normally or on abort): waits for
// a phase of asynchronous work this thread issued itself (a TMA load's
// complete_tx, an MMA commit) to land, ignoring the abort flag, for at most
// WAIT_LIMIT_NS.  Nothing of the CTA may still be written by the async proxy
// when it frees its tensor memory and exits.
__device__ __forceinline__ bool mbar_drain(uint64_t *bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long const t0 = globaltimer();
    while (!mbar_try_wait(bar, parity))
        if (globaltimer() - t0 > WAIT_LIMIT_NS) return false;
    return true;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y,
                                            uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// Drain of every tcgen05.mma the calling thread has issued: one more commit
// (it arrives once all earlier MMAs of this thread have completed) on a
// barrier used for nothing else, then a drain wait on it.
__device__ __forceinline__ void mma_drain(uint64_t *bar)
{
    tc_commit(bar);
    mbar_drain(bar, 0);
}

// The MMA issuer runs as a whole warp on warp-uniform values and only the MMAs
// and commits themselves are left to one elected lane (always the same one):
// tcgen05.mma takes its descriptors and addresses from uniform registers, and
// an issuer that had branched to a single lane first spent more time moving
// operands there, one by one, than the tensor core on the MMAs (a tile's 20
// MMAs took about 2000 cycles to issue, against 1020 to execute).
__device__ __forceinline__ bool elect_one()
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}
// Warp-wide probe and bounded wait of a phase (as mbar_wait).  Every branch of
// the wait is on a vote, so the lanes leave it together: the .aligned tensor-
// memory instructions that follow need a converged warp, and lanes that left a
// wait one by one need not be (a vote after the wait does not converge them).
__device__ __forceinline__ bool mbar_test_warp(uint64_t *bar, uint32_t parity)
{
    return __all_sync(0xffffffffu, mbar_test(bar, parity));
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag,
                                               uint32_t *err, uint32_t code, unsigned long long limit_ns)
{
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    PollLimit limit(limit_ns);
    for (;;) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        bool const stop = *abort_flag != 0, late = limit.expired();
        if (__any_sync(0xffffffffu, stop || late)) {
            if (!stop && threadIdx.x % 32 == 0) {
                *abort_flag = 1;
                atomicExch(err, code);
            }
            return false;
        }
    }
}
// A value that is the same in all lanes, in a uniform register.
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __reduce_max_sync(0xffffffffu, x); }

// Shared-memory descriptor with its start address moved on by `off` 16-byte units
// (no carry out of the address field: every operand lies below 256 KB).
__device__ __forceinline__ uint64_t desc_at(uint64_t base, uint32_t off)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"((uint32_t)base + off), "r"((uint32_t)(base >> 32)));
    return d;
}

// D (tensor memory) = or += A (tensor memory) x B (shared memory), kind::tf32.
template <bool ACC>
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "n"(ACC ? 1 : 0)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
            taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// tcgen05.wait::ld that also ties the loaded registers to the wait, so that no use of
// them can be scheduled before the load has completed.
__device__ __forceinline__ void tmem_wait_ld_dep(uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.wait::ld.sync.aligned;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
        :
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 1/x with rcp.approx.ftz.f32 (PTX: at most 1 ulp of error over the full range).
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Round to TF32 (10 mantissa bits), to nearest with ties away from zero, in
// two integer operations; equal to cvt.rna.tf32.f32 for finite inputs.
__device__ __forceinline__ float tf32_rna(float x)
{
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading / stride
// byte offsets (16-byte units), version 1, swizzle layout in bits 61-63.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout)
{
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)layout << 61;
    return d;
}

// kind::f16 instruction descriptor with BF16 A and B (K-major) and FP32 D.
__host__ __device__ constexpr uint32_t idesc_bf16xf32(uint32_t M, uint32_t N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

// D = or += A B, kind::f16, with A from tensor memory (two BF16 per 32-bit column, the
// lower K index in the low half) and B from shared memory.
template <bool ACC>
__device__ __forceinline__ void mma_ts_bf16(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "n"(ACC ? 1 : 0)
        : "memory");
}

// Instruction descriptor for kind::tf32 with FP32 accumulation, A K-major.
__host__ __device__ constexpr uint32_t idesc_tf32(uint32_t M, uint32_t N, uint32_t b_mn_major)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | (b_mn_major << 16) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

}  // namespace nmfb_tc
