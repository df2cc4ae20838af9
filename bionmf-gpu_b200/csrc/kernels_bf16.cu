// kernels_bf16.cu -- the BF16 fused half-iteration arms (NMFB_ARM_BF16,
// NMFB_ARM_SPLIT_BF16 and NMFB_ARM_BF16X3).
//
// Same method and data flow as the FP32 arm (kernels_fused.cu): for 128 rows
// of the factor X being updated and a range of the reduction dimension, each
// 64-row tile of the other factor Y and the matching V tile give
//   D   = X Y^T                      (MMA1, TMEM, FP32 accumulate)
//   R   = V / D                      (R warps, FP32 registers)
//   Acc = R Y                        (MMA2, TMEM, FP32 accumulate)
// and Acc is summed per tile into FP32 registers; k_finish (finish.cuh) then
// applies X = X .* (sum of splits) ./ colsum(Y) and writes X's BF16 copies and
// column sums for the next half-iteration.  What changes is the operand type of
// the two contractions (tcgen05.mma kind::f16, BF16 A and B, K = 16 per
// instruction, FP32 accumulation):
//   NMFB_ARM_BF16       : X, Y, R rounded to BF16 (one product each);
//   NMFB_ARM_SPLIT_BF16 : the WH denominator from a split-BF16 product,
//                         x = xh + xl (xh = BF16(x), xl = BF16(x - xh)),
//                         D = Xh Yh^T + Xh Yl^T + Xl Yh^T (16 significant bits:
//                         small WH entries amplify denominator error in the
//                         quotient); MMA2 stays one BF16 product;
//   NMFB_ARM_BF16X3     : both contractions split, MMA2 = Rh Yh + Rh Yl + Rl Yh
//                         (FP32-class results from BF16 tensor instructions,
//                         K = 16 per instruction against 8 for TF32).
// The quotient, the per-tile sums and the updates stay FP32.  BF16 keeps FP32's
// 8-bit exponent, so a per-column rescaling of the factors would change no
// rounding error and is not applied.
//
// All operands reach shared memory by TMA in the layout the MMA reads: BF16
// hi / lo copies of X and Y (rows x KP, K-major) and, per 64-row block, the
// transposed hi block followed by the transposed lo block (64 rows -> 2 KP rows
// of 64 values) that MMA2 reads K-major -- written by k_finish when the factor
// is updated, or on its own when it is not current (start of a run, after the
// test's EPS adjust of H).  The R warps work in two teams on alternate tiles.
// R replaces D in tensor memory, 16 columns of D becoming 8 of packed Rh and 8 of
// Rl, and is MMA2's A operand there.
//
// Warp roles: 0 = V producer, 1 = MMA issuer / TMEM owner,
// 2 = X and MMA1's Y producer, 3 = MMA2's Y producer, 4..19 (4..11 at
// rank 64) = R warps, the last four (eight) = accumulator warps.
// Persistent like the FP32 arm: every CTA takes an equal run of the list of all
// row blocks' tiles (TileSplit), loading X anew where the run enters a row block.
// Every wait is bounded (1 s); on expiry the kernel records an error word that
// the host turns into NMFB_ETIMEOUT.  No TMA multicast is used.
#include "nmfb_internal.cuh"
#include "fused_common.cuh"
#include "finish.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <float.h>

using nmfb::ConvState;
using namespace nmfb_tc;

namespace {

// D = or += A B, kind::f16, both operands from shared memory.
template <bool ACC>
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "n"(ACC ? 1 : 0)
        : "memory");
}

// MODE 0: BF16 x BF16 in both contractions; 1: split-BF16 WH denominator;
// 2: split-BF16 in both contractions.
template <int KP, int MODE>
struct GeoB {
    static constexpr int BR = 64;                           // reduction rows per tile
    static constexpr int ROWB = 2 * KP;                     // bytes per X / Y row
    static constexpr uint32_t LAYOUT = (KP == 16) ? 6u : (KP == 32) ? 4u : 2u;   // SW32 / SW64 / SW128
    static constexpr int XBYTES = BO * KP * 2;
    static constexpr int YBYTES = BR * KP * 2;              // = KP rows of 128 B: one Y^T part
    static constexpr int YTROWS = (MODE == 2 ? 2 : 1) * KP; // Y^T hi (and lo) rows per tile
    // A ring each for MMA1's and MMA2's Y operands, as in the FP32 kernel.
    static constexpr int Y1STAGE = (MODE >= 1 ? 2 : 1) * YBYTES;   // Yh (| Yl)
    static constexpr int Y2STAGE = YTROWS * 128;            // Y^T
    static constexpr int VBYTES = BO * BR * 4;
    static constexpr int Y1ST = (KP == 64 && MODE == 2) ? 2 : 3, Y2ST = 2;   // (2: room for a fourth V stage)
    static constexpr uint32_t NDB = 4;                      // D buffers in TMEM; R takes D's place
    static constexpr int FIXED = 1024 + 512;
    static constexpr int XALL = (MODE >= 1 ? 2 : 1) * XBYTES, YALL = Y1ST * Y1STAGE + Y2ST * Y2STAGE;
    static constexpr int VAVAIL = (SMEM_LIMIT - FIXED - XALL - YALL) / VBYTES;
    static constexpr int VST = VAVAIL > 6 ? 6 : VAVAIL;
    static_assert(VST >= 3, "shared-memory ring too small");
    // A team takes every other tile, so with an odd ring its uses of a V stage are two phases
    // apart and their parities the same: waiting for tile t it must not meet the stage before
    // tile t - VST (the other team's) has landed in it. D(t) is there only once R(t - NDB) was.
    static_assert(VST % 2 == 0 || VST >= (int)NDB, "vfull's parity would be ambiguous");
    static constexpr int SMEM = FIXED + XALL + YALL + VST * VBYTES;
    static constexpr int NR = (KP == 64) ? 8 : 16;          // R warps
    static constexpr int NA = (KP == 64) ? 2 : 1;           // accumulator warps: sets of four, KP / NA columns each
    static constexpr int NTHR = (4 + NR + 4 * NA) * 32;   // (a multiple of four warps: one more would cost 8 registers a thread)
    static constexpr uint32_t ACCW = (MODE == 2 ? 2 : 1) * KP;   // TMEM columns of one accumulator
    static constexpr uint32_t DB0 = 2 * ACCW;               // Acc[0..1] at 0 and ACCW; D[b] at DB0 + b*BR
    static_assert(DB0 + NDB * BR <= TMEM_COLS, "TMEM columns exceeded");
    static_assert(YBYTES % 1024 == 0 && Y1STAGE % 1024 == 0 && Y2STAGE % 1024 == 0 && XBYTES % 1024 == 0,
                  "1024-byte stage alignment");
};

struct MapsB {
    CUtensorMap v;        // V (FP32), as in the FP32 arm
    CUtensorMap xh, xl;   // X hi / lo (BF16, rows x KP), box [KP x 128]
    CUtensorMap yh, yl;   // Y hi / lo (BF16, rows x KP), box [KP x 64]
    CUtensorMap yt;       // Y^T blocks (BF16, [rows/64][hi, lo][KP][64]), box [64 x KP] or [64 x 2 KP]
};

struct ArgsB {
    uint32_t O, R;
    TileSplit ts;
    ColSum csy;           // column sums of the other factor
    float *part;                 // [slot][O][KP]
    uint32_t *err;
    const ConvState *st;
    unsigned long long wait_ns;  // limit of every bounded wait (%globaltimer ns)
};

template <bool HSIDE, int KP, int MODE>
__global__ void __launch_bounds__(GeoB<KP, MODE>::NTHR, 1)
    k_fused_bf16(const __grid_constant__ MapsB maps, const ArgsB args)
{
    using G = GeoB<KP, MODE>;
    constexpr int BR = G::BR;
    constexpr int NR = G::NR;
    constexpr bool SPLIT = MODE >= 1;                // MMA1 split
    constexpr bool SPLIT2 = MODE == 2;               // MMA2 split
    constexpr int NTERMS = SPLIT ? 3 : 1;

    extern __shared__ unsigned char smem_raw[];
    uint32_t const base_u32 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *const base = smem_raw + (base_u32 - smem_u32(smem_raw));
    unsigned char *const sX = base;                                  // Xh (| Xl)
    unsigned char *const sY1 = sX + G::XALL;                         // [Y1ST][Yh (| Yl)]
    unsigned char *const sY2 = sY1 + G::Y1ST * G::Y1STAGE;           // [Y2ST][Y^T]
    unsigned char *const sV = sY2 + G::Y2ST * G::Y2STAGE;            // [VST][V]
    uint64_t *const bars = reinterpret_cast<uint64_t *>(sV + G::VST * G::VBYTES);
    uint64_t *const vfull = bars;                    // [VST]  TMA -> R warps
    uint64_t *const vempty = vfull + G::VST;         // [VST]  R warps -> V producer
    uint64_t *const y1full = vempty + G::VST;        // [Y1ST] TMA -> MMA1
    uint64_t *const y1empty = y1full + G::Y1ST;      // [Y1ST] MMA1 commit -> Y1 producer
    uint64_t *const y2full = y1empty + G::Y1ST;      // [Y2ST] TMA -> MMA2
    uint64_t *const y2empty = y2full + G::Y2ST;      // [Y2ST] MMA2 commit -> Y2 producer
    uint64_t *const dfull = y2empty + G::Y2ST;       // [NDB]  MMA1 commit -> R warps
    uint64_t *const rfull = dfull + G::NDB;          // [NDB]  R warps -> MMA2
    uint64_t *const accrdy = rfull + G::NDB;         // [2]    MMA2 commit -> accumulator warps
    uint64_t *const accfree = accrdy + 2;            // [2]    accumulator warps -> MMA2
    uint64_t *const xfull = accfree + 2;             // [1]    TMA -> MMA1
    uint64_t *const xfree = xfull + 1;               // [1]    last MMA1 of a row block -> X producer
    uint64_t *const mdrain = xfree + 1;              // [1]    issuer's final commit (drain)
    uint32_t *const tmem_slot = reinterpret_cast<uint32_t *>(mdrain + 1);
    volatile uint32_t *const abort_flag = tmem_slot + 1;

    chain_next();
    uint32_t const warp = uniform(threadIdx.x / 32), lane = threadIdx.x % 32;
    // This CTA's run of tiles [g0, g0 + T) of the (row block, reduction tile) list.
    uint32_t const TB = args.ts.tb;
    uint32_t const g0 = blockIdx.x * args.ts.tpc;
    uint32_t T = min(args.ts.total - g0, args.ts.tpc);
    uint32_t const ob0 = g0 / TB, c00 = g0 - ob0 * TB;

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::VST; s++) {
            mbar_init(&vfull[s], 1);
            mbar_init(&vempty[s], NR / 2);   // one team reads each V tile
        }
        for (int s = 0; s < G::Y1ST; s++) {
            mbar_init(&y1full[s], 1);
            mbar_init(&y1empty[s], 1);
        }
        for (int s = 0; s < G::Y2ST; s++) {
            mbar_init(&y2full[s], 1);
            mbar_init(&y2empty[s], 1);
        }
        for (uint32_t b = 0; b < G::NDB; b++) {
            mbar_init(&dfull[b], 1);
            mbar_init(&rfull[b], NR / 2);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&accrdy[b], 1);
            mbar_init(&accfree[b], 4 * G::NA);
        }
        mbar_init(xfull, 1);
        mbar_init(xfree, 1);
        mbar_init(mdrain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t const tmem = *tmem_slot;
    chain_wait();   // nothing above reads or writes global memory
    if (args.st && *(volatile const uint32_t *)&args.st->converged) T = 0;   // every role's loop is empty

    if (warp == 0) {
        // ------------------------------------------------------------ V producer, then the column sums of Y
        uint32_t issued = 0;
        if (lane == 0) {
            uint64_t const pol = policy_evict_first();
            uint32_t ob = ob0, c = c00;
            for (uint32_t t = 0; t < T; t++, ob += (c + 1 == TB), c = (c + 1 == TB) ? 0 : c + 1) {
                uint32_t const s = t % G::VST;
                if (t >= (uint32_t)G::VST &&
                    !mbar_wait(&vempty[s], ((t / G::VST) - 1) & 1, abort_flag, args.err, 21u, args.wait_ns))
                    break;
                issued = t + 1;
                unsigned char *sv = sV + s * G::VBYTES;
                int const r0 = (int)(c * BR), o0 = (int)(ob * BO);
                mbar_expect_tx(&vfull[s], G::VBYTES);
                if (HSIDE) {
                    tma_load_2d(sv, &maps.v, &vfull[s], o0, r0, pol);          // V[r0:r0+BR][o0:o0+128]
                } else {
#pragma unroll
                    for (int b = 0; b < BR / 32; b++)                          // V[o0:o0+128][r0+32b : +32]
                        tma_load_2d(sv + b * (BO * 128), &maps.v, &vfull[s], r0 + 32 * b, o0, pol);
                }
            }
        }
        __syncwarp();
        if (T > 0) column_sums<KP>(args.csy);   // (while the last tiles are worked on; k_finish divides by them)
        if (lane == 0)
            // drain: the last load into every stage has landed
            for (uint32_t t = issued > (uint32_t)G::VST ? issued - G::VST : 0; t < issued; t++)
                mbar_drain(&vfull[t % G::VST], (t / G::VST) & 1);
    } else if (warp == 2) {
        // ------------------------------------------------------------ X and MMA1's Y producer
        if (lane == 0) {
            uint64_t const pol = policy_evict_last();
            uint32_t issued = 0, xs = 0, c = c00;   // xs: row blocks whose X has been requested
            for (uint32_t t = 0; t < T; t++, c = (c + 1 == TB) ? 0 : c + 1) {
                uint32_t const s = t % G::Y1ST;
                if (t >= (uint32_t)G::Y1ST &&
                    !mbar_wait(&y1empty[s], ((t / G::Y1ST) - 1) & 1, abort_flag, args.err, 22u, args.wait_ns))
                    break;
                issued = t + 1;
                unsigned char *sy = sY1 + s * G::Y1STAGE;
                int const r0 = (int)(c * BR);
                mbar_expect_tx(&y1full[s], G::Y1STAGE);
                tma_load_2d(sy, &maps.yh, &y1full[s], 0, r0, pol);
                if (SPLIT) tma_load_2d(sy + G::YBYTES, &maps.yl, &y1full[s], 0, r0, pol);
                if (t == 0 || c == 0) {   // X of the row block, once MMA1 has read the previous one's
                    if (xs > 0 && !mbar_wait(xfree, (xs - 1) & 1, abort_flag, args.err, 29u, args.wait_ns)) break;
                    int const o0 = (int)((ob0 + xs) * BO);
                    mbar_expect_tx(xfull, G::XALL);
                    tma_load_2d(sX, &maps.xh, xfull, 0, o0, pol);
                    if (SPLIT) tma_load_2d(sX + G::XBYTES, &maps.xl, xfull, 0, o0, pol);
                    xs++;
                }
            }
            // drain: the last X and the last load into every Y stage have landed
            if (xs > 0) mbar_drain(xfull, (xs - 1) & 1);
            for (uint32_t t = issued > (uint32_t)G::Y1ST ? issued - G::Y1ST : 0; t < issued; t++)
                mbar_drain(&y1full[t % G::Y1ST], (t / G::Y1ST) & 1);
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------ MMA2's Y producer
        if (lane == 0) {
            uint64_t const pol = policy_evict_last();
            uint32_t issued = 0, c = c00;
            for (uint32_t t = 0; t < T; t++, c = (c + 1 == TB) ? 0 : c + 1) {
                uint32_t const s = t % G::Y2ST;
                if (t >= (uint32_t)G::Y2ST &&
                    !mbar_wait(&y2empty[s], ((t / G::Y2ST) - 1) & 1, abort_flag, args.err, 30u, args.wait_ns))
                    break;
                issued = t + 1;
                mbar_expect_tx(&y2full[s], G::Y2STAGE);
                tma_load_2d(sY2 + s * G::Y2STAGE, &maps.yt, &y2full[s], 0, (int)(c * 2 * KP), pol);
            }
            for (uint32_t t = issued > (uint32_t)G::Y2ST ? issued - G::Y2ST : 0; t < issued; t++)
                mbar_drain(&y2full[t % G::Y2ST], (t / G::Y2ST) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        //   MMA2(n2): needs R(n2) in tensor memory, its Y operands and, for n2 >= 2,
        //             Acc[n2 % 2] read by the accumulator warps (tile n2-2);
        //   MMA1(n1): needs its Y operands, a free D buffer (n1 < n2 + NDB) and, for the
        //             first tile of a row block, its X; the last one's releases X.
        constexpr uint32_t IDESC1 = idesc_bf16xf32(BO, BR);
        constexpr uint32_t IDESC2 = idesc_bf16xf32(BO, KP);
        constexpr uint32_t IDESC2W = idesc_bf16xf32(BO, 2 * KP);
        uint32_t const y1_u32 = base_u32 + G::XALL, y2_u32 = y1_u32 + G::Y1ST * G::Y1STAGE;
        uint64_t const dX = smem_desc(base_u32, 16, 8 * G::ROWB, G::LAYOUT);   // Xh, then Xl
        uint64_t const dY0 = smem_desc(y1_u32, 16, 8 * G::ROWB, G::LAYOUT);
        uint64_t const dYT0 = smem_desc(y2_u32, 16, 1024, 2u);
        uint32_t const tm = uniform(tmem);
        bool ok = true, x_ok = false;
        uint32_t n1 = 0, n2 = 0, c1 = c00, xs = 0;   // c1: reduction tile of n1; xs: its row block, from the CTA's first
        PollLimit limit(args.wait_ns);
        while (ok && n2 < T) {
            bool progressed = false;
            if (n2 < n1 && mbar_test_warp(&rfull[n2 % G::NDB], (n2 / G::NDB) & 1) &&
                mbar_test_warp(&y2full[n2 % G::Y2ST], (n2 / G::Y2ST) & 1) &&
                (n2 < 2 || mbar_test_warp(&accfree[n2 & 1], ((n2 >> 1) - 1) & 1))) {
                tc_fence_after();
                uint32_t const ys = n2 % G::Y2ST, bp = n2 & 1;
                uint32_t const oyt = ys * (G::Y2STAGE >> 4);
                uint32_t const r = tm + G::DB0 + (n2 % G::NDB) * BR;   // k-step g: Rh at r + 16 g, Rl at r + 16 g + 8
                uint32_t const dacc = tm + bp * G::ACCW;
                if (elect_one()) {
                    // Acc[0:2KP] (+)= Rh [Y^T_hi; Y^T_lo];  Acc[0:KP] += Rl Y^T_hi  (MODE 2), or
                    // Acc (+)= Rh Y^T_hi
                    mma_ts_bf16<false>(dacc, r, desc_at(dYT0, oyt), SPLIT2 ? IDESC2W : IDESC2);
                    if (SPLIT2) mma_ts_bf16<true>(dacc, r + 8, desc_at(dYT0, oyt), IDESC2);
#pragma unroll
                    for (int ks = 1; ks < BR / 16; ks++) {
                        mma_ts_bf16<true>(dacc, r + ks * 16, desc_at(dYT0, oyt + ks * 2), SPLIT2 ? IDESC2W : IDESC2);
                        if (SPLIT2) mma_ts_bf16<true>(dacc, r + ks * 16 + 8, desc_at(dYT0, oyt + ks * 2), IDESC2);
                    }
                    tc_commit(&accrdy[bp]);
                    tc_commit(&y2empty[ys]);
                }
                n2++;
                progressed = true;
            }
            if (n1 < T && !x_ok) x_ok = mbar_test_warp(xfull, xs & 1);
            if (n1 < T && x_ok && n1 < n2 + G::NDB && mbar_test_warp(&y1full[n1 % G::Y1ST], (n1 / G::Y1ST) & 1)) {
                tc_fence_after();
                uint32_t const s = n1 % G::Y1ST, db = n1 % G::NDB;
                uint32_t const oy = s * (G::Y1STAGE >> 4);
                uint32_t const dcol = tm + G::DB0 + db * BR;
                bool const last = c1 + 1 == TB;   // the row block's last tile
                if (elect_one()) {
                    // D = Xl Yh^T + Xh Yl^T + Xh Yh^T (split arms; small terms first), K = KP in steps of 16.
#pragma unroll
                    for (int tt = 0; tt < NTERMS; tt++) {
                        int const term = NTERMS - 1 - tt;   // 2: Xl*Yh, 1: Xh*Yl, 0: Xh*Yh
                        uint32_t const xo = (term == 2) ? (G::XBYTES >> 4) : 0;
                        uint32_t const yo = oy + ((term == 1) ? (G::YBYTES >> 4) : 0);
                        if (tt == 0)
                            mma_bf16<false>(dcol, desc_at(dX, xo), desc_at(dY0, yo), IDESC1);
                        else
                            mma_bf16<true>(dcol, desc_at(dX, xo), desc_at(dY0, yo), IDESC1);
#pragma unroll
                        for (int ks = 1; ks < KP / 16; ks++)
                            mma_bf16<true>(dcol, desc_at(dX, xo + ks * 2), desc_at(dY0, yo + ks * 2), IDESC1);
                    }
                    tc_commit(&dfull[db]);
                    tc_commit(&y1empty[s]);
                    if (last) tc_commit(xfree);
                }
                n1++;
                c1 = last ? 0 : c1 + 1;
                xs += last;
                x_ok = !last;
                progressed = true;
            }
            if (progressed) {
                limit.reset();
            } else {
                bool const stop = *abort_flag != 0, late = limit.expired();
                if (__any_sync(0xffffffffu, stop || late)) {
                    if (!stop && lane == 0) {
                        *abort_flag = 1;
                        atomicExch(args.err, 24u);
                    }
                    ok = false;
                }
            }
        }
        // drain: every MMA issued above has completed before the CTA frees
        // the shared and tensor memory it reads and writes
        if (elect_one()) mma_drain(mdrain);
        __syncwarp();
    } else if (warp >= 4 && warp < 4 + NR) {
        // ------------------------------------------------------------ R warps
        // Two teams of NR/2 warps take alternate tiles (team 0 even, team 1 odd), so
        // one team's load latency overlaps the other's arithmetic; a warp handles
        // TMEM lanes 32 quad .. +31 and CW tile columns in chunks of 16.
        constexpr int GPT = NR / 8;                     // column groups per team
        constexpr int CW = BR / GPT;                    // tile columns per warp
        static_assert(CW % 16 == 0, "16-column chunks");
        uint32_t const quad = warp & 3;
        uint32_t const jg = (warp - 4) >> 2;
        uint32_t const team = jg / GPT, grp = jg % GPT;
        uint32_t const row = quad * 32 + lane;          // TMEM lane = output row within the block
        uint32_t const lane_addr = tmem + ((quad * 32) << 16);
        for (uint32_t t = team; t < T; t += 2) {
            uint32_t const s = t % G::VST, b = t % G::NDB;
            uint32_t const c = (c00 + t) % TB;              // reduction tile
            if (!mbar_wait_warp(&dfull[b], (t / G::NDB) & 1, abort_flag, args.err, 25u, args.wait_ns)) break;
            if (!mbar_wait_warp(&vfull[s], (t / G::VST) & 1, abort_flag, args.err, 26u, args.wait_ns)) break;
            tc_fence_after();
            const unsigned char *sv = sV + s * G::VBYTES;
            bool const edge = (c + 1) * BR > args.R;        // the partial last reduction tile
            int const valid = (int)(args.R - c * BR);       // its columns before R
#pragma unroll 1
            for (int ch = 0; ch < CW / 16; ch++) {
                int const col0 = grp * CW + ch * 16;
                uint32_t d[16];
                float v[16];
                tmem_ld16(lane_addr + G::DB0 + b * BR + col0, d);
                if (HSIDE) {
                    // V tile [BR rows][128 cols], row-major; this thread's column = row.
                    const float *vs = reinterpret_cast<const float *>(sv) + col0 * BO + row;
#pragma unroll
                    for (int c = 0; c < 16; c++) v[c] = vs[c * BO];
                } else {
                    // V boxes of [128 rows][32 floats], 128B swizzle.
                    int const qb = col0 / 32;
                    int const c0 = (col0 % 32) / 4;
                    const unsigned char *vb = sv + qb * (BO * 128) + row * 128;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        float4 const x = *reinterpret_cast<const float4 *>(vb + (((c + c0) ^ (row & 7)) << 4));
                        v[4 * c + 0] = x.x;
                        v[4 * c + 1] = x.y;
                        v[4 * c + 2] = x.z;
                        v[4 * c + 3] = x.w;
                    }
                }
                tmem_wait_ld_dep(d);
                if (edge) {
                    // Columns past R are zero-filled (V = 0, WH = 0): WH = 1 there makes R 0
                    // instead of 0 * inf, which the second contraction would carry into every row.
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if (col0 + c >= valid) {
                            d[c] = 0x3f800000u;
                            v[c] = 0.0f;
                        }
                }
                uint32_t pk[8], pl[8];
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    // R = V * (1/WH); a zero WH of the data behaves as in the reference's division.
                    float const r0 = v[c] * rcp_approx(__uint_as_float(d[c]));
                    float const r1 = v[c + 1] * rcp_approx(__uint_as_float(d[c + 1]));
                    pk[c / 2] = fin_bf16x2(r0, r1);
                    if (SPLIT2) {
                        float const h0 = __uint_as_float(pk[c / 2] << 16), h1 = __uint_as_float(pk[c / 2] & 0xffff0000u);
                        pl[c / 2] = fin_bf16x2(r0 - h0, r1 - h1);
                    }
                }
                // R over the 16 columns of D it came from: Rh packed in the first 8, Rl in the others.
                tmem_st8(lane_addr + G::DB0 + b * BR + col0, pk);
                if (SPLIT2) tmem_st8(lane_addr + G::DB0 + b * BR + col0 + 8, pl);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&vempty[s]);   // the values of V have been used (see the FP32 kernel)
                mbar_arrive(&rfull[b]);
            }
        }
    } else if (warp >= 4 + NR) {
        // ------------------------------------------------------------ accumulator warps
        uint32_t const quad = warp & 3;
        uint32_t const row = quad * 32 + lane;
        uint32_t const lane_addr = tmem + ((quad * 32) << 16);
        constexpr int KC = KP / G::NA;
        uint32_t const k0 = ((warp - 4 - NR) >> 2) * KC;   // first column
        float sum[KC];
#pragma unroll
        for (int c = 0; c < KC; c++) sum[c] = 0.0f;
        uint32_t ob = ob0, c1 = c00;   // row block and reduction tile of t
        bool gap_done = c00 == 0 || c00 % args.ts.run != 0;
        for (uint32_t t = 0; t < T; t++) {
            uint32_t const bp = t & 1;
            if (!mbar_wait_warp(&accrdy[bp], (t >> 1) & 1, abort_flag, args.err, 28u, args.wait_ns)) break;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < KC; c0 += 16) {
                uint32_t a[16], a2[16];
                tmem_ld16(lane_addr + bp * G::ACCW + k0 + c0, a);
                if (SPLIT2) tmem_ld16(lane_addr + bp * G::ACCW + KP + k0 + c0, a2);
                tmem_wait_ld_dep(a);
                if (SPLIT2) tmem_wait_ld_dep(a2);
#pragma unroll
                for (int c = 0; c < 16; c++)
                    sum[c0 + c] += SPLIT2 ? __uint_as_float(a[c]) + __uint_as_float(a2[c]) : __uint_as_float(a[c]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&accfree[bp]);
            bool const done = c1 + 1 == TB;   // the row block's last tile
            if (done || t + 1 == T || (c1 + 1) % args.ts.run == 0) {   // a partial of the row block
                uint32_t const o = ob * BO + row;
                if (o < args.O) {
                    float *dst = args.part + ((size_t)args.ts.slot(ob, blockIdx.x, c1) * args.O + o) * KP + k0;
#pragma unroll
                    for (int c = 0; c < KC; c += 4)
                        *reinterpret_cast<float4 *>(dst + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
                    if (!gap_done) {   // the unused slot (TileSplit::slot)
                        dst = args.part + ((size_t)(args.ts.slot(ob0, blockIdx.x, c00) - 1) * args.O + o) * KP + k0;
#pragma unroll
                        for (int c = 0; c < KC; c += 4) *reinterpret_cast<float4 *>(dst + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                }
                gap_done = true;
#pragma unroll
                for (int c = 0; c < KC; c++) sum[c] = 0.0f;
            }
            c1 = done ? 0 : c1 + 1;
            ob += done;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Host side
PFN_cuTensorMapEncodeTiled_v12000 encode_fn_b()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

int encode_map(nmfb_ctx *ctx, CUtensorMap *map, CUtensorMapDataType dt, const void *base, uint64_t inner,
               uint64_t outer, uint64_t row_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw)
{
    auto fn = encode_fn_b();
    if (!fn) return nmfb_fail(ctx, NMFB_ENODEV, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(map, dt, 2, (void *)base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return nmfb_fail(ctx, NMFB_ECUDA, "cuTensorMapEncodeTiled (bf16 arm) failed (%d)", (int)r);
    return NMFB_OK;
}

struct PlanB {
    MapsB mapsH, mapsW;
    __nv_bfloat16 *wsplit, *hsplit;   // hi | lo | transposed hi/lo blocks, for W and for H
    uint32_t *dErr;                   // shared with the FP32 arm's error word
    int arm;                          // arm the Y^T maps were encoded for
    double *dCsW, *dCsH;              // k_finish's column-sum partials of W and of H
};

template <int KP, int MODE>
int set_attrs_mode(nmfb_ctx *ctx)
{
    int const smem = GeoB<KP, MODE>::SMEM;
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_bf16<true, KP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_bf16<false, KP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return NMFB_OK;
}

template <int KP>
int set_attrs_b(nmfb_ctx *ctx)
{
    int rc = set_attrs_mode<KP, 0>(ctx);
    if (!rc) rc = set_attrs_mode<KP, 1>(ctx);
    if (!rc) rc = set_attrs_mode<KP, 2>(ctx);
    return rc;
}

template <bool HSIDE, int KP, int MODE>
int launch_b(nmfb_ctx *ctx, const MapsB &maps, PlanB *plan)
{
    using G = GeoB<KP, MODE>;
    static_assert(G::BR == 64, "plan_of");
    ArgsB args;
    args.O = HSIDE ? ctx->m : ctx->n;
    args.R = HSIDE ? ctx->n : ctx->m;
    args.ts = plan_of(ctx, !HSIDE);
    if ((size_t)args.ts.slots * args.O * KP > ctx->part_items)
        return nmfb_fail(ctx, NMFB_EINVAL, "bf16 arm: partial buffer too small (%u slots)", args.ts.slots);
    args.csy.cs = HSIDE ? plan->dCsW : plan->dCsH;
    args.csy.nblk = fin_blocks(args.R, fin_rpt(plan_of(ctx, HSIDE).slots));
    args.csy.acc = HSIDE ? ctx->dAccW : ctx->dAccH;
    args.part = ctx->dPart;
    args.err = plan->dErr;
    args.st = ctx->dState;
    args.wait_ns = ctx->wait_ns ? ctx->wait_ns : WAIT_LIMIT_NS;
    int const main = HSIDE ? 0 : 1;
    int rc = nmfb_prof_begin(ctx, main);
    if (rc) return rc;
    NMFB_CUDA_TRY(ctx, launch_chained(k_fused_bf16<HSIDE, KP, MODE>, args.ts.ctas(), G::NTHR, G::SMEM, ctx->stream, maps,
                                      args));
    NMFB_LAUNCH_CHECK(ctx);
    return nmfb_prof_end(ctx, main);
}

template <bool HSIDE, int KP>
int dispatch_kp(nmfb_ctx *ctx, const MapsB &maps, PlanB *plan)
{
    switch (ctx->arm) {
    case NMFB_ARM_BF16: return launch_b<HSIDE, KP, 0>(ctx, maps, plan);
    case NMFB_ARM_SPLIT_BF16: return launch_b<HSIDE, KP, 1>(ctx, maps, plan);
    default: return launch_b<HSIDE, KP, 2>(ctx, maps, plan);
    }
}

template <bool HSIDE>
int dispatch_b(nmfb_ctx *ctx, const MapsB &maps, PlanB *plan)
{
    switch (ctx->kp) {
    case 16: return dispatch_kp<HSIDE, 16>(ctx, maps, plan);
    case 32: return dispatch_kp<HSIDE, 32>(ctx, maps, plan);
    case 64: return dispatch_kp<HSIDE, 64>(ctx, maps, plan);
    default: return nmfb_fail(ctx, NMFB_EINVAL, "bf16 arms: unsupported padded rank %u", ctx->kp);
    }
}

int encode_maps_b(nmfb_ctx *ctx, PlanB *plan)
{
    uint32_t const kp = ctx->kp;
    size_t const wsz = (size_t)ctx->n * kp, hsz = (size_t)ctx->m * kp;
    uint64_t const wblk = (ctx->n + 63) / 64, hblk = (ctx->m + 63) / 64;
    uint32_t const ytrows = (ctx->arm == NMFB_ARM_BF16X3 ? 2 : 1) * kp;
    CUtensorMapSwizzle const fsw = (kp == 16) ? CU_TENSOR_MAP_SWIZZLE_32B
                                 : (kp == 32) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    CUtensorMapDataType const BF = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, F32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    uint64_t const vrow = ctx->ldv * sizeof(float), frow = (uint64_t)kp * 2;
    int rc;
    // update_H: X = H (rows m), Y = W (rows n)
    MapsB &mh = plan->mapsH;
    if ((rc = encode_map(ctx, &mh.v, F32, ctx->dV, ctx->m, ctx->n, vrow, BO, 64, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    if ((rc = encode_map(ctx, &mh.xh, BF, plan->hsplit, kp, ctx->m, frow, kp, BO, fsw))) return rc;
    if ((rc = encode_map(ctx, &mh.xl, BF, plan->hsplit + hsz, kp, ctx->m, frow, kp, BO, fsw))) return rc;
    if ((rc = encode_map(ctx, &mh.yh, BF, plan->wsplit, kp, ctx->n, frow, kp, 64, fsw))) return rc;
    if ((rc = encode_map(ctx, &mh.yl, BF, plan->wsplit + wsz, kp, ctx->n, frow, kp, 64, fsw))) return rc;
    if ((rc = encode_map(ctx, &mh.yt, BF, plan->wsplit + 2 * wsz, 64, wblk * 2 * kp, 128, 64, ytrows,
                         CU_TENSOR_MAP_SWIZZLE_128B)))
        return rc;
    // update_W: X = W (rows n), Y = H (rows m)
    MapsB &mw = plan->mapsW;
    if ((rc = encode_map(ctx, &mw.v, F32, ctx->dV, ctx->m, ctx->n, vrow, 32, BO, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
    if ((rc = encode_map(ctx, &mw.xh, BF, plan->wsplit, kp, ctx->n, frow, kp, BO, fsw))) return rc;
    if ((rc = encode_map(ctx, &mw.xl, BF, plan->wsplit + wsz, kp, ctx->n, frow, kp, BO, fsw))) return rc;
    if ((rc = encode_map(ctx, &mw.yh, BF, plan->hsplit, kp, ctx->m, frow, kp, 64, fsw))) return rc;
    if ((rc = encode_map(ctx, &mw.yl, BF, plan->hsplit + hsz, kp, ctx->m, frow, kp, 64, fsw))) return rc;
    if ((rc = encode_map(ctx, &mw.yt, BF, plan->hsplit + 2 * hsz, 64, hblk * 2 * kp, 128, 64, ytrows,
                         CU_TENSOR_MAP_SWIZZLE_128B)))
        return rc;
    plan->arm = ctx->arm;
    return NMFB_OK;
}

// k_finish on W (or H): its update from the partials, or, with update = false,
// only its BF16 copies and column-sum partials.
template <int KP>
int launch_finish_b(nmfb_ctx *ctx, bool w, bool update, int adjust)
{
    PlanB *plan = (PlanB *)ctx->bplan;
    FinishArgs fa = {};
    fa.O = w ? ctx->n : ctx->m;
    __nv_bfloat16 *xs = w ? plan->wsplit : plan->hsplit;
    size_t const sz = (size_t)fa.O * KP;
    fa.ts = plan_of(ctx, w);
    fa.k = ctx->k;
    fa.adjust = adjust;
    fa.part = update ? ctx->dPart : nullptr;
    fa.X = w ? ctx->dW : ctx->dH;
    fa.accY = w ? ctx->dAccH : ctx->dAccW;
    fa.bhi = xs;
    fa.blo = xs + sz;
    fa.bT = xs + 2 * sz;
    fa.bnblk64 = (fa.O + 63) / 64;
    fa.cs = w ? plan->dCsW : plan->dCsH;
    fa.st = ctx->dState;
    NMFB_CUDA_TRY(ctx, (fin_launch<KP, 64, 1>(fa, ctx->stream)));
    NMFB_LAUNCH_CHECK(ctx);
    ctx->fz_ok[w ? 0 : 1] = 1;
    return NMFB_OK;
}

int finish_b(nmfb_ctx *ctx, bool w, bool update, int adjust)
{
    switch (ctx->kp) {
    case 16: return launch_finish_b<16>(ctx, w, update, adjust);
    case 32: return launch_finish_b<32>(ctx, w, update, adjust);
    default: return launch_finish_b<64>(ctx, w, update, adjust);
    }
}

// One half-iteration: the fused BF16 kernel and k_finish (which writes X's BF16
// copies and column sums for the next half-iteration); the copies of X and Y
// are prepared first only when they are not current.
int bf16_half(nmfb_ctx *ctx, bool is_H, int adjust)
{
    PlanB *plan = (PlanB *)ctx->bplan;
    if (!plan) return nmfb_fail(ctx, NMFB_ESTATE, "bf16 arm not prepared");
    int rc;
    if (plan->arm != ctx->arm && (rc = encode_maps_b(ctx, plan))) return rc;
    int const whole = is_H ? 2 : 3;
    if ((rc = nmfb_prof_begin(ctx, whole))) return rc;
    if (!ctx->fz_ok[is_H ? 0 : 1] && (rc = finish_b(ctx, is_H, false, 0))) return rc;    // Y
    if (!ctx->fz_ok[is_H ? 1 : 0] && (rc = finish_b(ctx, !is_H, false, 0))) return rc;   // X
    rc = is_H ? dispatch_b<true>(ctx, plan->mapsH, plan) : dispatch_b<false>(ctx, plan->mapsW, plan);
    if (!rc) rc = finish_b(ctx, !is_H, true, adjust);
    if (rc) return rc;
    return nmfb_prof_end(ctx, whole);
}

}  // namespace

int nmfb_bf16_prepare(nmfb_ctx *ctx)
{
    if (ctx->bplan) return NMFB_OK;
    uint32_t const kp = ctx->kp;
    if (kp != 16 && kp != 32 && kp != 64)
        return nmfb_fail(ctx, NMFB_EINVAL, "the bf16 arms support ranks up to 64 (k=%u)", ctx->k);
    int rc = (kp == 16) ? set_attrs_b<16>(ctx) : (kp == 32) ? set_attrs_b<32>(ctx) : set_attrs_b<64>(ctx);
    if (rc) return rc;
    PlanB *plan = (PlanB *)calloc(1, sizeof(PlanB));
    if (!plan) return nmfb_fail(ctx, NMFB_ENOMEM, "bf16 plan");
    ctx->bplan = plan;
    plan->arm = -1;
    plan->dErr = nmfb_fused_err_word(ctx);
    if (!plan->dErr) return nmfb_fail(ctx, NMFB_ESTATE, "bf16 arm needs the fused error word");
    // per factor: hi (rows x kp) | lo (rows x kp) | transposed hi and lo blocks (ceil(rows/64) x 2 kp x 64)
    size_t const wsz = (size_t)ctx->n * kp, hsz = (size_t)ctx->m * kp;
    size_t const wt = (size_t)((ctx->n + 63) / 64) * 128 * kp, ht = (size_t)((ctx->m + 63) / 64) * 128 * kp;
    cudaError_t e = nmfb_malloc(ctx, (void **)&plan->wsplit, (2 * wsz + wt) * sizeof(__nv_bfloat16));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->hsplit, (2 * hsz + ht) * sizeof(__nv_bfloat16));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->dCsW, (size_t)fin_blocks(ctx->n, 1) * kp * sizeof(double));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->dCsH, (size_t)fin_blocks(ctx->m, 1) * kp * sizeof(double));
    if (e != cudaSuccess) return nmfb_fail(ctx, NMFB_ENOMEM, "bf16 split buffers: %s", cudaGetErrorString(e));
    return NMFB_OK;
}

int nmfb_bf16_release(nmfb_ctx *ctx)
{
    PlanB *plan = (PlanB *)ctx->bplan;
    if (!plan) return NMFB_OK;
    if (plan->wsplit) nmfb_free(ctx, plan->wsplit);
    if (plan->hsplit) nmfb_free(ctx, plan->hsplit);
    if (plan->dCsW) nmfb_free(ctx, plan->dCsW);
    if (plan->dCsH) nmfb_free(ctx, plan->dCsH);
    free(plan);
    ctx->bplan = nullptr;
    return NMFB_OK;
}

int nmfb_bf16_update_H(nmfb_ctx *ctx, int adjust) { return bf16_half(ctx, true, adjust); }
int nmfb_bf16_update_W(nmfb_ctx *ctx, int adjust) { return bf16_half(ctx, false, adjust); }

// Makes W's BF16 copies and column sums current (before a test block is
// replayed as a graph).
int nmfb_bf16_ready_W(nmfb_ctx *ctx)
{
    if (!ctx->bplan || ctx->fz_ok[0]) return NMFB_OK;
    return finish_b(ctx, true, false, 0);
}
