// kernels_fused.cu -- the fused half-iteration arm (NMFB_ARM_FUSED / _FUSED_TF32).
//
// One kernel computes, for a block of 128 rows of the factor being updated
// (X = W for update_W, X = H for update_H) and a range of the reduction
// dimension, the partial  Xaux = sum_r  (V ./ (X Y^T))[o][r] * Y[r][:]
// without ever materialising the n x m quotient:
//
//   TMA      : V tile (128 x BR, FP32) into a VST-deep ring; the Y tile
//              operands of MMA1 and of MMA2 into a ring each.
//   split    : k_finish, when it updates a factor, writes it as TF32 hi (round
//              to nearest) and the transposed hi/lo blocks that MMA2 reads K-major
//              (lo = y - hi, exact; an MN-major read of a TF32 operand returns
//              zeros on sm_100a), plus BF16 copies bf16(lo), bf16(y) and bf16(y)
//              transposed per tile; the Y producers TMA-load them per tile.  X (128 rows per CTA) is split
//              once per CTA by the accumulator warps.
//   MMA1     : D (TMEM, 128 x BR) = Xh Yh^T                    (kind::tf32, k-steps of 8)
//              + [bf16(Xh) | bf16(Xl)] [bf16(Yl) ; bf16(Y)]^T (kind::f16, K = 2 KP, k-steps of 16),
//              or at KP = 16 + Xh Yl^T + Xl Yh^T (kind::tf32).
//   epilogue : R = V / D in FP32 registers (V times an approximate reciprocal,
//              <= 1.5 ulp; the reference uses fdividef);  R = Rh + Rl with
//              Rh = TF32(R) written back over D and bf16(Rl) packed into a
//              separate TMEM region.
//   MMA2     : Acc[tile] (TMEM, 128 x 2 KP) = Rh [Yh | Yl]   (kind::tf32, N = 2 KP)
//              + bf16(Rl) bf16(Y) into Acc[0:KP]               (kind::f16, K = 16).
//   epilogue : adds Acc[tile] into FP32 registers (per-tile accumulation keeps
//              the tensor core's FP32 sums short) and writes the split's
//              partial; k_finish (one CTA per 32 rows) sums the splits, applies
//              X = X .* Xaux ./ colsum(Y) (and the EPS adjust when asked), and
//              writes X's split copies for the next half-iteration, whose V producers
//              sum its columns: two launches per half-iteration.
//
// Precision of the two contractions: x y = xh yh + xh yl + xl y with xh, yh
// TF32.  The large term xh yh (and, in MMA2, rh yl) is an exact TF32 product
// with FP32 accumulation; the small terms, each at most 2^-12 of the whole,
// are BF16 products (relative rounding 2^-9 of the term), so every product is
// accurate to about 2^-20 relative.  Against the 3 x TF32 form (12 + 16 MMAs
// per 64-column tile at k = 32, all at the tensor pipe's per-instruction floor
// of N <= 64) this issues 8 + 12, and the R warps' epilogue stays one TMEM load
// and one reciprocal per element.
//
// Reference equivalent: get_H_BLM / get_W_BLN (src/NMF_routines.c:376-525,
// 1014-1164): two cuBLAS SGEMMs around matrix_div_sub with WH in HBM.
//
// Warp roles: warp 0 = V producer (TMA), warp 1 = MMA issuer and TMEM owner,
// warps 2 and 3 = Y producers (TMA), warps 4-11 (or 4-19) = R warps in two teams that
// take alternate tiles (warp w reads TMEM lanes 32*(w%4)..+31), last 4 (or 8) warps
// = accumulator and split warps.
// V stages are released once the epilogue has used them, Y stages when the MMA
// that reads them has completed.
// Every mbarrier wait is bounded (1 s of %globaltimer); on expiry the kernel
// records an error word that the host turns into NMFB_ETIMEOUT.
// No TMA multicast is used anywhere.
#include "nmfb_internal.cuh"
#include "fused_common.cuh"
#include "finish.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <float.h>
#include <cudaTypedefs.h>
#include <type_traits>

using nmfb::ConvState;
using namespace nmfb_tc;

namespace {

// Swizzle of a K-major operand whose rows are `bytes` long: the UMMA layout code
// and the tensor-map mode (rows of 32 / 64 / 128 bytes).
__host__ __device__ constexpr uint32_t umma_layout(int bytes) { return bytes == 32 ? 6u : bytes == 64 ? 4u : 2u; }

struct FusedMaps {
    CUtensorMap v;       // V, box [128 x BR] (H side, no swizzle) or [32 x 128] (W side, 128B swizzle)
    CUtensorMap y;       // TF32 hi part of the other factor (rows x KP), box rows = BR
    CUtensorMap yt;      // its transposed split: per 32 rows, [hi^T (KP x 32) ; lo^T (KP x 32)]
    CUtensorMap ylb;     // BF16 copy of its lo part (KP = 16: the FP32 lo part; rows x KP), box [KP x BR]
    CUtensorMap yb;      // BF16 copy (rows x KP), box [KP x BR]
    CUtensorMap ybt;     // BF16 transposed tiles: per BR rows, KP rows of BR values; box [BR x KP]
};

struct FusedArgs {
    uint32_t O, R;        // output rows, reduction length
    TileSplit ts;
    ColSum csy;           // column sums of the other factor
    float *part;          // [slot][O][KP]
    uint32_t *err;        // device error word
    const ConvState *st;
    const float *X;       // factor being updated (O x KP), read once per row block into TMEM
    unsigned long long wait_ns;  // limit of every bounded wait (%globaltimer ns)
#ifdef NMFB_FUSED_DEBUG
    float *dbg;           // block 0, tile 0: D | V | Rh | Acc (debug builds only; 128 x 64 each)
#endif
};

// ---------------------------------------------------------------------------
template <int KP>
struct Geo {
    static constexpr int BR = 64;                         // reduction rows per tile
    static constexpr int CB = (KP == 16) ? 16 : 32;       // floats per swizzle column block
    static constexpr int NB = KP / CB;                     // column blocks
    static constexpr int ROWB = CB * 4;                    // bytes per row of a block
    static constexpr uint32_t LAYOUT = (KP == 16) ? 4u : 2u;  // SW64 : SW128
    static constexpr int YBLK = BR * ROWB;                 // bytes of one Yh column block
    static constexpr int YTBLK = KP * 128;                 // bytes of one Y^T part (32 reduction rows)
    static constexpr int YTPAIR = 2 * YTBLK;               // Y^T hi part followed by its lo part
    static constexpr int YBYTES = BR * KP * 4;
    static constexpr int VBYTES = BO * BR * 4;
    // Two rings for Y: MMA1's operands (released by MMA1, up to NDB tiles before the
    // tile's MMA2) and MMA2's.  With one ring for both a stage was held through the
    // whole distance between the two, and MMA1 could not run ahead of MMA2.
    static constexpr int YBB = BR * KP * 2;                // one BF16 tile of BR rows of 2 KP bytes
    static constexpr int YBTB = KP * BR * 2;               // bf16(Y)^T tile, KP rows of 2 BR bytes
    static constexpr int Y1STAGE = YBYTES + 2 * YBB;       // Yh (TF32, NB column blocks) | bf16(Yl) | bf16(Y)
    static constexpr int Y2STAGE = 2 * YBYTES + YBTB;      // YTh | YTl (per 32 rows) | bf16(Y)^T
    // MMA1's small terms Xh Yl + Xl Y: TF32 at KP = 16 (Xh Yl + Xl Yh, from an FP32 copy of
    // Yl that takes the place of the two BF16 tiles; 2 of 18 MMAs more, and MMAs do not bound
    // the small problems of these ranks), BF16 above (4 of 20 MMAs fewer at KP = 32).
    static constexpr bool LO32 = KP == 16;
    static_assert(!LO32 || YBYTES == 2 * YBB, "the FP32 tile of Yl takes the BF16 tiles' place");
    static constexpr uint32_t BLAYOUT = umma_layout(2 * KP);
    static constexpr uint32_t BTLAYOUT = umma_layout(2 * BR);
    static constexpr int Y1ST = (KP == 64) ? 2 : 3, Y2ST = 2;   // what is left goes to V
    static constexpr int FIXED = 1024 + 512;
    static constexpr int YALL = Y1ST * Y1STAGE + Y2ST * Y2STAGE;
    static constexpr int VAVAIL = (SMEM_LIMIT - FIXED - YALL) / VBYTES;
    static constexpr int VST = VAVAIL > 6 ? 6 : VAVAIL;    // V ring depth (HBM stream)
    static constexpr int SMEM = FIXED + YALL + VST * VBYTES;
    static_assert(VST >= 2, "shared-memory ring too small");
    static_assert(YBB % 1024 == 0 && Y1STAGE % 1024 == 0 && Y2STAGE % 1024 == 0, "1024-byte stage alignment");
    static constexpr int NR = (KP >= 64) ? 8 : 16;        // R warps
    // Accumulator warps: sets of four, KP / NA columns each.  At KP = 64 tensor memory
    // holds one accumulator besides three D buffers, so it has to be read fast.
    static constexpr int NA = (KP == 64) ? 2 : 1;
    static constexpr int NTHR = (4 + NR + 4 * NA) * 32;   // (a multiple of four warps: one more would cost 8 registers a thread)
    static constexpr uint32_t ACC = 2 * KP;                // TMEM columns of one per-tile accumulator
    static constexpr uint32_t NACC = (KP == 64) ? 1 : 2;   // accumulators
    static constexpr uint32_t NDB = (KP == 16) ? 4 : 3;    // D buffers (MMA1 runs NDB tiles ahead)
    // (a team takes every other tile: with an odd ring its uses of a V stage are two phases apart,
    // and D(t) has to imply that tile t - VST, the other team's, has landed)
    static_assert(VST % 2 == 0 || VST >= (int)NDB, "vfull's parity would be ambiguous");
    static constexpr uint32_t DA0 = NACC * ACC;            // D[b] (then Rh[b]) at DA0 + b BR
    static constexpr uint32_t NRL = (KP == 16) ? NDB : 2;  // bf16(Rl) buffers (2: one per R team)
    static_assert(NRL == NDB || (NRL == 2 && Y2ST == 2), "the R teams wait on y2empty for their Rl buffer");
    static constexpr uint32_t RL0 = DA0 + NDB * BR;        // bf16(Rl)[b] at RL0 + b BR/2
    static constexpr uint32_t NXB = (KP == 64) ? 1 : 2;    // X buffers (2: the next row block's X while this one is read)
    static constexpr uint32_t XC0 = RL0 + NRL * BR / 2;    // X hi (TF32, KP columns) | bf16(X hi) | bf16(X lo)
                                                           // (KP/2 each) or X lo (TF32, KP); buffer b at XC0 + 2 KP b
    static_assert(XC0 + NXB * 2 * KP <= 512, "TMEM columns exceeded");
};

// TMEM columns: per-tile accumulators Acc[b] at b*2KP, b < NACC (2KP columns: the Rh Yh +
// bf16(Rl) bf16(Y) sum and the Rh Yl part side by side); D[b] (BR columns, then
// Rh[b]) at DA0 + b*BR, b < NDB; bf16(Rl)[b] (BR/2 columns, column group g of
// 16 in its 8 columns RL0 + b*BR/2 + 8g), b < NRL; then, per X buffer, a row
// block's 128 rows of X as TF32 hi (KP columns) and bf16(X hi) | bf16(X lo)
// (KP/2 columns each), the A operands of MMA1 for every tile of that row block
// (so MMA1 reads only Y from shared memory).

// Warp roles: 0 = V producer (TMA), 1 = MMA issuer + TMEM owner, 2, 3 = Y
// producers (TMA), 4 .. 3 + NR = R warps (V / D, feed MMA2), the others =
// accumulator warps (sum the per-tile MMA2 results in FP32 registers; split X).
//
// Persistent, one CTA per SM: the tiles of all row blocks form one list and
// every CTA takes an equal run of it (TileSplit), so the launch is one wave
// whatever the shape and pays the pipeline's fill (about six tile times) once
// per CTA instead of once per (row block, split) pair.
template <bool HSIDE, int KP, int NTERMS>
__global__ void __launch_bounds__(Geo<KP>::NTHR, 1)
    k_fused_half(const __grid_constant__ FusedMaps maps, const FusedArgs args)
{
    using G = Geo<KP>;
    constexpr int BR = G::BR;
    constexpr int NR = G::NR;
    constexpr uint32_t ACC_COLS = G::ACC;

    extern __shared__ unsigned char smem_raw[];
    uint32_t const base_u32 = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *const base = smem_raw + (base_u32 - smem_u32(smem_raw));
    unsigned char *const sY1 = base;                                // [Y1ST][Yh | bf16 Yl | bf16 Y]
    unsigned char *const sY2 = sY1 + G::Y1ST * G::Y1STAGE;          // [Y2ST][YTh | YTl | bf16 Y^T]
    unsigned char *const sV = sY2 + G::Y2ST * G::Y2STAGE;           // [VST][VBYTES]
    uint64_t *const bars = reinterpret_cast<uint64_t *>(sV + G::VST * G::VBYTES);
    uint64_t *const vfull = bars;                   // [VST]  TMA -> epilogue
    uint64_t *const vempty = vfull + G::VST;        // [VST]  epilogue -> V producer
    uint64_t *const y1full = vempty + G::VST;       // [Y1ST] TMA -> MMA1
    uint64_t *const y1empty = y1full + G::Y1ST;     // [Y1ST] MMA1 commit -> Y1 producer
    uint64_t *const y2full = y1empty + G::Y1ST;     // [Y2ST] TMA -> MMA2
    uint64_t *const y2empty = y2full + G::Y2ST;     // [Y2ST] MMA2 commit -> Y2 producer
    uint64_t *const dfull = y2empty + G::Y2ST;      // [NDB]  MMA1 commit -> R warps
    uint64_t *const rfull = dfull + G::NDB;         // [NDB]  R warps -> MMA2
    uint64_t *const accrdy = rfull + G::NDB;        // [NACC] MMA2 commit -> accumulator warps
    uint64_t *const accfree = accrdy + G::NACC;     // [NACC] accumulator warps -> MMA2
    uint64_t *const xready = accfree + G::NACC;     // [NXB]  X split into TMEM -> MMA1
    uint64_t *const xfree = xready + G::NXB;        // [NXB]  last MMA1 of a row block -> accumulator warps
    uint64_t *const mdrain = xfree + G::NXB;        // [1]    issuer's final commit (drain)
    uint32_t *const tmem_slot = reinterpret_cast<uint32_t *>(mdrain + 1);
    volatile uint32_t *const abort_flag = tmem_slot + 1;

    chain_next();
    uint32_t const warp = uniform(threadIdx.x / 32), lane = threadIdx.x % 32;
    // This CTA's run of tiles [g0, g0 + T) of the whole (row block, reduction tile)
    // list, row-block-major: tile g is reduction tile g % TB of row block g / TB.
    uint32_t const TB = args.ts.tb;
    uint32_t const g0 = blockIdx.x * args.ts.tpc;
    uint32_t T = min(args.ts.total - g0, args.ts.tpc);
    uint32_t const ob0 = g0 / TB, c00 = g0 - ob0 * TB;
#ifdef NMFB_FUSED_DEBUG
    // Per-tile event times of block 0 (ns since kernel start), 8 events x 64 tiles.
    unsigned long long const ts0 = globaltimer();
    unsigned long long *const dts = args.dbg ? reinterpret_cast<unsigned long long *>(args.dbg + 4 * BO * 64) : nullptr;
#define DBG_TS(ev, t)                                                                              \
    do {                                                                                           \
        if (dts && blockIdx.x == 0 && (t) < 64) dts[(ev) * 64 + (t)] = globaltimer() - ts0;        \
    } while (0)
#define DBG_PH(ph, t)                                                                                 \
    do {                                                                                              \
        if (dts && blockIdx.x == 0 && warp == 5 && lane == 0 && (t) < 64)                             \
            dts[1536 + (ph) * 64 + (t)] = clock64();                                                  \
    } while (0)
#else
#define DBG_TS(ev, t) do { } while (0)
#define DBG_PH(ph, t) do { } while (0)
#endif

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
        for (uint32_t b = 0; b < G::NACC; b++) {
            mbar_init(&accrdy[b], 1);
            mbar_init(&accfree[b], 4 * G::NA);
        }
        for (uint32_t b = 0; b < G::NXB; b++) {
            mbar_init(&xready[b], 4 * G::NA);
            mbar_init(&xfree[b], 1);
        }
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
                    !mbar_wait(&vempty[s], ((t / G::VST) - 1) & 1, abort_flag, args.err, 1u, args.wait_ns))
                    break;
                issued = t + 1;
                unsigned char *sv = sV + s * G::VBYTES;
                int const r0 = (int)(c * BR), o0 = (int)(ob * BO);
                DBG_TS(0, t);
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
            // drain: the last load into every stage has landed (each earlier one
            // had to, before its stage was released for reuse)
            for (uint32_t t = issued > (uint32_t)G::VST ? issued - G::VST : 0; t < issued; t++)
                mbar_drain(&vfull[t % G::VST], (t / G::VST) & 1);
    } else if (warp == 2 || warp == 3) {
        // ------------------------------------------------------------ Y producers
        // warp 2: MMA1's operands, warp 3: MMA2's
        if (lane == 0) {
            bool const one = warp == 2;
            uint64_t const pol = policy_evict_last();
            uint64_t *const full = one ? y1full : y2full, *const empty = one ? y1empty : y2empty;
            uint32_t const nst = one ? G::Y1ST : G::Y2ST;
            uint32_t issued = 0, c = c00, s = 0, ph = 0;   // stage and its phase
            for (uint32_t t = 0; t < T; t++, c = (c + 1 == TB) ? 0 : c + 1) {
                if (t >= nst && !mbar_wait(&empty[s], ph ^ 1, abort_flag, args.err, 2u, args.wait_ns)) break;
                issued = t + 1;
                int const r0 = (int)(c * BR);
                if (one) {
                    unsigned char *sy = sY1 + s * G::Y1STAGE;
                    DBG_TS(1, t);
                    mbar_expect_tx(&full[s], G::YBYTES + (NTERMS == 3 ? 2 * G::YBB : 0));
                    for (int b = 0; b < G::NB; b++) tma_load_2d(sy + b * G::YBLK, &maps.y, &full[s], b * G::CB, r0, pol);
                    if (NTERMS == 3) {
                        tma_load_2d(sy + G::YBYTES, &maps.ylb, &full[s], 0, r0, pol);
                        if (!G::LO32) tma_load_2d(sy + G::YBYTES + G::YBB, &maps.yb, &full[s], 0, r0, pol);
                    }
                } else {
                    unsigned char *sy = sY2 + s * G::Y2STAGE;
                    mbar_expect_tx(&full[s], 2 * G::YBYTES + (NTERMS == 3 ? G::YBTB : 0));
                    // Y^T: the BR / 32 row blocks of this tile, 2 KP rows of 128 B each
                    tma_load_2d(sy, &maps.yt, &full[s], 0, (r0 / 32) * 2 * KP, pol);
                    if (NTERMS == 3) tma_load_2d(sy + 2 * G::YBYTES, &maps.ybt, &full[s], 0, (int)(c * KP), pol);
                }
                if (++s == nst) {
                    s = 0;
                    ph ^= 1;
                }
            }
            for (uint32_t t = issued > nst ? issued - nst : 0; t < issued; t++) mbar_drain(&full[t % nst], (t / nst) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // Two issue queues, polled without blocking:
        //   MMA2(n2): needs the R warps' R(n2), its Y operands and, for n2 >= NACC, the
        //             accumulator warps to have read Acc[n2 % NACC] of tile n2-NACC;
        //   MMA1(n1): needs its Y operands and a free D buffer (MMA2(n1-NDB)
        //             issued, i.e. n1 < n2 + NDB); A = X from TMEM, which for the
        //             first tile of a row block has to be ready, and whose buffer the
        //             last one's MMA1 releases.
        constexpr uint32_t IDESC1 = idesc_tf32(BO, BR, 0);
        constexpr uint32_t IDESC1B = idesc_bf16xf32(BO, BR);
        constexpr uint32_t IDESC2 = NTERMS == 3 ? idesc_tf32(BO, 2 * KP, 0) : idesc_tf32(BO, KP, 0);
        constexpr uint32_t IDESC2B = idesc_bf16xf32(BO, KP);
        uint64_t const dY0 = smem_desc(base_u32, 16, 8 * G::ROWB, G::LAYOUT);
        uint64_t const dYB0 = G::LO32 ? smem_desc(base_u32 + G::YBYTES, 16, 8 * G::ROWB, G::LAYOUT)
                                      : smem_desc(base_u32 + G::YBYTES, 16, 8 * 2 * KP, G::BLAYOUT);
        uint32_t const y2_u32 = base_u32 + G::Y1ST * G::Y1STAGE;
        uint64_t const dYT0 = smem_desc(y2_u32, 16, 1024, 2u);
        uint64_t const dYBT0 = smem_desc(y2_u32 + 2 * G::YBYTES, 16, 8 * 2 * BR, G::BTLAYOUT);
        uint32_t const tm = uniform(tmem);
        bool ok = true, x_ok = false;
        uint32_t n1 = 0, n2 = 0, c1 = c00, xs = 0;   // c1: reduction tile of n1; xs: its row block, counted from the CTA's first
        PollLimit limit(args.wait_ns);
        while (ok && n2 < T) {
            bool progressed = false;
            if (n2 < n1 && mbar_test_warp(&rfull[n2 % G::NDB], (n2 / G::NDB) & 1) &&
                mbar_test_warp(&y2full[n2 % G::Y2ST], (n2 / G::Y2ST) & 1) &&
                (n2 < G::NACC || mbar_test_warp(&accfree[n2 % G::NACC], ((n2 / G::NACC) - 1) & 1))) {
                tc_fence_after();
                uint32_t const sp = n2 % G::Y2ST, bp = n2 % G::NACC, db = n2 % G::NDB;
                uint32_t const rh = tm + G::DA0 + db * BR;
                uint32_t const rl = tm + G::RL0 + (n2 % G::NRL) * (BR / 2);
                uint32_t const dacc = tm + bp * ACC_COLS;
                uint32_t const oy = sp * (G::Y2STAGE >> 4);
                if (elect_one()) {
                    // MMA2 for this tile only, K = BR reduction rows:
                    //   Acc[bp][0:2KP] (+)= Rh [Y^T_hi; Y^T_lo]     (kind::tf32, N = 2 KP, k-steps of 8)
                    //   Acc[bp][0:KP]   += bf16(Rl) bf16(Y)^T      (kind::f16, N = KP, k-steps of 16;
                    //                      column group g of the R warps = k-step g, A at rl + 8 g)
                    // so Acc[0:KP] + Acc[KP:2KP] = Rh Yh + Rh Yl + Rl Y (summed by the
                    // accumulator warps in FP32 registers).
                    // Each MMA truncates its FP32 sums, so the small terms come while the sums are
                    // still small (after the first k-step, whose MMA also clears Acc[KP:2KP]).
                    mma_ts<false>(dacc, rh, desc_at(dYT0, oy), IDESC2);
                    if (NTERMS == 3) {
#pragma unroll
                        for (int g = 0; g < BR / 16; g++)
                            mma_ts_bf16<true>(dacc, rl + g * 8, desc_at(dYBT0, oy + g * 2), IDESC2B);
                    }
#pragma unroll
                    for (int ks = 1; ks < BR / 8; ks++)
                        mma_ts<true>(dacc, rh + ks * 8, desc_at(dYT0, oy + (((ks / 4) * G::YTPAIR + (ks % 4) * 32) >> 4)),
                                     IDESC2);
                    tc_commit(&accrdy[bp]);
                    tc_commit(&y2empty[sp]);
                    DBG_TS(3, n2);
                }
                n2++;
                progressed = true;
            }
            if (n1 < T && !x_ok) x_ok = mbar_test_warp(&xready[xs % G::NXB], (xs / G::NXB) & 1);
            if (n1 < T && x_ok && n1 < n2 + G::NDB && mbar_test_warp(&y1full[n1 % G::Y1ST], (n1 / G::Y1ST) & 1)) {
                tc_fence_after();
                uint32_t const s = n1 % G::Y1ST, db = n1 % G::NDB;
                uint32_t const dcol = tm + G::DA0 + db * BR;
                uint32_t const xh = tm + G::XC0 + (xs % G::NXB) * 2 * KP;
                uint32_t const oy = s * (G::Y1STAGE >> 4);
                bool const last = c1 + 1 == TB;   // the row block's last tile
                if (elect_one()) {
                    // MMA1, K = KP: D = Xh Yh^T (TF32, k-steps of 8 per column block) and the small
                    // terms [bf16(Xh) | bf16(Xl)] [bf16(Yl) ; bf16(Y)]^T (K = 2 KP, k-steps of 16:
                    // the first KP / 16 read bf16(Yl), the rest bf16(Y)), or Xh Yl^T + Xl Yh^T in TF32.
                    // Each MMA truncates its FP32 sums, so D comes out a little small, R = V / D
                    // large and MMA2's sum small again: the two offset each other.  MMA2 has
                    // more steps, so up to rank 32 the small terms come last here, where a step
                    // truncates most, and at 64 first: rms error of one update / 2^-24 with
                    // them first / last 3.8 / 2.2 (20000 x 1000 k = 16), 3.5 / 2.1
                    // (12007 x 1501 k = 20), 3.0 / 2.0 (60000 x 5000 k = 32) and
                    // 1.8 / 3.8 (40009 x 3001 k = 50).
                    constexpr int KPB = G::CB / 8;     // k-steps per swizzle column block
                    auto const main_term = [&](auto sum) {   // sum: added to D
#pragma unroll
                        for (int ks = 0; ks < KP / 8; ks++) {
                            uint64_t const b = desc_at(dY0, oy + (((ks / KPB) * G::YBLK + (ks % KPB) * 32) >> 4));
                            if (ks == 0)
                                mma_ts<decltype(sum)::value>(dcol, xh, b, IDESC1);
                            else
                                mma_ts<true>(dcol, xh + ks * 8, b, IDESC1);
                        }
                    };
                    auto const small_terms = [&](auto sum) {
                        if constexpr (G::LO32) {
                            mma_ts<decltype(sum)::value>(dcol, xh, desc_at(dYB0, oy), IDESC1);
                            mma_ts<true>(dcol, xh + KP, desc_at(dY0, oy), IDESC1);
#pragma unroll
                            for (int ks = 1; ks < KP / 8; ks++) {
                                mma_ts<true>(dcol, xh + ks * 8, desc_at(dYB0, oy + ks * 2), IDESC1);
                                mma_ts<true>(dcol, xh + KP + ks * 8, desc_at(dY0, oy + ks * 2), IDESC1);
                            }
                        } else {
                            mma_ts_bf16<decltype(sum)::value>(dcol, xh + KP, desc_at(dYB0, oy), IDESC1B);
#pragma unroll
                            for (int j = 1; j < KP / 8; j++)
                                mma_ts_bf16<true>(dcol, xh + KP + j * 8,
                                                  desc_at(dYB0, oy + (((j / (KP / 16)) * G::YBB + (j % (KP / 16)) * 32) >> 4)),
                                                  IDESC1B);
                        }
                    };
                    if constexpr (NTERMS != 3) {
                        main_term(std::false_type());
                    } else if constexpr (KP == 64) {
                        small_terms(std::false_type());
                        main_term(std::true_type());
                    } else {
                        main_term(std::false_type());
                        small_terms(std::true_type());
                    }
                    tc_commit(&dfull[db]);
                    tc_commit(&y1empty[s]);
                    if (last) tc_commit(&xfree[xs % G::NXB]);
                    DBG_TS(2, n1);
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
                        atomicExch(args.err, 4u);
                    }
                    ok = false;
                }
            }
        }
        // drain: every MMA issued above has completed (and with it its reads of
        // shared memory and writes of tensor memory) before the CTA frees them
        if (elect_one()) mma_drain(mdrain);
        __syncwarp();
    } else if (warp >= 4 && warp < 4 + NR) {
        // ------------------------------------------------------------ R warps
        // Two teams of NR/2 warps take alternate tiles (team 0 even, team 1 odd), so
        // one team's load latency overlaps the other's arithmetic.  Within a team,
        // warp (quad, grp) handles TMEM lanes 32 quad .. +31 and CW = BR / GPT tile
        // columns, in chunks of 16 (one BF16 k-step of MMA2 each).
        constexpr int TW = NR / 2;                     // warps per team
        constexpr int GPT = TW / 4;                    // column groups per team
        constexpr int CW = BR / GPT;                   // tile columns per warp
        static_assert(CW % 16 == 0, "16-column chunks");
        uint32_t const quad = warp & 3;
        uint32_t const jg = (warp - 4) >> 2;
        uint32_t const team = jg / GPT, grp = jg % GPT;
        uint32_t const row = quad * 32 + lane;        // TMEM lane = output row within the block
        uint32_t const lane_addr = tmem + ((quad * 32) << 16);
        for (uint32_t t = team; t < T; t += 2) {
            uint32_t const s = t % G::VST, b = t % G::NDB;
            uint32_t const c = (c00 + t) % TB;            // reduction tile
            if (warp == 4 && lane == 0) DBG_TS(4, t);
            DBG_PH(0, t);
            if (!mbar_wait_warp(&dfull[b], (t / G::NDB) & 1, abort_flag, args.err, 6u, args.wait_ns)) break;
            DBG_PH(1, t);
            if (!mbar_wait_warp(&vfull[s], (t / G::VST) & 1, abort_flag, args.err, 7u, args.wait_ns)) break;
            tc_fence_after();
            DBG_PH(2, t);
            if (warp == 4 && lane == 0) DBG_TS(5, t);
            const unsigned char *sv = sV + s * G::VBYTES;
            bool const edge = (c + 1) * BR > args.R;      // the partial last reduction tile
            int const valid = (int)(args.R - c * BR);     // its columns before R
            bool aborted = false;
#pragma unroll 1
            for (int ch = 0; ch < CW / 16; ch++) {
                int const col0 = grp * CW + ch * 16;                          // first tile column of the chunk
                uint32_t const dcol = G::DA0 + b * BR + col0;                 // its columns of D
                uint32_t const rlcol = G::RL0 + (t % G::NRL) * (BR / 2) + (col0 / 16) * 8;  // and of bf16(Rl)
                uint32_t d[16];   // D, then the TF32 hi part of R
                uint32_t v[16];   // V, then the lo part of R
                tmem_ld16(lane_addr + dcol, d);
                if (HSIDE) {
                    // V tile [BR rows][128 cols], row-major; this thread's column = row.
                    const float *vs = reinterpret_cast<const float *>(sv) + col0 * BO + row;
#pragma unroll
                    for (int c = 0; c < 16; c++) v[c] = __float_as_uint(vs[c * BO]);
                } else {
                    // V boxes of [128 rows][32 floats], 128B swizzle.
                    int const qb = col0 / 32;
                    int const c0 = (col0 % 32) / 4;      // 16-byte chunk offset within the box
                    const unsigned char *vb = sv + qb * (BO * 128) + row * 128;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint4 const x = *reinterpret_cast<const uint4 *>(vb + (((c + c0) ^ (row & 7)) << 4));
                        v[4 * c + 0] = x.x;
                        v[4 * c + 1] = x.y;
                        v[4 * c + 2] = x.z;
                        v[4 * c + 3] = x.w;
                    }
                }
                tmem_wait_ld_dep(d);
                if (ch == CW / 16 - 1) DBG_PH(4, t);
                if (edge) {
                    // Columns past R are zero-filled (V = 0, WH = 0): WH = 1 there makes R 0
                    // instead of 0 * inf, which MMA2 would carry into every row's sum.
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        if (col0 + c >= valid) {
                            d[c] = 0x3f800000u;
                            v[c] = 0u;
                        }
                }
                uint32_t pl[8];   // bf16(R lo), packed in column pairs
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    // R = V / WH as V * (1/WH): the approximate reciprocal (<= 1 ulp) runs at
                    // full rate, the fast-division intrinsic at a third of it.  A zero WH of
                    // the data behaves as in the reference's division (V / 0 = inf, 0 / 0 = NaN).
                    float const vv = __uint_as_float(v[c]);
                    float const wh = __uint_as_float(d[c]);
                    float const r = vv * rcp_approx(wh);
                    float const h = tf32_rna(r);
#ifdef NMFB_FUSED_DEBUG
                    if (args.dbg && blockIdx.x == 0 && t == 0) {
                        args.dbg[row * 64 + col0 + c] = wh;
                        args.dbg[BO * 64 + row * 64 + col0 + c] = vv;
                        args.dbg[2 * BO * 64 + row * 64 + col0 + c] = h;
                    }
#endif
                    d[c] = __float_as_uint(h);
                    v[c] = __float_as_uint(r - h);
                }
                if (NTERMS == 3) {
#pragma unroll
                    for (int j = 0; j < 8; j++) pl[j] = fin_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                }
                if (ch == CW / 16 - 1) DBG_PH(5, t);
                // this team's bf16(Rl) buffer: MMA2 of the team's previous tile has read it
                // (its commit to y2empty; the next one on that barrier waits for this tile)
                if (NTERMS == 3 && G::NRL < G::NDB && ch == 0 && t >= 2) {
                    if (!mbar_wait_warp(&y2empty[t & 1], ((t >> 1) - 1) & 1, abort_flag, args.err, 5u, args.wait_ns)) {
                        aborted = true;
                        break;
                    }
                    tc_fence_after();
                }
                tmem_st16(lane_addr + dcol, d);
                if (NTERMS == 3) tmem_st8(lane_addr + rlcol, pl);
            }
            if (aborted) break;
            // The V stage is released once its values have been used, not when their loads
            // have been issued: an arrive does not wait for the warp's loads in flight, and
            // the next TMA load could overwrite the stage under them.
            __syncwarp();
            if (lane == 0) mbar_arrive(&vempty[s]);
            DBG_PH(3, t);
            tmem_wait_st();
            DBG_PH(6, t);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&rfull[b]);
            DBG_PH(7, t);
            if (warp == 4 && lane == 0) DBG_TS(6, t);
#ifdef NMFB_FUSED_DEBUG
            if (lane == 0 && dts && blockIdx.x == 0 && t < 64 && warp < 12) dts[512 + (warp - 4) * 64 + t] = globaltimer() - ts0;
#endif
        }
    } else if (warp >= 4 + NR) {
        // ------------------------------------------------------------ accumulator warps
        // Warp 4+NR+4a+q owns TMEM lanes 32q..32q+31 and columns KC a..KC a + KC - 1: sums
        // the per-tile Acc into FP32 registers, writes the sum at the end of each row
        // block (of this CTA's run of tiles), and (all together) splits the X of every
        // row block into tensor memory, ahead of its tiles as soon as an X buffer is free.
        constexpr int KC = KP / G::NA;
        uint32_t const quad = warp & 3;
        uint32_t const k0 = ((warp - 4 - NR) >> 2) * KC;   // first column
        uint32_t const row = quad * 32 + lane;
        uint32_t const lane_addr = tmem + ((quad * 32) << 16);
        uint32_t const nseg = (g0 + T - 1) / TB - ob0 + 1;   // row blocks of the run
        float sum[KC];
#pragma unroll
        for (int c = 0; c < KC; c++) sum[c] = 0.0f;
        // this thread's part of its row of X in row block ob0 + xs as TF32 hi and bf16(hi) | bf16(lo), into TMEM lanes = rows
        auto write_X = [&](uint32_t xs) {
            uint32_t const o = (ob0 + xs) * BO + row;
            const float *xr = args.X + (size_t)o * KP;
            uint32_t const xc = lane_addr + G::XC0 + (xs % G::NXB) * 2 * KP;
#pragma unroll 1   // the sums leave registers for 16 columns at a time
            for (uint32_t c0 = k0; c0 < k0 + KC; c0 += 16) {
                float x[16];
#pragma unroll
                for (int c = 0; c < 16; c += 4) {
                    float4 const v = (o < args.O) ? *reinterpret_cast<const float4 *>(xr + c0 + c)
                                                  : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    x[c] = v.x;
                    x[c + 1] = v.y;
                    x[c + 2] = v.z;
                    x[c + 3] = v.w;
                }
                uint32_t h[8], b8[8];
#pragma unroll
                for (int half = 0; half < 2; half++) {
#pragma unroll
                    for (int c = 0; c < 8; c++) h[c] = __float_as_uint(tf32_rna(x[8 * half + c]));
                    tmem_st8(xc + c0 + 8 * half, h);
                }
                if (NTERMS == 3 && G::LO32) {
#pragma unroll
                    for (int half = 0; half < 2; half++) {
#pragma unroll
                        for (int c = 0; c < 8; c++) h[c] = __float_as_uint(x[8 * half + c] - tf32_rna(x[8 * half + c]));
                        tmem_st8(xc + KP + c0 + 8 * half, h);
                    }
                } else if (NTERMS == 3) {
#pragma unroll
                    for (int c = 0; c < 8; c++) b8[c] = fin_bf16x2(tf32_rna(x[2 * c]), tf32_rna(x[2 * c + 1]));
                    tmem_st8(xc + KP + c0 / 2, b8);
#pragma unroll
                    for (int c = 0; c < 8; c++)
                        b8[c] = fin_bf16x2(x[2 * c] - tf32_rna(x[2 * c]), x[2 * c + 1] - tf32_rna(x[2 * c + 1]));
                    tmem_st8(xc + KP + KP / 2 + c0 / 2, b8);
                }
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&xready[xs % G::NXB]);
        };
        bool ok = true;
        uint32_t xw = 0, ob = ob0, c1 = c00;   // X blocks written; row block and reduction tile of t
        bool gap_done = c00 == 0 || c00 % args.ts.run != 0;
        for (uint32_t t = 0; ok && t < T; t++) {
            uint32_t const bp = t % G::NACC;
            PollLimit limit(args.wait_ns);
            for (;;) {
                // the next row block's X first: MMA1 of its first tile waits for it
                if (xw < nseg &&
                    (xw < G::NXB || __all_sync(0xffffffffu, mbar_test(&xfree[xw % G::NXB], ((xw / G::NXB) - 1) & 1)))) {
                    tc_fence_after();
                    write_X(xw);
                    xw++;
                    limit.reset();
                    continue;
                }
                if (__all_sync(0xffffffffu, mbar_try_wait(&accrdy[bp], (t / G::NACC) & 1))) break;
                bool const stop = *abort_flag != 0;
                bool const late = limit.expired();
                if (__any_sync(0xffffffffu, stop || late)) {
                    if (!stop && lane == 0) {
                        *abort_flag = 1;
                        atomicExch(args.err, 8u);
                    }
                    ok = false;
                    break;
                }
            }
            if (!ok) break;
            tc_fence_after();
            // Acc columns [0, KP) plus, for the 3-term arm, [KP, 2 KP): the tile's sum, added
            // to the running one in one rounding.
#pragma unroll
            for (int c0 = 0; c0 < KC; c0 += 16) {
                uint32_t a[16], a2[16];
                tmem_ld16(lane_addr + bp * ACC_COLS + k0 + c0, a);
                if (NTERMS == 3) tmem_ld16(lane_addr + bp * ACC_COLS + KP + k0 + c0, a2);
                tmem_wait_ld_dep(a);
                if (NTERMS == 3) tmem_wait_ld_dep(a2);
#pragma unroll
                for (int c = 0; c < 16; c++)
                    sum[c0 + c] += NTERMS == 3 ? __uint_as_float(a[c]) + __uint_as_float(a2[c]) : __uint_as_float(a[c]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&accfree[bp]);
            if (warp == 4 + NR && lane == 0) DBG_TS(7, t);
#ifdef NMFB_FUSED_DEBUG
            if (lane == 0 && dts && blockIdx.x == 0 && t < 64) dts[1024 + (warp - 4 - NR) * 64 + t] = globaltimer() - ts0;
            if (args.dbg && blockIdx.x == 0 && t + 1 == T)
                for (int c = 0; c < KC; c++) args.dbg[3 * BO * 64 + row * KP + k0 + c] = sum[c];
#endif
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
PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
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

int encode_2d(nmfb_ctx *ctx, CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint64_t row_bytes,
              uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw,
              CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT32)
{
    auto fn = encode_fn();
    if (!fn) return nmfb_fail(ctx, NMFB_ENODEV, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(map, dt, 2, (void *)base, dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return nmfb_fail(ctx, NMFB_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return NMFB_OK;
}

// Layout of one factor's split copies (k_finish's outputs), in one buffer:
// hi (rows x kp FP32) | transposed hi/lo per 32 rows | bf16(lo) (rows x kp) |
// bf16(y) (rows x kp) | bf16(y) transposed per br rows; at kp = 16 lo itself (FP32)
// in place of bf16(lo) | bf16(y).
struct SplitLayout {
    size_t t, bl, b, bt, floats;   // offsets in floats (bl, b, bt: start of the BF16 parts)
    uint32_t br, nblk32, nblkbr;
    SplitLayout(uint32_t rows, uint32_t kp)
    {
        br = 64;
        nblk32 = (rows + 31) / 32;
        nblkbr = (rows + br - 1) / br;
        size_t const f = (size_t)rows * kp;
        t = f;
        bl = t + (size_t)nblk32 * 64 * kp;
        b = bl + f / 2;                                   // rows * kp BF16 = f / 2 floats (kp is even)
        bt = b + f / 2;
        floats = bt + ((size_t)nblkbr * kp * br + 1) / 2;
    }
};

struct FusedPlan {
    FusedMaps mapsH, mapsW;  // update_H (HSIDE) and update_W
    uint32_t *dErr;
    float *dSplitW, *dSplitH;  // split copies of W and of H (SplitLayout)
    double *dCsW, *dCsH;       // [CTAs of k_finish][kp] column-sum partials of W and of H
#ifdef NMFB_FUSED_DEBUG
    float *dDbg;
#endif
};

// k_finish on W (or H): its update from the partials, or, with update = false,
// only its split copies and column-sum partials.
template <int KP>
int launch_finish(nmfb_ctx *ctx, bool w, bool update, int adjust)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    FinishArgs fa = {};
    float *xsp = w ? plan->dSplitW : plan->dSplitH;
    fa.O = w ? ctx->n : ctx->m;
    SplitLayout const L(fa.O, KP);
    fa.ts = plan_of(ctx, w);
    fa.k = ctx->k;
    fa.adjust = adjust;
    fa.part = update ? ctx->dPart : nullptr;
    fa.X = w ? ctx->dW : ctx->dH;
    fa.accY = w ? ctx->dAccH : ctx->dAccW;
    fa.xhi = xsp;
    fa.xT = xsp + L.t;
    fa.xBl = reinterpret_cast<__nv_bfloat16 *>(xsp + L.bl);
    fa.xB = reinterpret_cast<__nv_bfloat16 *>(xsp + L.b);
    fa.xBT = reinterpret_cast<__nv_bfloat16 *>(xsp + L.bt);
    fa.xnblk32 = L.nblk32;
    fa.xnblkbr = L.nblkbr;
    fa.cs = w ? plan->dCsW : plan->dCsH;
    fa.st = ctx->dState;
    NMFB_CUDA_TRY(ctx, (fin_launch<KP, 64, 0>(fa, ctx->stream)));
    NMFB_LAUNCH_CHECK(ctx);
    return NMFB_OK;
}

template <bool HSIDE, int KP, int NTERMS>
int launch_fused(nmfb_ctx *ctx, const FusedMaps &maps, int adjust)
{
    using G = Geo<KP>;
    static_assert(G::BR == 64, "plan_of");
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    FusedArgs args;
    args.O = HSIDE ? ctx->m : ctx->n;
    args.R = HSIDE ? ctx->n : ctx->m;
    args.ts = plan_of(ctx, !HSIDE);
    if ((size_t)args.ts.slots * args.O * KP > ctx->part_items)
        return nmfb_fail(ctx, NMFB_EINVAL, "fused: partial buffer too small (%u slots)", args.ts.slots);
    args.csy.cs = HSIDE ? plan->dCsW : plan->dCsH;
    args.csy.nblk = fin_blocks(args.R, fin_rpt(plan_of(ctx, HSIDE).slots));
    args.csy.acc = HSIDE ? ctx->dAccW : ctx->dAccH;
    args.part = ctx->dPart;
    args.err = plan->dErr;
    args.st = ctx->dState;
    args.X = HSIDE ? ctx->dH : ctx->dW;
    args.wait_ns = ctx->wait_ns ? ctx->wait_ns : WAIT_LIMIT_NS;
#ifdef NMFB_FUSED_DEBUG
    args.dbg = plan->dDbg;
#endif
    int const main = HSIDE ? 0 : 1;
    int rc = nmfb_prof_begin(ctx, main);
    if (rc) return rc;
    NMFB_CUDA_TRY(ctx, launch_chained(k_fused_half<HSIDE, KP, NTERMS>, args.ts.ctas(), G::NTHR, G::SMEM, ctx->stream, maps,
                                      args));
    NMFB_LAUNCH_CHECK(ctx);
    if ((rc = nmfb_prof_end(ctx, main))) return rc;
    return launch_finish<KP>(ctx, !HSIDE, true, adjust);
}

template <bool HSIDE>
int dispatch(nmfb_ctx *ctx, const FusedMaps &maps, int adjust)
{
    bool const x3 = ctx->arm == NMFB_ARM_FUSED;
    switch (ctx->kp) {
    case 16: return x3 ? launch_fused<HSIDE, 16, 3>(ctx, maps, adjust) : launch_fused<HSIDE, 16, 1>(ctx, maps, adjust);
    case 32: return x3 ? launch_fused<HSIDE, 32, 3>(ctx, maps, adjust) : launch_fused<HSIDE, 32, 1>(ctx, maps, adjust);
    case 64: return x3 ? launch_fused<HSIDE, 64, 3>(ctx, maps, adjust) : launch_fused<HSIDE, 64, 1>(ctx, maps, adjust);
    default: return nmfb_fail(ctx, NMFB_EINVAL, "fused arm: unsupported padded rank %u", ctx->kp);
    }
}

// Split copies and column-sum partials of a factor, for a half-iteration that
// reads it as Y when the previous one's k_finish did not leave them.
int prepare_factor(nmfb_ctx *ctx, bool w)
{
    int const rc = ctx->kp == 16   ? launch_finish<16>(ctx, w, false, 0)
                   : ctx->kp == 32 ? launch_finish<32>(ctx, w, false, 0)
                                   : launch_finish<64>(ctx, w, false, 0);
    if (!rc) ctx->fz_ok[w ? 0 : 1] = 1;
    return rc;
}

// One half-iteration: two launches when the other factor's split copies and
// column-sum partials are current (the previous half-iteration's k_finish left them).
int fused_half(nmfb_ctx *ctx, bool is_H, int adjust)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    if (!plan) return nmfb_fail(ctx, NMFB_ESTATE, "fused arm not prepared");
    int const whole = is_H ? 2 : 3;
    int rc = nmfb_prof_begin(ctx, whole);
    if (rc) return rc;
    bool const yw = is_H;   // Y = W for update_H
    if (!ctx->fz_ok[yw ? 0 : 1] && (rc = prepare_factor(ctx, yw))) return rc;
    rc = is_H ? dispatch<true>(ctx, plan->mapsH, adjust) : dispatch<false>(ctx, plan->mapsW, adjust);
    if (rc) return rc;
    ctx->fz_ok[is_H ? 1 : 0] = 1;
    return nmfb_prof_end(ctx, whole);
}

}  // namespace

template <int KP>
int set_smem_attrs(nmfb_ctx *ctx)
{
    int const smem = Geo<KP>::SMEM;
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_half<true, KP, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_half<false, KP, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_half<true, KP, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NMFB_CUDA_TRY(ctx, cudaFuncSetAttribute(k_fused_half<false, KP, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return NMFB_OK;
}

int nmfb_fused_prepare(nmfb_ctx *ctx)
{
    if (ctx->tmaps) return NMFB_OK;
    uint32_t const kp = ctx->kp;
    if (kp != 16 && kp != 32 && kp != 64)
        return nmfb_fail(ctx, NMFB_EINVAL, "the fused arm supports ranks up to 64 (k=%u); use the plain arm", ctx->k);
    int rc = (kp == 16) ? set_smem_attrs<16>(ctx) : (kp == 32) ? set_smem_attrs<32>(ctx) : set_smem_attrs<64>(ctx);
    if (rc) return rc;
    FusedPlan *plan = (FusedPlan *)calloc(1, sizeof(FusedPlan));
    if (!plan) return nmfb_fail(ctx, NMFB_ENOMEM, "fused plan");
    ctx->tmaps = plan;
    cudaError_t e = nmfb_malloc(ctx, (void **)&plan->dErr, sizeof(uint32_t));
    if (e != cudaSuccess) return nmfb_fail(ctx, NMFB_ENOMEM, "fused error word: %s", cudaGetErrorString(e));
    NMFB_CUDA_TRY(ctx, cudaMemsetAsync(plan->dErr, 0, sizeof(uint32_t), ctx->own_stream));
#ifdef NMFB_FUSED_DEBUG
    NMFB_CUDA_TRY(ctx, nmfb_malloc(ctx, (void **)&plan->dDbg, (4 * BO * 64 + 8192) * sizeof(float)));
    NMFB_CUDA_TRY(ctx, cudaMemsetAsync(plan->dDbg, 0, (4 * BO * 64 + 8192) * sizeof(float), ctx->own_stream));
#endif
    uint32_t const cb = (kp == 16) ? 16 : 32;
    CUtensorMapSwizzle const fsw = (kp == 16) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    auto const sw_for = [](uint32_t bytes) {
        return bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    };
    CUtensorMapDataType const BF16 = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    uint64_t const vrow = ctx->ldv * sizeof(float), frow = (uint64_t)kp * sizeof(float);
    SplitLayout const LW(ctx->n, kp), LH(ctx->m, kp);
    uint32_t const br = LW.br;
    e = nmfb_malloc(ctx, (void **)&plan->dSplitW, LW.floats * sizeof(float));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->dSplitH, LH.floats * sizeof(float));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->dCsW, (size_t)fin_blocks(ctx->n, 1) * kp * sizeof(double));
    if (e == cudaSuccess) e = nmfb_malloc(ctx, (void **)&plan->dCsH, (size_t)fin_blocks(ctx->m, 1) * kp * sizeof(double));
    if (e != cudaSuccess) return nmfb_fail(ctx, NMFB_ENOMEM, "fused split buffers: %s", cudaGetErrorString(e));
    // Maps over one factor's split copies: Y (the other factor, `rows` rows).
    auto const y_maps = [&](FusedMaps &mp, const float *sp, const SplitLayout &L, uint32_t rows) -> int {
        int r;
        if ((r = encode_2d(ctx, &mp.y, sp, kp, rows, frow, cb, br, fsw))) return r;
        if (kp == 16)
            r = encode_2d(ctx, &mp.ylb, sp + L.bl, kp, rows, frow, cb, br, fsw);
        else
            r = encode_2d(ctx, &mp.ylb, sp + L.bl, kp, rows, (uint64_t)kp * 2, kp, br, sw_for(2 * kp), BF16);
        if (r) return r;
        if ((r = encode_2d(ctx, &mp.yt, sp + L.t, 32, (uint64_t)L.nblk32 * 2 * kp, 128, 32, 2 * kp * (br / 32),
                           CU_TENSOR_MAP_SWIZZLE_128B)))
            return r;
        if ((r = encode_2d(ctx, &mp.yb, sp + L.b, kp, rows, (uint64_t)kp * 2, kp, br, sw_for(2 * kp), BF16))) return r;
        return encode_2d(ctx, &mp.ybt, sp + L.bt, br, (uint64_t)L.nblkbr * kp, (uint64_t)br * 2, br, kp,
                         sw_for(2 * br), BF16);
    };
    // update_H: X = H (rows m), Y = W (rows n); V tile [br rows of V][128 cols].
    FusedMaps &mh = plan->mapsH;
    if ((rc = encode_2d(ctx, &mh.v, ctx->dV, ctx->m, ctx->n, vrow, BO, br, CU_TENSOR_MAP_SWIZZLE_NONE))) return rc;
    if ((rc = y_maps(mh, plan->dSplitW, LW, ctx->n))) return rc;
    // update_W: X = W (rows n), Y = H (rows m); V tile [128 rows][32 cols] x (br/32), 128B swizzle.
    FusedMaps &mw = plan->mapsW;
    if ((rc = encode_2d(ctx, &mw.v, ctx->dV, ctx->m, ctx->n, vrow, 32, BO, CU_TENSOR_MAP_SWIZZLE_128B))) return rc;
    if ((rc = y_maps(mw, plan->dSplitH, LH, ctx->m))) return rc;
    return NMFB_OK;
}

int nmfb_fused_release(nmfb_ctx *ctx)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    if (!plan) return NMFB_OK;
    if (plan->dErr) nmfb_free(ctx, plan->dErr);
    if (plan->dSplitW) nmfb_free(ctx, plan->dSplitW);
    if (plan->dSplitH) nmfb_free(ctx, plan->dSplitH);
    if (plan->dCsW) nmfb_free(ctx, plan->dCsW);
    if (plan->dCsH) nmfb_free(ctx, plan->dCsH);
    free(plan);
    ctx->tmaps = nullptr;
    return NMFB_OK;
}

int nmfb_fused_update_H(nmfb_ctx *ctx, int adjust) { return fused_half(ctx, true, adjust); }

// Makes W's split copies and column sums current (before a test block is
// replayed as a graph, which holds no preparation launch).
int nmfb_fused_ready_W(nmfb_ctx *ctx)
{
    if (!ctx->tmaps || ctx->fz_ok[0]) return NMFB_OK;
    return prepare_factor(ctx, true);
}
int nmfb_fused_update_W(nmfb_ctx *ctx, int adjust) { return fused_half(ctx, false, adjust); }

uint32_t *nmfb_fused_err_word(nmfb_ctx *ctx)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    return plan ? plan->dErr : nullptr;
}

// Reads the fused kernels' error word (the site of the first bounded wait that
// ran out, 0 if none) and clears it, so each expiry is reported once and the
// context stays usable.
int nmfb_fused_error(nmfb_ctx *ctx, uint32_t *code)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    *code = 0;
    if (!plan) return NMFB_OK;
    NMFB_CUDA_TRY(ctx, cudaMemcpyAsync(code, plan->dErr, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
    NMFB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    if (*code) {
        // an aborted launch leaves factor copies behind that match no factor
        NMFB_CUDA_TRY(ctx, cudaMemsetAsync(plan->dErr, 0, sizeof(uint32_t), ctx->stream));
        ctx->fz_ok[0] = ctx->fz_ok[1] = 0;
        NMFB_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return NMFB_OK;
}

#ifdef NMFB_FUSED_DEBUG
extern "C" int nmfb_debug_dump(nmfb_ctx *ctx, float *host)
{
    FusedPlan *plan = (FusedPlan *)ctx->tmaps;
    NMFB_CUDA_TRY(ctx, cudaMemcpy(host, plan->dDbg, (4 * BO * 64 + 8192) * sizeof(float), cudaMemcpyDeviceToHost));
    return NMFB_OK;
}
#endif
