// cs_kernels_split_tc3d.cu — split-precision sweep for dense 3x3x3 (27-point)
// kernels on the fifth-generation tensor cores (tcgen05.mma, TMEM).
//
// Arithmetic: as in the 2D tcgen05 kernel (cs_kernels_split_tc.cu). Inputs
// (hi, lo) are scaled by a power of two per input plane of a tile and cut
// into five balanced 9-bit digits held exactly in FP16; the weights are cut
// the same way with one scale. Products of digit k of x and digit e of w with
// k + e = L land in one FP32 accumulator per level L, input plane and output
// plane; such a level sums at most 9 * 5 products below 2^16, so it is exact
// in any order, and the levels are recombined error-free into (hi, lo).
//
// Mapping (M = 128, K = 16):
//   * A work item is a column of output tiles, 16 rows x 64 columns on zc
//     consecutive planes. The CTA loads each input plane of the column once
//     (planes z0-1 .. z0+zc), by one 3D TMA load of rows y0-1 .. y0+16 and
//     columns x0-4 .. x0+67, and cuts it into five digit planes (18 rows of
//     72 halves).
//   * Row m of A is the 16-wide window of block b = m % 8 (8 output columns)
//     in output row r = m / 8: a K-major, non-swizzled descriptor with a
//     16-byte K-chunk stride and a stride of one plane row between 8-row
//     groups reads it out of the digit plane in place; window row offset i
//     (0..2) is the same descriptor started i rows lower.
//   * Input plane P feeds output planes P+1, P and P-1 as their z taps
//     dz = 0, 1, 2, and its MMAs serve all three at once: column n of B_i is
//     (weight digit e, tap plane dz, column c), n = 24 e + 8 dz + c, with
//     B[k][n] = w_e[dz][i][k - c - 3]. For input digit d one MMA with
//     N = 24 (5 - d), rounded up to 16s, feeds levels d..4 of the plane's TMEM
//     block: 3 row offsets x 5 digits = 15 MMAs per input plane and 1024
//     outputs.
//   * Each input plane has its own 128-column TMEM block (ring of four), so
//     every plane keeps its own scale. (Levels of 32 columns, one in four of
//     them padding, took rings of three and, FP64, of two; GB300, us a sweep:
//     split 128^3 20.8 and 19.8, 512^3 740 and 734; FP64 512^3 1112 and 1107.) The
//     epilogue
//     reads a block once, as soon as its MMAs are done, hands it back, and
//     adds its three tap-plane parts to the running sums of output planes
//     P+1 (dz = 0), P (dz = 1) and P-1 (dz = 2, its last: stored). Parts of
//     one output with the same plane scale (the usual case) are added as
//     exact level sums and recombined once; otherwise as (hi, lo) pairs
//     relative to the largest scale.
//   * Roles: one warp issues the window loads (six stage buffers), one
//     thread issues the MMAs, three groups of four warps cut every third
//     input plane into digit planes (ring of seven; a plane is too small for
//     many warps to share without waiting on each other; only the window
//     columns that meet nonzero weights are cut), and eight warps (a TMEM
//     lane quarter and half of the 8 columns each) drain the blocks,
//     recombine, scale once and store. No slicer shares the MMA thread's
//     warp scheduler.
//
// Every mbarrier wait is bounded (WaitCfg, 2 s by default). An expired wait is
// counted in g_tc3d_wait_timeouts; the CTA then waits, again bounded, for the
// TMA copies and the MMAs it still has in flight, frees its TMEM and leaves.
#include "cs_internal.h"
#include "cs_split_common.cuh"
#include "cs_tc_common.cuh"
#include "cs_tc_f64.cuh"

#include <algorithm>
#include <type_traits>

namespace cs {

__device__ unsigned int g_tc3d_wait_timeouts;

namespace {

using split::kDigitBits;
using split::SliceWeights;
using split::slice_digits;
using split::two_sum;
using namespace tc;

// Number formats: split (FP32 (hi, lo) grids, five digits, a ring of four
// 128-column TMEM blocks) and FP64 (FP64 grids, six digits cut with integer
// operations as in the 2D kernel, a ring of three 160-column blocks). LV: levels
// kept; kBlk: TMEM columns from one input plane's block to the next.
//
// FP64 is bound by its epilogue and the slicers' integer operations: 155
// instructions an output, 0.6 of the schedulers' slots (GB300, star3d1r 512^3, 861
// us a sweep). Not faster: conversions to FP64 by integer operations (1200 us
// against 1112 then), two columns a step with the next ones' loads in flight
// (1277), all three parts loaded first with 112 registers for the epilogue by
// setmaxnreg (1287; split 826 against 738), sixteen epilogue warps (1171 against
// 1126), two planes per loop iteration (930 against 897, spills).
// Again: what computes an output again (Redo).
struct NoAgain {
};
struct SumAgain {
    const double *in;  // interior point (0, 0, 0) of the source
    int pattern, redo;
    double w[27];
};
struct F3Split {
    static constexpr bool kF64 = false;
    static constexpr int D = split::kDigits, LV = D;  // 5
    static constexpr int NBLK = 4, kBlk = 128;
    using Out = float2;
    using Digits = SliceWeights;
    using Again = NoAgain;
};
struct F3F64 {
    static constexpr bool kF64 = true;
    static constexpr int D = 6, LV = 6;
    static constexpr int NBLK = 3, kBlk = 160;
    using Out = double;
    using Digits = F64Weights;
    using Again = NoAgain;
};
// FP64 with level 6 too, inputs rounded to even and the weights' sum kept, as
// the 2D kernel's FmtF64Fine: errors no larger than those of FP64 FMA sweeps
// (box3d1r, uniform data, error of the norm: 64 x 60 x 66 x 30 sweeps 3.0e-15 with
// six levels, 7.5e-17 so, FP64 FMA 1.4e-16; 128 x 130 x 125 x 100 9.9e-15, 8.0e-17,
// 1.4e-16. star3d1r 160 x 128 x 125 x 100 1.25e-16 against 9.2e-17 of its seven FMA, so
// the server keeps it on those).
struct F3F64Fine : F3F64 {
    static constexpr int LV = 7, kBlk = 168;
    using Again = SumAgain;
};

// Warp roles. Warp w issues from the SM's scheduler w % 4, and an epilogue
// warp can read only TMEM lanes 32 (w % 4) .. + 31, so each scheduler hosts
// two epilogue warps. The MMA thread stalls on every tcgen05.mma until the
// tensor core takes it, so every issue slot it loses to a busy neighbour
// stretches the MMA stream: it shares scheduler 1 with the TMA warp, the two
// epilogue warps of lane quarter 1 and two idle warps, and the twelve slicer
// warps sit on schedulers 0, 2 and 3 (box3d1r 512^3 on GB300: 135 -> 148
// GStencil/s against slicers spread over all four). 24 warps, six per
// scheduler, leave 80 registers a thread.
constexpr int kGroups = 3, kGroupWarps = 4;  // slicer groups of four warps take every third plane
constexpr int kSliceWarps = kGroups * kGroupWarps, kEpiWarps = 8;
constexpr int kWarpTma = 1, kWarpMma = 5;
constexpr unsigned kEpiMask = (1u << 0) | (1u << 2) | (1u << 3) | (1u << 4) | (1u << 6) | (1u << 7) | (1u << 9) |
                              (1u << 13);
constexpr unsigned kSliceMask = (1u << 8) | (1u << 10) | (1u << 11) | (1u << 12) | (1u << 14) | (1u << 15) |
                                (1u << 16) | (1u << 18) | (1u << 19) | (1u << 20) | (1u << 22) | (1u << 23);
constexpr int kThreads = 32 * 24;  // warps 17 and 21 idle
constexpr int kGroupThreads = 32 * kGroupWarps;
static_assert(__builtin_popcount(kSliceMask) == kSliceWarps && __builtin_popcount(kEpiMask) == kEpiWarps &&
                  (kSliceMask & kEpiMask) == 0 && ((kSliceMask | kEpiMask) & ((1u << kWarpTma) | (1u << kWarpMma))) == 0,
              "warp roles overlap");
static_assert((kSliceMask & 0x22222222u) == 0 && (kWarpMma & 3) == 1, "no slicer beside the MMA thread");
constexpr int kSliceBarrier = 1;             // named barriers 1 .. kGroups: one per slicer group

constexpr int G = 16;                        // output rows per tile (M = G x 8 blocks = 128)
constexpr int TX = 64, TY = G;               // output tile 16 x 64
constexpr int ST_X = TX + 8, ST_Y = TY + 2;  // window: columns x0-4 .. x0+67, rows y0-1 .. y0+16
constexpr int PL = ST_X * ST_Y;              // halves per digit plane (2,592 bytes)
constexpr unsigned kRowBytes = ST_X * 2;     // 144
constexpr int NOFF = 3;                      // window row offsets
constexpr int NLV = 24;                      // TMEM columns per level: 3 tap planes x 8
// N of an MMA that feeds `levels` levels: M = 128 wants multiples of 16, so odd
// counts take 8 columns more, of a level that does not exist; they lie behind
// the block's last level and are not read.
// With seven levels there is no room behind it: the 8 columns come first, from 8
// zero rows before B_i's (kFront).
__host__ __device__ constexpr int mma_n(int levels) { return (NLV * levels + 15) / 16 * 16; }
template <class F>
constexpr int kFront = F::LV > F::D ? 8 : 0;
template <class F>
constexpr int kNcol = kFront<F> + mma_n(F::D);  // rows of B_i: 128 split, 144 FP64 (152)
constexpr int kTmemCols = 512;
constexpr int kStages = 2 * kGroups;         // TMA window buffers (two per slicer group)
constexpr int NPL = 7;                       // digit-plane sets (ring); also keeps one CTA per SM
constexpr int kScaleRing = 32;               // per-input-plane scale exponents (ring)
constexpr unsigned kStageBytes = ST_X * ST_Y * 8;  // 10,368 (8-byte points)
// Column pairs of a window row. Only window columns 3..68 meet a nonzero
// weight (block b reads columns 8b .. 8b+15, taps at k = c+3 .. c+5), so the
// slicers cut pairs 1..34 (columns 2..69); the digit planes' columns 0, 1, 70
// and 71 keep the zeros they are initialised with (the MMAs multiply them by
// zero weights, so they only need to be finite).
constexpr int PAIRS = ST_X / 2, CUT0 = 1, NCUTX = 34, NCUT = ST_Y * NCUTX;  // 36, 612
constexpr int PER = (NCUT + kGroupThreads - 1) / kGroupThreads;            // 5
static_assert(F3Split::NBLK * F3Split::kBlk <= kTmemCols && F3F64::NBLK * F3F64::kBlk <= kTmemCols &&
                  F3F64Fine::NBLK * F3F64Fine::kBlk <= kTmemCols && NLV * F3F64Fine::LV <= F3F64Fine::kBlk,
              "TMEM blocks exceed the allocation");
static_assert(kEpiWarps == 8, "two epilogue warps per TMEM lane quarter, four columns each");
static_assert(kStageBytes % 128 == 0, "TMA destinations stay 128-byte aligned");

template <class F>
struct Smem {
    uint4 stage[kStages][ST_Y * PAIRS];        // TMA destinations: pairs of 8-byte points
    __half planes[NPL][F::D][PL];              // digit planes of input planes (ring)
    __half bmat[NOFF][kNcol<F> * 16];          // B_i, K-major 8x16-byte core matrices
    unsigned long long stage_full[kStages], stage_empty[kStages];
    unsigned long long planes_full[NPL], planes_empty[NPL];
    unsigned long long blk_full[F::NBLK], blk_empty[F::NBLK];
    unsigned tmem;                             // TMEM base column
    int abort;                                 // set by the first expired wait
    int scale_exp[kScaleRing];                 // input-plane scale exponents by plane sequence
    float red[kGroups][2][kGroupWarps];           // split: per-warp max |hi|
    int redi[kGroups][2][kGroupWarps];            // FP64: per-warp max biased exponent
    std::conditional_t<F::LV == 7, Redo, NoRedo> redo;  // input planes that hold an Inf or NaN
};
static_assert(sizeof(Smem<F3F64Fine>) + 128 <= 232448 && sizeof(Smem<F3Split>) + 128 <= 232448,
              "shared memory of one CTA must stay within 227 KB");

// The MMAs of one input plane: window row offset I, input digit D. `a`
// addresses digit 0, row 0 of the plane's digit planes; descriptor
// addresses advance in 16-byte units.
template <class F, int I, int D>
__device__ __forceinline__ void plane_mma(unsigned d_base, unsigned long long a, unsigned long long b0)
{
    constexpr int NCOL = kNcol<F>;
    constexpr unsigned long long a_off = ((unsigned long long)D * PL * 2 + I * kRowBytes) >> 4;
    constexpr unsigned long long b_off = ((unsigned long long)I * NCOL * 16 * 2) >> 4;
    static_assert(((unsigned long long)D * PL * 2 + I * kRowBytes) % 16 == 0 && (NCOL * 16 * 2) % 16 == 0,
                  "descriptor offsets must be 16-byte multiples");
    if constexpr (F::LV == F::D) {
        mma_f16(d_base + (unsigned)(NLV * D), a + a_off, b0 + b_off, instr_desc(mma_n(F::D - D)),
                (I | D) != 0 ? 1u : 0u);
    } else {
        // Levels D .. D + W - 1 (fewer: level 6 of the first row offset comes
        // from an MMA of its own, below).
        static_assert(F::LV == 7 && F::D == 6 && kFront<F> == 8);
        constexpr int W = (I == 0 && D == 1) ? 5 : F::LV - D < F::D ? F::LV - D : F::D, pad = NLV * W % 16;
        constexpr unsigned long long row = (unsigned long long)(kFront<F> - pad) * 32 >> 4;  // 8 rows: 256 bytes
        if constexpr (I == 0 && D == 0) {
            // Digit 1 with the weights' digit 5 initialises level 6, and with it
            // the 8 columns before it, which digit 0 initialises next.
            mma_f16(d_base + (unsigned)(NLV * 6 - 8), a + (PL * 2 >> 4), b0 + (unsigned long long)((8 + NLV * 5 - 8) * 32 >> 4),
                    instr_desc(32), 0u);
        }
        mma_f16(d_base + (unsigned)(NLV * D - pad), a + a_off, b0 + b_off + row, instr_desc(NLV * W + pad),
                (I | D) != 0 ? 1u : 0u);
    }
    if constexpr (D + 1 < F::D)
        plane_mma<F, I, D + 1>(d_base, a, b0);
    else if constexpr (I + 1 < NOFF)
        plane_mma<F, I + 1, 0>(d_base, a, b0);
}

// Work item `item` of the sweep: output tile column (x0, y0) on planes
// zs .. zs + zn - 1. Items run x fastest, then y, then the plane chunk, so
// CTAs working at the same time share window rows in L2.
struct Item {
    int x0, y0, zs, zn;
};

__device__ __forceinline__ Item item_of(int item, int tiles_x, int tiles_y, int zc, int h)
{
    const int txy = tiles_x * tiles_y;
    const int chunk = item / txy, rem = item - chunk * txy;
    const int ty = rem / tiles_x;
    Item it;
    it.x0 = (rem - ty * tiles_x) * TX;
    it.y0 = ty * TY;
    it.zs = chunk * zc;
    it.zn = min(zc, h - it.zs);
    return it;
}

__device__ __forceinline__ void tmem_ld4(unsigned taddr, float (&v)[4])
{
    unsigned r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(r[j]);
}

// Recombines five exact level sums (level L in units of 2^-9L) into a
// double-float pair.
__device__ __forceinline__ void recombine(const float (&acc)[split::kDigits], float &hi, float &lo)
{
    float h1, e1, h2, e2;
    two_sum(acc[0], acc[1] * 0x1p-9f, h1, e1);
    two_sum(h1, acc[2] * 0x1p-18f, h2, e2);
    const float tail = fmaf(acc[3], 0x1p-27f, acc[4] * 0x1p-36f);
    two_sum(h2, (e1 + e2) + tail, hi, lo);
}

template <class F>
__global__ void __launch_bounds__(kThreads, 1)
    k3d_tc(const __grid_constant__ CUtensorMap tmap, typename F::Out *__restrict__ out, int h, int m, int n,
           long long ldy, long long ldz, int tiles_x, int tiles_y, int zc, int items, int map_x, int map_y,
           int map_z, typename F::Digits sw, WaitCfg wc, const __grid_constant__ typename F::Again again)
{
    constexpr int D = F::D, NBLK = F::NBLK, NCOL = kNcol<F>;
    extern __shared__ unsigned char smem_raw[];
    Smem<F> &S = *reinterpret_cast<Smem<F> *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_allow_dependents();
    volatile int *abort = &S.abort;
    auto bar = [](unsigned long long *b, int i) { return smem_addr(&b[i]); };
    const unsigned long long limit = wc.limit_ns;
    auto wait = [abort, limit](unsigned b, unsigned parity) {
        return mbar_wait(b, parity, abort, &g_tc3d_wait_timeouts, limit);
    };
    const int first = blockIdx.x, step = gridDim.x;

    int issued = 0, committed = 0;  // window loads issued / input planes committed (one thread each)
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(bar(S.stage_full, i), 1);
            mbar_init(bar(S.stage_empty, i), kGroupWarps);
        }
        for (int i = 0; i < NPL; ++i) {
            mbar_init(bar(S.planes_full, i), kGroupWarps);
            mbar_init(bar(S.planes_empty, i), 1);
        }
        for (int i = 0; i < NBLK; ++i) {
            mbar_init(bar(S.blk_full, i), 1);
            mbar_init(bar(S.blk_empty, i), kEpiWarps);
        }
        S.abort = 0;
        if constexpr (F::LV == 7) S.redo.count = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarpTma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&S.tmem)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // B_i: N row nn = NLV e + 8 dz + c (digit e of w, z tap dz, column c of the
    // block), K index k; a thread takes 8 k at a time. (One at a time, and
    // the planes zeroed by words: GB300, 64^3 12.7 us a sweep FP64 and 10.6 split,
    // so 10.2 and 8.0.)
    for (int idx = tid; idx < NOFF * NCOL * 2; idx += kThreads) {
        const int i = idx / (NCOL * 2), rem = idx - i * (NCOL * 2), kc = rem / NCOL, nn = rem - kc * NCOL;
        const int n0 = nn - kFront<F>, e = n0 / NLV, dz = n0 % NLV >> 3, c = nn & 7;
        unsigned long long lo = 0, hi = 0;
#pragma unroll
        for (int tj = 0; tj < 3; ++tj) {
            const int k = c + 3 + tj - 8 * kc;
            if (n0 < 0 || e >= D || k < 0 || k >= 8) continue;
            const unsigned long long v = __half_as_ushort(sw.d[e][(dz * 3 + i) * 3 + tj]);
            if (k < 4)
                lo |= v << 16 * k;
            else
                hi |= v << 16 * (k - 4);
        }
        *reinterpret_cast<ulonglong2 *>(&S.bmat[i][(nn >> 3) * 128 + (nn & 7) * 8 + kc * 64]) = make_ulonglong2(lo, hi);
    }
    for (int i = tid; i < NPL * D * PL / 8; i += kThreads)
        reinterpret_cast<uint4 *>(&S.planes[0][0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // All 512 columns are this CTA's, so they start at column 0: as a constant
    // it costs the MMA thread no move into a uniform register per MMA.
    const unsigned tmem = 0;

    if (warp == kWarpTma) {
        // ------------------------------------------------ TMA producer
        if (lane == 0 && !wc.skip_loads) {
            pdl_wait();  // the previous sweep has finished with both buffers
            int q = 0;  // input-plane sequence number
            bool ok = true;
            for (int item = first; item < items && ok; item += step) {
                const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
                for (int p = 0; p < wi.zn + 2; ++p, ++q) {
                    const int sb = q % kStages;
                    if (!(ok = wait(bar(S.stage_empty, sb), ((q / kStages) & 1) ^ 1))) break;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_expect_tx(bar(S.stage_full, sb), kStageBytes);
                    tma_load_3d(smem_addr(S.stage[sb]), &tmap, map_x + wi.x0 - 4, map_y + wi.y0 - 1,
                                map_z + wi.zs - 1 + p, bar(S.stage_full, sb));
                    issued = q + 1;
                }
            }
        }
    } else if (warp == kWarpMma) {
        // ------------------------------------------------ MMA issuer
        const unsigned long long a_desc0 = smem_desc(smem_addr(S.planes[0][0]), 16, kRowBytes);
        constexpr unsigned long long kSetUnits = (unsigned long long)D * PL * 2 / 16;
        const unsigned long long b_desc0 = smem_desc(smem_addr(S.bmat[0]), 128, 256);
        int q = 0;
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            for (int p = 0; p < wi.zn + 2; ++p, ++q) {
                const int slot = q % NPL, blk = q % NBLK;
                if (!(ok = __all_sync(0xffffffffu, wait(bar(S.planes_full, slot), (q / NPL) & 1) &&
                                                       wait(bar(S.blk_empty, blk), ((q / NBLK) & 1) ^ 1))))
                    break;
                tc_fence_after();
                if (elect_one()) {
                    plane_mma<F, 0, 0>(tmem + (unsigned)(F::kBlk * blk), a_desc0 + kSetUnits * slot, b_desc0);
                    mma_commit(bar(S.blk_full, blk));       // block ready for the epilogue
                    mma_commit(bar(S.planes_empty, slot));  // digit planes may be overwritten
                }
                committed = q + 1;
            }
        }
    } else if ((kSliceMask >> warp) & 1u) {
        // ------------------------------------------------ slicers
        // Group grp (four warps) cuts the planes with q % kGroups == grp, from
        // stage buffers grp and grp + kGroups; the groups work on consecutive
        // planes at the same time.
        const int sidx = __popc(kSliceMask & ((1u << warp) - 1u));  // 0 .. kSliceWarps - 1
        const int grp = sidx / kGroupWarps, gw = sidx % kGroupWarps;
        const int st = 32 * gw + lane;
        const bool leader = st == 0;
        // Of a sequence of planes that runs through all items the group takes
        // numbers grp + kGroups j, with `slot` and `lap` their remainder by NPL
        // and the parity of the quotient.
        int slot = grp, lap = 0;
        long long planes = 0;  // of all items of this CTA
        for (int item = first; item < items; item += step) planes += item_of(item, tiles_x, tiles_y, zc, h).zn + 2;
        {
            const int own = (int)((planes - grp + kGroups - 1) / kGroups);
            for (int j = 0; j < own; ++j) {
                const int q = grp + kGroups * j, set = j & 1, sb = grp + kGroups * set;
                // (a) window landed? Every thread waits for itself; one barrier
                // per plane, at (c), makes the group agree to go on.
                const bool landed = wait(bar(S.stage_full, sb), (j >> 1) & 1);
                // (b) window -> registers, then release the stage to the next load.
                const uint4 *stg = S.stage[sb];
                uint4 v[PER];
                float vmax = 0.f;   // split: largest |hi|
                unsigned emax = 0;  // FP64: largest upper word without its sign, then biased exponent
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int u = st + k * kGroupThreads;
                    v[k] = make_uint4(0u, 0u, 0u, 0u);
                    if (u < NCUT) {
                        v[k] = stg[(u / NCUTX) * PAIRS + CUT0 + u % NCUTX];
                        if constexpr (F::kF64)
                            emax = max(emax, max(v[k].y & 0x7FFFFFFFu, v[k].w & 0x7FFFFFFFu));
                        else
                            vmax = max_nan(vmax, max_nan(fabsf(__uint_as_float(v[k].x)), fabsf(__uint_as_float(v[k].z))));
                    }
                }
                if constexpr (F::kF64) {
                    emax = __reduce_max_sync(0xffffffffu, emax) >> 20;
                } else {
                    vmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(vmax)));
                    if (!(vmax <= 3.402823466e38f)) {  // an Inf or a NaN: the largest of the numbers, with a sign
                        vmax = 0.f;
#pragma unroll
                        for (int k = 0; k < PER; ++k)
                            vmax = fmaxf(vmax, fmaxf(fabsf(__uint_as_float(v[k].x)), fabsf(__uint_as_float(v[k].z))));
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
                        vmax = -vmax;
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    if constexpr (F::kF64)
                        S.redi[grp][set][gw] = (int)emax;
                    else
                        S.red[grp][set][gw] = vmax;
                    mbar_arrive(bar(S.stage_empty, sb));
                }
                // (c) digit-plane set free (the MMAs that read it are done)?
                // The barrier also publishes the maxima; the group's next
                // plane's are in the other set.
                const bool free = landed && wait(bar(S.planes_empty, slot), lap ^ 1);
                if (bar_any(kSliceBarrier + grp, kGroupThreads, !free)) break;
                int ex;
                bool finite = true;  // split: no Inf or NaN in the plane
                if constexpr (F::kF64) {
                    int eb = S.redi[grp][set][0];
#pragma unroll
                    for (int i = 1; i < kGroupWarps; ++i) eb = max(eb, S.redi[grp][set][i]);
                    ex = max(eb, 1);
                } else {
                    vmax = 0.f;
#pragma unroll
                    for (int i = 0; i < kGroupWarps; ++i) {
                        const float w = S.red[grp][set][i];
                        vmax = fmaxf(vmax, fabsf(w));
                        finite = finite && __float_as_int(w) >= 0;
                    }
                    ex = split::tile_exponent(vmax);
                }
                if (leader) S.scale_exp[(unsigned)q % kScaleRing] = (F::kF64 && ex == 2047) ? kNonFiniteTile : ex;
                if constexpr (F::LV == 7)
                    if (leader && ex == 2047 && again.redo) S.redo.add(q);
                unsigned *dst0 = reinterpret_cast<unsigned *>(&S.planes[slot][0][0]);
                if constexpr (F::kF64) {
                    if (ex >= kFastExp) {
#pragma unroll
                        for (int k = 0; k < PER; ++k) {
                            const int u = st + k * kGroupThreads;
                            if (u < NCUT)
                                f64_cut_fast<(F::LV > 6), PL / 2>(v[k], ex, dst0 + (u / NCUTX) * PAIRS + CUT0 + u % NCUTX);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < PER; ++k) {
                            const int u = st + k * kGroupThreads;
                            if (u < NCUT)
                                f64_cut_any<(F::LV > 6), PL / 2>(v[k], ex, dst0 + (u / NCUTX) * PAIRS + CUT0 + u % NCUTX);
                        }
                    }
                } else {
                    const float to_digits = ldexpf(1.0f, kDigitBits - ex);
                    if (finite) {
                        split::f2x s2;
                        asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(to_digits));
#pragma unroll
                        for (int k = 0; k < PER; ++k) {
                            const int u = st + k * kGroupThreads;
                            if (u < NCUT) {
                                split::f2x a, b;
                                asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(v[k].x), "r"(v[k].z));
                                asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "r"(v[k].y), "r"(v[k].w));
                                unsigned wd[D];
                                split::slice_digit_pairs_x2(split::f2_mul(a, s2), split::f2_mul(b, s2), wd);
                                unsigned *dst = dst0 + (u / NCUTX) * PAIRS + CUT0 + u % NCUTX;
#pragma unroll
                                for (int dg = 0; dg < D; ++dg) dst[dg * (PL / 2)] = wd[dg];
                            }
                        }
                    } else {  // digits of an Inf or NaN are NaN here
#pragma unroll
                        for (int k = 0; k < PER; ++k) {
                            const int u = st + k * kGroupThreads;
                            if (u < NCUT) {
                                float d0[D], d1[D];
                                slice_digits(__uint_as_float(v[k].x) * to_digits, __uint_as_float(v[k].y) * to_digits, d0);
                                slice_digits(__uint_as_float(v[k].z) * to_digits, __uint_as_float(v[k].w) * to_digits, d1);
                                unsigned *dst = dst0 + (u / NCUTX) * PAIRS + CUT0 + u % NCUTX;
#pragma unroll
                                for (int dg = 0; dg < D; ++dg) dst[dg * (PL / 2)] = split::pack_h2(d0[dg], d1[dg]);
                            }
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(S.planes_full, slot));
                slot += kGroups;
                if (slot >= NPL) {
                    slot -= NPL;
                    lap ^= 1;
                }
            }
        }
    } else if ((kEpiMask >> warp) & 1u) {
        // ------------------------------------------------ epilogue
        // Warp w reads TMEM lanes 32 (w % 4) ..; lane -> D row m = (output
        // row er, block eb); of the two warps of a lane quarter (w < 4 and
        // w >= 4 for quarters 0, 2, 3; 9 and 13 for quarter 1) hh = 0, 1
        // takes columns 8 eb + 4 hh .. + 3.
        // Each input plane's block is read once, as soon as its MMAs are
        // done, and handed back at once: its three tap-plane partial sums go
        // to the running sums of the output planes it feeds. Output j of the
        // column receives input plane j (dz = 0), j+1 (dz = 1) and j+2
        // (dz = 2) in that order and is stored after the last.
        const int quarter = warp & 3, hh = (warp >> 2) & 1;
        const int mrow = 32 * quarter + lane;
        const int er = mrow >> 3, eb = mrow & 7;
        const unsigned lane_bits = (unsigned)(32 * quarter) << 16;
        unsigned q = 0;    // input plane, of a sequence through all items
        int blk = 0, full = 0;  // its TMEM block, and the parity of its turn
        auto release = [&] {  // the block is drained: hand it back
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(S.blk_empty, blk));
        };
        auto next = [&] {
            ++q;
            if (++blk == NBLK) {
                blk = 0;
                full ^= 1;
            }
        };
        if constexpr (F::kF64) {
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            const int xb = wi.x0 + 8 * eb + 4 * hh, yy = wi.y0 + er;
            const bool whole = yy < m && xb + 3 < n;
            typename F::Out *op = out + (long long)(wi.zs - 2) * ldz + (long long)yy * ldy + xb;  // plane p - 2
            // Running sums of outputs p - 2 (a) and p - 1 (b). A part's six
            // level sums combine into one 64-bit integer T (value T 2^c,
            // c = plane exponent + ew - 1080, as in the 2D kernel); while every
            // part of a sum had the same plane exponent (ea, eb2) the sum stays
            // an exact integer (27 taps: |T| < 2^63), rounded once at the end.
            // A part with another exponent turns the sum into an FP64 value
            // (fa, fb: the bits live in the same words); a part from a window
            // with an Inf or NaN makes the output NaN (na, nb).
            long long a[4], b[4];
            int ea = 0, eb2 = 0;
            bool fa = false, fb = false, na = false, nb = false;
            const int ew = sw.ew;
            // Integer sums start at -3 kRawBias, so that they are right once
            // all three parts are in; `left` parts are missing before this one.
            constexpr unsigned long long bias = kRawBias<F::LV == 7 ? 0 : 3>;
            auto add_raw = [&](long long (&sm)[4], const float (&acc)[F::LV][4]) {
#pragma unroll
                for (int c = 0; c < 4; c += 2) {
                    if constexpr (F::LV == 7) {
                        float u[7], v[7];
#pragma unroll
                        for (int L = 0; L < 7; ++L) u[L] = acc[L][c], v[L] = acc[L][c + 1];
                        f64_add_raw2(u, v, sw.rest, sm[c], sm[c + 1]);
                        continue;
                    }
                    const float u[6] = {acc[0][c], acc[1][c], acc[2][c], acc[3][c], acc[4][c], acc[5][c]};
                    const float v[6] = {acc[0][c + 1], acc[1][c + 1], acc[2][c + 1],
                                        acc[3][c + 1], acc[4][c + 1], acc[5][c + 1]};
                    f64_add_raw2(u, v, sm[c], sm[c + 1]);
                }
            };
            auto add_part = [&](long long (&sm)[4], int &se, bool &fl, bool &nf, const float (&acc)[F::LV][4],
                                int ex, int left) {
                if (nf) return;
                if (ex == kNonFiniteTile) {
                    nf = true;
                    return;
                }
                if (!fl && ex == se) {
                    add_raw(sm, acc);
                    return;
                }
                if (!fl) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        sm[c] = __double_as_longlong(f64_from_fixed((long long)((unsigned long long)sm[c] + left * bias), se + ew - 1080));
                    fl = true;
                }
                const long long none = (long long)(0 - bias);
                long long t[4] = {none, none, none, none};
                add_raw(t, acc);
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    sm[c] = __double_as_longlong(__longlong_as_double(sm[c]) + f64_from_fixed(t[c], ex + ew - 1080));
            };
            auto load_issue = [&](int dz, float (&acc)[F::LV][4]) {
                const unsigned col = (unsigned)(F::kBlk * blk + 8 * dz + 4 * hh);
#pragma unroll
                for (int L = 0; L < F::LV; ++L) tmem_ld4(tmem + lane_bits + col + NLV * L, acc[L]);
            };
            auto load_part = [&](int dz, float (&acc)[F::LV][4]) {
                load_issue(dz, acc);
                tmem_wait_ld();
            };
            for (int p = 0; p < wi.zn + 2; ++p, op += ldz, next()) {
                if (!(ok = wait(bar(S.blk_full, blk), full))) break;
                tc_fence_after();
                const int ex = S.scale_exp[q % kScaleRing];
                float acc[F::LV][4];
                // The usual plane: every sum it goes to has its exponent, and
                // nothing rare is under way. (All of this is the same in the
                // whole CTA: the loads want full warps.)
                const int sc_q = ex + ew - 1080;
                if (ex == ea && ex == eb2 && p >= 2 && p <= wi.zn && !(fa | fb | na | nb) &&
                    ex != kNonFiniteTile && f64_scale_is_plain(sc_q)) {
                    load_part(1, acc);
                    add_raw(b, acc);
                    load_part(2, acc);
                    add_raw(a, acc);
                    // The conversions, 64 cycles each on the FP64 unit, run
                    // beside the last part's load and sum (one after the other
                    // before the store: star3d1r 512^3, GB300, 897 us, so 861).
                    load_issue(0, acc);
                    long long d[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) d[c] = f64_bits_of(a[c]);
                    tmem_wait_ld();
                    release();
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        a[c] = b[c];
                        b[c] = (long long)(0 - 3 * bias);
                    }
                    add_raw(b, acc);
                    double res[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) res[c] = f64_scaled(d[c], sc_q);
                    if (whole) {
                        *reinterpret_cast<double2 *>(op) = make_double2(res[0], res[1]);
                        *reinterpret_cast<double2 *>(op + 2) = make_double2(res[2], res[3]);
                    } else if (yy < m) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (xb + c < n) op[c] = res[c];
                    }
                    __syncwarp();
                    continue;
                }
                // z tap 2 of output p - 2: its last part; store.
                load_part(2, acc);
                if (p >= 2) {
                    add_part(a, ea, fa, na, acc, ex, 1);
                    if (yy < m) {
                        double res[4];
                        const int sc = ea + ew - 1080;
                        if (!na && !fa && f64_scale_is_plain(sc)) {
#pragma unroll
                            for (int c = 0; c < 4; ++c) res[c] = f64_from_fixed_plain(a[c], sc);
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c)
                                res[c] = na ? __longlong_as_double(0x7FF8000000000000ll)
                                     : fa ? __longlong_as_double(a[c])
                                          : f64_from_fixed(a[c], sc);
                        }
#pragma unroll
                        for (int c = 0; c < 4; c += 2) {
                            if (xb + c + 1 < n)
                                *reinterpret_cast<double2 *>(op + c) = make_double2(res[c], res[c + 1]);
                            else if (xb + c < n)
                                op[c] = res[c];
                        }
                    }
                }
                // z tap 1 of output p - 1.
                load_part(1, acc);
                if (p >= 1 && p - 1 < wi.zn) add_part(b, eb2, fb, nb, acc, ex, 2);
                // z tap 0 of output p: its first part. The block is then
                // drained and handed back.
                load_part(0, acc);
                release();
#pragma unroll
                for (int c = 0; c < 4; ++c) {  // rotate: p - 1 becomes p - 2, p starts
                    a[c] = b[c];
                    b[c] = (long long)(0 - 3 * bias);
                }
                ea = eb2;
                fa = fb;
                na = nb;
                eb2 = ex;
                fb = false;
                nb = ex == kNonFiniteTile;
                if (!nb) add_raw(b, acc);
            }
        }
        } else {
        float scale = 0.f;  // 2^scale_e
        int scale_e = -(1 << 20);
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            const int xb = wi.x0 + 8 * eb + 4 * hh, yy = wi.y0 + er;
            const bool whole = yy < m && xb + 3 < n;
            typename F::Out *op = out + (long long)(wi.zs - 2) * ldz + (long long)yy * ldy + xb;  // plane p - 2
            // Running sums of outputs p - 2 (a) and p - 1 (b). While every
            // part added to a sum had the same plane scale (2^ea, 2^eb2), the
            // sum is kept as level sums: S0, S1, S2 exact (three parts of at
            // most 45 digit products below 2^16 each stay below 2^24) and the
            // tail T = S3 2^-27 + S4 2^-36 (its rounding weighs below 2^-50 of
            // S0's unit); the output is then recombined once. A part with
            // another scale turns the sum into a (hi, lo) pair in [0], [1]
            // relative to the largest scale seen (fa, fb set), which takes its
            // later parts as recombined pairs. Plane scales are the same for
            // the whole CTA, so the choice never diverges.
            float a[4][4], b[4][4];
            int ea = 0, eb2 = 0;
            bool fa = false, fb = false;
            auto tail = [](float s3, float s4) { return fmaf(s3, 0x1p-27f, s4 * 0x1p-36f); };
            // Level sums -> (hi, lo) in [0], [1].
            auto to_pair = [](float (&sm)[4][4]) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float h1, e1, h2, e2, hi, lo;
                    two_sum(sm[0][c], sm[1][c] * 0x1p-9f, h1, e1);
                    two_sum(h1, sm[2][c] * 0x1p-18f, h2, e2);
                    two_sum(h2, (e1 + e2) + sm[3][c], hi, lo);
                    sm[0][c] = hi;
                    sm[1][c] = lo;
                }
            };
            // Adds a tap plane's part (five levels per column, relative to
            // 2^ex) to a running sum.
            auto add_part = [&](float (&sm)[4][4], int &se, bool &fl, const float (&acc)[D][4], int ex) {
                if (!fl && ex == se) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        sm[0][c] += acc[0][c];
                        sm[1][c] += acc[1][c];
                        sm[2][c] += acc[2][c];
                        sm[3][c] += tail(acc[3][c], acc[4][c]);
                    }
                    return;
                }
                if (!fl) to_pair(sm);
                fl = true;
                float ra = 1.0f, rb = 1.0f;
                if (ex > se) {
                    ra = ldexpf(1.0f, se - ex);
                    se = ex;
                } else {
                    rb = ldexpf(1.0f, ex - se);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float lv[D], ph, pl, s2, e2;
#pragma unroll
                    for (int L = 0; L < D; ++L) lv[L] = acc[L][c];
                    recombine(lv, ph, pl);
                    two_sum(sm[0][c] * ra, ph * rb, s2, e2);
                    sm[1][c] = sm[1][c] * ra + (e2 + pl * rb);
                    sm[0][c] = s2;
                }
            };
            auto load_part = [&](int dz, float (&acc)[D][4]) {
                const unsigned col = (unsigned)(F::kBlk * blk + 8 * dz + 4 * hh);
#pragma unroll
                for (int L = 0; L < D; ++L) tmem_ld4(tmem + lane_bits + col + NLV * L, acc[L]);
                tmem_wait_ld();
            };
            for (int p = 0; p < wi.zn + 2; ++p, op += ldz, next()) {
                if (!(ok = wait(bar(S.blk_full, blk), full))) break;
                tc_fence_after();
                const int ex = S.scale_exp[q % kScaleRing];
                float acc[D][4];
                // The usual plane: every sum it goes to has its scale.
                if (ex == ea && ex == eb2 && p >= 2 && p <= wi.zn && !(fa | fb)) {
                    if (ex != scale_e) {
                        scale_e = ex;
                        scale = ldexpf(1.0f, ex + sw.ew - 2 * kDigitBits);
                    }
                    load_part(2, acc);
                    float2 res[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float s0 = a[0][c] + acc[0][c], s1 = a[1][c] + acc[1][c], s2 = a[2][c] + acc[2][c];
                        const float s3 = a[3][c] + tail(acc[3][c], acc[4][c]);
                        float h1, e1, h2, e2, hi, lo;
                        two_sum(s0, s1 * 0x1p-9f, h1, e1);
                        two_sum(h1, s2 * 0x1p-18f, h2, e2);
                        two_sum(h2, (e1 + e2) + s3, hi, lo);
                        res[c] = make_float2(hi * scale, lo * scale);
                    }
                    if (whole) {
                        *reinterpret_cast<float4 *>(op) = make_float4(res[0].x, res[0].y, res[1].x, res[1].y);
                        *reinterpret_cast<float4 *>(op + 2) = make_float4(res[2].x, res[2].y, res[3].x, res[3].y);
                    } else if (yy < m) {
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (xb + c < n) op[c] = res[c];
                    }
                    __syncwarp();
                    load_part(1, acc);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        a[0][c] = b[0][c] + acc[0][c];
                        a[1][c] = b[1][c] + acc[1][c];
                        a[2][c] = b[2][c] + acc[2][c];
                        a[3][c] = b[3][c] + tail(acc[3][c], acc[4][c]);
                    }
                    load_part(0, acc);
                    release();
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        b[0][c] = acc[0][c];
                        b[1][c] = acc[1][c];
                        b[2][c] = acc[2][c];
                        b[3][c] = tail(acc[3][c], acc[4][c]);
                    }
                    continue;
                }
                // z tap 2 of output p - 2: its last part; store.
                load_part(2, acc);
                if (p >= 2) {
                    add_part(a, ea, fa, acc, ex);
                    if (!fa) to_pair(a);
                    if (yy < m) {
                        const float scale = ldexpf(1.0f, ea + sw.ew - 2 * kDigitBits);
                        float2 res[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            float hi, lo;
                            two_sum(a[0][c], a[1][c], hi, lo);
                            res[c] = make_float2(hi * scale, lo * scale);
                        }
#pragma unroll
                        for (int c = 0; c < 4; c += 2) {
                            if (xb + c + 1 < n)
                                *reinterpret_cast<float4 *>(op + c) =
                                    make_float4(res[c].x, res[c].y, res[c + 1].x, res[c + 1].y);
                            else if (xb + c < n)
                                op[c] = res[c];
                        }
                    }
                }
                // z tap 1 of output p - 1.
                load_part(1, acc);
                if (p >= 1 && p - 1 < wi.zn) add_part(b, eb2, fb, acc, ex);
                // z tap 0 of output p: its first part. The block is then
                // drained and handed back.
                load_part(0, acc);
                release();
#pragma unroll
                for (int c = 0; c < 4; ++c) {  // rotate: p - 1 becomes p - 2, p starts
#pragma unroll
                    for (int k = 0; k < 4; ++k) a[k][c] = b[k][c];
                    b[0][c] = acc[0][c];
                    b[1][c] = acc[1][c];
                    b[2][c] = acc[2][c];
                    b[3][c] = tail(acc[3][c], acc[4][c]);
                }
                ea = eb2;
                fa = fb;
                eb2 = ex;
                fb = false;
            }
        }
        }
    }

    // Exit: every role is done or has given up. Let the last window loads and
    // the last MMA batch finish (they have normally finished already) before
    // the shared memory and TMEM are released.
    tc_fence_before();
    __syncthreads();
    if (warp == kWarpTma && lane == 0)
        for (int l = max(0, issued - kStages); l < issued; ++l)
            mbar_drain(bar(S.stage_full, l % kStages), (l / kStages) & 1, &g_tc3d_wait_timeouts);
    if (warp == kWarpMma && lane == 0 && committed > 0)
        mbar_drain(bar(S.blk_full, (committed - 1) % NBLK), ((committed - 1) / NBLK) & 1,
                   &g_tc3d_wait_timeouts);
    __syncthreads();
    tc_fence_after();
    if (warp == kWarpTma)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(kTmemCols));
    if constexpr (F::LV == 7) {
        if (S.redo.count > 0 && !S.abort) {  // output planes j with an Inf or NaN in their three input planes
            int q = 0;
            for (int item = first; item < items; item += step) {
                const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
                for (int j = 0; j < wi.zn; ++j) {
                    if (!S.redo.holds(q + j, q + j + 2)) continue;
                    for (int i = tid; i < TX * TY; i += kThreads) {
                        const int y = wi.y0 + i / TX, x = wi.x0 + i % TX;
                        const long long at = (long long)(wi.zs + j) * ldz + (long long)y * ldy + x;
                        if (y < m && x < n)
                            out[at] = fma_sum_3d<1>(again.in + at, ldy, ldz, again.w, again.pattern);
                    }
                }
                q += wi.zn + 2;
            }
        }
    }
}

}  // namespace

bool split_tc3d_layout_ok(const GridView &g, long long origin, const void *in_base, const void *out_base)
{
    if (g.dims != 3) return false;
    const long long ldy = g.pitch[1], ldz = g.pitch[0];
    return ldy % 2 == 0 && ldz % 2 == 0 && ldz % ldy == 0 && (origin % ldy) % 2 == 0 &&
           reinterpret_cast<uintptr_t>(in_base) % 16 == 0 && reinterpret_cast<uintptr_t>(out_base) % 16 == 0;
}

namespace {

template <class F>
cudaError_t launch_tc3d(const GridView &g, const typename F::Digits &digits, long long origin, long long elements,
                        const void *in_base, void *out_base, const TcWait &wt, cudaStream_t st,
                        const typename F::Again &again = typename F::Again{})
{
    const long long ldy = g.pitch[1], ldz = g.pitch[0];
    CUtensorMap map;
    // The map copies 8-byte points whatever they hold ((hi, lo) pairs or FP64).
    cudaError_t e = encode_split_window_map_3d(&map, reinterpret_cast<const float2 *>(in_base), ldy, ldz,
                                               elements / ldz, ST_X, ST_Y);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(Smem<F>) + 128;
    static const cudaError_t attr_err =
        cudaFuncSetAttribute(k3d_tc<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (attr_err != cudaSuccess) return attr_err;
    const int h = (int)g.ext[0], m = (int)g.ext[1], n = (int)g.ext[2];
    const int tiles_x = (n + TX - 1) / TX, tiles_y = (m + TY - 1) / TY;
    // Planes per work item: a column of zc output planes loads and cuts
    // zc + 2 input planes, and the busiest CTA takes ceil(items / SMs) items,
    // so zc (up to 32) minimises ceil(items / SMs) * (zc + 2).
    const int sms = device_sm_count();
    const long long txy = (long long)tiles_x * tiles_y;
    int zc = 1;
    long long best = -1;
    for (int c = 1; c <= std::min(32, h); ++c) {
        const long long it = txy * ((h + c - 1) / c);
        const long long cost = ((it + sms - 1) / sms) * (c + 2);
        if (best < 0 || cost < best) best = cost, zc = c;
    }
    const int items = (int)(txy * ((h + zc - 1) / zc));
    const int grid = std::min(items, sms);
    note_launch();
    return launch_programmatic(k3d_tc<F>, grid, kThreads, smem, st, map,
                               reinterpret_cast<typename F::Out *>(out_base) + origin, h, m, n, ldy, ldz, tiles_x,
                               tiles_y, zc, items, (int)(origin % ldy), (int)((origin % ldz) / ldy),
                               (int)(origin / ldz), digits, WaitCfg{wt.limit_ns, wt.skip_loads}, again);
}

}  // namespace

cudaError_t launch_split_sweep_tc3d(const GridView &g, const Weights &w, long long origin,
                                    long long elements, const float2 *in_base, float2 *out_base,
                                    const TcWait &wt, cudaStream_t st)
{
    return launch_tc3d<F3Split>(g, split::slice_weights(w, 27), origin, elements, in_base, out_base, wt, st);
}

cudaError_t launch_fp64_sweep_tc3d(const GridView &g, const Weights &w, long long origin, long long elements,
                                   const double *in_base, double *out_base, const TcWait &wt, cudaStream_t st,
                                   const TcForm *form)
{
    if (form) {
        SumAgain again{in_base + origin, form->pattern, form->redo, {}};
        for (int i = 0; i < 27; ++i) again.w[i] = w.v[i];
        return launch_tc3d<F3F64Fine>(g, f64_slice_weights(w, 27, &tap_order(Taps::kCube3)), origin, elements, in_base,
                                      out_base, wt, st, again);
    }
    return launch_tc3d<F3F64>(g, f64_slice_weights(w, 27), origin, elements, in_base, out_base, wt, st);
}

cudaError_t tc3d_wait_counter(unsigned **counter)
{
    return cudaGetSymbolAddress((void **)counter, g_tc3d_wait_timeouts);
}

cudaError_t split_tc3d_wait_timeouts(unsigned *count, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(count, g_tc3d_wait_timeouts, sizeof(unsigned));
    if (e != cudaSuccess || !reset) return e;
    const unsigned zero = 0;
    return cudaMemcpyToSymbol(g_tc3d_wait_timeouts, &zero, sizeof(unsigned));
}

}  // namespace cs
