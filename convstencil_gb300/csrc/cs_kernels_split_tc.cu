// cs_kernels_split_tc.cu — dense 7x7 sweeps on the fifth-generation tensor
// cores (tcgen05.mma, accumulators in TMEM), in two number formats that share
// one pipeline:
//
//   * split precision (FmtSplit): grids of FP32 (hi, lo) pairs. Every input
//     pair of a tile is scaled by a power of two and cut into five balanced
//     9-bit digits held exactly in FP16; the weights likewise. Products of
//     digit k of x and digit e of w with k + e = L land in one FP32
//     accumulator per level L. Every product is an integer below 2^16 and a
//     level sums at most 49 * 5 of them, so each level is exact (< 2^24)
//     whatever the summation order; the five levels are recombined
//     error-free into a new (hi, lo) pair.
//   * FP64 (FmtF64): FP64 grids, the drop-in form. Each FP64 input is turned
//     into a 52-bit fixed-point integer relative to its tile's largest
//     exponent and cut into six balanced 9-bit digits with integer
//     operations only (no FP64 instruction: this GPU's FP64 pipe runs at
//     about 1/1000 of its FP16 tensor rate); the weights into six digits of a
//     fixed point below 1/4, so the top digits of both stay within 128.
//     Levels 0..5 (21 digit pairs per tap) are kept: level L sums at most
//     49 * (4 * 2^16 + 2 * 2^15) < 2^24, so each is again exact. The levels
//     are combined into one 64-bit integer and rounded once to FP64 by
//     integer operations. Error per sweep: the inputs carry 52 bits below
//     the tile maximum, the weights 53 below the largest weight, and the
//     dropped levels >= 6 weigh below 2^-48 of (tile max x largest weight)
//     in the worst case (about 2^-53 for data without adversarial digits).
//
//   * FP64 with seven levels (FmtF64Fine): the forms that AUTO takes in the
//     place of FP64 FMA sweeps (several steps per launch, odd layouts, 1D, small
//     served grids), whose errors must not be larger than those sweeps'. Level
//     6 is kept too, inputs round to even and the weights keep their sum, so a
//     launch errs by its inputs' and its outputs' rounding.
//   * split with six digits (FmtSplit6): the launches of several steps, below,
//     of split plans, whose errors would otherwise grow with the steps' weights.
//
// Modes (MODE): one sweep of a 2D grid (kModeGrid); three steps of a radius-1
// 2D grid as one sweep of its three times self-convolved kernel, the frame two
// points wide computed step by step (kModeSteps); up to 23 steps of a 1D grid
// (kMode1d). BATCH: many grids in one launch. ODD: grids whose rows TMA cannot
// address one by one (OddRows).
//
// Mapping onto tcgen05 (M = 128, K = 16, N = 32 per level):
//   * A CTA owns a 64 x 64 output tile: 16 row groups of 4 rows, 8 blocks
//     of 8 columns. Its input window (70 x 72 points, columns x0-4 ..
//     x0+67) arrives by one 2D TMA load and is cut into digit planes in
//     shared memory, one row of 72 halves (144 bytes) per window row.
//   * Row m of the A operand is the 16-wide window of block b = m % 8 in
//     row group r = m / 8. A K-major, non-swizzled shared-memory descriptor
//     with a 16-byte K-chunk stride and a stride of four plane rows between
//     8-row groups reads exactly that sliding window out of the plane in
//     place: element (m, k) sits at plane row 4r, column 8b + k. Window row
//     offset i (0..9) is the same descriptor started i plane rows lower, so
//     no im2col copy exists.
//   * Column n of B_i is output (row 4r + rho, column 8b + c), n = 8 rho + c;
//     B_i[k][n] = w[i - rho][k - c - 1] where that tap exists, else 0.
//   * For input digit d the B operand is [B_i(e=0) | ... | B_i(e=D-1-d)]
//     (the first 32 (D-d) rows of one K-major matrix) and the accumulator
//     starts at TMEM column 32 d, so one MMA feeds levels d..D-1 at once:
//     per tile 10 offsets x D digits MMAs (50 split, 60 FP64) into 32 D FP32
//     columns.
//   * The tile shape serves as many outputs per MMA as shared memory allows:
//     4 rows per group give 4096 outputs per tile (2 rows: 2048 per 40
//     MMAs). The issuing thread stalls on each MMA until the tensor core
//     accepts it, so the MMAs are unrolled with compile-time descriptor
//     offsets (measured on GB300: 56 cycles per MMA for the split N =
//     160..32 sequence, 70 with the descriptors computed in the loop).
//   * One persistent CTA per SM (about 188 KB of shared memory split, 219 KB
//     FP64) with warp roles joined by mbarriers: one warp issues the TMA
//     window loads, one thread issues the MMAs (tcgen05.mma issue blocks
//     while the tensor core is busy, so it must not sit in anyone else's
//     barrier), eight warps read a window into registers, release the stage
//     to the next load and cut the digit planes, and four (split) or eight
//     (FP64) warps drain the accumulators, recombine and store. Two
//     accumulators (TMEM columns 0 and 256) and two sets of digit planes let
//     slicing of tile t+1, the MMAs of tile t and the stores of tile t-1 run at
//     the same time.
//   * Bound: the shared memory that the MMAs read (354 KB of operands a tile
//     split, 455 KB FP64, at 128 bytes a cycle 2,770 and 3,560 cycles) beside
//     the slicers' and the TMA unit's ~120 KB. That is about 70 % of the cycles
//     a tile takes (5,400 split); the rest is the roles waiting for each other,
//     with no unit above 60 %. GB300, 8192^2: split 280 us a sweep, FP64 321, three
//     steps of radius 1 362.
//
// Every mbarrier wait is bounded (WaitCfg, 2 s by default). An expired wait
// is counted in g_tc_wait_timeouts; the CTA then waits, again bounded, for
// the TMA copy and the MMAs it still has in flight, frees its TMEM and
// leaves.
#include "cs_internal.h"
#include "cs_split_common.cuh"
#include "cs_split_ff.cuh"
#include "cs_tc_common.cuh"
#include "cs_tc_f64.cuh"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace cs {

__device__ unsigned int g_tc_wait_timeouts;

namespace {

using split::kDigitBits;
using split::slice_digits;
using split::two_sum;
using namespace tc;

// Number formats.
// kEpiWarps: epilogue warps, one or two per TMEM lane quarter. Every warp the
// epilogue runs takes issue slots from the slicers, which bound the split
// kernel, so its light recombination runs on four warps (8192^2 on GB300:
// 192 -> 204 GStencil/s against eight); the FP64 recombination (integer
// operations) needs eight (120 GStencil/s on four, 169 on eight).
// kCols: columns drained at a time. Four leave the FP64 kernels' registers
// free of spills (three-step 8192^2 launch, GB300: 370 us with eight, 359 with
// four; with twelve or sixteen slicer warps, 80 or 72 registers, 403 and 420).
// kLevels: levels kept, from 0; digits d of x and e of w meet in level d + e.
struct FmtSplit {
    static constexpr bool kF64 = false;
    static constexpr int kDigits = split::kDigits, kLevels = split::kDigits;  // 5
    static constexpr int kEpiWarps = 4, kSliceWarps = 8, kCols = 8;
    using Out = float2;
    using Digits = split::SliceWeights;
};

// Split grids cut into six digits, for launches of several steps (radius-1 and
// 1D stencils, whose single steps run in double-float arithmetic): the input
// pairs keep 52 bits below their tile's largest value, more than the (hi, lo)
// format holds, so a launch's error is the rounding of its results to pairs.
struct FmtSplit6 {
    static constexpr bool kF64 = false;
    static constexpr int kDigits = 6, kLevels = 6;
    static constexpr int kEpiWarps = 4, kSliceWarps = 8, kCols = 8;
    using Out = float2;
    using Digits = F64Weights;
};

struct FmtF64 {
    static constexpr bool kF64 = true;
    static constexpr int kDigits = 6, kLevels = 6;
    static constexpr int kEpiWarps = 8, kSliceWarps = 8, kCols = 4;
    using Out = double;
    using Digits = F64Weights;
};

// Level 6 (27 digit pairs per tap) costs an MMA and 24 % more columns of B, no
// shared memory (rows of B that are there). Without it what the dropped pairs
// weigh, 2^-53 of the tile's largest value on average, is a launch's largest
// error. (Error of the norm with six levels, with seven and of FP64 FMA sweeps,
// uniform data: star2d1r 1024^2 x 100 5.7e-16, 1.06e-16, 1.12e-16; odd box2d3r x 20
// 2.3e-16, 6.5e-17, 1.7e-16; 1d2r 1,000,000 x 100 4.1e-16, 1.2e-16, 1.5e-16. GB300, us
// a solve: star2d1r 476 and 476, box2d1r 2047 x 1531 x 60 516 and 524, 1d2r
// 10,240,000 x 100 563 and 563: set by the slicers, not the MMAs.)
struct FmtF64Fine : FmtF64 {
    static constexpr int kLevels = 7;
};

// Formats whose launches may stand for kernels without digits (Redo).
template <class F>
constexpr bool kRedoable = F::kDigits == 6 && (F::kLevels == 7 || !F::kF64);

// Warp roles.
constexpr int kWarpTma = 0, kWarpMma = 1, kWarpSlice0 = 2;
template <class F>
constexpr int kThreads = 32 * (kWarpSlice0 + F::kSliceWarps + F::kEpiWarps);  // 448 split, 576 FP64
constexpr int kMaxSliceWarps = 8;
constexpr int kSliceBarrier = 1;           // named barrier of the slicer warps
constexpr int kBuildBarrier = 2;           // named barrier of the warps that build B

constexpr int R = 4;                       // output rows per row group (N dimension)
constexpr int G = 16;                      // row groups per tile (M = G x 8 blocks = 128)
constexpr int TX = 64, TY = G * R;         // output tile 64 x 64
constexpr int ST_X = TX + 8, ST_Y = TY + 6;  // window: columns x0-4 .. x0+67, rows y0-3 .. y0+66
constexpr int PL = ST_X * ST_Y;            // halves per digit plane (10,080 bytes)
constexpr unsigned kRowBytes = ST_X * 2;   // 144
constexpr int NOFF = R + 6;                // window row offsets per row group
constexpr int NLV = 8 * R;                 // accumulator columns per level
constexpr int kWz = 24;                    // halves per staged weight row: taps at 8 .. 14
constexpr int kAccStride = 256;            // TMEM columns between the two accumulators
constexpr int kTmemCols = 512;
constexpr unsigned kStageBytes = ST_X * ST_Y * 8;  // 40,320 (8-byte points)
constexpr int PAIRS = ST_X / 2, NPAIR = ST_Y * PAIRS;           // 36, 2,520
// Windows of odd layouts (OddRows): a spare pair per row, even and odd rows apart.
constexpr int kOddRow = 8 * ST_X + 16, kOddHalf = (ST_Y / 2 * kOddRow + 127) / 128 * 128;  // bytes
constexpr int kStageF64 = (kOddHalf + ST_Y / 2 * kOddRow) / 16;
// 1D (kMode1d): a tile is 4096 outputs, 128 rows of 32; row m of A is the 80
// points around output row m, read in five K steps. The window is 4096 + 48
// points, 518 chunks of 8; chunk j sits in phase j % 4 at place j / 4, so the
// rows' chunks of one K step (two phases, places m .. m + 2) are core matrices
// of consecutive 16-byte rows: the canonical non-swizzled layout again, each
// point stored once. The reach is the largest whose 2 * 24 + 1 taps keep the
// level sums exact, as the 49 of a 7x7 do (with a reach of 16, four K steps,
// a launch took the same time, set by the slicers, for two thirds of the
// steps: 1d2r 10,240,000 x 100, GB300, 852 us, so 597 then).
constexpr int kReach1d = kTcReach1d;                // points either side of an output: 24
constexpr int kOut1d = 4096, kWin1d = kOut1d + 2 * kReach1d, NPAIR1D = kWin1d / 2;
constexpr int kSteps1d = (32 + 2 * kReach1d) / 16;  // K steps
// bytes between phases: 130 chunks; the words a slicer warp stores (16 per
// phase pair) then fall into different banks
constexpr int kPhase1d = 2080;
constexpr unsigned kBytes1d = kWin1d * 8;
constexpr int kFrame1d = 2 * kReach1d;              // points of an end computed step by step (frame_end_1d)
static_assert(2 * kReach1d + 1 <= 49, "level sums are exact for 49 taps");
static_assert(4 * kPhase1d <= PL * 2 && kBytes1d <= kStageBytes && NPAIR1D <= NPAIR &&
                  kPhase1d >= (kWin1d + 31) / 32 * 16 && kPhase1d / 4 % 32 == 8,
              "the 1D window and digits fit the 2D buffers");
static_assert(FmtSplit::kEpiWarps == 4 && FmtF64::kEpiWarps == 8 && R == 4,
              "one or two epilogue warps per TMEM lane quarter, R / (warps per quarter) rows each");

template <class F>
struct Smem {
    static constexpr int D = F::kDigits;
    static constexpr int NCOL = NLV * D;       // rows of B: digit e at NLV * e
    static_assert(NLV * F::kLevels <= kAccStride, "an accumulator must fit between the two TMEM bases");
    uint4 stage[F::kF64 ? kStageF64 : NPAIR];  // windows: pairs of 8-byte points
    __half planes[2][D][PL];                   // digit planes, two tiles
    __half bmat[NOFF][NCOL * 16];              // B_i, K-major 8x16-byte core matrices
    __half wz[D][7][kWz];                      // weight digits, rows padded with zeros
    unsigned long long stage_full, stage_empty;
    unsigned long long planes_full[2], planes_empty[2];
    unsigned long long acc_full[2], acc_empty[2];
    unsigned long long ends[2][2][kFrame1d];   // 1D: the two ends, two levels
    unsigned tmem;                             // TMEM base column
    int abort;                                 // set by the first expired wait
    int scale_exp[4];                          // per-tile input scale, ring of 4
    float red[2][kMaxSliceWarps];                 // split: per-warp max |hi|, by tile parity
    int redi[2][kMaxSliceWarps];                  // FP64: per-warp max biased exponent
    std::conditional_t<kRedoable<F>, Redo, NoRedo> redo;  // tiles to compute again
};

static_assert(sizeof(Smem<FmtF64Fine>) + 128 <= 232448 && sizeof(Smem<FmtSplit>) + 128 <= 232448 &&
                  sizeof(Smem<FmtSplit6>) + 128 <= 232448,
              "shared memory of one CTA must stay within 227 KB");

// The MMAs of one tile: window row offsets and input digits DG. Descriptor
// addresses advance in 16-byte units: digit planes are PL halves apart, row
// offsets one plane row, B_i matrices NCOL * 16 halves.
//
// Offset I serves output rows rho with 0 <= I - rho <= 6 only. Of the 32 columns
// (8 rho + c) of a level that leaves the first 16 at offsets 0 and 1 and the last
// 16 at 8 and 9; their MMAs stop 16 columns before the last level's end, or
// start 16 after the first's beginning. The first offset issued, 3, is a whole
// one: it initialises the accumulator. (6 %
// of the columns; GB300, 8192^2: split 284.0 -> 281.8 us a sweep, FP64 three steps
// 358.0 -> 357.1.)
//
// With more levels than digits, digit 1 is the first to reach the last level:
// its first MMA stops short of it and one of its own initialises it.
__host__ __device__ constexpr int nth_offset(int j) { return j == 0 ? 3 : j <= 3 ? j - 1 : j; }
// Levels that digit DG feeds, from level DG on: the B rows of as many digits of w.
template <class F>
__host__ __device__ constexpr int levels_of(int dg)
{
    return F::kLevels - dg < F::kDigits ? F::kLevels - dg : F::kDigits;
}
template <class F, int J, int DG>
__device__ __forceinline__ void tile_mma(unsigned d_base, unsigned long long a0, unsigned long long b0)
{
    constexpr int D = F::kDigits, L = F::kLevels, W = levels_of<F>(DG);
    constexpr int NCOL = NLV * D, I = nth_offset(J), LO = I >= 8 ? 16 : 0, HI = I <= 1 ? 16 : 0;
    constexpr unsigned long long a_off = ((unsigned long long)DG * PL * 2 + I * kRowBytes) >> 4;
    constexpr unsigned long long b_off = ((unsigned long long)I * NCOL * 16 * 2 + LO / 8 * 256) >> 4;
    static_assert(((unsigned long long)DG * PL * 2 + I * kRowBytes) % 16 == 0 && (NCOL * 16 * 2) % 16 == 0,
                  "descriptor offsets must be 16-byte multiples");
    static_assert(L <= D + 1);
    if constexpr (L > D && J == 0 && DG == 1) {
        mma_f16(d_base + (unsigned)NLV, a0 + a_off, b0 + b_off, instr_desc(NLV * (W - 1)), 1u);
        mma_f16(d_base + (unsigned)(NLV * D), a0 + a_off, b0 + b_off + (NLV * (W - 1) * 16 * 2 >> 4), instr_desc(NLV), 0u);
    } else {
        mma_f16(d_base + (unsigned)(NLV * DG + LO), a0 + a_off, b0 + b_off, instr_desc(NLV * W - LO - HI),
                (J | DG) != 0 ? 1u : 0u);
    }
    if constexpr (DG + 1 < D)
        tile_mma<F, J, DG + 1>(d_base, a0, b0);
    else if constexpr (J + 1 < NOFF)
        tile_mma<F, J + 1, 0>(d_base, a0, b0);
}

// The MMAs of one 1D tile: K step KK, input digit DG.
template <class F, int KK, int DG>
__device__ __forceinline__ void tile_mma_1d(unsigned d_base, unsigned long long a0, unsigned long long b0)
{
    constexpr int D = F::kDigits, L = F::kLevels, W = levels_of<F>(DG);
    constexpr unsigned long long a_off =
        ((unsigned long long)DG * PL * 2 + (KK & 1) * 2 * kPhase1d + (KK >> 1) * 16) >> 4;
    constexpr unsigned long long b_off = ((unsigned long long)KK * NLV * D * 16 * 2) >> 4;
    if constexpr (L > D && KK == 0 && DG == 1) {
        mma_f16(d_base + (unsigned)NLV, a0 + a_off, b0 + b_off, instr_desc(NLV * (W - 1)), 1u);
        mma_f16(d_base + (unsigned)(NLV * D), a0 + a_off, b0 + b_off + (NLV * (W - 1) * 16 * 2 >> 4), instr_desc(NLV), 0u);
    } else {
        mma_f16(d_base + (unsigned)(NLV * DG), a0 + a_off, b0 + b_off, instr_desc(NLV * W), (KK | DG) != 0 ? 1u : 0u);
    }
    if constexpr (DG + 1 < D)
        tile_mma_1d<F, KK, DG + 1>(d_base, a0, b0);
    else if constexpr (KK + 1 < kSteps1d)
        tile_mma_1d<F, KK + 1, 0>(d_base, a0, b0);
}

// One grid of a batch (batch mode): its tensor map, output, sizes, tile
// numbering and weight digits. Records live in a device array.
template <class F>
struct alignas(128) TcGrid {
    CUtensorMap map;          // window map over the source buffer
    typename F::Out *out;     // interior point (0, 0) of the destination
    long long ld;
    int m, n, tiles_x, tile_begin, map_x, map_y;
    int digits_id;            // grids with the same id have the same weights
    typename F::Digits digits;
};

// The weight digits as B_i needs them: row ti of digit e at wz[e][ti][8 ..
// 14], zeros around it. Threads t0, t0 + nt, ... fill it; a barrier of those
// threads belongs between this and build_bmat.
template <class F>
__device__ __forceinline__ void stage_digits(Smem<F> &S, const typename F::Digits &sw, int t0, int nt)
{
    for (int idx = t0; idx < F::kDigits * 7 * kWz; idx += nt) {
        const int row = idx / kWz, j = idx - row * kWz - 8, e = row / 7, ti = row - 7 * e;
        S.wz[e][ti][j + 8] = j >= 0 && j < 7 ? sw.d[e][ti * 7 + j] : __float2half(0.f);
    }
}

// B_i: N row nn = NLV e + 8 rho + c (digit e of w, output row rho of the
// group, column c of the block), K index k; threads t0, t0 + nt, ... fill it,
// a 16-byte chunk of eight k at a time: chunk kh of a row holds
// w_e[i - rho][8 kh - c - 1 ..], consecutive halves of the staged row. (One
// half at a time, each from the kernel parameters at an address of its own,
// the set-up took 16,500 cycles, 8 us of every launch; so it takes 4,000.
// box2d3r 1024^2 on GB300: 20.9 us a launch before, 14.9 so.)
template <class F>
__device__ __forceinline__ void build_bmat(Smem<F> &S, int t0, int nt)
{
    constexpr int NCOL = NLV * F::kDigits;
    for (int idx = t0; idx < NOFF * NCOL * 2; idx += nt) {
        const int i = idx / (NCOL * 2), rem = idx - i * (NCOL * 2);
        const int nn = rem >> 1, kh = rem & 1;
        const int e = nn / NLV, rho = (nn % NLV) >> 3, c = nn & 7;
        const int ti = i - rho;
        __align__(16) __half v[8];
        if (ti >= 0 && ti < 7) {
            const __half *src = &S.wz[e][ti][8 * kh + 7 - c];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = src[k];
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __float2half(0.f);
        }
        *reinterpret_cast<uint4 *>(&S.bmat[i][(nn >> 3) * 128 + (nn & 7) * 8 + kh * 64]) =
            *reinterpret_cast<const uint4 *>(v);
    }
}

// The same for 1D: the 49 taps of digit e at wz1[e][32 .. 80] (the rows of wz,
// laid end to end), and B of K step kk: N row nn = 32 e + c (output c of a
// row), tap 16 kk + k - c.
constexpr int kWz1d = 112;
static_assert(FmtF64::kDigits * kWz1d <= FmtF64::kDigits * 7 * kWz, "the 1D rows fit wz");
template <class F>
__device__ __forceinline__ void stage_digits_1d(Smem<F> &S, const typename F::Digits &sw, int t0, int nt)
{
    __half *wz = &S.wz[0][0][0];
    for (int idx = t0; idx < F::kDigits * kWz1d; idx += nt) {
        const int e = idx / kWz1d, j = idx - e * kWz1d - 32;
        wz[idx] = j >= 0 && j <= 2 * kReach1d ? sw.d[e][j] : __float2half(0.f);
    }
}
template <class F>
__device__ __forceinline__ void build_bmat_1d(Smem<F> &S, int t0, int nt)
{
    constexpr int NCOL = NLV * F::kDigits;
    const __half *wz = &S.wz[0][0][0];
    for (int idx = t0; idx < kSteps1d * NCOL * 2; idx += nt) {
        const int kk = idx / (NCOL * 2), rem = idx - kk * (NCOL * 2);
        const int nn = rem >> 1, kh = rem & 1;
        const __half *src = wz + (nn / NLV) * kWz1d + 32 + 16 * kk + 8 * kh - nn % NLV;
        __align__(16) __half v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = src[k];
        *reinterpret_cast<uint4 *>(&S.bmat[kk][(nn >> 3) * 128 + (nn & 7) * 8 + kh * 64]) =
            *reinterpret_cast<const uint4 *>(v);
    }
}

// Batch mode: the grid of global tile `tile` (last record whose tile_begin
// is not above it).
template <class F>
__device__ __forceinline__ int grid_of(const TcGrid<F> *grids, int ngrids, int tile)
{
    int lo = 0, hi = ngrids - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (grids[mid].tile_begin <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// What one launch computes.
constexpr int kModeGrid = 0;    // one sweep of a 2D grid
constexpr int kMode1d = 1;      // several steps of a 1D grid
constexpr int kModeSteps = 2;   // several steps of a 2D radius-1 grid

// kModeSteps: T steps of a 3x3 stencil are one sweep of its T-fold
// self-convolution (7x7 at T = 3) wherever the window of every intermediate
// step stays inside the grid, that is for outputs at least T - 1 points from
// the boundary. Those come from the digit pipeline (`sw` holds the convolved
// weights); the frame of T - 1 points along the boundary is computed step by
// step with FP64 FMA by the epilogue warps before their first accumulator is
// ready, from the same input, with the halo each single sweep would read. A
// launch costs what one step on the 7x7 pipeline costs (its limit is the
// digits, not the taps): box2d1r 2047 x 1531, 60 steps, GB300: 1818 us at a
// step per launch, 525 at three; star2d1r 1024^2, 100 steps: 1295 us on the
// FP64 FMA kernel (the FP64 pipe takes 10 us of each step's 13), 478 so.
constexpr int kMaxSteps = 3;

// Grids of odd pitch or odd first column, whose rows are not all 16-byte
// aligned: the rows of each parity have a map of their own, its pitch two rows
// and its base a 16-byte boundary at the first of them or one point before it.
// A window's even and odd rows come by one load each, from the even column at
// or before the window's first, so that they may lie one point late in the
// stage. (GB300, 8192^2 box2d3r: 412 us a sweep, one point at a time by
// cp.async 570 from one warp and 607 from the slicers, row by row 508 by bulk
// copies; 6237 on FP64 FMA, 326 on an even layout. The output's 8-byte stores
// alone cost 60 of those us.)
struct OddRows {
    CUtensorMap map[2];  // rows 0, 2, .. and 1, 3, .. of a window
    int x[2], y[2];      // where tile (0, 0)'s window starts in them
    unsigned late[2];    // points by which its rows are late
};

template <class F, int MODE>
struct StepArgs {
    const typename F::Out *in;  // interior point (0, 0) of the source
    int steps;                  // T
    int radius;                 // of one step
    int aligned;                // 1D: the buffers and the interior are 16-byte aligned
    unsigned taps;              // 2D steps, bit t: weight t belongs to the pattern
    int frame_cta;              // CTAs from this one on compute the frame
    typename F::Out w[MODE == kModeGrid ? 49 : 9];  // weights of one step (kModeGrid: at the centre of a 7x7)
    OddRows rows;               // odd layouts
    int above, below;           // odd layouts: rows of the grid before and after the ones swept
    int pattern;                // of the weights
    int redo;                   // tiles that hold an Inf or NaN are computed again (else: NaN)
};

// The frame's arithmetic, that of single sweeps: FP64 FMA, or double-float.
__device__ __forceinline__ void tap_acc(double &a, double w, double x) { a = fma(w, x, a); }
// (ff::ff_tap's operations as intrinsics, which the compiler does not contract:
// a product folded into the TwoSum that follows it would count its rounding
// error twice.)
__device__ __forceinline__ void tap_acc(float2 &a, float2 w, float2 x)
{
    const float p = __fmul_rn(w.x, x.x), ep = __fmaf_rn(w.x, x.x, -p);
    const float s = __fadd_rn(a.x, p), bb = __fsub_rn(s, a.x);
    const float q = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    a.y = __fmaf_rn(w.y, x.x, __fmaf_rn(w.x, x.y, __fadd_rn(__fadd_rn(a.y, q), ep)));
    a.x = s;
}
__device__ __forceinline__ double tap_sum(double a) { return a; }
__device__ __forceinline__ float2 tap_sum(float2 a) { return ff::ff_finish(a.x, a.y); }
__device__ __forceinline__ double prev_lane(double x) { return __shfl_up_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ double next_lane(double x) { return __shfl_down_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ float2 prev_lane(float2 x)
{
    return make_float2(__shfl_up_sync(0xffffffffu, x.x, 1), __shfl_up_sync(0xffffffffu, x.y, 1));
}
__device__ __forceinline__ float2 next_lane(float2 x)
{
    return make_float2(__shfl_down_sync(0xffffffffu, x.x, 1), __shfl_down_sync(0xffffffffu, x.y, 1));
}
// One strip of the frame, by one warp: T steps for the T - 1 points next to
// an edge, at positions l0 .. l0 + 25 along it. `edge` is the offset of
// the edge's first point, `sa` the step away from the edge, `sl` the step
// along it (`len` points, outputs before `end`); w and taps are the 3x3 weights turned the same
// way. Lane l holds position l0 - 3 + l; neighbours along the edge come by
// shuffles, and every level's outermost lanes fall out of use. A halo cell
// keeps the value of the buffer that the sweep of its level would read.
// (The loops over levels and strips stay rolled: the code runs once or a few
// times per launch, and unrolled its instruction fetches took most of 13,000
// cycles, more than the first tile needs to reach the epilogue.)
template <class V>
__device__ __forceinline__ void frame_strip(const V *__restrict__ in, V *__restrict__ out, long long edge,
                                            long long sa, long long sl, int len, int l0, int end, int steps,
                                            const V (&w)[9], unsigned taps)
{
    constexpr int T = kMaxSteps;
    const int lane = threadIdx.x & 31, p = l0 - T + lane;
    const bool inside = p >= 0 && p < len, halo = p == -1 || p == len;
    const long long at = edge + (long long)p * sl;
    V even[2 * T], odd[2 * T - 1], u[2 * T];  // row k of the strip is u[k + 1]
#pragma unroll
    for (int j = 0; j < 2 * T; ++j) u[j] = even[j] = inside || halo ? in[at + (j - 1) * sa] : V{};
#pragma unroll
    for (int j = 0; j < 2 * T - 1; ++j) odd[j] = halo || (inside && j == 0) ? out[at + (j - 1) * sa] : V{};
#pragma unroll 1
    for (int level = 1; level <= steps; ++level) {
        const int rows = 2 * steps - 1 - level;  // rows of this level that count
        V v[2 * T - 2];
#pragma unroll
        for (int k = 0; k < 2 * T - 2; ++k) v[k] = V{};
#pragma unroll
        for (int j = 0; j < 2 * T; ++j) {
            const V x[3] = {prev_lane(u[j]), u[j], next_lane(u[j])};
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int k = j - t / 3;  // row k takes u[k + da] through weight row da
                if (k >= 0 && k < 2 * T - 2 && k < rows && (taps >> t & 1u)) tap_acc(v[k], w[t], x[t % 3]);
            }
        }
        // the next level's input
        u[0] = (level & 1) ? odd[0] : even[0];
#pragma unroll
        for (int k = 0; k < 2 * T - 2; ++k)
            u[k + 1] = halo ? ((level & 1) ? odd[k + 1] : even[k + 1]) : inside ? tap_sum(v[k]) : V{};
    }
    if (p < end && lane >= T && lane < 32 - T) {
#pragma unroll
        for (int k = 0; k < T - 1; ++k)
            if (k < steps - 1) out[at + k * sa] = u[k + 1];
    }
}

// The frame of an m x n grid, strip by strip, shared by `nwarps` warps.
template <class F>
__device__ __noinline__ void frame_steps(const StepArgs<F, kModeSteps> &s, typename F::Out *__restrict__ out, int m, int n,
                                         long long ld, int warp, int nwarps)
{
    constexpr int S = 32 - 2 * kMaxSteps;  // outputs per strip
    const int fw = s.steps - 1;            // frame width
    if (fw == 0) return;
    const int nx = (n + S - 1) / S, ny = (m - 2 * fw + S - 1) / S;
#pragma unroll 1
    for (int i = warp; i < 2 * (nx + ny); i += nwarps) {
        const bool horiz = i < 2 * nx;  // top and bottom rows, whole length
        const int q = horiz ? i : i - 2 * nx, cnt = horiz ? nx : ny;
        const bool far = q >= cnt;
        const int l0 = (far ? q - cnt : q) * S + (horiz ? 0 : fw);
        typename F::Out w[9];
        unsigned taps = 0;
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const int da = far ? 2 - t / 3 : t / 3, dl = t % 3;
            const int src = horiz ? 3 * da + dl : 3 * dl + da;
            w[t] = s.w[src];
            taps |= (s.taps >> src & 1u) << t;
        }
        // columns end fw short of the corners, which belong to the rows
        frame_strip(s.in, out, far ? (horiz ? (long long)(m - 1) * ld : n - 1) : 0,
                    horiz ? (far ? -ld : ld) : (far ? -1 : 1), horiz ? 1 : ld, horiz ? n : m, l0, horiz ? n : m - fw,
                    s.steps, w, taps);
    }
}

// The (T - 1) r outputs next to one end of a 1D grid (T r <= 24), by one warp:
// points -r .. 2 T r - r - 1 counted from that end, two per lane, in `buf`
// (level l's in buf[l % 2]); every level's last r points fall out of use.
template <class F>
__device__ __noinline__ void frame_end_1d(const StepArgs<F, kMode1d> &s, typename F::Out *__restrict__ out, long long n, bool left,
                                          typename F::Out (*buf)[kFrame1d])
{
    using V = typename F::Out;
    const int lane = threadIdx.x & 31, r = s.radius, points = 2 * s.steps * r;
    auto at = [&](int i) { return left ? i - r : n - 1 - (i - r); };  // point i - r from this end
    for (int i = lane; i < points; i += 32) {
        buf[0][i] = s.in[at(i)];
        if (i < r) buf[1][i] = out[at(i)];  // the halo that odd levels read
    }
    __syncwarp();
#pragma unroll 1
    for (int level = 1; level <= s.steps; ++level) {
        const V *u = buf[(level & 1) ^ 1];
        for (int i = r + lane; i < points - level * r; i += 32) {
            V v{};
#pragma unroll 1
            for (int t = 0; t <= 2 * r; ++t) tap_acc(v, s.w[left ? t : 2 * r - t], u[i - r + t]);
            buf[level & 1][i] = tap_sum(v);
        }
        __syncwarp();
    }
    for (int i = r + lane; i < s.steps * r; i += 32) out[at(i)] = buf[s.steps & 1][i];
}

// A tile's outputs computed again (Redo), by the whole CTA: FP64 FMA or double-
// float sums of single steps on windows in shared memory (`a`, then `b` and `a`
// by turns). Points outside the grid and its halo are zeros that meet no output:
// those next to the boundary are the frame's.
template <class F, int MODE>
__device__ __forceinline__ void redo_tile(const StepArgs<F, MODE> &s, typename F::Out *__restrict__ out, int m, int n,
                                          long long ld, int tiles_x, int tile, typename F::Out *a, typename F::Out *b)
{
    using V = typename F::Out;
    const int tid = threadIdx.x, nt = blockDim.x, r = s.radius;
    if constexpr (MODE == kMode1d) {
        const int reach = s.steps * r, frame = reach - r;
        const long long at = (long long)tile * kOut1d;
        for (int i = tid; i < kOut1d + 2 * reach; i += nt) {
            const long long x = at + i - reach;
            a[i] = x >= -r && x < (long long)n + r ? s.in[x] : V{};
        }
        __syncthreads();
        for (int level = 1, len = kOut1d + 2 * (reach - r); level <= s.steps; ++level, len -= 2 * r) {
            for (int i = tid; i < len; i += nt) {
                V v{};
                for (int t = 0; t <= 2 * r; ++t) tap_acc(v, s.w[t], a[i + t]);
                b[i] = tap_sum(v);
                if (level == s.steps && at + i >= frame && at + i < (long long)n - frame) out[at + i] = b[i];
            }
            __syncthreads();
            V *const c = a;
            a = b;
            b = c;
        }
    } else {
        constexpr bool STEPS = MODE == kModeSteps;
        constexpr int W = TX + 2 * 3, K = STEPS ? 3 : 7;
        const int y0 = tile / tiles_x * TY, x0 = tile % tiles_x * TX;
        static_assert(TX == TY && W * W * 8 <= F::kDigits * PL * 2, "square tiles, whose windows fit a plane set");
        const int steps = STEPS ? s.steps : 1, reach = STEPS ? steps : 3, frame = STEPS ? steps - 1 : 0;
        const int top = STEPS ? -r : -r - s.above, bottom = STEPS ? m + r : m + r + s.below;
        for (int i = tid; i < (TX + 2 * reach) * (TX + 2 * reach); i += nt) {
            const int p = i / (TX + 2 * reach), q = i - p * (TX + 2 * reach);
            const int y = y0 - reach + p, x = x0 - reach + q;
            a[p * W + q] = y >= top && y < bottom && x >= -r && x < n + r ? s.in[(long long)y * ld + x] : V{};
        }
        __syncthreads();
        for (int level = 1; level <= steps; ++level) {
            const int side = TX + 2 * (steps - level);
            for (int i = tid; i < side * side; i += nt) {
                const int p = i / side, q = i - p * side;
                V v{};
                for (int t = 0; t < K * K; ++t) {
                    const int dy = t / K, dx = t - dy * K;
                    const bool tap = STEPS ? s.taps >> t & 1u
                                           : max(abs(dy - 3), abs(dx - 3)) <= r &&
                                                 in_pattern(s.pattern, 0, dy - 3, dx - 3, r);
                    if (tap) tap_acc(v, s.w[t], a[(p + dy) * W + q + dx]);
                }
                b[p * W + q] = tap_sum(v);
                const int y = y0 + p, x = x0 + q;
                if (level == steps && y >= frame && y < m - frame && x >= frame && x < n - frame)
                    out[(long long)y * ld + x] = b[p * W + q];
            }
            __syncthreads();
            V *const c = a;
            a = b;
            b = c;
        }
    }
}

template <class F, int MODE>
__device__ __noinline__ void redo_tiles(const StepArgs<F, MODE> &s, typename F::Out *__restrict__ out, int m, int n,
                                        long long ld, int tiles_x, int tiles, Smem<F> &S)
{
    using V = typename F::Out;
    for (int it = 0, tile = blockIdx.x; tile < tiles; ++it, tile += gridDim.x)
        if (S.redo.holds(it, it))
            redo_tile<F, MODE>(s, out, m, n, ld, tiles_x, tile, reinterpret_cast<V *>(S.planes[0][0]),
                               reinterpret_cast<V *>(S.planes[1][0]));
}

// One grid (BATCH = false: kernel parameters describe it, tiles are dealt
// round-robin) or a batch of grids (BATCH = true: `grids` describes them,
// each CTA takes a contiguous run of the batch's tiles, and the MMA warp
// rebuilds its B matrices when the run crosses into the next grid, after
// the MMAs of the previous tile have completed).
template <class F, bool BATCH, int MODE = kModeGrid, bool ODD = false>
__global__ void __launch_bounds__(kThreads<F>, 1)
    k2d_tc(const __grid_constant__ CUtensorMap tmap, typename F::Out *__restrict__ out, int m, int n,
           long long ld, int tiles_x, int tiles, int map_x, int map_y, typename F::Digits sw, WaitCfg wc,
           const TcGrid<F> *__restrict__ grids, int ngrids, const __grid_constant__ StepArgs<F, MODE> sa)
{
    constexpr bool ONED = MODE == kMode1d, STEPS = MODE == kModeSteps;
    static_assert(!BATCH || (MODE == kModeGrid && !ODD), "batches run one sweep of 7x7 grids");
    constexpr int D = F::kDigits, kSliceWarps = F::kSliceWarps, kSliceThreads = 32 * kSliceWarps;
    constexpr int kWarpEpi0 = kWarpSlice0 + kSliceWarps;
    constexpr int PER = (NPAIR + kSliceThreads - 1) / kSliceThreads;  // pairs of points a slicer holds
    using SM = Smem<F>;
    extern __shared__ unsigned char smem_raw[];
    SM &S = *reinterpret_cast<SM *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_allow_dependents();
    int my_tiles, first = 0;
    if constexpr (BATCH) {
        const int per = tiles / (int)gridDim.x, extra = tiles % (int)gridDim.x, b = (int)blockIdx.x;
        first = b * per + min(b, extra);
        my_tiles = per + (b < extra ? 1 : 0);
    } else {
        my_tiles = (int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    }
    // Where tile `it` of this CTA lies: its grid and output origin.
    auto tile_at = [&](int it, int &g, int &x0, int &y0) {
        if constexpr (BATCH) {
            const int tile = first + it;
            g = grid_of(grids, ngrids, tile);
            const int local = tile - grids[g].tile_begin, tx = grids[g].tiles_x;
            const int ty = local / tx;
            x0 = (local - ty * tx) * TX;
            y0 = ty * TY;
        } else {
            const int tile = blockIdx.x + it * gridDim.x;
            const int ty = tile / tiles_x;
            g = 0;
            x0 = (tile - ty * tiles_x) * TX;
            y0 = ty * TY;
        }
    };
    auto load_window = [&](int it, unsigned bar) {
        int g, x0, y0;
        tile_at(it, g, x0, y0);
        const CUtensorMap *map = &tmap;
        int mx = map_x, my = map_y;
        if constexpr (BATCH) {
            map = &grids[g].map;
            mx = grids[g].map_x;
            my = grids[g].map_y;
        }
        const int x = mx + x0 - 4, y = my + y0 - 3;
        if constexpr (ODD) {
            mbar_expect_tx(bar, ST_Y * kOddRow);
            tma_load_2d(smem_addr(S.stage), &sa.rows.map[0], sa.rows.x[0] + x0, sa.rows.y[0] + y0 / 2, bar);
            tma_load_2d(smem_addr(S.stage) + kOddHalf, &sa.rows.map[1], sa.rows.x[1] + x0, sa.rows.y[1] + y0 / 2, bar);
        } else {
            mbar_expect_tx(bar, kStageBytes);
            tma_load_2d(smem_addr(S.stage), map, x, y, bar);
        }
    };
    volatile int *abort = &S.abort;
    const unsigned stage_full = smem_addr(&S.stage_full), stage_empty = smem_addr(&S.stage_empty);
    auto bar2 = [](unsigned long long (&b)[2], int i) { return smem_addr(&b[i]); };
    const unsigned long long limit = wc.limit_ns;
    auto wait = [abort, limit](unsigned bar, unsigned parity) {
        return mbar_wait(bar, parity, abort, &g_tc_wait_timeouts, limit);
    };

    if (warp == kWarpTma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&S.tmem)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    int issued = 0, committed = 0;  // window loads issued / MMA batches committed (one thread each)
    if (tid == 0) {
        mbar_init(stage_full, 1);
        mbar_init(stage_empty, kSliceWarps);
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar2(S.planes_full, i), kSliceWarps);
            mbar_init(bar2(S.planes_empty, i), 1);
            mbar_init(bar2(S.acc_full, i), 1);
            mbar_init(bar2(S.acc_empty, i), F::kEpiWarps);
        }
        S.abort = 0;
        if constexpr (kRedoable<F>) S.redo.count = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!ONED && my_tiles > 0 && !wc.skip_loads) {  // the first window load overlaps the set-up below
            pdl_wait();
            load_window(0, stage_full);
            issued = 1;
        }
    }
    // B matrices of the first tile's grid (batch mode: the MMA warp rebuilds
    // them whenever its run of tiles enters another grid), by every warp but
    // the first, which may be waiting for the previous kernel's end.
    constexpr int kBuilders = kThreads<F> - 32;
    int g_bmat = 0;
    if constexpr (BATCH) {
        if (my_tiles > 0) {
            int x0, y0;
            tile_at(0, g_bmat, x0, y0);
            if (warp != 0) stage_digits<F>(S, grids[g_bmat].digits, tid - 32, kBuilders);
        }
    } else {
        if (warp != 0) {
            if constexpr (ONED)
                stage_digits_1d<F>(S, sw, tid - 32, kBuilders);
            else
                stage_digits<F>(S, sw, tid - 32, kBuilders);
        }
    }
    if (warp != 0) {
        asm volatile("bar.sync %0, %1;" ::"n"(kBuildBarrier), "n"(kBuilders) : "memory");
        if constexpr (ONED)
            build_bmat_1d<F>(S, tid - 32, kBuilders);
        else
            build_bmat<F>(S, tid - 32, kBuilders);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // All 512 columns are this CTA's, so they start at column 0: as a constant
    // it costs the MMA thread no move into a uniform register per MMA.
    const unsigned tmem = 0;

    if (warp == kWarpTma) {
        // ------------------------------------------------ TMA producer
        if constexpr (ONED) {
            // A window inside the halo and 16-byte aligned is one bulk copy;
            // others are copied in 8-byte pieces, with zeros past the halo.
            pdl_wait();
            bool ok = !wc.skip_loads;
            const long long end = (long long)n + sa.radius;  // (2^31 and more for the longest arrays)
            for (int it = 0; it < my_tiles && ok; ++it) {
                ok = lane != 0 || wait(stage_empty, (it & 1) ^ 1);
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                const long long x = (long long)(blockIdx.x + it * gridDim.x) * kOut1d - kReach1d;
                const unsigned dst = smem_addr(S.stage);
                if (sa.aligned && x >= -sa.radius && x + kWin1d <= end) {
                    if (lane == 0) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        mbar_expect_tx(stage_full, kBytes1d);
                        bulk_load(dst, sa.in + x, kBytes1d, stage_full);
                        issued = it + 1;
                    }
                } else {
                    for (int i = lane; i < kWin1d; i += 32) {
                        const bool take = x + i >= -sa.radius && x + i < end;
                        cp_async8(dst + 8u * i, take ? sa.in + x + i : sa.in, take);
                    }
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(stage_full);
                        issued = it + 1;
                    }
                }
            }
        } else if (lane == 0 && !wc.skip_loads) {
            for (int it = issued; it < my_tiles; ++it) {
                if (!wait(stage_empty, (it & 1) ^ 1)) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                load_window(it, stage_full);
                issued = it + 1;
            }
        }
    } else if (warp == kWarpMma) {
        // ------------------------------------------------ MMA issuer
        constexpr unsigned lbo = ONED ? kPhase1d : 16, sbo = ONED ? 128 : R * kRowBytes;
        const unsigned long long a_desc_buf0 = smem_desc(smem_addr(S.planes[0][0]), lbo, sbo);
        const unsigned long long a_desc_buf1 = smem_desc(smem_addr(S.planes[1][0]), lbo, sbo);
        const unsigned long long b_desc0 = smem_desc(smem_addr(S.bmat[0]), 128, 256);
        for (int it = 0; it < my_tiles; ++it) {
            const int buf = it & 1, use = it >> 1;
            if constexpr (BATCH) {
                int g, x0, y0;
                tile_at(it, g, x0, y0);
                if (g != g_bmat) {
                    // New grid with other weights: once the MMAs of the
                    // previous tile (and so all earlier ones) are done reading
                    // B, the warp rewrites it. Grids that share the weights
                    // (the same digits_id) keep it.
                    if (grids[g].digits_id != grids[g_bmat].digits_id) {
                        int ok = 1;
                        if (lane == 0 && it > 0) ok = wait(bar2(S.acc_full, (it - 1) & 1), ((it - 1) >> 1) & 1);
                        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
                        tc_fence_after();
                        stage_digits<F>(S, grids[g].digits, lane, 32);
                        __syncwarp();
                        build_bmat<F>(S, lane, 32);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    }
                    g_bmat = g;
                }
            }
            if (!__all_sync(0xffffffffu, wait(bar2(S.planes_full, buf), use & 1) &&
                                             wait(bar2(S.acc_empty, buf), (use & 1) ^ 1)))
                break;
            tc_fence_after();
            if (elect_one()) {
                // The issuing thread stalls on every MMA until the tensor core
                // takes it, so nothing else sits between them: all MMAs are
                // unrolled, each descriptor one add of a compile-time offset.
                const unsigned d_base = tmem + (unsigned)(kAccStride * buf);
                const unsigned long long a0 = buf ? a_desc_buf1 : a_desc_buf0;
                if constexpr (ONED)
                    tile_mma_1d<F, 0, 0>(d_base, a0, b_desc0);
                else
                    tile_mma<F, 0, 0>(d_base, a0, b_desc0);
                mma_commit(bar2(S.planes_empty, buf));  // planes may be overwritten
                mma_commit(bar2(S.acc_full, buf));      // accumulator ready
            }
            committed = it + 1;
        }
    } else if (warp < kWarpEpi0) {
        // ------------------------------------------------ slicers
        constexpr int kPairs = ONED ? NPAIR1D : NPAIR;
        const int st = tid - 32 * kWarpSlice0;
        const bool leader = st == 0;
        auto stage_pair = [&](int idx) {  // pair idx of a 2D window
            if constexpr (ODD) {
                const int row = idx / PAIRS, half = row & 1;
                return reinterpret_cast<uint2 *>(S.stage) + half * (kOddHalf / 8) + (row >> 1) * (kOddRow / 8) +
                       2 * (idx % PAIRS) + (half ? sa.rows.late[1] : sa.rows.late[0]);
            } else {
                return reinterpret_cast<uint2 *>(S.stage + idx);
            }
        };
        for (int it = 0; it < my_tiles; ++it) {
            const int buf = it & 1, use = it >> 1;
            // (a) window landed? Every thread waits for itself; one barrier
            // per tile, at (c), makes them agree to go on. (Before, one thread
            // waited and three barriers shared its answers and the maxima.
            // GB300, launch before and after: 1d2r 10,240,000 66.9 and 55.8
            // us, box2d1r 8192^2 three steps 381 and 359, box2d3r 8192^2
            // split 305 and 295; FP64, bound by the MMAs, 335 and 338.)
            const bool landed = wait(stage_full, it & 1);
            // (b) window -> registers, then release the stage to the next load.
            if constexpr (STEPS || ODD) {
                // Points past the halo meet zero weights in every output kept,
                // but must not set the tile's scale either: tiles at the
                // boundary first zero them in the stage (a thread the points
                // that it reads next).
                const int r = STEPS ? 1 : sa.radius;
                // (A band's neighbouring rows are in, so that its tiles see the
                // windows, and take the scales, of a whole sweep.)
                const int top = STEPS ? -r : -r - sa.above, bottom = STEPS ? m + r : m + r + sa.below;
                int g, x0, y0;
                tile_at(it, g, x0, y0);
                if (x0 - 4 < -r || y0 - 3 < top || x0 + ST_X - 4 >= n + r || y0 + ST_Y - 3 >= bottom) {
#pragma unroll 1
                    for (int idx = st; idx < kPairs; idx += kSliceThreads) {
                        const int yy = y0 - 3 + idx / PAIRS, xx = x0 - 4 + 2 * (idx % PAIRS);
                        const bool row = yy >= top && yy < bottom;
                        uint2 *at = stage_pair(idx);
                        if (!row || xx < -r || xx >= n + r) at[0] = make_uint2(0u, 0u);
                        if (!row || xx + 1 < -r || xx + 1 >= n + r) at[1] = make_uint2(0u, 0u);
                    }
                }
            }
            uint4 v[PER];
            float vmax = 0.f;   // split: largest |hi|
            unsigned emax = 0;  // FP64: largest upper word without its sign, then biased exponent
            // (three steps: exponents at once; shifted after, that kernel spills: 378 us, so 353)
            auto size_of = [](unsigned hi) { return STEPS ? (hi >> 20) & 0x7FFu : hi & 0x7FFFFFFFu; };
            if constexpr (!ODD) {
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    const int idx = st + q * kSliceThreads;
                    v[q] = idx < kPairs ? S.stage[idx] : make_uint4(0u, 0u, 0u, 0u);
                }
            } else {
                // pair q of this thread lies 7 q rows and 4 q pairs on, or one row more
                static_assert(kSliceThreads == 7 * PAIRS + 4 && PER <= 10);
                unsigned u = st;
                asm volatile("" : "+r"(u));  // what follows is not kept in registers over a tile
                const unsigned row0 = u / PAIRS, col0 = u % PAIRS, at0 = smem_addr(S.stage) + 16 * col0;
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    v[q] = make_uint4(0u, 0u, 0u, 0u);
                    if (st + q * kSliceThreads < kPairs) {
                        const unsigned next = col0 + 4 * q >= PAIRS ? 1u : 0u, row = row0 + 7 * q + next;
                        const unsigned at = at0 + 64 * q - next * (16 * PAIRS) + (row >> 1) * kOddRow +
                                            ((row & 1) ? kOddHalf + 8 * sa.rows.late[1] : 8 * sa.rows.late[0]);
                        asm volatile("ld.shared.v2.b32 {%0, %1}, [%4];\n\tld.shared.v2.b32 {%2, %3}, [%4 + 8];"
                                     : "=r"(v[q].x), "=r"(v[q].y), "=r"(v[q].z), "=r"(v[q].w)
                                     : "r"(at)
                                     : "memory");
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                if constexpr (F::kF64)
                    emax = max(emax, max(size_of(v[q].y), size_of(v[q].w)));
                else if constexpr (kRedoable<F>)
                    vmax = max_nan(vmax, max_nan(fabsf(__uint_as_float(v[q].x)), fabsf(__uint_as_float(v[q].z))));
                else
                    vmax = fmaxf(vmax, fmaxf(fabsf(__uint_as_float(v[q].x)), fabsf(__uint_as_float(v[q].z))));
            }
            if constexpr (F::kF64) {
                emax = __reduce_max_sync(0xffffffffu, emax) >> (STEPS ? 0 : 20);
            } else if constexpr (kRedoable<F>) {  // (not negative: ordered as integers, a NaN above Inf)
                vmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(vmax)));
            } else {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
            }
            __syncwarp();
            if (lane == 0) {
                if constexpr (F::kF64)
                    S.redi[buf][warp - kWarpSlice0] = (int)emax;
                else
                    S.red[buf][warp - kWarpSlice0] = vmax;
                mbar_arrive(stage_empty);
            }
            // (c) planes of this buffer free (MMAs two tiles back done)? The
            // barrier also publishes the maxima; their next tile's are in the
            // other set, and the one after that comes after its barrier.
            const bool free = landed && wait(bar2(S.planes_empty, buf), (use & 1) ^ 1);
            if (bar_any(kSliceBarrier, kSliceThreads, !free)) break;
            int ex;
            bool finite = true;
            if constexpr (F::kF64) {
                int eb = S.redi[buf][0];
#pragma unroll
                for (int i = 1; i < kSliceWarps; ++i) eb = max(eb, S.redi[buf][i]);
                ex = max(eb, 1);
                finite = ex != 2047;
            } else {
                vmax = S.red[buf][0];
                if constexpr (kRedoable<F>) {
#pragma unroll
                    for (int i = 1; i < kSliceWarps; ++i) vmax = max_nan(vmax, S.red[buf][i]);
                    finite = vmax <= 3.402823466e38f;
                    if (!finite) vmax = 0.f;
                } else {
#pragma unroll
                    for (int i = 1; i < kSliceWarps; ++i) vmax = fmaxf(vmax, S.red[buf][i]);
                }
                // six digits: |x| / 2^ex < 1/4, the top digit within 128
                ex = split::tile_exponent(vmax) + (D == 6 ? 1 : 0);
            }
            if (leader) S.scale_exp[it & 3] = (F::kF64 && !finite) ? kNonFiniteTile : ex;
            if constexpr (kRedoable<F>)
                if (leader && !finite && sa.redo) S.redo.add(it);
            unsigned *dst0 = reinterpret_cast<unsigned *>(&S.planes[buf][0][0]);
            // 1D: chunk idx / 4 in phase (idx / 4) % 4
            auto word = [](int idx) {
                return ONED ? (idx >> 2 & 3) * (kPhase1d / 4) + (idx >> 4) * 4 + (idx & 3) : idx;
            };
            if constexpr (F::kF64) {
                constexpr bool EVEN = F::kLevels > 6;
                if (ex >= kFastExp) {
#pragma unroll
                    for (int q = 0; q < PER; ++q) {
                        const int idx = st + q * kSliceThreads;
                        if (idx < kPairs) f64_cut_fast<EVEN, PL / 2>(v[q], ex, dst0 + word(idx));
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < PER; ++q) {
                        const int idx = st + q * kSliceThreads;
                        if (idx < kPairs) f64_cut_any<EVEN, PL / 2>(v[q], ex, dst0 + word(idx));
                    }
                }
            } else {
                const float to_digits = ldexpf(1.0f, kDigitBits - ex);
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    const int idx = st + q * kSliceThreads;
                    if (idx < kPairs) {
                        split::f2x a, b, s2;
                        asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "r"(v[q].x), "r"(v[q].z));
                        asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "r"(v[q].y), "r"(v[q].w));
                        asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(to_digits));
                        unsigned wd[D];
                        split::slice_digit_pairs_x2(split::f2_mul(a, s2), split::f2_mul(b, s2), wd);
                        unsigned *dst = dst0 + word(idx);
#pragma unroll
                        for (int k = 0; k < D; ++k) dst[k * (PL / 2)] = wd[k];
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar2(S.planes_full, buf));
        }
    } else {
        // ------------------------------------------------ epilogue
        // Warp w reads TMEM lanes 32 (w % 4) ..; lane -> D row m = (row group
        // er, block eb); warp h of a quarter (one warp per quarter split,
        // two FP64) stores rows kRowsPerWarp h .. of the group, columns
        // 8 eb .. 8 eb + 7.
        if constexpr (STEPS) {
            const int fc = (int)blockIdx.x - sa.frame_cta, fn = (int)gridDim.x - sa.frame_cta;
            if (fc >= 0) {
                pdl_wait();
                frame_steps<F>(sa, out, m, n, ld, (warp - kWarpEpi0) * fn + fc, F::kEpiWarps * fn);
            }
        }
        if constexpr (ONED) {  // the ends, on the last CTA (no other has fewer tiles)
            if (blockIdx.x == gridDim.x - 1 && warp < kWarpEpi0 + 2 && sa.steps > 1) {
                pdl_wait();
                frame_end_1d<F>(sa, out, n, warp == kWarpEpi0,
                                reinterpret_cast<typename F::Out(*)[kFrame1d]>(S.ends[warp - kWarpEpi0][0]));
            }
        }
        const int quarter = warp & 3, h = (warp - kWarpEpi0) >> 2;
        const int mrow = 32 * quarter + lane;
        const int er = mrow >> 3, eb = mrow & 7;
        const unsigned lane_bits = (unsigned)(32 * quarter) << 16;
        const int frame = STEPS || ONED ? (sa.steps - 1) * sa.radius : 0;
        for (int it = 0; it < my_tiles; ++it) {
            const int buf = it & 1, use = it >> 1;
            if (!wait(bar2(S.acc_full, buf), use & 1)) break;
            tc_fence_after();
            int g, x0, y0;
            tile_at(it, g, x0, y0);
            typename F::Out *o_base = out;
            long long o_ld = ld;
            int o_m = m, o_n = n, ew = sw.ew;
            if constexpr (BATCH) {
                o_base = grids[g].out;
                o_ld = grids[g].ld;
                o_m = grids[g].m;
                o_n = grids[g].n;
                ew = grids[g].digits.ew;
            }
            const int ex = S.scale_exp[it & 3];
            const int xb = x0 + 8 * eb;
            constexpr int kRowsPerWarp = R * 4 / F::kEpiWarps;  // 4 split, 2 FP64
            constexpr int C = F::kCols, kPasses = kRowsPerWarp * 8 / C;
#pragma unroll 1
            for (int pass = 0; pass < kPasses; ++pass) {
                const int rho = kRowsPerWarp * h + pass * C / 8;
                const int c0 = pass * C % 8;  // first of the C columns of this pass
                float acc[F::kLevels][C];
#pragma unroll
                for (int L = 0; L < F::kLevels; ++L)
                    tmem_ldc(tmem + lane_bits + (unsigned)(kAccStride * buf + NLV * L + 8 * rho + c0), acc[L]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (pass == kPasses - 1) {  // accumulator drained: hand it back to the MMA warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar2(S.acc_empty, buf));
                }
                typename F::Out res[C];
                if constexpr (F::kF64) {
                    // value = T 2^c with T from the levels (f64_combine) and
                    // c = (input scale) + (weight scale) - 1080.
                    const int c = ex + ew - 1080;
                    long long t[C];
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        if constexpr (F::kLevels == 7) {
                            const float lv[7] = {acc[0][j], acc[1][j], acc[2][j], acc[3][j],
                                                 acc[4][j], acc[5][j], acc[6][j]};
                            t[j] = f64_combine(lv, sw.rest);
                        } else {
                            const float lv[6] = {acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4][j], acc[5][j]};
                            t[j] = f64_combine(lv);
                        }
                    }
                    if (f64_scale_is_plain(c)) {
#pragma unroll
                        for (int j = 0; j < C; ++j) res[j] = f64_from_fixed_plain(t[j], c);
                    } else {
#pragma unroll
                        for (int j = 0; j < C; ++j)
                            res[j] = ex == kNonFiniteTile ? __longlong_as_double(0x7FF8000000000000ll)
                                                          : f64_from_fixed(t[j], c);
                    }
                } else {
                    const float scale = ldexpf(1.0f, ex + ew - 2 * kDigitBits);
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        float h1, e1, h2, e2, hi, lo;
                        two_sum(acc[0][j], acc[1][j] * 0x1p-9f, h1, e1);
                        two_sum(h1, acc[2][j] * 0x1p-18f, h2, e2);
                        float tail = acc[4][j] * 0x1p-36f;
                        if constexpr (D == 6) tail = fmaf(acc[D - 1][j], 0x1p-45f, tail);
                        tail = fmaf(acc[3][j], 0x1p-27f, tail);
                        two_sum(h2, (e1 + e2) + tail, hi, lo);
                        res[j] = make_float2(hi * scale, lo * scale);
                    }
                }
                auto store2 = [](typename F::Out *o, typename F::Out u, typename F::Out v) {
                    if constexpr (F::kF64)
                        *reinterpret_cast<double2 *>(o) = make_double2(u, v);
                    else
                        *reinterpret_cast<float4 *>(o) = make_float4(u.x, u.y, v.x, v.y);
                };
                if constexpr (ONED) {
                    // Outputs 32 mrow + 8 rho .. + 7 of the tile: every lane's
                    // store has a line of its own, so it is 32 bytes where the
                    // grid allows them. (GB300, launch of 10,240,000 x 11 steps
                    // with 16 and 32 bytes: FP64 58.0 and 55.8 us, split 61.8
                    // and 53.7. In 2D, whose lanes share lines, no difference.)
                    const long long x = (long long)(blockIdx.x + it * gridDim.x) * kOut1d + 32 * mrow + 8 * rho + c0;
                    if (reinterpret_cast<unsigned long long>(out) % 32 == 0 && x >= frame && x + C <= n - frame) {
#pragma unroll
                        for (int j = 0; j < C; j += 4) store_32(out + x + j, res + j);
                    } else if (sa.aligned && x >= frame && x + C <= n - frame) {
#pragma unroll
                        for (int j = 0; j < C; j += 2) store2(out + x + j, res[j], res[j + 1]);
                    } else {
#pragma unroll
                        for (int j = 0; j < C; ++j)
                            if (x + j >= frame && x + j < n - frame) out[x + j] = res[j];
                    }
                } else {
                    const int yy = y0 + R * er + rho, xc = xb + c0;
                    if (yy >= o_m) continue;
                    if (STEPS && (yy < frame || yy >= o_m - frame)) continue;
                    typename F::Out *o = o_base + (long long)yy * o_ld + xc;
                    if (STEPS && (xc < frame || xc + C > o_n - frame)) {
#pragma unroll
                        for (int j = 0; j < C; ++j)
                            if (xc + j >= frame && xc + j < o_n - frame) o[j] = res[j];
                        continue;
                    }
                    if constexpr (ODD) {  // all rows of a warp start on the same side of a 16-byte boundary
                        const int late = (int)(reinterpret_cast<unsigned long long>(o) >> 3 & 1);
                        if (xc + C > o_n) {
#pragma unroll
                            for (int j = 0; j < C; ++j)
                                if (xc + j < o_n) o[j] = res[j];
                        } else if (late) {
                            o[0] = res[0];
#pragma unroll
                            for (int j = 1; j + 1 < C; j += 2) store2(o + j, res[j], res[j + 1]);
                            o[C - 1] = res[C - 1];
                        } else {
#pragma unroll
                            for (int j = 0; j < C; j += 2) store2(o + j, res[j], res[j + 1]);
                        }
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < C; j += 2) {
                        if (xc + j + 1 < o_n)
                            store2(o + j, res[j], res[j + 1]);
                        else if (xc + j < o_n)
                            o[j] = res[j];
                    }
                }
            }
        }
    }

    // Exit: every role is done or has given up. Let the last window load and
    // the last MMA batch finish (they have normally finished already) before
    // the shared memory and TMEM are released.
    tc_fence_before();
    __syncthreads();
    if (warp == kWarpTma && lane == 0 && issued > 0)
        mbar_drain(stage_full, (issued - 1) & 1, &g_tc_wait_timeouts);
    if (warp == kWarpMma && lane == 0 && committed > 0)
        mbar_drain(bar2(S.acc_full, (committed - 1) & 1), ((committed - 1) >> 1) & 1, &g_tc_wait_timeouts);
    __syncthreads();
    tc_fence_after();
    if (warp == kWarpTma)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(kTmemCols));
    if constexpr (kRedoable<F>) {
        if (S.redo.count > 0 && !S.abort) redo_tiles<F, MODE>(sa, out, m, n, ld, tiles_x, tiles, S);
    }
}

template <class F, bool BATCH, int MODE = kModeGrid, bool ODD = false>
cudaError_t set_smem_attr()
{
    static const cudaError_t err = cudaFuncSetAttribute(
        k2d_tc<F, BATCH, MODE, ODD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(Smem<F>) + 128));
    return err;
}

template <class F, int MODE = kModeGrid, bool ODD = false>
cudaError_t launch_tc(const GridView &g, const typename F::Digits &digits, long long origin, long long elements,
                      const void *in_base, void *out_base, const WaitCfg &wc, cudaStream_t st,
                      const StepArgs<F, MODE> &sa = StepArgs<F, MODE>{})
{
    const long long ld = g.pitch[0];
    CUtensorMap map = {};
    StepArgs<F, MODE> args = sa;
    cudaError_t e = cudaSuccess;
    // The maps copy 8-byte points whatever they hold ((hi, lo) pairs or FP64).
    const float2 *points = reinterpret_cast<const float2 *>(in_base);
    if constexpr (ODD) {
        const long long rows = elements / ld, x = origin % ld - 4, y = origin / ld - 3;
        const int first = (int)(y & 1), late = (int)(ld & 1);  // rows 1, 3, .. of an odd pitch: one point late
        for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
            const int q = k ^ first, shift = q * late;
            const long long start = x + shift;
            args.rows.x[k] = (int)(start - (start & 1));
            args.rows.late[k] = (unsigned)(start & 1);
            args.rows.y[k] = (int)((y + k - q) / 2);
            e = encode_split_window_map(&args.rows.map[k], points + q * ld - shift, 2 * ld, (rows + 1 - q) / 2,
                                        ST_X + 2, ST_Y / 2, ld + shift);
        }
    } else {
        e = encode_split_window_map(&map, points, ld, elements / ld, ST_X, ST_Y);
    }
    if (e != cudaSuccess) return e;
    if ((e = set_smem_attr<F, false, MODE, ODD>()) != cudaSuccess) return e;
    const int tiles_x = (int)((g.ext[1] + TX - 1) / TX);
    const int tiles = tiles_x * (int)((g.ext[0] + TY - 1) / TY);
    // One CTA per SM (its shared-memory footprint admits no second one, so
    // the TMEM allocation never waits).
    const int grid = std::min(tiles, device_sm_count());
    note_launch();
    return launch_programmatic(k2d_tc<F, false, MODE, ODD>, grid, kThreads<F>, sizeof(Smem<F>) + 128, st, map,
                               reinterpret_cast<typename F::Out *>(out_base) + origin, (int)g.ext[0],
                               (int)g.ext[1], ld, tiles_x, tiles, (int)(origin % ld), (int)(origin / ld), digits,
                               wc, static_cast<const TcGrid<F> *>(nullptr), 0, args);
}

template <class F>
cudaError_t fill_record(void *rec, const GridView &g, const Weights &w, long long origin, long long elements,
                        const void *in_base, void *out_base, int tile_begin, int digits_id, int *tiles,
                        typename F::Digits (*slice)(const Weights &))
{
    TcGrid<F> r;
    std::memset(&r, 0, sizeof r);
    const long long ld = g.pitch[0];
    cudaError_t e = encode_split_window_map(&r.map, reinterpret_cast<const float2 *>(in_base), ld, elements / ld,
                                            ST_X, ST_Y);
    if (e != cudaSuccess) return e;
    r.out = reinterpret_cast<typename F::Out *>(out_base) + origin;
    r.ld = ld;
    r.m = (int)g.ext[0];
    r.n = (int)g.ext[1];
    r.tiles_x = (int)((g.ext[1] + TX - 1) / TX);
    r.tile_begin = tile_begin;
    r.map_x = (int)(origin % ld);
    r.map_y = (int)(origin / ld);
    r.digits_id = digits_id;
    r.digits = slice(w);
    *tiles = r.tiles_x * (int)((g.ext[0] + TY - 1) / TY);
    std::memcpy(rec, &r, sizeof r);
    return cudaSuccess;
}

template <class F>
cudaError_t launch_batch(const void *records, int ngrids, int total, const WaitCfg &wc, cudaStream_t st)
{
    cudaError_t e = set_smem_attr<F, true>();
    if (e != cudaSuccess) return e;
    CUtensorMap unused;
    std::memset(&unused, 0, sizeof unused);
    const int grid = std::min(total, device_sm_count());
    note_launch();
    // The records were written before the previous kernel of the stream ran,
    // so the set-up may read them before pdl_wait().
    return launch_programmatic(k2d_tc<F, true>, grid, kThreads<F>, sizeof(Smem<F>) + 128, st, unused,
                               static_cast<typename F::Out *>(nullptr), 0, 0, 0LL, 0, total, 0, 0,
                               typename F::Digits{}, wc, reinterpret_cast<const TcGrid<F> *>(records), ngrids,
                               StepArgs<F, kModeGrid>{});
}

split::SliceWeights split_digits(const Weights &w) { return split::slice_weights(w); }
F64Weights f64_digits(const Weights &w) { return f64_slice_weights(w); }

}  // namespace

cudaError_t launch_split_sweep_tc(const GridView &g, const Weights &w, long long origin,
                                  long long elements, const float2 *in_base, float2 *out_base,
                                  const TcWait &wt, cudaStream_t st)
{
    return launch_tc<FmtSplit>(g, split::slice_weights(w), origin, elements, in_base, out_base,
                               WaitCfg{wt.limit_ns, wt.skip_loads}, st);
}

cudaError_t launch_fp64_sweep_tc(const GridView &g, const Weights &w, long long origin, long long elements,
                                 const double *in_base, double *out_base, const TcWait &wt, cudaStream_t st,
                                 const TcForm *form)
{
    const WaitCfg wc{wt.limit_ns, wt.skip_loads};
    if (!form) return launch_tc<FmtF64>(g, f64_slice_weights(w), origin, elements, in_base, out_base, wc, st);
    const F64Weights digits = f64_slice_weights(w, 49, &tap_order(Taps::kSquare7));
    StepArgs<FmtF64Fine, kModeGrid> sa{};
    sa.in = in_base + origin;
    sa.radius = form->radius;
    sa.above = (int)std::min(form->above, 3LL);
    sa.below = (int)std::min(form->below, 3LL);
    sa.pattern = form->pattern;
    sa.redo = form->redo;
    for (int i = 0; i < 49; ++i) sa.w[i] = w.v[i];
    if (!form->odd) return launch_tc<FmtF64Fine>(g, digits, origin, elements, in_base, out_base, wc, st, sa);
    return launch_tc<FmtF64Fine, kModeGrid, true>(g, digits, origin, elements, in_base, out_base, wc, st, sa);
}

namespace {

inline double step_weight(double w, double) { return w; }
inline float2 step_weight(double w, float2)
{
    const float h = (float)w;
    return make_float2(h, (float)(w - (double)h));
}

template <class F>
cudaError_t launch_steps_2d(const GridView &g, const Weights &wT, const Weights &w3x3, int steps, long long origin,
                            long long elements, const void *in_base, void *out_base, const TcWait &wt, cudaStream_t st,
                            const TcForm &form)
{
    using Out = typename F::Out;
    StepArgs<F, kModeSteps> sa{reinterpret_cast<const Out *>(in_base) + origin, steps, 1, 0, 0u, 0, {}};
    // The frame's strips go to the CTAs that have no tile in the last round,
    // or to all CTAs where that is sooner. A strip keeps one of an SM's four
    // FP64 pipes for about 9,000 cycles; an epilogue warp is idle that long
    // before its first accumulator, and for a tile (6,500 cycles) more in a
    // CTA that has one tile less (star2d1r 1024^2: 256 tiles, 104 CTAs with
    // two and 48 with one, 158 strips).
    const long long m = g.ext[0], n = g.ext[1];
    const int tiles = (int)(((m + TY - 1) / TY) * ((n + TX - 1) / TX)), ctas = std::min(tiles, device_sm_count());
    const long long strips = 2 * ((n + 25) / 26 + (m + 25) / 26), extra = tiles % ctas;
    auto rounds = [&](long long c) { return (strips + 4 * c - 1) / (4 * c); };
    if (extra > 0 && 9000 * rounds(ctas - extra) - 6500 < 9000 * rounds(ctas)) sa.frame_cta = (int)extra;
    for (int t = 0; t < 9; ++t) {
        sa.w[t] = step_weight(w3x3.v[t], Out{});
        if (form.pattern == PAT_DENSE || t / 3 == 1 || t % 3 == 1) sa.taps |= 1u << t;
    }
    sa.pattern = form.pattern;
    sa.redo = form.redo;
    const F64Weights digits = f64_slice_weights(wT, 49, &tap_order(Taps::kSquare7));
    const WaitCfg wc{wt.limit_ns, wt.skip_loads};
    if constexpr (F::kF64)
        if (form.odd) return launch_tc<F, kModeSteps, true>(g, digits, origin, elements, in_base, out_base, wc, st, sa);
    return launch_tc<F, kModeSteps>(g, digits, origin, elements, in_base, out_base, wc, st, sa);
}

template <class F>
cudaError_t launch_steps_1d(long long n, const double *taps, int radius, const double *w, int steps, long long origin,
                            const void *in_base, void *out_base, const TcWait &wt, cudaStream_t st, bool redo)
{
    using Out = typename F::Out;
    if (steps < 1 || steps * radius > kReach1d || n < 64) return cudaErrorInvalidValue;
    cudaError_t e = set_smem_attr<F, false, kMode1d>();
    if (e != cudaSuccess) return e;
    Weights wT;
    for (int i = 0; i < 49; ++i) wT.v[i] = taps[i];
    StepArgs<F, kMode1d> sa{reinterpret_cast<const Out *>(in_base) + origin, steps, radius, 0, 0u, 0, {}};
    sa.aligned = origin % 2 == 0 && reinterpret_cast<uintptr_t>(in_base) % 16 == 0 &&
                 reinterpret_cast<uintptr_t>(out_base) % 16 == 0;
    for (int t = 0; t <= 2 * radius; ++t) sa.w[t] = step_weight(w[t], Out{});
    sa.redo = redo;
    CUtensorMap unused;
    std::memset(&unused, 0, sizeof unused);
    const int tiles = (int)((n + kOut1d - 1) / kOut1d);
    note_launch();
    return launch_programmatic(k2d_tc<F, false, kMode1d>, std::min(tiles, device_sm_count()), kThreads<F>,
                               sizeof(Smem<F>) + 128, st, unused, reinterpret_cast<Out *>(out_base) + origin, 1,
                               (int)n, 0LL, 1, tiles, 0, 0, f64_slice_weights(wT, 49, &tap_order(Taps::kLine49)),
                               WaitCfg{wt.limit_ns, wt.skip_loads}, static_cast<const TcGrid<F> *>(nullptr), 0, sa);
}

}  // namespace

cudaError_t launch_steps_tc(bool fp64, const GridView &g, const Weights &wT, const Weights &w3x3, int steps,
                            long long origin, long long elements, const void *in_base, void *out_base,
                            const TcWait &wt, cudaStream_t st, const TcForm &form)
{
    return fp64 ? launch_steps_2d<FmtF64Fine>(g, wT, w3x3, steps, origin, elements, in_base, out_base, wt, st, form)
                : launch_steps_2d<FmtSplit6>(g, wT, w3x3, steps, origin, elements, in_base, out_base, wt, st, form);
}

cudaError_t launch_steps_tc_1d(bool fp64, long long n, const double *taps, int radius, const double *w, int steps,
                               long long origin, const void *in_base, void *out_base, const TcWait &wt,
                               cudaStream_t st, bool redo)
{
    return fp64 ? launch_steps_1d<FmtF64Fine>(n, taps, radius, w, steps, origin, in_base, out_base, wt, st, redo)
                : launch_steps_1d<FmtSplit6>(n, taps, radius, w, steps, origin, in_base, out_base, wt, st, redo);
}

size_t tc_batch_record_bytes(bool fp64) { return fp64 ? sizeof(TcGrid<FmtF64>) : sizeof(TcGrid<FmtSplit>); }

cudaError_t tc_batch_fill_record(bool fp64, void *rec, const GridView &g, const Weights &w, long long origin,
                                 long long elements, const void *in_base, void *out_base, int tile_begin,
                                 int digits_id, int *tiles)
{
    return fp64 ? fill_record<FmtF64>(rec, g, w, origin, elements, in_base, out_base, tile_begin, digits_id, tiles,
                                      f64_digits)
                : fill_record<FmtSplit>(rec, g, w, origin, elements, in_base, out_base, tile_begin, digits_id,
                                        tiles, split_digits);
}

cudaError_t launch_tc_batch(bool fp64, const void *records, int ngrids, int total_tiles, const TcWait &wt,
                            cudaStream_t st)
{
    const WaitCfg wc{wt.limit_ns, wt.skip_loads};
    return fp64 ? launch_batch<FmtF64>(records, ngrids, total_tiles, wc, st)
                : launch_batch<FmtSplit>(records, ngrids, total_tiles, wc, st);
}

cudaError_t split_tc_wait_timeouts(unsigned *count, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(count, g_tc_wait_timeouts, sizeof(unsigned));
    if (e != cudaSuccess || !reset) return e;
    const unsigned zero = 0;
    return cudaMemcpyToSymbol(g_tc_wait_timeouts, &zero, sizeof(unsigned));
}

}  // namespace cs
