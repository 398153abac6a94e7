// cs_kernels_tc3d_r3.cu — FP64 sweeps of 3D radius-3 kernels (7x7x7 boxes and
// their sparse forms: the fused 3D stencils) on the fifth-generation tensor
// cores. On the FP64 pipe such a sweep costs 343 FMA per point (63 for the
// octahedron); here it costs exact digit products on tcgen05.
//
// Arithmetic: the FP64 digit format of cs_tc_f64.cuh. Each input plane of a
// tile is cut into six balanced 9-bit digits relative to its largest exponent;
// the weights likewise with one scale. One z tap of an output (49 taps of one
// input plane) has level sums below 2^24, exact in FP32 in any order; they
// combine into one 64-bit integer, and the seven z taps are added as integers
// relative to the largest plane exponent among them (the weights' scale keeps
// sum |w| <= 16, so |sum| <= 2^62) and rounded once to FP64. Error: relative to the
// largest value of the output's 3D window times the largest weight, and no
// larger in the norm than that of FP64 FMA sweeps (40 sweeps of 64 x 60 x 66, uniform
// data: box 1.9e-16, FMA 5.1e-16; octahedron 1.5e-16, 2.2e-16). Planes with an Inf or
// NaN are computed again (Redo).
//
// Mapping (M = 128, K = 16):
//   * A work item is a column of output tiles, 16 rows x 64 columns on zc
//     consecutive planes; its zc + 6 input planes (22 rows x 72 columns) are
//     each loaded and cut once. Row m of A is the 16-wide window of column
//     block m % 8 in output row m / 8, read out of the digit plane in place
//     (the descriptors of cs_kernels_split_tc3d.cu); window row offset i
//     (0..6) starts i plane rows lower.
//   * Input plane P feeds outputs P .. P - 6 (counted from the column's first)
//     as their z taps 0 .. 6. The taps go to N in two halves, dz 0..3 and
//     4..6: column n of B_{half,i} is (digit e, dz % 4, column c), n = 32 e
//     (24 e) + 8 (dz % 4) + c, and one MMA with N = 32 (24) x (6 - d) feeds levels
//     d..5, so a half is 7 row offsets x 6 digits = 42 MMAs into 192 (144) TMEM
//     columns. (With the second half padded to 32 a level: 200 x 184 x 192, GB300,
//     185 us a sweep, so 177.) The two halves are the two TMEM blocks: one is drained while the other is
//     being computed. (All seven taps in one N would need 384 columns, one
//     block of the 512, and a wait for the epilogue after every plane.)
//   * Bound: the MMA stream and the shared memory it reads. An MMA reads 4 KB
//     of A and N x 32 bytes of B, 60 cycles on average at 128 bytes a cycle;
//     issued from registers the compiler knows to be uniform (elect_one, the
//     TMEM base a constant) the 84 MMAs of a plane (1024 outputs) take 5,500
//     cycles, of 6,100 per plane (issued under lane == 0: 7,260 of 8,350).
//   * Roles (27 warps, seven per scheduler, one idle, 72 registers): one loads
//     windows (four stages), one thread issues the MMAs, two groups of four
//     cut every second plane (ring of four digit-plane sets), sixteen drain
//     the blocks and keep the seven running sums of two columns each. No
//     slicer shares the MMA thread's scheduler. (Eight draining four columns:
//     7,000 cycles a plane, mostly waiting for their own TMEM loads, longer
//     than the MMAs.) GB300, box 256^3: 545 us a sweep with lane == 0 and
//     eight, 466 with elect_one, 398 with sixteen, 391 with the second half's
//     24 columns a level: 43 G outputs/s; the FP64 FMA kernel 1.5 (box), 8.3
//     (octahedron).
//   * Windows arrive by TMA where the layout allows it (even pitches,
//     16-byte aligned base, the halo in whole rows and planes); the window then starts 4 columns left of the
//     tile, or 3 where the interior's first column is odd, so that its
//     address is a multiple of 16 bytes. Other layouts (odd pitches among them) are
//     loaded by the same warp with 8-byte cp.async (its 50 copies a lane and
//     plane hide behind the MMAs: 200 x 184 x 193 runs at the rate of its tiles).
//
// Every mbarrier wait is bounded (WaitCfg, 2 s by default); an expired wait is
// counted beside those of the radius-1 kernels (one counter, so that the
// synchronous runs read no further one) and the CTA leaves as in those.
#include "cs_internal.h"
#include "cs_split_common.cuh"
#include "cs_tc_common.cuh"
#include "cs_tc_f64.cuh"

#include <algorithm>

namespace cs {

namespace {

using split::kDigitBits;
using namespace tc;

constexpr int D = 6, TAPS = 343;

struct Weights7 {
    __half d[D][TAPS];
    int ew;
    float rest;  // what the digits' sum lacks (f64_combine)
    int pattern, redo;
    double w[TAPS];  // the weights themselves (Redo)
};

constexpr int kGroups = 2, kGroupWarps = 4, kGroupThreads = 32 * kGroupWarps;
constexpr int kEpiWarps = 16;
constexpr int kWarpTma = 1, kWarpMma = 5;
constexpr unsigned kEpiMask = 0x0000DDDDu | (1u << 9) | (1u << 13) | (1u << 17) | (1u << 21);
constexpr unsigned kSliceMask = (1u << 16) | (1u << 18) | (1u << 19) | (1u << 20) | (1u << 22) | (1u << 23) |
                                (1u << 24) | (1u << 26);
constexpr int kWarps = 27, kThreads = 32 * kWarps;  // warp 25 idle
static_assert(__builtin_popcount(kSliceMask) == kGroups * kGroupWarps && __builtin_popcount(kEpiMask) == kEpiWarps &&
                  (kSliceMask & kEpiMask) == 0 &&
                  ((kSliceMask | kEpiMask) & ((1u << kWarpTma) | (1u << kWarpMma))) == 0 &&
                  (kSliceMask & 0x22222222u) == 0,
              "warp roles overlap, or a slicer shares the MMA thread's scheduler");
constexpr int kSliceBarrier = 1;             // named barriers 1 .. kGroups

constexpr int TX = 64, TY = 16;              // output tile
constexpr int ST_X = TX + 8, ST_Y = TY + 6;  // window: 72 columns, rows y0-3 .. y0+18
constexpr int PL = ST_X * ST_Y;              // halves per digit plane
constexpr unsigned kRowBytes = ST_X * 2;     // 144
constexpr int NOFF = 7, NCOL = 32 * D;       // rows of B: 192, and 144 of the second half
// TMEM columns per level: four tap planes x 8, three in the second half; and N
// of an MMA that feeds `levels` levels (M = 128 wants multiples of 16; the 8
// columns of an odd count lie behind the block's last level and are not read).
__host__ __device__ constexpr int nlv(int half) { return half ? 24 : 32; }
__host__ __device__ constexpr int mma_n(int half, int levels) { return (nlv(half) * levels + 15) / 16 * 16; }
constexpr int kBlkStride = 256, kTmemCols = 512;
constexpr int kStages = 4, NPL = 4;
constexpr int kScaleRing = 32;               // planes in flight stay below it
constexpr unsigned kStageBytes = PL * 8;     // 12,672
constexpr int NPAIR = PL / 2, PAIRS = ST_X / 2;                    // 792, 36
constexpr int PER = (NPAIR + kGroupThreads - 1) / kGroupThreads;  // 7
constexpr int kWz = 24;                      // halves per staged weight row: taps at 8 .. 14
static_assert(kStageBytes % 128 == 0, "TMA destinations stay 128-byte aligned");

struct Smem {
    uint4 stage[kStages][NPAIR];
    __half planes[NPL][D][PL];               // digit planes; first the staged weight rows
    __half bmat[2][NOFF][NCOL * 16];         // B_{half,i}, K-major 8x16-byte core matrices
    unsigned long long stage_full[kStages], stage_empty[kStages];
    unsigned long long planes_full[NPL], planes_empty[NPL];
    unsigned long long blk_full[2], blk_empty[2];
    unsigned tmem;
    int abort;
    int scale_exp[kScaleRing];
    int redi[kGroups][2][kGroupWarps];
    Redo redo;                               // input planes that hold an Inf or NaN
};
static_assert(sizeof(Smem) + 128 <= 232448, "shared memory of one CTA must stay within 227 KB");
static_assert(D * 49 * kWz * 2 <= (int)sizeof(Smem::planes), "the staged weights fit the digit planes");

template <int HZ, int I, int DG>
__device__ __forceinline__ void half_mma(unsigned d_base, unsigned long long a, unsigned long long b0)
{
    constexpr unsigned long long a_off = ((unsigned long long)DG * PL * 2 + I * kRowBytes) >> 4;
    constexpr unsigned long long b_off = ((unsigned long long)(HZ * NOFF + I) * NCOL * 16 * 2) >> 4;
    static_assert(((unsigned long long)DG * PL * 2 + I * kRowBytes) % 16 == 0, "descriptor offsets");
    mma_f16(d_base + (unsigned)(nlv(HZ) * DG), a + a_off, b0 + b_off, instr_desc(mma_n(HZ, D - DG)),
            (I | DG) != 0 ? 1u : 0u);
    if constexpr (DG + 1 < D)
        half_mma<HZ, I, DG + 1>(d_base, a, b0);
    else if constexpr (I + 1 < NOFF)
        half_mma<HZ, I + 1, 0>(d_base, a, b0);
}

struct Item {
    int x0, y0, zs, zn;
};

__device__ __forceinline__ Item item_of(int item, int tiles_x, int tiles_y, int zc, int h)
{
    const int txy = tiles_x * tiles_y;
    const int chunk = item / txy, rem = item - chunk * txy;
    const int ty = rem / tiles_x;
    return Item{(rem - ty * tiles_x) * TX, ty * TY, chunk * zc, min(zc, h - chunk * zc)};
}

__device__ __forceinline__ void tmem_ld2(unsigned taddr, float (&v)[2])
{
    unsigned r[2];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 2; ++j) v[j] = __uint_as_float(r[j]);
}

// x 2^-k, k >= 0 (the low bits lie far below the result's last one).
__device__ __forceinline__ long long shift_down(long long x, int k) { return x >> min(k, 63); }

template <bool TMA>
__global__ void __launch_bounds__(kThreads, 1)
    k3d_tc_r3(const __grid_constant__ CUtensorMap tmap, const double *__restrict__ in, double *__restrict__ out, int h,
              int m, int n, long long ldy, long long ldz, int tiles_x, int tiles_y, int zc, int items, int map_x,
              int map_y, int map_z, int left, int vec2, const __grid_constant__ Weights7 sw, WaitCfg wc,
              unsigned *timeouts)
{
    extern __shared__ unsigned char smem_raw[];
    Smem &S = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_allow_dependents();
    volatile int *abort = &S.abort;
    auto bar = [](unsigned long long *b, int i) { return smem_addr(&b[i]); };
    const unsigned long long limit = wc.limit_ns;
    auto wait = [abort, limit, timeouts](unsigned b, unsigned parity) {
        return mbar_wait(b, parity, abort, timeouts, limit);
    };
    const int first = blockIdx.x, step = gridDim.x;

    int issued = 0, committed = 0;  // window loads issued / planes committed
    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(bar(S.stage_full, i), TMA ? 1 : 32);
            mbar_init(bar(S.stage_empty, i), kGroupWarps);
        }
        for (int i = 0; i < NPL; ++i) {
            mbar_init(bar(S.planes_full, i), kGroupWarps);
            mbar_init(bar(S.planes_empty, i), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar(S.blk_full, i), 1);
            mbar_init(bar(S.blk_empty, i), kEpiWarps);
        }
        S.abort = 0;
        S.redo.count = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarpTma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&S.tmem)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // B_{half,i}: N row nn = 32 e (24 e) + 8 dzl + c, K index k, tap column tj = k - c
    // - (left - 3). The weight rows are staged first, padded with zeros (row
    // (e, dz, ti) by one warp: uniform parameter reads), then written in
    // 16-byte chunks of eight k, consecutive halves of a staged row.
    __half *wz = &S.planes[0][0][0];
    for (int row = warp; row < D * 49; row += kWarps) {
        const int e = row / 49, t0 = (row - 49 * e) * 7;
        __half v = __float2half(0.f);
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            const __half x = sw.d[e][t0 + j];
            if (lane == 8 + j) v = x;
        }
        if (lane < kWz) wz[row * kWz + lane] = v;
    }
    __syncthreads();
    for (int idx = tid; idx < 2 * NOFF * NCOL * 2; idx += kThreads) {
        const int hi = idx / (NCOL * 2), rem = idx - hi * (NCOL * 2);
        const int hz = hi / NOFF, i = hi - hz * NOFF;
        const int nn = rem >> 1, kh = rem & 1;
        const int e = nn / nlv(hz), dz = 4 * hz + ((nn % nlv(hz)) >> 3), c = nn & 7;
        __align__(16) __half v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = e < D ? wz[(e * 49 + dz * 7 + i) * kWz + 8 * kh + 11 - left - c + k] : __float2half(0.f);
        *reinterpret_cast<uint4 *>(&S.bmat[hz][i][(nn >> 3) * 128 + (nn & 7) * 8 + kh * 64]) =
            *reinterpret_cast<const uint4 *>(v);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // All 512 columns are this CTA's, so they start at column 0: as a constant
    // it costs the MMA thread no move into a uniform register per MMA.
    const unsigned tmem = 0;

    if (warp == kWarpTma) {
        // ------------------------------------------------ window loads
        if (!wc.skip_loads && (!TMA || lane == 0)) {
            pdl_wait();  // the previous sweep has finished with both buffers
            int q = 0;   // input-plane sequence number
            bool ok = true;
            for (int item = first; item < items && ok; item += step) {
                const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
                for (int p = 0; p < wi.zn + 6; ++p, ++q) {
                    const int sb = q % kStages;
                    ok = lane != 0 || wait(bar(S.stage_empty, sb), ((q / kStages) & 1) ^ 1);
                    if constexpr (!TMA) ok = __shfl_sync(0xffffffffu, ok, 0);
                    if (!ok) break;
                    if constexpr (TMA) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        mbar_expect_tx(bar(S.stage_full, sb), kStageBytes);
                        tma_load_3d(smem_addr(S.stage[sb]), &tmap, map_x + wi.x0 - left, map_y + wi.y0 - 3,
                                    map_z + wi.zs - 3 + p, bar(S.stage_full, sb));
                    } else {
                        __syncwarp();
                        const double *src = in + (long long)(wi.zs - 3 + p) * ldz + (long long)(wi.y0 - 3) * ldy +
                                            wi.x0 - left;
                        const unsigned dst = smem_addr(S.stage[sb]);
                        for (int row = 0; row < ST_Y; ++row, src += ldy) {
                            const bool rok = wi.y0 - 3 + row <= m + 2;
#pragma unroll
                            for (int b = 0; b < 3; ++b) {
                                const int col = lane + 32 * b, x = wi.x0 - left + col;
                                if (b == 2 && col >= ST_X) continue;
                                const bool take = rok && x >= -3 && x <= n + 2;
                                cp_async8(dst + 8u * (row * ST_X + col), take ? src + col : in, take);
                            }
                        }
                        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar(S.stage_full, sb))
                                     : "memory");
                    }
                    issued = q + 1;
                }
            }
        }
    } else if (warp == kWarpMma) {
        // ------------------------------------------------ MMA issuer
        const unsigned long long a_desc0 = smem_desc(smem_addr(S.planes[0][0]), 16, kRowBytes);
        constexpr unsigned long long kSetUnits = (unsigned long long)D * PL * 2 / 16;
        const unsigned long long b_desc0 = smem_desc(smem_addr(S.bmat[0][0]), 128, 256);
        int q = 0;
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            for (int p = 0; p < wi.zn + 6; ++p, ++q) {
                const int slot = q % NPL;
                const unsigned long long a = a_desc0 + kSetUnits * slot;
                if (!(ok = __all_sync(0xffffffffu, wait(bar(S.planes_full, slot), (q / NPL) & 1) &&
                                                       wait(bar(S.blk_empty, 0), (q & 1) ^ 1))))
                    break;
                tc_fence_after();
                if (elect_one()) {
                    half_mma<0, 0, 0>(tmem, a, b_desc0);
                    mma_commit(bar(S.blk_full, 0));
                }
                committed = 2 * q + 1;
                if (!(ok = __all_sync(0xffffffffu, wait(bar(S.blk_empty, 1), (q & 1) ^ 1)))) break;
                tc_fence_after();
                if (elect_one()) {
                    half_mma<1, 0, 0>(tmem + kBlkStride, a, b_desc0);
                    mma_commit(bar(S.blk_full, 1));
                    mma_commit(bar(S.planes_empty, slot));  // digit planes may be overwritten
                }
                committed = 2 * q + 2;
            }
        }
    } else if ((kSliceMask >> warp) & 1u) {
        // ------------------------------------------------ slicers
        const int sidx = __popc(kSliceMask & ((1u << warp) - 1u));
        const int grp = sidx / kGroupWarps, gw = sidx % kGroupWarps;
        const int st = 32 * gw + lane;
        const bool leader = st == 0;
        int q = 0;
        bool go = true;
        for (int item = first; item < items && go; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            // Points past the halo of three meet zero weights or outputs that
            // are not kept, but must not set the plane's scale either.
            const bool edge = TMA && (wi.x0 == 0 || wi.x0 - left + ST_X > n + 3 || wi.y0 - 3 + ST_Y > m + 3);
            for (int p = 0; p < wi.zn + 6; ++p, ++q) {
                if (q % kGroups != grp) continue;
                const int sb = q % kStages, slot = q % NPL;
                // (a) window landed? Every thread waits for itself; one barrier
                // per plane, at (c), makes the group agree to go on.
                const bool landed = wait(bar(S.stage_full, sb), (q / kStages) & 1);
                const int set = (q / kGroups) & 1;
                // (b) window -> registers, then release the stage to the next load.
                const uint4 *stg = S.stage[sb];
                uint4 v[PER];
                unsigned emax = 0;  // largest biased exponent
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int u = st + k * kGroupThreads;
                    v[k] = make_uint4(0u, 0u, 0u, 0u);
                    if (u < NPAIR) {
                        v[k] = stg[u];
                        if (edge) {
                            const int yy = wi.y0 - 3 + u / PAIRS, xx = wi.x0 - left + 2 * (u % PAIRS);
                            const bool row = yy <= m + 2;
                            if (!row || xx < -3 || xx > n + 2) v[k].x = v[k].y = 0u;
                            if (!row || xx + 1 < -3 || xx + 1 > n + 2) v[k].z = v[k].w = 0u;
                        }
                        emax = max(emax, max(v[k].y & 0x7FFFFFFFu, v[k].w & 0x7FFFFFFFu));
                    }
                }
                emax = __reduce_max_sync(0xffffffffu, emax) >> 20;
                __syncwarp();
                if (lane == 0) {
                    S.redi[grp][set][gw] = (int)emax;
                    mbar_arrive(bar(S.stage_empty, sb));
                }
                // (c) digit-plane set free (the MMAs that read it are done)?
                // The barrier also publishes the maxima; the group's next
                // plane's are in the other set.
                const bool free = landed && wait(bar(S.planes_empty, slot), ((q / NPL) & 1) ^ 1);
                go = !bar_any(kSliceBarrier + grp, kGroupThreads, !free);
                if (!go) break;
                int ex = 1;
#pragma unroll
                for (int i = 0; i < kGroupWarps; ++i) ex = max(ex, S.redi[grp][set][i]);
                if (leader) {
                    S.scale_exp[q % kScaleRing] = ex == 2047 ? kNonFiniteTile : ex;
                    if (ex == 2047 && sw.redo) S.redo.add(q);
                }
                unsigned *dst0 = reinterpret_cast<unsigned *>(&S.planes[slot][0][0]);
                if (ex >= kFastExp) {
#pragma unroll
                    for (int k = 0; k < PER; ++k) {
                        const int u = st + k * kGroupThreads;
                        if (u < NPAIR) f64_cut_fast<true, PL / 2>(v[k], ex, dst0 + u);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < PER; ++k) {
                        const int u = st + k * kGroupThreads;
                        if (u < NPAIR) f64_cut_any<true, PL / 2>(v[k], ex, dst0 + u);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(S.planes_full, slot));
            }
        }
    } else if ((kEpiMask >> warp) & 1u) {
        // ------------------------------------------------ epilogue
        // Warp w reads TMEM lanes 32 (w % 4) ..; lane -> D row m = (output row
        // er, block eb); of the four warps of a lane quarter hh = 0 .. 3 takes
        // columns 8 eb + 2 hh, + 1. s[dz] is the running sum of the output
        // whose z tap dz the current input plane is, in units of its largest
        // plane exponent so far, se[dz] (the same in every thread).
        const int quarter = warp & 3, hh = quarter == 1 ? (warp - 9) >> 2 : warp >> 2;
        const int mrow = 32 * quarter + lane;
        const int er = mrow >> 3, eb = mrow & 7;
        const unsigned taddr = tmem + ((unsigned)(32 * quarter) << 16) + 2u * hh;
        int q = 0;
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            const int xb = wi.x0 + 8 * eb + 2 * hh, yy = wi.y0 + er;
            double *op = out + (long long)(wi.zs - 6) * ldz + (long long)yy * ldy + xb;
            long long s[7][2];
            int se[7];
#pragma unroll
            for (int dz = 0; dz < 7; ++dz) {
                se[dz] = 1;
#pragma unroll
                for (int c = 0; c < 2; ++c) s[dz][c] = 0;
            }
            unsigned bad = 0;  // bit k: the plane k back holds an Inf or NaN
            for (int p = 0; p < wi.zn + 6; ++p, ++q, op += ldz) {
                int ex = 1;
#pragma unroll
                for (int hz = 0; hz < 2; ++hz) {
                    if (!(ok = wait(bar(S.blk_full, hz), q & 1))) break;
                    tc_fence_after();
                    if (hz == 0) {
                        ex = S.scale_exp[q % kScaleRing];
                        bad = bad << 1 | (ex == kNonFiniteTile ? 1u : 0u);
                        if (ex == kNonFiniteTile) ex = 1;
                    }
#pragma unroll
                    for (int dl = 0; dl < (hz ? 3 : 4); ++dl) {
                        const int dz = 4 * hz + dl;
                        float acc[D][2];
#pragma unroll
                        for (int L = 0; L < D; ++L) tmem_ld2(taddr + kBlkStride * hz + nlv(hz) * L + 8 * dl, acc[L]);
                        tmem_wait_ld();
                        if (dl == (hz ? 2 : 3)) {  // block drained: hand it back
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar(S.blk_empty, hz));
                        }
                        long long t[2];
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float lv[6] = {acc[0][c], acc[1][c], acc[2][c], acc[3][c], acc[4][c], acc[5][c]};
                            t[c] = f64_combine(lv, sw.rest);
                        }
                        if (dz == 0) {
                            se[0] = ex;
#pragma unroll
                            for (int c = 0; c < 2; ++c) s[0][c] = t[c];
                        } else {
                            if (ex != se[dz]) {
                                const int up = max(ex - se[dz], 0), down = max(se[dz] - ex, 0);
#pragma unroll
                                for (int c = 0; c < 2; ++c) {
                                    s[dz][c] = shift_down(s[dz][c], up);
                                    t[c] = shift_down(t[c], down);
                                }
                                se[dz] += up;
                            }
#pragma unroll
                            for (int c = 0; c < 2; ++c) s[dz][c] += t[c];
                        }
                    }
                }
                if (!ok) break;
                if (p >= 6 && yy < m) {  // output p - 6 of the column has all its taps
                    double res[2];
                    const int sc = se[6] + sw.ew - 1080;
                    if (!(bad & 0x7Fu) && f64_scale_is_plain(sc)) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) res[c] = f64_from_fixed_plain(s[6][c], sc);
                    } else {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            res[c] = (bad & 0x7Fu) ? __longlong_as_double(0x7FF8000000000000ll)
                                                   : f64_from_fixed(s[6][c], sc);
                    }
                    if (vec2 && xb + 1 < n) {
                        *reinterpret_cast<double2 *>(op) = make_double2(res[0], res[1]);
                    } else {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
                            if (xb + c < n) op[c] = res[c];
                    }
                }
#pragma unroll
                for (int dz = 6; dz > 0; --dz) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) s[dz][c] = s[dz - 1][c];
                    se[dz] = se[dz - 1];
                }
            }
        }
    }

    // Exit: every role is done or has given up. Let the loads and MMAs still
    // in flight finish before shared memory and TMEM are released.
    tc_fence_before();
    __syncthreads();
    if (warp == kWarpTma && lane == 0)
        for (int l = max(0, issued - kStages); l < issued; ++l)
            mbar_drain(bar(S.stage_full, l % kStages), (l / kStages) & 1, timeouts);
    if (warp == kWarpMma && lane == 0 && committed > 0)
        mbar_drain(bar(S.blk_full, (committed - 1) & 1), ((committed - 1) / 2) & 1, timeouts);
    __syncthreads();
    tc_fence_after();
    if (warp == kWarpTma)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(S.tmem), "r"(kTmemCols));
    if (S.redo.count > 0 && !S.abort) {  // output planes j with an Inf or NaN in their seven input planes
        int q = 0;
        for (int item = first; item < items; item += step) {
            const Item wi = item_of(item, tiles_x, tiles_y, zc, h);
            for (int j = 0; j < wi.zn; ++j) {
                if (!S.redo.holds(q + j, q + j + 6)) continue;
                for (int i = tid; i < TX * TY; i += kThreads) {
                    const int y = wi.y0 + i / TX, x = wi.x0 + i % TX;
                    const long long at = (long long)(wi.zs + j) * ldz + (long long)y * ldy + x;
                    if (y < m && x < n) out[at] = fma_sum_3d<3>(in + at, ldy, ldz, sw.w, sw.pattern);
                }
            }
            q += wi.zn + 6;
        }
    }
}

// Digits of the 343 weights: as f64_slice_weights with the sum and the moments
// kept, and a scale that also holds sum |w| / 2^ew to 16. (The sum alone kept, each
// error carried on to the next tap, and level 5 cut off at T's unit: 40 sweeps of
// the octahedron, smooth data, erred by 3.2e-16 of the norm, FP64 FMA by 2.3e-16.)
Weights7 slice_weights7(const Weights &w, const TcForm &form)
{
    Weights7 s{};
    s.pattern = form.pattern;
    s.redo = form.redo;
    for (int i = 0; i < TAPS; ++i) s.w[i] = w.v[i];
    double mx = 0.0, sum = 0.0;
    for (int i = 0; i < TAPS; ++i) mx = std::fmax(mx, std::fabs(w.v[i]));
    int e = 0;
    if (mx > 0.0) {
        std::frexp(mx, &e);
        e += 2;  // |w| / 2^ew < 1/4
        for (int i = 0; i < TAPS; ++i) sum += std::ldexp(std::fabs(w.v[i]), -e);
        for (; sum > 16.0; sum *= 0.5) ++e;
    }
    s.ew = e;
    const TapOrder &at = tap_order(Taps::kCube7);
    KeepSums kept;
    sum = 0.0;
    double size = 0.0;
    for (int j = 0; j < TAPS; ++j) {
        const int i = at.tap[j];
        const double t = std::ldexp(w.v[i], kDigitBits - e);
        if (t == 0.0) continue;
        sum += t;
        size += std::fabs(t);
        double a = std::ldexp(kept.round(std::ldexp(t, 45), at.x[j], at.y[j], at.z[j]), -45);
        for (int k = 0; k < D; ++k) {
            const double d = std::rint(a);
            s.d[k][i] = __float2half_rn((float)d);
            a = (a - d) * 512.0;
        }
    }
    s.rest = rest_of(kept, sum, size);
    return s;
}

}  // namespace

cudaError_t launch_fp64_sweep_tc3d_r3(const GridView &g, const Weights &w, long long origin, long long elements,
                                      const double *in_base, double *out_base, bool rows_whole, const TcForm &form,
                                      const TcWait &wt, cudaStream_t st)
{
    const long long ldy = g.pitch[1], ldz = g.pitch[0];
    const bool tma = rows_whole && ldy % 2 == 0 && ldz % ldy == 0 && reinterpret_cast<uintptr_t>(in_base) % 16 == 0;
    const int map_x = (int)(origin % ldy);
    const int left = tma && map_x % 2 != 0 ? 3 : 4;  // the window's address stays a multiple of 16 bytes
    const bool vec2 = ldy % 2 == 0 && ldz % 2 == 0 && origin % 2 == 0 && reinterpret_cast<uintptr_t>(out_base) % 16 == 0;
    CUtensorMap map = {};
    if (tma) {
        const cudaError_t e = encode_split_window_map_3d(&map, reinterpret_cast<const float2 *>(in_base), ldy, ldz,
                                                         elements / ldz, ST_X, ST_Y);
        if (e != cudaSuccess) return e;
    }
    unsigned *timeouts = nullptr;
    const cudaError_t ce = tc3d_wait_counter(&timeouts);
    if (ce != cudaSuccess) return ce;
    const size_t smem = sizeof(Smem) + 128;
    auto kernel = tma ? k3d_tc_r3<true> : k3d_tc_r3<false>;
    static const cudaError_t attr[2] = {
        cudaFuncSetAttribute(k3d_tc_r3<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
        cudaFuncSetAttribute(k3d_tc_r3<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)};
    if (attr[0] != cudaSuccess || attr[1] != cudaSuccess) return attr[0] != cudaSuccess ? attr[0] : attr[1];
    const int h = (int)g.ext[0], m = (int)g.ext[1], n = (int)g.ext[2];
    const int tiles_x = (n + TX - 1) / TX, tiles_y = (m + TY - 1) / TY;
    // Planes per work item: a column of zc output planes takes zc + 6 input
    // planes' work, and the busiest CTA ceil(items / SMs) items.
    const int sms = device_sm_count();
    const long long txy = (long long)tiles_x * tiles_y;
    int zc = 1;
    long long best = -1;
    for (int c = 1; c <= std::min(64, h); ++c) {
        const long long it = txy * ((h + c - 1) / c), cost = ((it + sms - 1) / sms) * (c + 6);
        if (best < 0 || cost < best) best = cost, zc = c;
    }
    const int items = (int)(txy * ((h + zc - 1) / zc));
    note_launch();
    return launch_programmatic(kernel, std::min(items, sms), kThreads, smem, st, map, in_base + origin,
                               out_base + origin, h, m, n, ldy, ldz, tiles_x, tiles_y, zc, items, map_x,
                               (int)((origin % ldz) / ldy), (int)(origin / ldz), left, vec2 ? 1 : 0, slice_weights7(w, form),
                               WaitCfg{wt.limit_ns, wt.skip_loads}, timeouts);
}

}  // namespace cs
