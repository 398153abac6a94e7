// cs_tc_f64.cuh — the FP64 number format of the tcgen05 digit kernels
// (cs_kernels_split_tc.cu for 2D, cs_kernels_split_tc3d.cu for 3D): weights
// and inputs cut into six balanced 9-bit digits held exactly in FP16 (the
// inputs with integer operations only), and the exact integer recombination
// of the level sums with one rounding to FP64.
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "cs_internal.h"
#include "cs_split_common.cuh"

namespace cs {
namespace tc {

// Six balanced base-512 digits of w / 2^ew (|w| / 2^ew < 1/4, so the top
// digit stays within 128) for the 49 taps of a 7x7 kernel, or for the first
// `taps` (27: a 3x3x3 kernel).
struct F64Weights {
    __half d[6][49];
    int ew;
    float rest;  // see keep_sum
};

// The taps of a line of 49, of a 7x7, a 3x3x3 or a 7x7x7, farthest first.
struct TapOrder {
    std::vector<int> tap;
    std::vector<double> x, y, z;  // where it lies
};
enum class Taps { kLine49, kSquare7, kCube3, kCube7 };
inline const TapOrder &tap_order(Taps t)
{
    auto make = [](int nx, int ny, int nz) {
        TapOrder o;
        auto px = [=](int i) { return i % nx - nx / 2; };
        auto py = [=](int i) { return i / nx % ny - ny / 2; };
        auto pz = [=](int i) { return i / (nx * ny) - nz / 2; };
        auto far = [&](int i) { return px(i) * px(i) + py(i) * py(i) + pz(i) * pz(i); };
        for (int i = 0; i < nx * ny * nz; ++i) o.tap.push_back(i);
        std::stable_sort(o.tap.begin(), o.tap.end(), [&](int a, int b) { return far(a) > far(b); });
        for (int i : o.tap) o.x.push_back(px(i)), o.y.push_back(py(i)), o.z.push_back(pz(i));
        return o;
    };
    static const TapOrder orders[4] = {make(49, 1, 1), make(7, 7, 1), make(3, 3, 3), make(7, 7, 7)};
    return orders[(int)t];
}

// Rounds weights to integers (units of their last digit) so that their sum and
// first moments keep their values. An error of the sum scales a smooth grid by
// the same factor in every sweep, one of the moments moves it, where the errors
// of single weights average out; so each weight, from the farthest in, goes up
// or down as the sums of the errors so far want it. (To the nearest, each error
// carried on to the next tap, the moment along a row of a 7x7 was off by 3.8
// units; so all three by 0.4 to 0.5.)
struct KeepSums {
    double r0 = 0.0, rx = 0.0, ry = 0.0, rz = 0.0;  // errors so far
    double round(double v, double x, double y, double z)
    {
        const double below = std::floor(v), d = below - v, u = d + 1.0;
        auto miss = [&](double q) {
            return (r0 + q) * (r0 + q) + (rx + q * x) * (rx + q * x) + (ry + q * y) * (ry + q * y) +
                   (rz + q * z) * (rz + q * z);
        };
        const bool down = d == 0.0 || miss(d) <= miss(u);
        const double q = down ? d : u;
        r0 += q, rx += q * x, ry += q * y, rz += q * z;
        return down ? below : below + 1.0;
    }
};

// What is left of a sum, as a factor of the level-0 sum: r0 is in units of 2^-45,
// the number it goes to in units of 2^-42 of level 0's.
inline float rest_of(const KeepSums &k, double sum, double size)
{
    return std::fabs(sum) > size * 0x1p-6 ? (float)(-k.r0 * 0.125 / sum) : 0.0f;
}

// keep: where the taps lie whose sum and first moments keep their values
// (KeepSums; six digits hold a weight to 2^-45 of the top digit's unit), or null.
// What is then left of the sum goes to the recombination as `rest`, the factor
// of the level-0 sum that makes up for it there (f64_combine; 0 where the
// weights cancel). 100 steps of star2d1r 1024^2, uniform data: error of the norm
// 5.7e-16 with six levels, 1.3e-16 with seven and carried errors, 1.06e-16 so.
inline F64Weights f64_slice_weights(const Weights &w, int taps = 49, const TapOrder *keep = nullptr)
{
    F64Weights s{};
    double mx = 0.0;
    for (int i = 0; i < taps; ++i) mx = std::fmax(mx, std::fabs(w.v[i]));
    int e = 0;
    if (mx > 0.0) {
        std::frexp(mx, &e);  // mx < 2^e
        e += 2;              // |w| / 2^ew < 1/4
    }
    s.ew = e;
    KeepSums kept;
    double sum = 0.0, size = 0.0;
    for (int k = 0; k < taps; ++k) {
        const int i = keep ? keep->tap[k] : k;
        double a = std::ldexp(w.v[i], split::kDigitBits - e);  // |a| < 128, exact
        sum += a;
        size += std::fabs(a);
        if (keep && a != 0.0)
            a = std::ldexp(kept.round(std::ldexp(a, 45), keep->x[k], keep->y[k], keep->z[k]), -45);
        for (int t = 0; t < 6; ++t) {
            const double d = std::rint(a);
            s.d[t][i] = __float2half_rn((float)d);
            a = (a - d) * 512.0;  // exact: a - d is a multiple of a's last bit
        }
    }
    s.rest = keep ? rest_of(kept, sum, size) : 0.0f;
    return s;
}

// ---- FP64 digits and recombination (integer operations only)

// 256 in each of six 9-bit fields: Y = X + kF64Bias has fields u in [0, 511]
// (top field up to 384) with X = sum (u_k - 256) 512^(5-k).
constexpr unsigned long long kF64Bias = 256ull * ((1ull << 54) - 1) / 511;

// Biased-digit word of one FP64 value (bits lo, hi) of a tile whose largest
// biased exponent is eb1 (at least 1): X = round(x / 2^(eb1 - 1074)), so
// |X| <= 2^52, returned as 2 (X + kF64Bias), whose lowest bit says nothing. The
// shift is clamped at 63: any mantissa (< 2^53) shifted by 55 or more rounds to
// 0 as it should.
// EVEN rounds ties to even. They are frequent: half of the values of the largest
// exponent (which lose one bit), a quarter of those of the next, 2^-(sh + 1) of
// those sh below. Half up adds a quarter unit to every value of the largest
// exponent on average, an eighth to the next, the same way each sweep (30
// steps of a 9-point average of uniform data, 520 x 512, against quad
// precision: 3.7e-15 half up and one step per launch), and costs less.
// f64_ties_down: takes one unit off a mantissa (lo its lower word) whose last
// bit kept, number sh + 1, is clear: ties then round down, which is to even, and
// nothing else changes. (Of the lower word only: bits of the upper one are
// reached from sh = 31, where a value in 2^32 is a tie. To even at sh = 0 alone,
// 100 steps of star2d1r 1024^2 erred by 1.2e-15, so by 5.7e-16; GB300, box2d1r
// 2047 x 1531 x 60 515 us a solve and 517, 1d2r 10,240,000 x 100 560 and 563.)
__device__ __forceinline__ unsigned f64_ties_down(unsigned lo, int sh)
{
    unsigned last;
    asm("shl.b32 %0, %1, %2;" : "=r"(last) : "r"(2u), "r"(sh));  // 0 from 31 on
    return (lo & last) == 0u && lo != 0u ? lo - 1u : lo;
}
template <bool EVEN = false>
__device__ __forceinline__ unsigned long long f64_biased_fixed(unsigned lo, unsigned hi, int eb1)
{
    const int e = (int)((hi >> 20) & 0x7FFu);
    const int ee = max(e, 1);  // subnormals: no implicit bit, exponent 1
    const int sh = min(eb1 - ee, 63);
    if (EVEN) lo = f64_ties_down(lo, sh);
    const unsigned long long mant =
        ((unsigned long long)((hi & 0xFFFFFu) | (e ? 0x100000u : 0u)) << 32) | lo;
    const unsigned long long x = ((mant >> sh) + 1) >> 1;
    const unsigned long long neg = (unsigned long long)(long long)((int)hi >> 31);  // 0 or all ones
    return ((kF64Bias - neg) + (x ^ neg)) << 1;  // kF64Bias + x, or kF64Bias - x = (kF64Bias + 1) + ~x
}

// The same for tiles whose largest biased exponent is at least kFastExp (all
// but tiles of values below 2^-895): a zero or subnormal then shifts out
// whether or not it is given the implicit bit, so neither needs a test, and
// PTX defines a shift by more than 63 (C++ does not). Half up in magnitude with
// the sign applied first: with t = floor(m / 2^sh), the arithmetic shift of ~m
// is -t - 1 whether or not bits were lost, and (-t - 1 + 1) >> 1 = -((t + 1) >> 1).
// (Four of 15 integer operations less per point than with the sign
// at the end; GB300, us a launch:
// star3d1r 512^3 933 and 897, box2d1r 8192^2 in threes 358 and 353.)
constexpr int kFastExp = 128;
template <bool EVEN = false>
__device__ __forceinline__ unsigned long long f64_biased_fixed_fast(unsigned lo, unsigned hi, int eb1)
{
    const int sh = eb1 - (int)((hi >> 20) & 0x7FFu);
    if (EVEN) lo = f64_ties_down(lo, sh);
    const unsigned neg = (unsigned)((int)hi >> 31);
    const unsigned long long m = ((unsigned long long)(((hi & 0xFFFFFu) | 0x100000u) ^ neg) << 32) | (lo ^ neg);
    unsigned long long t;
    asm("shr.s64 %0, %1, %2;" : "=l"(t) : "l"(m), "r"(sh));
    return t + (2 * kF64Bias + 1);
}

// Digit k (0 = most significant) of two biased words, as an FP16 pair:
// FP16 (1024 + u) has the bits 0x6400 | u, and (1024 + u) - 1280 = u - 256
// is exact in FP16. (The top field is at most 384, so masking it is harmless.)
template <int K>
__device__ __forceinline__ unsigned f64_digit_pair(unsigned long long ya, unsigned long long yb)
{
    constexpr int sh = split::kDigitBits * (5 - K) + 1;
    const unsigned ta = (unsigned)(ya >> sh);
    const unsigned tb = sh >= 16 ? (unsigned)(yb >> (sh - 16)) : (unsigned)(yb << (16 - sh));
    const unsigned w = ((ta & 0x1FFu) | (tb & 0x1FF0000u)) | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&w), __halves2half2(__ushort_as_half(0x6500),
                                                                                     __ushort_as_half(0x6500)));
    return *reinterpret_cast<const unsigned *>(&h);
}

// T = sum over levels of S_L 2^(42 - 9L), level 5 without its last three
// bits: |T| < 2^63. Multiply-adds on the FMA pipe (the integer ALU pipe is
// this kernel's busiest).
__device__ __forceinline__ long long f64_combine(const float (&lv)[6])
{
    long long t = (long long)(__float2int_rn(lv[5]) >> 3);
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[4])), "r"(1 << 6));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[3])), "r"(1 << 15));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[2])), "r"(1 << 24));
    unsigned tl, th;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(tl), "=r"(th) : "l"(t));
    // levels 0 and 1 sit wholly in the upper word: S1 2^33 + S0 2^42
    th += (unsigned)(__float2int_rn(lv[1]) * 2 + __float2int_rn(lv[0]) * 1024);
    asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "r"(tl), "r"(th));
    return t;
}

// The same with what the weights' sum lacks (F64Weights::rest), of six levels or
// seven: the last ones come in as one number, rounded to T's unit (2^-42 of level
// 0's, below 2^-52 of T itself but for sums that cancel).
template <int LV>
__device__ __forceinline__ long long f64_combine(const float (&lv)[LV], float rest)
{
    static_assert(LV == 6 || LV == 7);
    float last = lv[0] * rest;
    if constexpr (LV == 7) last = fmaf(lv[6], 0x1p-12f, last);
    long long t = __float2int_rn(fmaf(lv[5], 0.125f, last));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[4])), "r"(1 << 6));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[3])), "r"(1 << 15));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(__float2int_rn(lv[2])), "r"(1 << 24));
    unsigned tl, th;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(tl), "=r"(th) : "l"(t));
    th += (unsigned)(__float2int_rn(lv[1]) * 2 + __float2int_rn(lv[0]) * 1024);
    asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "r"(tl), "r"(th));
    return t;
}

// f64_combine for two outputs whose level sums are below 2^22 in magnitude
// (one z tap of a 3D input plane: 9 taps, so level L sums at most 9 * 5 * 2^16 <
// 2^22), added to their running 64-bit sums: an FP32 addition of 1.5 * 2^23
// (exact in that range: the sum lands in [2^23, 2^24), where the spacing is 1)
// leaves kRaw + S in the bits of S's float, and the multiply-adds take those
// bits as they are. Every call therefore adds kRawBias too (modulo 2^64; kRaw is
// a multiple of 8, so level 5's shift leaves it whole), which the caller takes
// off once per sum. (GB300, star3d1r 512^3: 1128 us a sweep with the bias taken
// off every level, 1112 so.)
constexpr unsigned kRaw = 0x4B400000u;
// LOW: level 5's bits below T's unit (none of seven levels' sum, below).
template <int LOW = 3>
constexpr unsigned long long kRawBias = (kRaw >> LOW) +
                                        (unsigned long long)kRaw * ((1u << 6) + (1u << 15) + (1u << 24)) +
                                        ((unsigned long long)(kRaw * 1026u) << 32);
template <int LOW = 3>
__device__ __forceinline__ void f64_add_raw2(const float (&u)[6], const float (&v)[6], long long &su, long long &sv)
{
    int a[6], b[6];
#pragma unroll
    for (int L = 0; L < 6; ++L) {
        unsigned long long x;
        asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(u[L]), "f"(v[L]));
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(0x4B4000004B400000ull));
        asm("mov.b64 {%0, %1}, %2;" : "=r"(a[L]), "=r"(b[L]) : "l"(x));
    }
    auto sum = [](const int (&r)[6], long long &t) {
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(r[5] >> LOW), "r"(1));
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(r[4]), "r"(1 << 6));
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(r[3]), "r"(1 << 15));
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(t) : "r"(r[2]), "r"(1 << 24));
        unsigned tl, th;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(tl), "=r"(th) : "l"(t));
        th += (unsigned)r[1] * 2u + (unsigned)r[0] * 1024u;
        asm("mov.b64 %0, {%1, %2};" : "=l"(t) : "r"(tl), "r"(th));
    };
    sum(a, su);
    sum(b, sv);
}
// The same of seven levels: level 5, level 6 and what the weights' sum lacks
// (F64Weights::rest) come in as one number, rounded to T's unit: cut off there, as
// above, every part loses half a unit, the same way each sweep (star3d1r 160 x 128 x
// 125, 100 sweeps: 9.5e-16 of the norm so). A call adds kRawBias<0>.
__device__ __forceinline__ void f64_add_raw2(const float (&u)[7], const float (&v)[7], float rest, long long &su,
                                             long long &sv)
{
    const float p[6] = {u[0], u[1], u[2], u[3], u[4], fmaf(u[5], 0.125f, fmaf(u[6], 0x1p-12f, u[0] * rest))};
    const float q[6] = {v[0], v[1], v[2], v[3], v[4], fmaf(v[5], 0.125f, fmaf(v[6], 0x1p-12f, v[0] * rest))};
    f64_add_raw2<0>(p, q, su, sv);
}

// Results outside the normal FP64 range (subnormal or overflowing): FP64
// arithmetic, kept out of line so that the common path carries no FP64
// instruction (the compiler cannot if-convert a call).
static __device__ __noinline__ double f64_from_fixed_rare(long long t, int c)
{
    return scalbn((double)t, c);
}

// FP64 value of T * 2^c, rounded to nearest even: the 64-bit integer is
// converted once (cvt.rn.f64.s64, exact rounding) and the power of two is
// added to the exponent field; results outside the normal range take the
// out-of-line FP64 route.
__device__ __forceinline__ double f64_from_fixed(long long t, int c)
{
    const double d = __ll2double_rn(t);
    const long long bits = __double_as_longlong(d);
    const int e = (int)((bits >> 52) & 0x7FF);
    const int ne = e + c;
    if (e == 0) return d;  // t == 0
    if (ne >= 1 && ne <= 2046) return __longlong_as_double(bits + ((long long)c << 52));
    return f64_from_fixed_rare(t, c);
}

// Whether every T != 0 times 2^c is a normal number (|T| < 2^63), and then its
// value: no range tests per output.
__device__ __forceinline__ bool f64_scale_is_plain(int c) { return c >= -1022 && c <= 960; }
// f64_bits_of converts where it is written, f64_scaled does the rest.
__device__ __forceinline__ long long f64_bits_of(long long t)
{
    double d;
    asm volatile("cvt.rn.f64.s64 %0, %1;" : "=d"(d) : "l"(t));
    return __double_as_longlong(d);
}
__device__ __forceinline__ double f64_scaled(long long bits, int c)
{
    const int hi = (int)(bits >> 32);
    return __hiloint2double(hi != 0 ? hi + (c << 20) : 0, (int)bits);
}
__device__ __forceinline__ double f64_from_fixed_plain(long long t, int c)
{
    return f64_scaled(__double_as_longlong(__ll2double_rn(t)), c);
}

// Cuts one pair of points (v: lo, hi words of both) into six digit planes
// PW words apart.
template <int PW>
__device__ __forceinline__ void f64_cut_pair(unsigned long long ya, unsigned long long yb, unsigned *dst)
{
    dst[0 * PW] = f64_digit_pair<0>(ya, yb);
    dst[1 * PW] = f64_digit_pair<1>(ya, yb);
    dst[2 * PW] = f64_digit_pair<2>(ya, yb);
    dst[3 * PW] = f64_digit_pair<3>(ya, yb);
    dst[4 * PW] = f64_digit_pair<4>(ya, yb);
    dst[5 * PW] = f64_digit_pair<5>(ya, yb);
}
template <bool EVEN, int PW>
__device__ __forceinline__ void f64_cut_fast(const uint4 &v, int ex, unsigned *dst)
{
    f64_cut_pair<PW>(f64_biased_fixed_fast<EVEN>(v.x, v.y, ex), f64_biased_fixed_fast<EVEN>(v.z, v.w, ex), dst);
}
// Tiles of tiny values. (Inline although rare: as a call it made the compiler
// keep the cutting loop's values where a call leaves them; the 3D radius-3
// sweep took 586 us on 256^3, GB300, against 539 so.)
template <bool EVEN, int PW>
__device__ __forceinline__ void f64_cut_any(const uint4 &v, int ex, unsigned *dst)
{
    f64_cut_pair<PW>(f64_biased_fixed<EVEN>(v.x, v.y, ex), f64_biased_fixed<EVEN>(v.z, v.w, ex), dst);
}

// Marks a tile whose window holds an Inf or NaN (its outputs become NaN).
constexpr int kNonFiniteTile = -100000;

}  // namespace tc
}  // namespace cs
