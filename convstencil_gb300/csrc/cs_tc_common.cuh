// cs_tc_common.cuh — building blocks shared by the tcgen05 split kernels
// (cs_kernels_split_tc.cu for 2D, cs_kernels_split_tc3d.cu for 3D): bounded
// mbarrier waits, shared-memory matrix and instruction descriptors for
// kind::f16 MMAs with TMEM accumulators, TMEM loads and TMA tile loads.
//
// Every wait is bounded by WaitCfg::limit_ns of %globaltimer (2 s unless the
// plan sets another limit). An expired wait adds one to the caller's device
// counter and raises the CTA's abort flag, so every role of the CTA stops at
// its next wait; mbar_drain is the bounded wait used at exit for copies and
// MMAs still in flight. The host reads the counter after synchronous runs and
// reports CS_ERR_TIMEOUT.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <utility>

namespace cs {
namespace tc {

constexpr unsigned long long kWaitNs = 2000000000ull;  // default bound of one wait

// Per-launch wait settings (kernel parameter).
struct WaitCfg {
    unsigned long long limit_ns;  // bound of every mbarrier wait
    int skip_loads;               // test hook: the producer issues no TMA loads, so the
                                  // consumers' first wait runs out and the CTA leaves
};

// Programmatic dependent launch. A sweep launched with the programmatic
// stream serialization attribute may be scheduled while the previous kernel
// of its stream is still finishing: it sets up (barriers, TMEM, B matrices)
// at once and calls pdl_wait(), which returns once the previous grid has
// completed and its writes are visible, before its first global-memory
// access (the first window load; every store comes after loads). Launched
// without the attribute, pdl_wait() returns at once. pdl_allow_dependents()
// lets the next such kernel be scheduled as this one's CTAs leave.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_allow_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches a sweep kernel, with the programmatic stream serialization
// attribute (see pdl_wait) where `overlap` is set.
template <typename... Exp, typename... Act>
cudaError_t launch_overlapped(bool overlap, void (*kernel)(Exp...), dim3 grid, int block, size_t smem,
                              cudaStream_t st, Act &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}
template <typename... Exp, typename... Act>
cudaError_t launch_programmatic(void (*kernel)(Exp...), int grid, int block, size_t smem, cudaStream_t st,
                                Act &&...args)
{
    return launch_overlapped(true, kernel, dim3((unsigned)grid), block, smem, st, std::forward<Act>(args)...);
}

__device__ __forceinline__ unsigned smem_addr(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A waiting warp sleeps up to 2 us at a time: with the default limit the waits
// of the slicers and the producer take more of the others' issue slots and
// shared-memory cycles (GB300, us a launch: box2d3r 8192^2 327 and 319, split
// box3d1r 512^3 732 and 724).
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// The polling loop of mbar_wait, out of line: it is entered only when the
// phase is not complete at the first test.
static __device__ __noinline__ bool mbar_wait_slow(unsigned bar, unsigned parity, volatile int *abort,
                                                   unsigned *timeouts, unsigned long long limit_ns)
{
    const unsigned long long t0 = globaltimer();
    for (;;) {
        for (int i = 0; i < 16; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
        if (globaltimer() - t0 > limit_ns) {
            atomicAdd(timeouts, 1u);
            *abort = 1;
            return false;
        }
    }
}

// Waits for the phase with the given parity. Gives up after limit_ns
// (counted in *timeouts, and *abort raised so every other role stops too) or
// as soon as another role has raised *abort. The first test is inline: a call
// costs the issuing role several hundred cycles under load (measured on the
// 3D kernel's MMA thread), and most waits find their phase complete.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int *abort, unsigned *timeouts,
                                          unsigned long long limit_ns = kWaitNs)
{
    return mbar_try_wait(bar, parity) || mbar_wait_slow(bar, parity, abort, timeouts, limit_ns);
}

// Bounded wait used only at exit for copies / MMAs still in flight.
static __device__ __noinline__ bool mbar_drain(unsigned bar, unsigned parity, unsigned *timeouts,
                                               unsigned long long limit_ns = kWaitNs)
{
    const unsigned long long t0 = globaltimer();
    while (!mbar_try_wait(bar, parity))
        if (globaltimer() - t0 > limit_ns) {
            atomicAdd(timeouts, 1u);
            return false;
        }
    return true;
}

__device__ __forceinline__ void mbar_arrive(unsigned bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Named barrier of `threads` threads that also tells all of them whether any
// came with `fail` set: a role whose threads wait on mbarriers one by one
// decides with it, the same way in all of them, whether to go on.
__device__ __forceinline__ bool bar_any(int id, int threads, bool fail)
{
    unsigned any;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %3, 0;\n"
        " barrier.cta.red.or.pred.aligned q, %1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(any)
        : "r"(id), "r"(threads), "r"((unsigned)fail)
        : "memory");
    return any != 0;
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, no swizzle; lbo = byte stride of
// the 16-byte K chunks, sbo = byte stride of the 8-row groups.
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo)
{
    return (unsigned long long)((addr & 0x3FFFFu) >> 4) | ((unsigned long long)(lbo >> 4) << 16) |
           ((unsigned long long)(sbo >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP16 A and B, FP32 D, both K-major, M = 128.
__host__ __device__ constexpr unsigned instr_desc(int n)
{
    return (1u << 4) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}

// One thread of a converged warp, the same one every time. The MMA warp walks
// its loop as a whole and issues under this: under lane == 0 the compiler must
// move every descriptor of every MMA from a thread's registers to the uniform
// ones the instruction takes, and the issuing thread, not the tensor core, set
// the pace (GB300, cycles per MMA beside the other roles, before and after:
// 3D radius 1 106 and 80, radius 3 86 and 65; split box3d1r 512^3 930 and 750
// us a sweep, box2d3r 8192^2 FP64 337 and 327).
__device__ __forceinline__ bool elect_one()
{
    unsigned leader;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(leader));
    return leader != 0;
}

__device__ __forceinline__ void mma_f16(unsigned d_tmem, unsigned long long a, unsigned long long b,
                                        unsigned idesc, unsigned accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(unsigned bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ldc(unsigned taddr, float (&v)[4])
{
    unsigned r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void tmem_ldc(unsigned taddr, float (&v)[8])
{
    unsigned r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap *map, int x, int y, unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// The larger, or NaN where one is.
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Work of a CTA (tiles, or input planes, numbered in its order) whose window
// held an Inf or a NaN. Digits cannot hold one, so the outputs are computed
// again after the rest, with the plan's own weights one by one as the kernels
// without digits do: a point that is not finite then reaches the outputs that
// read it and no other. Lies in shared memory; work is added by the slicers'
// leaders, who look at its scale. (Cost on finite grids, GB300, us a solve:
// star2d1r 1024^2 x 100 481.6 and 486.7, box2d1r 2047 x 1531 x 60 525 and 529, 1d2r
// 10,240,000 x 100 562.5 and 563.7, fused box3d1r none; noted by the epilogue
// instead 485, 536, 574.)
struct NoRedo {
};
struct Redo {
    static constexpr int kMost = 64;
    int count, item[kMost];
    __device__ __forceinline__ void add(int i)
    {
        const int k = atomicAdd(&count, 1);
        if (k < kMost) item[k] = i;
    }
    // Whether one of lo .. hi is in it (more than it holds: any may be).
    __device__ __forceinline__ bool holds(int lo, int hi) const
    {
        if (count > kMost) return true;
        for (int k = 0; k < count; ++k)
            if (item[k] >= lo && item[k] <= hi) return true;
        return false;
    }
};

// Whether a tap at these offsets belongs to a kernel's pattern of radius r.
__device__ __forceinline__ bool in_pattern(int pattern, int dz, int dy, int dx, int r)
{
    return pattern == PAT_DENSE  ? true
           : pattern == PAT_STAR ? (dz != 0) + (dy != 0) + (dx != 0) <= 1
                                 : abs(dz) + abs(dy) + abs(dx) <= r;
}

// FP64 FMA sum of a (2r+1)^3 kernel's pattern at one point of a grid.
template <int R>
__device__ __forceinline__ double fma_sum_3d(const double *__restrict__ at, long long ldy, long long ldz,
                                             const double *w, int pattern)
{
    constexpr int K = 2 * R + 1;
    double v = 0.0;
    for (int t = 0; t < K * K * K; ++t) {
        const int dz = t / (K * K) - R, dy = t / K % K - R, dx = t % K - R;
        if (in_pattern(pattern, dz, dy, dx, R)) v = fma(w[t], at[dz * ldz + dy * ldy + dx], v);
    }
    return v;
}

// Untiled bulk copy: 16-byte aligned addresses, a multiple of 16 bytes.
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Four 8-byte points to a 32-byte boundary.
template <class T>
__device__ __forceinline__ void store_32(T *dst, const T *v)
{
    static_assert(sizeof(T) == 8);
    unsigned long long w[4];
    memcpy(w, v, sizeof w);
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(dst), "l"(w[0]), "l"(w[1]), "l"(w[2]), "l"(w[3])
                 : "memory");
}

// 8 bytes from global to shared memory, or zeros.
__device__ __forceinline__ void cp_async8(unsigned dst, const void *src, bool take)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(take ? 8 : 0) : "memory");
}

__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap *map, int x, int y, int z,
                                            unsigned bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

}  // namespace tc
}  // namespace cs
