// common.cuh - device helpers shared by every kernel file of libglm53f_b200 (sm_100a only).
//
// Number formats follow the reference engine (josesilva05/glm-5.3-flash-in-c):
//   E4M3FN decode  src/core/glm53f_ops.c:51-72   (bias 7, subnormals, s.1111.111 = NaN, no inf)
//   BF16 widen     include/glm53f/glm53f.h:150-155 (a 16-bit left shift)
//   sigmoid        src/core/glm53f_ops.c:46       (1.0f / (1.0f + expf(-x)), three float roundings)
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace g5b {

constexpr int DT_F32 = 0, DT_BF16 = 1, DT_FP8 = 2;
constexpr int WARP = 32;

// Host-side count of kernels launched by this library (reported by the benchmark).
extern unsigned long long g_launches;

#define G5B_LAUNCH(kernel, grid, block, smem, stream, ...)                     \
    do {                                                                       \
        kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);            \
        ++::g5b::g_launches;                                                   \
    } while (0)

// The same launch with programmatic stream serialization: the grid may be scheduled while the
// kernel before it in the stream is still draining (once all of that kernel's CTAs have passed
// pdl_trigger() or exited), so its launch latency and whatever it does before pdl_wait() overlap
// that kernel's tail. Only for kernels that call pdl_wait() before they read anything an earlier
// kernel wrote. (A kernel launched the ordinary way may call both: they do nothing then.)
#define G5B_LAUNCH_PDL(kernel, grid, block, smem, strm_, ...)                                      \
    do {                                                                                        \
        cudaLaunchConfig_t cfg_{};                                                              \
        cfg_.gridDim = (grid); cfg_.blockDim = (block);                                         \
        cfg_.dynamicSmemBytes = (smem); cfg_.stream = (strm_);                                  \
        cudaLaunchAttribute at_[1];                                                             \
        at_[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;                         \
        at_[0].val.programmaticStreamSerializationAllowed = 1;                                  \
        cfg_.attrs = at_; cfg_.numAttrs = 1;                                                    \
        if (cudaLaunchKernelEx(&cfg_, kernel, __VA_ARGS__) != cudaSuccess) {                    \
            cudaGetLastError();                                                                 \
            kernel<<<(grid), (block), (smem), (strm_)>>>(__VA_ARGS__);                          \
        }                                                                                       \
        ++::g5b::g_launches;                                                                    \
    } while (0)

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 16-byte streaming load: weights are read once per token, so they bypass L1 allocation and
// leave it to the activations that every row re-reads.
__device__ __forceinline__ uint4 ld_stream16(const void *p)
{
    uint4 v;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p));
    return v;
}

// Four E4M3 codes (one 32-bit word, lowest byte first) to four floats, exactly: the hardware
// conversion to f16 is exact for every E4M3 value (f16 holds 2^-9 as a normal number) and
// f16 -> f32 is exact; NaN codes stay NaN.
__device__ __forceinline__ void e4m3x4_to_f32(uint32_t w, float &a, float &b, float &c, float &d)
{
    uint32_t lo, hi;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(lo) : "h"((unsigned short)(w & 0xffffu)));
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(hi) : "h"((unsigned short)(w >> 16)));
    const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&lo));
    const float2 f1 = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
    a = f0.x; b = f0.y; c = f1.x; d = f1.y;
}

__device__ __forceinline__ float e4m3_to_f32(uint8_t code)
{
    float a, b, c, d;
    e4m3x4_to_f32((uint32_t)code, a, b, c, d);
    return a;
}

__device__ __forceinline__ float bf16_to_f32(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }
__device__ __forceinline__ void bf16x2_to_f32(uint32_t w, float &lo, float &hi)
{
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xffff0000u);
}

// expf as the host C library computes it: the double-precision exp rounded once to float agrees
// with a correctly rounded expf except on rare double-rounding cases.
__device__ __forceinline__ float expf_host(float x) { return (float)exp((double)x); }

// The reference's sigmoid: 1.0f / (1.0f + expf(-x)), each step rounded to float, never fused.
__device__ __forceinline__ float sigmoid_host(float x)
{
    return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf_host(-x)));
}

// v 2^k for the exponential of x: k is the low part of t's bits (t = k + 1.5 2^23); in two steps, so that a subnormal result is rounded once
__device__ __forceinline__ float exp_scaled(float v, float t, float x)
{
    const int k = __float_as_int(t) - 0x4b400000, k0 = k >> 1;
    v = v * __int_as_float((k0 + 127) << 23) * __int_as_float((k - k0 + 127) << 23);
    return x > 89.0f ? INFINITY : x < -104.0f ? 0.0f : v;
}

// exp(x) to 0.53 units in the last place (the double-precision route above: 0.5), in thirty FP32
// instructions: Cody and Waite's reduction x = n ln 2 + r with ln 2 cut after 14 bits (n times that is exact),
// Taylor's series of e^r to r^9 with its terms up to r^2 / 2 as pairs of floats, one rounding at the end. For
// places that take millions: FP64 instructions issue at half of the FP32 rate here, conversions to and from doubles at an eighth, and an
// exponential is about thirty instructions of either. Equal to the correctly rounded result for 99.75 % of the arguments when they are spread evenly over
// -87 .. 88, for 99.98 % when they are spread evenly over the floats there (the test of both is a sweep of either kind);
// subnormal results are off by less than one of their units.
__device__ __forceinline__ float expf_near(float x)
{
    const float t = fmaf(x, 1.44269504f, 0x1.8p23f), n = __fsub_rn(t, 0x1.8p23f);      // rounded to an integer, which also lies in t's low bits
    const float rh = fmaf(n, -0.693115234375f, x);
    const float sh = fmaf(n, -3.19461849453e-05f, rh), sl = fmaf(n, -3.19461849453e-05f, __fsub_rn(rh, sh));
    float q = fmaf(sh, 1.0f / 362880.0f, 1.0f / 40320.0f);
    q = fmaf(sh, q, 1.0f / 5040.0f);
    q = fmaf(sh, q, 1.0f / 720.0f);
    q = fmaf(sh, q, 1.0f / 120.0f);
    q = fmaf(sh, q, 1.0f / 24.0f);
    q = fmaf(sh, q, 1.0f / 6.0f);
    const float sq = __fmul_rn(sh, sh), sqe = fmaf(sh, sh, -sq), h = 0.5f * sq;
    const float c = fmaf(__fmul_rn(sq, sh), q, fmaf(0.5f, sqe, fmaf(sh, sl, sl)));
    const float a = __fadd_rn(h, c), ae = __fadd_rn(__fsub_rn(h, a), c);
    const float b = __fadd_rn(sh, a), be = __fadd_rn(__fsub_rn(sh, b), a);
    const float d = __fadd_rn(1.0f, b), de = __fadd_rn(__fsub_rn(1.0f, d), b);
    return exp_scaled(__fadd_rn(d, __fadd_rn(de, __fadd_rn(be, ae))), t, x);
}

// 1 / d rounded to nearest, d from 1 on: the estimate and one step of Newton's, whose residual is exact in a fused product, without the
// branch that a division has for its special cases - a dozen of them in a row waited for each other. Equal to the division for every
// mantissa (the test goes through all 2^23); 0 for an infinite d, NaN for NaN; from 2^126 on (subnormal results) off by less than one of their units.
// (Taken of d / 2^26, so that neither the argument nor the estimate leaves the range of normal numbers.)
__device__ __forceinline__ float rcp_estimate(float d)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
}
__device__ __forceinline__ float recip_from_one(float d)
{
    const float ds = d * 0x1p-26f, r = rcp_estimate(ds);
    return d == INFINITY ? 0.0f : fmaf(r, fmaf(-ds, r, 1.0f), r) * 0x1p-26f;
}

// The sigmoid of the function above, with this exponential: three roundings, 1.53 units of 2^-23 at most relative to the exact
// value (0.53 of the exponential, a half each of the sum and the quotient).
__device__ __forceinline__ float sigmoid_near(float x) { return recip_from_one(__fadd_rn(1.0f, expf_near(-x))); }

// Two floats side by side: one instruction for both (rounded like two of the scalar ones).
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float x, float y) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y)); return r; }
__device__ __forceinline__ void f2_get(F2 a, float &x, float &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, f2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float f2_sum(F2 a) { float x, y; f2_get(a, x, y); return __fadd_rn(x, y); }

// expf_near of two arguments, step by step the same operations: equal to it bit for bit.
__device__ __forceinline__ void expf_near2(float x0, float x1, float &e0, float &e1)
{
    auto both = [](float v) { return f2(v, v); };
    const F2 x = f2(x0, x1), t = f2_fma(x, both(1.44269504f), both(0x1.8p23f)), n = f2_add(t, both(-0x1.8p23f));
    const F2 c2 = both(-3.19461849453e-05f), rh = f2_fma(n, both(-0.693115234375f), x);
    const F2 sh = f2_fma(n, c2, rh), sl = f2_fma(n, c2, f2_sub(rh, sh));
    F2 q = f2_fma(sh, both(1.0f / 362880.0f), both(1.0f / 40320.0f));
    q = f2_fma(sh, q, both(1.0f / 5040.0f));
    q = f2_fma(sh, q, both(1.0f / 720.0f));
    q = f2_fma(sh, q, both(1.0f / 120.0f));
    q = f2_fma(sh, q, both(1.0f / 24.0f));
    q = f2_fma(sh, q, both(1.0f / 6.0f));
    const F2 nsh = f2_mul(sh, both(-1.0f)), nsq = f2_mul(sh, nsh), sqe = f2_fma(sh, sh, nsq), h = f2_mul(both(-0.5f), nsq);
    const F2 c = f2_fma(f2_mul(nsq, nsh), q, f2_fma(both(0.5f), sqe, f2_fma(sh, sl, sl)));
    const F2 a = f2_add(h, c), ae = f2_add(f2_sub(h, a), c);
    const F2 b = f2_add(sh, a), be = f2_add(f2_sub(sh, b), a);
    const F2 d = f2_add(both(1.0f), b), de = f2_add(f2_sub(both(1.0f), d), b);
    float v0, v1, t0, t1;
    f2_get(f2_add(d, f2_add(de, f2_add(be, ae))), v0, v1);
    f2_get(t, t0, t1);
    e0 = exp_scaled(v0, t0, x0); e1 = exp_scaled(v1, t1, x1);
}
__device__ __forceinline__ void sigmoid_near2(float x0, float x1, float &s0, float &s1)
{
    float d0, d1;
    expf_near2(-x0, -x1, s0, s1);
    const F2 d = f2_add(f2(s0, s1), f2(1.0f, 1.0f)), nds = f2_mul(d, f2(-0x1p-26f, -0x1p-26f));
    f2_get(d, d0, d1);
    f2_get(nds, s0, s1);
    const F2 r = f2(rcp_estimate(-s0), rcp_estimate(-s1));
    f2_get(f2_mul(f2_fma(r, f2_fma(nds, r, f2(1.0f, 1.0f)), r), f2(0x1p-26f, 0x1p-26f)), s0, s1);
    if (d0 == INFINITY) s0 = 0.0f;
    if (d1 == INFINITY) s1 = 0.0f;
}

// a*b + c with two float roundings, as C compiled without FMA contraction evaluates it.
__device__ __forceinline__ float mul_add_unfused(float a, float b, float c)
{
    return __fadd_rn(__fmul_rn(a, b), c);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over a whole CTA (blockDim.x a multiple of 32, at most 1024). `red` holds 32 doubles of
// shared memory. Every thread receives the total; the order of the sum is fixed.
__device__ __forceinline__ double block_sum(double v, double *red)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < nw; i++) t += red[i];
    return t;
}

// 1 / sqrt(x) to a few units of FP64: the single-precision estimate and two Newton steps (the exact sequence of square root
// and division is a chain of forty FP64 instructions, 0.7 us; what takes this rounds it to float).
__device__ __forceinline__ double rsqrt_newton(double x)
{
    if (!(x > 1e-30 && x < 1e38)) return 1.0 / sqrt(x);              // outside the estimate's range
    double r = (double)rsqrtf((float)x);
    r = fma(r, fma(-0.5 * x * r, r, 0.5), r);
    return fma(r, fma(-0.5 * x * r, r, 0.5), r);
}

// 16 bytes from global to shared memory, without a register on the way; both addresses 16-byte aligned
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- thread-block clusters
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_cta_rank()
{
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the shared variable `p` of CTA `rank` of this cluster
__device__ __forceinline__ double ld_cluster_f64(const double *p, uint32_t rank)
{
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t theirs;
    double v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(theirs) : "r"(mine), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(theirs) : "memory");
    return v;
}

// System-scope acquire / release on 64-bit words that another GPU writes or reads.
__device__ __forceinline__ unsigned long long ld_acquire_sys(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_sys(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}


// One more on a 64-bit counter another GPU waits on, with release semantics at system scope.
__device__ __forceinline__ void red_release_sys_add(unsigned long long *p, unsigned long long v)
{
    asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait until the 64-bit word another GPU publishes reaches `want`. The limit is wall-clock time
// (the ranks are separate host processes: ordinary host skew must not look like a lost peer), with
// an iteration cap behind it in case the timer does not advance. False when the wait ran out.
__device__ __forceinline__ bool wait_word_sys(const unsigned long long *p, unsigned long long want,
                                              unsigned long long limit_ns)
{
    if (ld_acquire_sys(p) >= want) return true;
    const unsigned long long t0 = global_ns();
    for (long long i = 0; i < (1ll << 28); i++) {
        if (ld_acquire_sys(p) >= want) return true;
        if (global_ns() - t0 > limit_ns) return false;
        __nanosleep(100);
    }
    return false;
}

}  // namespace g5b
