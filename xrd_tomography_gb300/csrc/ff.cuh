// ff.cuh -- double-float arithmetic: a value as an unevaluated sum hi + lo of
// two floats (about 48 significant bits).
//
// GB300 runs FP64 at 1/64 of its FP32 rate (1.24 vs 78 TFLOP/s measured), so
// the quantities that need more than FP32 -- 1 - cos(theta) and sin(theta/2)
// for small scattering angles, where the Gaussian q resolution amplifies
// relative error several hundredfold -- are carried as float pairs.  The
// algorithms are the classical error-free transformations: Knuth's TwoSum,
// Dekker's FastTwoSum, TwoProduct through a fused multiply-add, and one
// Newton correction of the SFU's reciprocal and reciprocal root.  Only additions and
// explicit fmaf appear where the error terms are formed, so FMA contraction
// cannot change them.
#pragma once

#include <cuda_runtime.h>

namespace xrdt {

struct ff {
    float hi, lo;
};

__host__ __device__ inline ff ff_from_double(double d)
{
    const float h = (float)d;
    return {h, (float)(d - (double)h)};
}

__device__ __forceinline__ ff fast_two_sum(float a, float b)
{
    const float s = a + b;
    return {s, b - (s - a)};
}

__device__ __forceinline__ ff two_sum(float a, float b)
{
    const float s = a + b;
    const float bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}

__device__ __forceinline__ ff ff_add(ff a, ff b)
{
    ff s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ ff ff_neg(ff a) { return {-a.hi, -a.lo}; }

__device__ __forceinline__ ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }

// exact float minus a pair
__device__ __forceinline__ ff ff_fsub(float a, ff b)
{
    ff s = two_sum(a, -b.hi);
    s.lo -= b.lo;
    return fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ ff ff_mul(ff a, ff b)
{
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ ff ff_mulf(ff a, float b)
{
    const float p = a.hi * b;
    float e = fmaf(a.hi, b, -p);
    e = fmaf(a.lo, b, e);
    return fast_two_sum(p, e);
}

// ---- loose pairs ----
// The same operations without the last FastTwoSum: the low part may reach a
// few ulps of the high one.  Every function here takes such pairs (their
// errors stay near 2^-44); ff_tight restores the bound where the high part is
// used as the value rounded to float.
__device__ __forceinline__ ff ff_tight(ff a) { return fast_two_sum(a.hi, a.lo); }

__device__ __forceinline__ ff ffl_add(ff a, ff b)
{
    const ff s = two_sum(a.hi, b.hi);
    return {s.hi, s.lo + (a.lo + b.lo)};
}

__device__ __forceinline__ ff ffl_sub(ff a, ff b) { return ffl_add(a, ff_neg(b)); }

__device__ __forceinline__ ff ffl_mul(ff a, ff b)
{
    const float p = __fmul_rn(a.hi, b.hi);
    return {p, fmaf(a.lo, b.hi, fmaf(a.hi, b.lo, fmaf(a.hi, b.hi, -p)))};
}

// a1 b1 + a2 b2
__device__ __forceinline__ ff ffl_dot2(ff a1, ff b1, ff a2, ff b2)
{
    const ff p = ffl_mul(a1, b1), q = ffl_mul(a2, b2);
    const ff s = two_sum(p.hi, q.hi);
    return {s.hi, s.lo + (p.lo + q.lo)};
}

// a1 b1 + a2 b2 + a3 b3
__device__ __forceinline__ ff ffl_dot3(ff a1, ff b1, ff a2, ff b2, ff a3, ff b3)
{
    const ff p = ffl_mul(a1, b1), q = ffl_mul(a2, b2), r = ffl_mul(a3, b3);
    const ff s = two_sum(p.hi, q.hi), t = two_sum(s.hi, r.hi);
    return {t.hi, (s.lo + t.lo) + ((p.lo + q.lo) + r.lo)};
}

// 1 / a: the SFU's reciprocal and one correction, about 2^-45 relative.  From
// correctly rounded float quotients and roots the pairs would be no better for
// several times the instructions.
__device__ __forceinline__ ff ffl_rcp(ff a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a.hi));
    return {r, r * fmaf(-a.lo, r, fmaf(-a.hi, r, 1.f))};
}

// sqrt(a), a > 0, from the SFU's reciprocal root with one correction
__device__ __forceinline__ ff ffl_sqrt(ff a)
{
    float rs;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(a.hi));
    const float x = __fmul_rn(a.hi, rs);
    return {x, 0.5f * (fmaf(-x, x, a.hi) + a.lo) * rs};
}

__device__ __forceinline__ ff ff_rcp(ff a) { return ff_tight(ffl_rcp(a)); }
__device__ __forceinline__ ff ff_sqrt(ff a) { return ff_tight(ffl_sqrt(a)); }
__device__ __forceinline__ ff ff_div(ff a, ff b) { return ff_mul(a, ffl_rcp(b)); }
__device__ __forceinline__ ff ff_dot2(ff a1, ff b1, ff a2, ff b2) { return ff_tight(ffl_dot2(a1, b1, a2, b2)); }

} // namespace xrdt
