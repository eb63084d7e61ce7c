/* Single-precision pieces shared by the link kernels that keep their matrix in
 * registers: reciprocals and roots without branches, the fused forms of the
 * Householder step, the bias-corrected coherence of one entry.
 */
#ifndef TC_LINK_FLOAT_CUH
#define TC_LINK_FLOAT_CUH

#include "tcoh_internal.h"

#include <float.h>

/* A value that the compiler cannot follow: the addresses formed from it are
   not kept in registers from one pixel pair to the next (there are more of
   them than registers; they would be spilled). */
__device__ __forceinline__ int opaque(int v)
{
    asm volatile("" : "+r"(v));
    return v;
}

/* The hardware's approximate reciprocal, within two ulps. Zero and denormal
   operands give an infinity: where a caller can have them (a tridiagonal's
   sub-diagonal, the square of a zero coherence), a select drops the result. */
__device__ __forceinline__ float rcp_approx(float x)
{
    float y;

    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* The approximate reciprocal square root, likewise: zero and denormal operands
   give an infinity. */
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;

    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

/* 1 / x correctly rounded, by one Newton step with fused multiply-adds from the
   approximate reciprocal (Markstein, IBM Journal of Research and Development
   34, 1990), and the square root by his iteration from the approximate
   reciprocal root. Equal to __frcp_rn and sqrtf for every significand and
   every exponent from -90 to 90 (all of them compared once; tests/
   link_float_check.cu compares some); the caller keeps to exponents within 80,
   or drops what they give (not a number for 0). They have no branches: with the intrinsics a
   Householder step took 17 % longer (2.48k against 2.14k cycles, eight warps,
   30 dates). */
__device__ __forceinline__ float rcp_rn(float x)
{
    const float y = rcp_approx(x);

    return fmaf(y, fmaf(-x, y, 1.0f), y);
}

__device__ __forceinline__ float sqrt_rn(float a)
{
    const float y = rsqrt_approx(a);
    float s = __fmul_rn(a, y), h = 0.5f * y;
    const float e = fmaf(-s, h, 0.5f);

    h = fmaf(h, e, h);
    s = fmaf(s, e, s);
    return fmaf(fmaf(-s, s, a), h, s);
}

/* T_ij / |T_ij| of the goodness of fit (tcoh.cl:734-738); 1 for |T_ij| below
   1e-37 (|T_ij| is at most 1). The factor 2^60, which changes no rounding, keeps
   the square normal: without it the approximate root flushed the square of
   |T_ij| < 1.1e-19 (dates whose energy lies in different pixels) to zero, and the
   phasor was infinite. */
__device__ __forceinline__ float2 unit_phasor(float2 t)
{
    const float x = t.x * 0x1p60f, y = t.y * 0x1p60f;
    const float m2 = x * x + y * y;
    const bool some = m2 >= FLT_MIN;
    const float s = some ? rsqrt_approx(m2) : 0.f;

    return make_float2(some ? x * s : 1.f, y * s);
}

/* Fused products with the roundings written out, so that what a pixel gets does
   not depend on how the compiler contracts the expressions around them. */
__device__ __forceinline__ float2 cscale(float2 a, float2 b) /* a b */
{
    return make_float2(fmaf(a.x, b.x, -__fmul_rn(a.y, b.y)), fmaf(a.y, b.x, __fmul_rn(a.x, b.y)));
}

/* One element of the rank-2 update: t - (v conj(wj) + w conj(vj)), with
   nv = -v and nw = -w (four FMAs per component). */
__device__ __forceinline__ float2 r2(float2 t, float2 nv, float2 nw, float4 q)
{
    t.x = fmaf(nv.x, q.z, t.x);
    t.x = fmaf(nv.y, q.w, t.x);
    t.x = fmaf(nw.x, q.x, t.x);
    t.x = fmaf(nw.y, q.y, t.x);
    t.y = fmaf(nv.y, q.z, t.y);
    t.y = fmaf(-nv.x, q.w, t.y);
    t.y = fmaf(nw.y, q.x, t.y);
    t.y = fmaf(-nw.x, q.y, t.y);
    return t;
}

/* a / b correctly rounded, from y = 1 / b correctly rounded and Markstein's
   correction of the quotient: equal to __fdiv_rn for quotients of 2^-30 to 2
   with divisors of 2^-67 to 2^67 (2.6 x 10^9 random pairs, tests/
   link_float_check.cu), the date sums' products that load_T divides by this
   way. */
__device__ __forceinline__ float div_rn(float a, float b, float y)
{
    const float q = __fmul_rn(a, y);

    return fmaf(fmaf(-b, q, a), y, q);
}

/* T_ij (i < j) from its Gram sum g and the date norms (tcoh.cl:611-636),
   in IEEE float without contraction; near: the bias decision lies within
   TC_BIAS_BAND of its threshold. */
static __device__ __noinline__ float2 t_entry_any(float2 g, float nrm_i, float nrm_j, float fl,
                                           bool debias, bool &near)
{
    const float dd = __fmul_rn(nrm_i, nrm_j);
    float re = 0.f, im = 0.f;

    if (dd > 0.f) {
        re = __fdiv_rn(g.x, dd);
        im = __fdiv_rn(g.y, dd);
        if (debias) {
            const float m2 = __fadd_rn(__fmul_rn(re, re), __fmul_rn(im, im));
            const float lm1 = __fsub_rn(__fmul_rn(fl, m2), 1.0f);
            const float m2c = __fdiv_rn(lm1, __fsub_rn(fl, 1.0f));

            near |= fabsf(lm1) < TC_BIAS_BAND * fl * m2;
            const float f = (m2 > 0.f && m2c > 0.f) ? __fsqrt_rn(__fdiv_rn(m2c, m2)) : 0.f;

            re = __fmul_rn(re, f);
            im = __fmul_rn(im, f);
        }
    }
    return make_float2(re, im);
}

/* The same without branches, for date norms and looks of ordinary size. */
__device__ __forceinline__ float2 t_entry(float2 g, float nrm_i, float nrm_j, float fl, float ilm1,
                                          bool debias, bool &near)
{
    const float dd = __fmul_rn(nrm_i, nrm_j), y = rcp_rn(dd);
    float re = dd > 0.f ? div_rn(g.x, dd, y) : 0.f, im = dd > 0.f ? div_rn(g.y, dd, y) : 0.f;
    const float m2 = __fadd_rn(__fmul_rn(re, re), __fmul_rn(im, im));
    const float lm1 = __fsub_rn(__fmul_rn(fl, m2), 1.0f);
    const float m2c = div_rn(lm1, __fsub_rn(fl, 1.0f), ilm1);
    const bool some = m2 > 0.f && m2c > 0.f;
    const float f = some ? sqrt_rn(div_rn(m2c, m2, rcp_rn(m2))) : 0.f;

    near |= debias & (fabsf(lm1) < TC_BIAS_BAND * fl * m2);
    re = debias ? __fmul_rn(re, f) : re;
    im = debias ? __fmul_rn(im, f) : im;
    return make_float2(re, im);
}

#endif
