/* artful_cuda — double-float arithmetic: a value as the unevaluated sum of two floats, about 48 significant bits
 * from FP32 instructions, which this GPU issues 64 times as fast as FP64 ones; and what the mixed trace forms in
 * it: a ray's constants of motion (lens.inc:125-142) and a coordinate's motion over a step (lens.inc:165-192).
 *
 * Sums by Knuth's error-free TwoSum, products by an FMA's residual (the exact error of a rounded product); each
 * result is renormalised by Dekker's fast two-sum, so that hi is the pair's value rounded to float and |lo| at most
 * half its ulp; the reciprocal and the reciprocal square root are the float estimates refined by one
 * Newton-Raphson step.  No step contracts: every product is its own or an explicit FMA's.
 *
 * Renormalising is a third of the work.  It is left out (the operations named Open, whose low part may be an ulp or
 * two of the high one) only where the value goes on into a sum it is a small part of, or meets roundings larger than
 * it would save: there the error against exact values is the same with and without, to a per cent in every quantile
 * from the median (2^-46.9 for the coefficients) to 99.9 %, over spins, inclinations and distances of the scenes'
 * range (the host test measures it).  A 1080p x 4 frame takes 1364 us so, 64 views 4600-4700; with every result
 * renormalised and the sums in their plain form 1451 and 5200.  Left out everywhere it was 1306 and 4480, and the
 * coefficients' errors half as large again in the median and twice at 99.9 %.
 * Compiles on the host too, where the test runs it. */
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define ARTF_PAIR __host__ __device__ __forceinline__
#else
#define ARTF_PAIR inline
#endif

namespace artf {

struct Ff {
    float hi, lo;
};

/* The float operations, each rounded to nearest by itself (the device's flush subnormals as the unit's flags say). */
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float addF(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float mulF(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fmaF(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float recipEstimate(float x) { return __fdividef(1.f, x); }
__device__ __forceinline__ float rsqrtEstimate(float x) { return rsqrtf(x); }
#else
ARTF_PAIR float addF(float a, float b) { return a + b; }
ARTF_PAIR float mulF(float a, float b) { return a * b; }
ARTF_PAIR float fmaF(float a, float b, float c) { return fmaf(a, b, c); }
ARTF_PAIR float recipEstimate(float x) { return 1.f / x; }
ARTF_PAIR float rsqrtEstimate(float x) { return 1.f / sqrtf(x); }
#endif

ARTF_PAIR Ff ffNorm(float s, float e) {
    const float hi = addF(s, e);
    return Ff{hi, addF(e, -addF(hi, -s))};
}
/* a + b and a b of floats: the rounded result and its error */
ARTF_PAIR Ff ffSum(float a, float b) {
    const float s = addF(a, b), bb = addF(s, -a);
    return Ff{s, addF(addF(a, -addF(s, -bb)), addF(b, -bb))};
}
ARTF_PAIR Ff ffProd(float a, float b) {
    const float p = mulF(a, b);
    return Ff{p, fmaF(a, b, -p)};
}
ARTF_PAIR Ff ffNorm(Ff open) { return ffNorm(open.hi, open.lo); }
ARTF_PAIR Ff ffNeg(Ff a) { return Ff{-a.hi, -a.lo}; }

/* a + m b, m a power of two (m b is exact, and goes into the sums as it is formed) */
ARTF_PAIR Ff ffAddOpen(Ff a, Ff b, float m = 1.f) {
    const float s = fmaF(m, b.hi, a.hi), bb = addF(s, -a.hi);
    const float e = addF(addF(a.hi, -addF(s, -bb)), fmaF(m, b.hi, -bb));
    return Ff{s, addF(e, fmaF(m, b.lo, a.lo))};
}
ARTF_PAIR Ff ffAdd(Ff a, Ff b, float m = 1.f) { return ffNorm(ffAddOpen(a, b, m)); }
ARTF_PAIR Ff ffSub(Ff a, Ff b) { return ffAdd(a, ffNeg(b)); }
/* The same where |a| is at least |m b|: the sum's error in two operations (Dekker's) for five */
ARTF_PAIR Ff ffAddLessOpen(Ff a, Ff b, float m = 1.f) {
    const float s = fmaF(m, b.hi, a.hi);
    return Ff{s, addF(fmaF(m, b.hi, -addF(s, -a.hi)), fmaF(m, b.lo, a.lo))};
}
ARTF_PAIR Ff ffAddLess(Ff a, Ff b, float m = 1.f) { return ffNorm(ffAddLessOpen(a, b, m)); }

ARTF_PAIR Ff ffMulOpen(Ff a, Ff b) {
    const Ff p = ffProd(a.hi, b.hi);
    return Ff{p.hi, fmaF(a.hi, b.lo, fmaF(a.lo, b.hi, p.lo))};
}
ARTF_PAIR Ff ffMul(Ff a, Ff b) { return ffNorm(ffMulOpen(a, b)); }
ARTF_PAIR Ff ffMulFOpen(Ff a, float b) {
    const Ff p = ffProd(a.hi, b);
    return Ff{p.hi, fmaF(a.lo, b, p.lo)};
}
ARTF_PAIR Ff ffMulF(Ff a, float b) { return ffNorm(ffMulFOpen(a, b)); }
ARTF_PAIR Ff ffSquareOpen(Ff a) {
    const Ff p = ffProd(a.hi, a.hi);
    return Ff{p.hi, fmaF(a.hi, addF(a.lo, a.lo), p.lo)};
}
ARTF_PAIR Ff ffSquare(Ff a) { return ffNorm(ffSquareOpen(a)); }
ARTF_PAIR Ff ffRecip(Ff x) {
    const float y = recipEstimate(x.hi);
    const float r = fmaF(-x.lo, y, fmaF(-x.hi, y, 1.f)); /* 1 - x y */
    return ffNorm(y, mulF(y, r));
}
ARTF_PAIR Ff ffRsqrt(Ff x) {
    const float y = rsqrtEstimate(x.hi);
    const Ff q = ffMulOpen(x, ffProd(y, y)); /* x y^2, next to 1 */
    return ffNorm(y, mulF(.5f * y, addF(addF(1.f, -q.hi), -q.lo)));
}

/* A double as the float it rounds to and what is left of its bits in a word: all 53, where a pair's low float would
 * keep 48.  restOf: of x beside `wide`, its float widened; withRest: x again. */
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ int64_t bitsOf(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double ofBits(int64_t b) { return __longlong_as_double(b); }
#else
ARTF_PAIR int64_t bitsOf(double x) {
    int64_t b;
    memcpy(&b, &x, sizeof b);
    return b;
}
ARTF_PAIR double ofBits(int64_t b) {
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
}
#endif
ARTF_PAIR int32_t restOf(double x, double wide) { return (int32_t)(bitsOf(x) - bitsOf(wide)); }
ARTF_PAIR double withRest(double wide, int32_t rest) { return ofBits(bitsOf(wide) + rest); }

/* x (A + x (B + x C)): what u'' is of u, and n_z'' of n_z with A = a^2 - K, B = 0 and C = -2 a^2
 * (a^2 n_z - (K + 2 a^2 n_z^2) n_z). */
struct Cubic {
    Ff A, B, C;
};
ARTF_PAIR Ff ffCubic(const Cubic& f, Ff x) {
    return ffMul(x, ffAdd(f.A, ffMul(x, ffAdd(f.B, ffMulOpen(x, f.C)))));
}
ARTF_PAIR Ff ffCubicF(const Cubic& f, float x) {
    return ffMulF(ffAdd(f.A, ffMulF(ffAdd(f.B, ffMulFOpen(f.C, x)), x)), x);
}
/* One Nystrom step (lens.inc:165-192) of x'' = cubic(x), from x and its rate v in float: the motion of u at a
 * radial turning point and of n_z at a polar one are this same step, so a warp runs it once for the lanes at
 * either.  The next x and v, and the first stage; their high parts are what the ray goes on with.  For a step that
 * turns: v changes sign in it, so h |v| is at most h^2 |x''|, and that, by the step's rule, a fifth of |x|: the sums
 * onto x know which part is greater, and the stages' share in x is small. */
struct Motion {
    Ff x, v, first;
};
ARTF_PAIR Motion motionFf(const Cubic& f, float step, float x, float v) {
    const Ff step2 = ffProd(step, step), hv = ffProd(step, v), at{x, 0.f};
    const Ff k1 = ffCubicF(f, x);
    const Ff k2 = ffCubic(f, ffAddLess(ffAddLessOpen(at, hv, .5f), ffMulOpen(step2, k1), .125f));
    const Ff xv = ffAddLessOpen(at, hv);
    const Ff k3 = ffCubic(f, ffAddLess(xv, ffMulOpen(step2, k2), .5f));
    const Ff nextX = ffAddLess(xv, ffMulOpen(ffMulFOpen(step2, 1.f / 6.f), ffAddOpen(k1, k2, 2.f)));
    const Ff nextV = ffAdd(ffMul(ffProd(step, 1.f / 6.f), ffAdd(ffAdd(k1, k3), k2, 4.f)), Ff{v, 0.f});
    return Motion{nextX, nextV, k1};
}

/* n_z's cubic.  A = a^2 - K is the constants' uA; where the constants are float (no MOTION guard) uA carries a
 * float's rounding of that difference, and A is formed from a^2 and the float K. */
ARTF_PAIR Cubic axisCubic(Ff a2, Ff uA, float K, bool pairedConstants) {
    return Cubic{pairedConstants ? uA : ffSub(a2, Ff{K, 0.f}), Ff{0.f, 0.f}, Ff{-2.f * a2.hi, -2.f * a2.lo}};
}

/* What a ray's set-up takes from the view: the eye's basis, the metric's four factors, rho, a and the start
 * terms. */
struct MotionTermsFf {
    Ff forward[3], right[3], up[3], metric[4], rho, a, a2, mu0Squared, minusTwoA2;
};

/* The constants of motion alone, for an eye at rest (lens.inc:125-142 without the aberration of 110-122), in
 * rayStartWith's order of operations with the direction normalised first: 1 / E, the axial momentum xi,
 * K = eta + xi^2, the radial equation's coefficients and a xi, and the factors the first state is made of (d_x,
 * 1 / (|d| E), across and the axial component of the direction over E). */
struct MotionFf {
    Ff invEnergy, xi, big, uA, uB, uC, xiA, dx, over, across, xiAxis;
};
ARTF_PAIR MotionFf motionConstantsFf(const MotionTermsFf& t, float nx, float ny) {
    MotionFf m;
    Ff d[3];
    for (int k = 0; k < 3; ++k)
        d[k] = ffAddOpen(ffAddOpen(t.forward[k], ffMulFOpen(t.right[k], nx)), ffMulFOpen(t.up[k], ny));
    const Ff invLength = ffRsqrt(ffAdd(ffAddOpen(ffSquareOpen(d[0]), ffSquareOpen(d[1])), ffSquareOpen(d[2])));
    const Ff dz = ffMul(d[2], invLength);
    m.invEnergy = ffRecip(ffSub(t.metric[0], ffMulOpen(t.metric[1], dz)));
    m.dx = ffNorm(d[0]);
    m.over = ffMul(invLength, m.invEnergy);
    m.xi = ffNeg(ffMul(ffMul(t.metric[2], dz), m.invEnergy));
    m.xiAxis = ffMul(ffMul(t.metric[3], d[2]), m.over);
    m.across = ffMul(ffMul(t.rho, d[1]), m.over);
    const Ff eta = ffAdd(ffSquare(m.across), ffMulOpen(t.mu0Squared, ffAddOpen(ffSquare(m.xiAxis), ffNeg(t.a2))));
    m.big = ffAdd(eta, ffSquare(m.xi));
    m.uA = ffSub(t.a2, m.big);
    m.uB = ffMulF(ffAddOpen(eta, ffSquare(ffSub(m.xi, t.a))), 3.f);
    m.uC = ffMul(t.minusTwoA2, eta);
    m.xiA = ffMul(m.xi, t.a);
    return m;
}

}  // namespace artf
