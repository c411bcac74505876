/* artful_cuda — the mixed-precision trace: FP32 for the bulk of each geodesic, extended precision
 * (about FP64's) only where stability needs it.  "Wide" work runs as double-float pairs on the FP32 pipe
 * (Dekker's double-length arithmetic, about 48 bits), or in FP64 where it divides:
 *
 *   MOTION   the constants of motion (E, xi = L_z / E, Carter's eta, K and the radial equation's
 *            coefficients) come from the ray at the eye in double-float, from the frame's doubles split
 *            into pairs; the first state's w and v and the step, the integrator's FP32 quantities, are
 *            formed from them in FP32 (the step by the reference's rule from the rounded K, so every
 *            sub-step of a ray, FP32 or wide, takes the same one);
 *   HORIZON  within a band of the outer horizon (u > band * 0.995 / r+) the radial sub-step of
 *            (u, du/ds, psi) runs in FP64: Delta / r^2 in the frame-drag rate loses most of its bits to
 *            cancellation there;
 *   RADIAL   the step in which du/ds changes sign (the radial potential's zero) has its motion of
 *            (u, du/ds) in double-float (psi and its rate, smooth there, stay the FP32 step's);
 *   POLAR    the step in which the axis part of dn/ds changes sign (the polar potential's zero) has
 *            the axis component (n_z, dn_z/ds) in double-float: n_z'' depends on n_z alone, and the
 *            turning point is its (the components about the axis stay the FP32 step's);
 *   PSI      psi, the frame-drag angle, is summed with a compensated (two-sum) accumulator, and the
 *            endpoint's Mino time is formed in FP64 from the step count: neither drifts over 192 steps.
 * The radial and polar sub-steps are independent (u'' depends on u alone, n'' on n alone), so a guard
 * costs wide work only for the part that needs it; and u'' and n_z'' are the same cubic with other
 * coefficients, so one wide step in the code serves both turning points, and a warp runs it once for the
 * lanes at either.  The disc and sky shading stay in FP32.  Built with the fast FP32 flags; in double,
 * + - * are IEEE and / and sqrt are refined hardware estimates (within an ulp or two, lensCore.cuh), as in
 * the plain FP64 trace.  At the headline frame the double-float sub-steps give the FP64 ones' bits, rounded
 * to float, for every pixel.
 *
 * Scheduling (mixedTiles): a persistent grid of warps takes slots from one device queue (a slot: one ray of
 * each pixel of an 8 x 4 tile; heavy tiles first; views of uneven size share the queue), and a warp traces
 * its 32 rays together, each step's wide sub-steps at once.  Neighbouring rays turn within a step or two of
 * one another, so a wide step serves most of a warp at a time, and a ray's step costs nothing for the
 * schedule's sake.  (Lanes that waited for full rounds of wide steps and were refilled one by one, as an
 * FP64 wide step wanted, paid 80 thread instructions a step in votes and flags: 2.15 against 1.61 ms for the
 * 1080p x 4 frame, 7.63 against 5.51 for 64 views.)  What a step costs is issue slots (75 % of them used, FMA
 * pipe 55 % busy), so the FP32 step runs its coordinates in pairs with packed instructions (nystromStep: 1.86
 * -> 1.76 ms), the wide step is one code path (1.74 -> 1.61 with the counts out of registers) and each float
 * rounding is written out or pinned (ARTF_PINNED_FMA): whatever registers a kernel is given, its images are
 * the same bits.  A frame of fewer rays than the GPU's warps could take is bound by its longest ray's
 * latency; there warps take fewer rays each (mixedGrid). */
#define ARTF_PINNED_FMA 1 /* every float sum of two products rounds the same in every kernel (lensCore.cuh) */
#define ARTF_FAST_FP64 1 /* FP64 division and square roots by refined hardware estimates (lensCore.cuh) */
#define ARTF_FP64_NEWTON_STEPS 1 /* one refinement: ~40 bits, far below float's rounding (3.4 % faster) */
#include "lensKernel.cuh"
#include "lensMixed.h"
#include "lensPairs.cuh"
#include "lensParts.h"

#include <string.h>

namespace artf {

/* A view as the kernels read it, from the device view table or as a parameter. */
struct MixedView {
    Frame<float> f;
    Frame<double> d;
    ArtfCudaHoleFrame h; /* sample positions come from the FP32 frame, as the reference's */
    const float* map;
    const float* fluid;
    float4* hdr;
    ArtfCudaRayEnd* ends;
    /* Rays of the view's pixels, plane k for ray k (radiance, class bits), or NULL.  With planes, a work
     * unit is one ray and combinePlanes sums each pixel's rays afterwards; without, a unit is a pixel
     * whose rays one lane traces in turn. */
    float4* rayOut;
    double wideA2;            /* a^2 in double, for the horizon band's FP64 sub-step */
    StartTerms<double> start64; /* what a moving eye's rays' FP64 set-up takes from the view alone */
    MotionTermsFf motion;       /* the same and the frame's, for the set-up of an eye at rest, as pairs */
    float startNarrow[4];     /* the eye's e_r and 1/r in float, where every ray's set-up starts */
    float wScaleNarrow;       /* -u0^2 sqrt(Delta) sqrt(Sigma), in float: w's factor from the eye */
    float stepBaseNarrow;     /* the step rule's (pi / 24) x step scale, in float */
    float rhoScale, uGuard, share;
    int tilesX, pixelUnits, units, unitBase, tileBase, rays, jitter;
    int rowBegin, rows; /* the pixel rows this launch traces (a band of the frame, or all of it) */
    uint32_t seed;
};
static_assert(sizeof(MixedView) <= kMixedViewBytesMax, "a view table slot outgrew kMixedViewBytesMax");

namespace {

struct MixedParams {
    const MixedView* views;
    int viewCount;
    int totalUnits;
    /* the queue's slots (32 units: one ray plane of one tile) in the order handed out, each (view | plane
     * << 12, tile); NULL: pixel order, view after view */
    const uint2* order;
    unsigned long long* counters;
    float stepScale;
    int maxSteps;
    int lanesLog2;    /* a warp's rays at a time: 2^lanesLog2 of its lanes */
    int cornersLog2;  /* the probe's rays a tile: 1, or one at each corner */
    /* the order's slots a weight class; of the heavy classes' slots (its first), mostHeavy at most, a warp takes
     * eight rays at a time (the kernels that split) */
    const unsigned* classes;
    int mostHeavy;
    uint32_t guards;  /* ARTF_CUDA_GUARD_* */
};

/* One ray's state between steps. */
struct MixedRay {
    RayConst<float> c;
    int32_t stepRest;                      /* c.step's double: a moving eye's has more bits (withRest) */
    float uALo, uBLo, uCLo, xiALo;         /* the low halves of the coefficients the wide sub-steps use */
    RayState<float> s;                 /* s.psi stays 0: a step returns psi's increment */
    float psiHi, psiLo, through, sum[3];
    int i;
    unsigned crossings;                /* and bit 31 once the disc lit the ray */
    unsigned wide, turns;              /* wide steps and those in the horizon's band, radial and polar turning
                                        * points: two counts a word, a ray's 384 steps at most */
};
constexpr unsigned kLit = 0x80000000u;

/* Float <-> double conversions on the integer pipe.  On this GPU a conversion to double costs an FP64
 * instruction and one to float two, on the narrow FP64 pipe, while the integer pipe idles: these take a
 * handful of integer instructions instead, for the same bits as the hardware's conversions under this
 * unit's flags (flush-to-zero; round to nearest even), NaN aside (a NaN stays a NaN, its payload is not
 * kept).  artfCudaCheckConversions checks them against the hardware's.  The narrowing is a call, not
 * inlined at its sites in the FP64 paths: inlined, those copies overflowed the instruction cache (warps
 * stalled waiting for instructions; 3.97 ms against 3.50 at 1080p x 4). */
__device__ __forceinline__ double widen(float f) {
    const uint32_t b = __float_as_uint(f), sign = b & 0x80000000u, mag = b & 0x7fffffffu, e = mag >> 23;
    uint32_t hi = sign | ((mag >> 3) + 0x38000000u), lo = mag << 29;  /* rebias 127 -> 1023 */
    if (e == 0u) hi = sign, lo = 0u;                                    /* zero (a subnormal flushes) */
    if (e == 255u) hi = sign | 0x7ff00000u | ((mag & 0x7fffffu) >> 3);  /* infinity, NaN */
    return __hiloint2double((int)hi, (int)lo);
}

__device__ __noinline__ float narrow(double d) {
    const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
    const uint32_t sign = hi & 0x80000000u, e = (hi >> 20) & 0x7ffu;
    /* the top 23 bits of the 52-bit fraction, and the 29 below them that rounding looks at */
    const uint32_t keep = ((hi & 0xfffffu) << 3) | (lo >> 29), rest = lo & 0x1fffffffu;
    uint32_t bits;
    if (e >= 897u && e <= 1150u) {
        bits = ((e - 896u) << 23) | keep;
        bits += (rest > 0x10000000u || (rest == 0x10000000u && (keep & 1u))) ? 1u : 0u; /* (may carry to inf) */
    } else if (e == 896u) {
        /* in [2^-127, 2^-126): rounded to 24 significant bits as if the exponent went on, only what then
         * reaches 2^-126 is not flushed (the fraction's top 23 bits all ones, and the rest half or more) */
        bits = (keep == 0x7fffffu && rest >= 0x10000000u) ? 0x00800000u : 0u;
    } else if (e < 896u) {
        bits = 0u;
    } else if (e == 0x7ffu && ((hi & 0xfffffu) | lo)) {
        bits = 0x7fffffffu; /* NaN */
    } else {
        bits = 0x7f800000u; /* too large, or infinite */
    }
    return __uint_as_float(sign | bits);
}

/* ---- pairs (lensPairs.cuh) to and from double ---------------------------------------------------------- */

/* hi + lo as a double: exact, since the pair holds at most 48 significant bits. */
__device__ __forceinline__ double ffWide(Ff a) { return widen(a.hi) + widen(a.lo); }
__device__ __forceinline__ Ff ffSplit(double x) {
    const float hi = narrow(x);
    return Ff{hi, narrow(x - widen(hi))};
}

/* The wide coefficients, their high halves the FP32 ones. */
__device__ __forceinline__ void setWide(MixedRay& r, Ff uA, Ff uB, Ff uC, Ff xiA) {
    r.c.uA = uA.hi, r.c.uB = uB.hi, r.c.uC = uC.hi, r.c.xiA = xiA.hi;
    r.uALo = uA.lo, r.uBLo = uB.lo, r.uCLo = uC.lo, r.xiALo = xiA.lo;
}

/* The helpers below take the guards apart from the parameters, so that a kernel built for all of them
 * passes a constant and its tests fold away. */

/* A ray's start: its constants of motion and first state, in double-float under the MOTION guard. */
__device__ __forceinline__ void mixedStart(const MixedParams& p, uint32_t guards, const MixedView& v, float nx,
                                           float ny, float time, MixedRay& r) {
    if ((guards & ARTF_CUDA_GUARD_MOTION) && v.d.boost[3] > 1.0) {
        /* a moving eye: the whole set-up with its aberration in FP64 */
        RayConst<double> cd;
        RayState<double> sd;
        rayStartWith(v.d, v.start64, widen(nx), widen(ny), widen(time), cd, sd);
        r.c.invEnergy = narrow(cd.invEnergy), r.c.xi = narrow(cd.xi), r.c.moved = narrow(cd.moved);
        r.c.big = narrow(cd.big);
        r.c.step = narrow(cd.step);
        r.stepRest = restOf(cd.step, widen(r.c.step));
        setWide(r, ffSplit(cd.uA), ffSplit(cd.uB), ffSplit(cd.uC), ffSplit(cd.xiA));
        r.s.u = v.startNarrow[3], r.s.w = narrow(sd.w);
        for (int k = 0; k < 3; ++k) r.s.n[k] = v.startNarrow[k], r.s.v[k] = narrow(sd.v[k]);
    } else if (guards & ARTF_CUDA_GUARD_MOTION) {
        /* in double-float; the first state and the step, the integrator's FP32 quantities, from them in FP32 */
        const MotionFf m = motionConstantsFf(v.motion, nx, ny);
        r.c.invEnergy = m.invEnergy.hi, r.c.xi = m.xi.hi, r.c.moved = 1.f, r.c.big = m.big.hi;
        setWide(r, m.uA, m.uB, m.uC, m.xiA);
        r.c.step = divSqrtR(v.stepBaseNarrow, maxX(r.c.big, 4.f));
        r.stepRest = 0;
        /* (u and n start at the eye's: the view's, narrowed once) */
        r.s.u = v.startNarrow[3];
        r.s.w = v.wScaleNarrow * m.dx.hi * m.over.hi;
        for (int k = 0; k < 3; ++k)
            r.s.n[k] = v.startNarrow[k], r.s.v[k] = sum2(m.across.hi, v.f.etheta[k], m.xiAxis.hi, v.f.ephi[k]);
    } else {
        rayStart(v.f, nx, ny, time, p.stepScale, r.c, r.s);
        r.stepRest = 0;
        r.uALo = r.uBLo = r.uCLo = r.xiALo = 0.f;
    }
    r.c.time = time;
    r.s.psi = 0.f;
    r.s.drag = v.f.a != 0.f ? dragAt(v.f.a, v.f.a * v.f.a, r.c.xiA, r.s.u) : 0.f;
    r.psiHi = r.psiLo = 0.f;
    r.through = 1.f;
    r.sum[0] = r.sum[1] = r.sum[2] = 0.f;
    r.i = 0;
    r.crossings = r.wide = r.turns = 0;
}

/* A ray's step in double.  (Read as the float's alone where an eye rests: 1364 us at 1080p x 4, 1378 through the
 * rest, which is 0 there.) */
__device__ __forceinline__ double stepOf(const MixedView& v, const MixedRay& r) {
    return v.d.boost[3] > 1.0 ? withRest(widen(r.c.step), r.stepRest) : widen(r.c.step);
}

/* The sub-steps of an FP32 step that its guards ask for again, wide.  Radial, in the horizon's band: the
 * whole sub-step in FP64 (the frame-drag rate's Delta / r^2 cancels there, and it divides).  At a turning
 * point, of u or of n_z, that coordinate's motion in double-float: psi and its rate, and the components
 * about the axis, smooth there, stay the FP32 step's.  A step that turns both runs the motion twice. */
__device__ __forceinline__ void mixedGuards(uint32_t guards, const MixedView& v, MixedRay& r, bool band, bool turnR,
                                            bool turnP, StepOut<float>& o, unsigned& rounds) {
    if (!(band || turnR || turnP)) return;
    turnR = turnR && !band;
    r.wide += 1u | (band ? 0x10000u : 0u);
    r.turns += (turnR ? 1u : 0u) | (turnP ? 0x10000u : 0u);
    const unsigned first = (threadIdx.x & 31) == __ffs((int)__activemask()) - 1;
    rounds += first;
    if (band) {
        RayConst<double> c;
        c.step = stepOf(v, r), c.uA = ffWide(Ff{r.c.uA, r.uALo}), c.uB = ffWide(Ff{r.c.uB, r.uBLo});
        c.uC = ffWide(Ff{r.c.uC, r.uCLo}), c.xiA = ffWide(Ff{r.c.xiA, r.xiALo});
        c.invEnergy = c.xi = c.moved = c.time = c.big = 0.0; /* (not read by the sub-step) */
        double k1;
        RayState<double> s, next;
        s.u = widen(r.s.u), s.w = widen(r.s.w), s.psi = 0.0, s.drag = widen(r.s.drag);
        const double step = widen(r.c.step);
        radialStepWith(v.d.a, v.wideA2, c, stepTerms(step), s, next, k1);
        o.next.u = narrow(next.u), o.next.w = narrow(next.w), o.next.psi = narrow(next.psi);
        o.next.drag = narrow(next.drag);
        o.k1 = narrow(k1);
    }
    while (turnR || turnP) {
        Cubic f = axisCubic(v.motion.a2, Ff{r.c.uA, r.uALo}, r.c.big, guards & ARTF_CUDA_GUARD_MOTION);
        if (turnR) f = Cubic{Ff{r.c.uA, r.uALo}, Ff{r.c.uB, r.uBLo}, Ff{r.c.uC, r.uCLo}};
        const Motion m = motionFf(f, r.c.step, turnR ? r.s.u : r.s.n[2], turnR ? r.s.w : r.s.v[2]);
        if (turnR) {
            o.next.u = m.x.hi, o.next.w = m.v.hi, o.k1 = m.first.hi;
            turnR = false;
        } else {
            o.next.n[2] = m.x.hi, o.next.v[2] = m.v.hi, o.a1[2] = m.first.hi;
            turnP = false;
        }
    }
}

/* What a step meets: the disc crossing, escape, horizon and opacity.  Returns the end's kind
 * (ARTF_CUDA_END_*) + 1, or 0 when the ray goes on. */
__device__ __forceinline__ unsigned mixedMeets(bool compensated, const MixedView& v, MixedRay& r,
                                               const StepOut<float>& o, ArtfCudaRayEnd* end) {
    const Frame<float>& f = v.f;
    const float increment = o.next.psi;
    Crossing<float> x;
    bool opaque = false;
    if (crossingOf(f, v.rhoScale, r.c, r.s, o, x)) {
        x.psiC = compensated ? r.psiHi + (r.psiLo + x.part * increment) : r.psiHi + x.part * increment;
        ++r.crossings;
        float turn;
        const float light = shadeCrossing(f, v.rhoScale, v.map, v.fluid, r.c, x, r.through, r.sum, &turn);
        if (light > 0.f && !(r.crossings & kLit)) {
            r.crossings |= kLit;
            if (end) end->hitR = recipR(x.uc), end->hitPhi = turn - floorf(turn);
        }
        /* (the transmission only changes here) */
        opaque = !(r.through > .004f);
    }
    if (0.f > o.next.u) {
        const float part = divR(r.s.u, r.s.u - o.next.u);
        float away[3], dir[3];
        for (int k = 0; k < 3; ++k) away[k] = r.s.n[k] + part * (o.next.n[k] - r.s.n[k]);
        const float awayPsi = compensated ? r.psiHi + (r.psiLo + part * increment) : r.psiHi + part * increment;
        skyDirection(away, awayPsi, dir);
        if (f.stars > 0.f) shadeSky(f, v.map, r.c, dir, r.through, r.sum);
        /* (the escape's direction and moment travel in the slots the ray no longer needs) */
        r.s.n[0] = dir[0], r.s.n[1] = dir[1], r.s.n[2] = dir[2];
        r.s.w = part;
        return ARTF_CUDA_END_SKY + 1;
    }
    if (o.next.u > f.uHorizon) return ARTF_CUDA_END_HORIZON + 1;
    if (opaque) return ARTF_CUDA_END_OPAQUE + 1;
    return 0;
}

/* What a thread counts over its rays, in shared memory: touched once a ray, it would hold ten registers
 * through the stepping loop. */
enum { kMixedRays, kMixedSteps, kMixedCrossings, kMixedEscapes, kMixedWide, kMixedBand, kMixedRadial, kMixedPolar, kMixedCount };

/* The end record of a finished ray, and its tallies. */
__device__ __forceinline__ unsigned mixedFinish(const MixedView& v, const MixedRay& r, unsigned ended, ArtfCudaRayEnd* end,
                                                unsigned (*tally)[256]) {
    unsigned kind = ended - 1;
    if (r.crossings & kLit) kind |= ARTF_CUDA_END_LIT;
    const unsigned crossings = r.crossings & ~kLit;
    const bool sky = (kind & 15u) == ARTF_CUDA_END_SKY;
    const unsigned add[kMixedCount] = {1u, (unsigned)r.i, crossings, sky ? 1u : 0u, r.wide & 0xFFFFu, r.wide >> 16,
                                       r.turns & 0xFFFFu, r.turns >> 16};
    for (int k = 0; k < kMixedCount; ++k) tally[k][threadIdx.x] += add[k];
    if (end) {
        const double step = stepOf(v, r);
        for (int k = 0; k < 3; ++k) end->dir[k] = sky ? r.s.n[k] : 0.f;
        end->mino = (float)(sky ? ((double)(r.i - 1) + (double)r.s.w) * step : (double)r.i * step);
        end->steps = (uint16_t)r.i;
        end->crossings = (uint8_t)(crossings > 255u ? 255u : crossings);
        end->kind = (uint8_t)kind;
        end->fp64Steps = (uint16_t)(r.wide & 0xFFFFu);
        end->reserved = 0;
    }
    return kind;
}

/* One ray from start to end, each step's wide sub-steps at once.  kAll: every guard on (the default), the
 * step's tests of them as constants. */
template <bool kAll>
__device__ __forceinline__ unsigned traceRayMixed(const MixedParams& p, const MixedView& v, float nx, float ny,
                                                  float time, float* sum, ArtfCudaRayEnd* end, unsigned (*tally)[256],
                                                  unsigned& rounds) {
    const uint32_t guards = kAll ? (uint32_t)ARTF_CUDA_GUARD_ALL : p.guards;
    MixedRay r;
    mixedStart(p, guards, v, nx, ny, time, r);
    if (end) end->hitR = end->hitPhi = NAN;
    const bool compensated = guards & ARTF_CUDA_GUARD_PSI;
    unsigned ended = ARTF_CUDA_END_CAP + 1;
    for (;;) {
        StepOut<float> o;
        nystromStep(v.f.a, r.c, r.s, o);
        ++r.i;
        /* Most steps need no guard and meet nothing, which one branch decides (all its tests made: 1464 us with
         * a branch for each, 1372 with the tests in turn, 1331 so, at 1080p x 4). */
        const bool band = (guards & ARTF_CUDA_GUARD_HORIZON) && r.s.u > v.uGuard;
        const bool turnR = (guards & ARTF_CUDA_GUARD_RADIAL) && ((r.s.w > 0.f) != (o.next.w > 0.f));
        const bool turnP = (guards & ARTF_CUDA_GUARD_POLAR) && ((r.s.v[2] > 0.f) != (o.next.v[2] > 0.f));
        if (band | turnR | turnP | (r.s.n[2] * o.next.n[2] < 0.f) | (0.f > o.next.u) | (o.next.u > v.f.uHorizon)) {
            mixedGuards(guards, v, r, band, turnR, turnP, o, rounds);
            if (const unsigned met = mixedMeets(compensated, v, r, o, end)) {
                ended = met;
                break;
            }
        }
        const float increment = o.next.psi;
        if (compensated) {
            const float sumHi = r.psiHi + increment, back = sumHi - r.psiHi;
            r.psiLo += (r.psiHi - (sumHi - back)) + (increment - back);
            r.psiHi = sumHi;
        } else {
            r.psiHi += increment;
        }
        r.s = o.next;
        r.s.psi = 0.f;
        if (r.i >= p.maxSteps) break;
    }
    for (int k = 0; k < 3; ++k) sum[k] = sum[k] + r.sum[k];
    return mixedFinish(v, r, ended, end, tally);
}

__device__ __forceinline__ void clearMixed(unsigned (*tally)[256]) {
    for (int k = 0; k < kMixedCount; ++k) tally[k][threadIdx.x] = 0;
}

/* A warp's tallies to the launch's counters; the whole warp calls it. */
__device__ __forceinline__ void flushMixed(unsigned (*tally)[256], unsigned rounds, unsigned long long* counters) {
    const int to[kMixedCount] = {CRays, CSteps, CCrossings, CEscapes, CFp64Steps, CFp64Horizon, CFp64Radial, CFp64Polar};
    const bool first = (threadIdx.x & 31) == 0;
    for (int k = 0; k < kMixedCount; ++k) {
        const unsigned n = __reduce_add_sync(0xFFFFFFFFu, tally[k][threadIdx.x]);
        if (first && n) atomicAdd(counters + to[k], (unsigned long long)n);
    }
    rounds = __reduce_add_sync(0xFFFFFFFFu, rounds);
    if (first && rounds) atomicAdd(counters + CFp64Rounds, (unsigned long long)rounds);
}

/* The view a queue unit belongs to: the last whose first unit is at or below it. */
__device__ __forceinline__ int viewOf(const MixedParams& p, int unit) {
    int lo = 0, hi = p.viewCount - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&p.views[mid].unitBase) <= unit) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* ---- heavy first --------------------------------------------------------------------------------
 * After the queue empties the persistent grid drains, and a lane that took a long ray late holds its SM
 * while the others idle (a photon-ring ray runs to the step cap, ten times a sky ray's steps).  So the
 * queue hands out the heaviest tiles first and leaves short rays for the end.  A tile's weight is the
 * step count of one FP32 ray through its middle, stepped without shading (the disc is thin: it seldom
 * ends a ray) up to 64 steps (a sky ray takes about 25; what goes on longer is heavy); tiles are
 * counting-sorted by weight class, heaviest first.  The order changes when a ray is traced, never what
 * it computes, so the frame is the same bits in any order.
 *
 * A frame of few slots a resident warp is bound by its heavy tiles alone: a warp of 32 rays that part ways
 * runs all they need one after another, some 100 us of a 512 x 288 frame's 126.  There the heavy tiles come
 * apart, eight rays a warp, and each tile's weight is the most steps of its four corners' rays: the photon
 * ring is thinner than a tile, and one ray misses tiles whose long rays then start last.  Every heavy tile
 * costs more warps so; with the frame's size it gains less, and at six slots a warp nothing (mixedGrid). */

constexpr int kWeightClasses = 9; /* steps / 8 up to 64: the probe stops there (all heavier tiles, class 8) */
constexpr int kProbeSteps = 64;
constexpr int kHeavyClass = 5; /* 40 steps or more at a corner */
constexpr int kCornersLog2 = 2;

/* The view a batch-wide tile belongs to: the last whose first tile is at or below it. */
__device__ __forceinline__ int tileView(const MixedParams& p, int tile) {
    int lo = 0, hi = p.viewCount - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(&p.views[mid].tileBase) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* The probe, the order, the trace and the sum of planes follow one another at once (programmatic dependent
 * launch): each may start while the one before it drains, and waits here, before it reads or writes what others
 * do, until that one has finished, and with it all before (1080p x 4 1321 -> 1308 us, one ray a pixel 374 -> 364,
 * 512 x 288 102 -> 98). */
__device__ __forceinline__ void chained() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

/* Each tile's weight class, and each class's count of queue slots (a tile has one a ray plane), counted
 * in the block first so that each class takes one global atomic a block. */
template <bool kOne>
__device__ __forceinline__ void probeTiles(const MixedParams& p, const MixedView* one, int totalTiles, int* weights,
                                           unsigned* classes) {
    __shared__ unsigned counts[kWeightClasses];
    chained();
    if (threadIdx.x < kWeightClasses) counts[threadIdx.x] = 0;
    __syncthreads();
    const int at = (int)(blockIdx.x * 128 + threadIdx.x), g = at >> p.cornersLog2;
    const int corner = at & ((1 << p.cornersLog2) - 1);
    int w = 0;
    unsigned planes = 0;
    if (g < totalTiles) {
        const MixedView& v = kOne ? *one : p.views[tileView(p, g)];
        const int tile = g - v.tileBase;
        const int dx = p.cornersLog2 ? (corner & 1) * 7 : 4, dy = p.cornersLog2 ? (corner >> 1) * 3 : 2;
        const int x = min((tile % v.tilesX) * 8 + dx, (int)v.f.width - 1);
        const int y = min(v.rowBegin + (tile / v.tilesX) * 4 + dy, v.rowBegin + v.rows - 1);
        float nx, ny, moment;
        samplePosition(v.h, v.jitter, v.seed, x, y, 0, &nx, &ny, &moment);
        RayConst<float> c;
        RayState<float> s;
        rayStart(v.f, nx, ny, v.h.disc[2] + v.h.spin[3] * moment, p.stepScale, c, s);
        const float a = v.f.a;
        if (a != 0.f) s.drag = dragAt(a, a * a, c.xiA, s.u);
        const int most = min(p.maxSteps, kProbeSteps);
        int i = 0;
        while (i < most) {
            StepOut<float> o;
            nystromStep(a, c, s, o);
            ++i;
            if (0.f > o.next.u || o.next.u > v.f.uHorizon) break;
            s = o.next;
        }
        w = min(i >> 3, kWeightClasses - 1);
        planes = v.rayOut ? (unsigned)v.rays : 1u;
    }
    for (int off = 1; off < 1 << p.cornersLog2; off <<= 1) w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, off));
    if (g < totalTiles && corner == 0) {
        weights[g] = w;
        atomicAdd(counts + w, planes);
    }
    __syncthreads();
    if (threadIdx.x < kWeightClasses && counts[threadIdx.x]) atomicAdd(classes + threadIdx.x, counts[threadIdx.x]);
}

/* Each tile's slots into the order, its planes together, heavier classes first (within a class in the
 * order the atomics give): a block reserves each class's run with one global atomic, its tiles take
 * places within the run by shared ones. */
template <bool kOne>
__device__ __forceinline__ void placeTiles(const MixedParams& p, const MixedView* one, int totalTiles,
                                           const int* weights, const unsigned* classes, unsigned* cursors,
                                           uint2* order) {
    __shared__ unsigned counts[kWeightClasses], runs[kWeightClasses];
    chained();
    if (threadIdx.x < kWeightClasses) counts[threadIdx.x] = 0;
    __syncthreads();
    const int g = (int)(blockIdx.x * 128 + threadIdx.x);
    const bool active = g < totalTiles;
    int vi = 0, w = 0;
    unsigned planes = 0, within = 0;
    if (active) {
        vi = kOne ? 0 : tileView(p, g);
        w = weights[g];
        const MixedView& v = kOne ? *one : p.views[vi];
        planes = v.rayOut ? (unsigned)v.rays : 1u;
        within = atomicAdd(counts + w, planes);
    }
    __syncthreads();
    if (threadIdx.x < kWeightClasses) {
        unsigned before = 0;
        for (int c = kWeightClasses - 1; c > (int)threadIdx.x; --c) before += classes[c];
        runs[threadIdx.x] = counts[threadIdx.x] ? before + atomicAdd(cursors + threadIdx.x, counts[threadIdx.x]) : 0u;
    }
    __syncthreads();
    if (!active) return;
    const unsigned at = runs[w] + within;
    const unsigned tile = (unsigned)(g - (kOne ? one->tileBase : p.views[vi].tileBase));
    for (unsigned k = 0; k < planes; ++k) order[at + k] = make_uint2((unsigned)vi | k << 12, tile);
}

__global__ void __launch_bounds__(128) probeTable(const MixedParams p, int totalTiles, int* weights, unsigned* classes) {
    probeTiles<false>(p, nullptr, totalTiles, weights, classes);
}
__global__ void __launch_bounds__(128) probeOne(const MixedParams p, const __grid_constant__ MixedView view,
                                                int totalTiles, int* weights, unsigned* classes) {
    probeTiles<true>(p, &view, totalTiles, weights, classes);
}
__global__ void __launch_bounds__(128) placeTable(const MixedParams p, int totalTiles, const int* weights,
                                                  const unsigned* classes, unsigned* cursors, uint2* order) {
    placeTiles<false>(p, nullptr, totalTiles, weights, classes, cursors, order);
}
__global__ void __launch_bounds__(128) placeOne(const MixedParams p, const __grid_constant__ MixedView view,
                                                int totalTiles, const int* weights, const unsigned* classes,
                                                unsigned* cursors, uint2* order) {
    placeTiles<true>(p, &view, totalTiles, weights, classes, cursors, order);
}

/* The persistent trace: each warp takes slots from the queue, one ray plane of one 8 x 4 tile of pixels a
 * slot, and traces a slot's 32 rays together.  kOne: a single view, read from `one` (a kernel parameter)
 * rather than from the view table.  kSplit: the heavy slots in parts of eight rays (kernels of their own: the
 * test in the loop costs a large frame 1 %). */
template <bool kOne, bool kAll, bool kSplit = false>
__device__ __forceinline__ void mixedTiles(const MixedParams& p, const MixedView* one) {
    __shared__ unsigned tally[kMixedCount][256];
    const int lane = threadIdx.x & 31;
    unsigned rounds = 0;
    clearMixed(tally);
    chained();
    unsigned heavySlots = 0;
    if (kSplit)
        for (int c = kHeavyClass; c < kWeightClasses; ++c) heavySlots += __ldcg(p.classes + c); /* (not __ldg: a read-only load could move above the wait) */
    const MixedParts q = partsOf<kSplit>((unsigned)p.totalUnits, heavySlots, (unsigned)p.mostHeavy, p.lanesLog2);
    for (;;) {
        unsigned part = 0;
        if (lane == 0) part = (unsigned)atomicAdd(p.counters + CQueue, 1ull);
        part = __shfl_sync(0xFFFFFFFFu, part, 0);
        if (part >= q.parts) break;
        /* (a tile's rays row by row: 8 x 4 pixels a part, 8 x 2, 8 x 1, 4 x 1 or 2 x 1) */
        int lanesLog2;
        const unsigned first = partFirst<kSplit>(q, part, p.lanesLog2, lanesLog2);
        const unsigned within = (first & 31u) + (unsigned)lane;
        const int slot = (int)(first >> 5);
        const MixedView* v = kOne ? one : p.views;
        int plane, tile;
        if (p.order) {
            const uint2 s = __ldcg(p.order + slot);
            if (!kOne) v = p.views + (s.x & 4095u);
            plane = v->rayOut ? (int)(s.x >> 12) : 0;
            tile = (int)s.y;
        } else {
            const int unit = slot << 5;
            if (!kOne) v = p.views + viewOf(p, unit);
            int local = unit - v->unitBase;
            plane = v->rayOut ? local / v->pixelUnits : 0;
            local -= plane * v->pixelUnits;
            tile = local >> 5;
        }
        const int x = (tile % v->tilesX) * 8 + (int)(within & 7u);
        const int y = v->rowBegin + (tile / v->tilesX) * 4 + (int)(within >> 3);
        if (lane >> lanesLog2 == 0 && x < v->f.width && y < v->rowBegin + v->rows) {
            const size_t index = (size_t)y * (size_t)v->f.width + (size_t)x;
            const int64_t pixels = (int64_t)v->f.width * v->f.height;
            float sum[3] = {0.f, 0.f, 0.f};
            unsigned bits = 0;
            const int last = v->rayOut ? plane + 1 : v->rays;
            for (int k = plane; k < last; ++k) {
                float nx, ny, moment;
                samplePosition(v->h, v->jitter, v->seed, x, y, k, &nx, &ny, &moment);
                ArtfCudaRayEnd* end = v->ends && inBounds(v->f.fault, kBoundsRayEnd,
                                                          (int64_t)(index * (size_t)v->rays + (size_t)k),
                                                          pixels * v->rays)
                                          ? v->ends + index * (size_t)v->rays + (size_t)k
                                          : nullptr;
                bits |= classBits(traceRayMixed<kAll>(p, *v, nx, ny, v->h.disc[2] + v->h.spin[3] * moment, sum, end, tally,
                                                    rounds));
            }
            if (v->rayOut) {
                const size_t planeSize = (size_t)v->f.width * (size_t)v->rows;
                const size_t inBand = (size_t)(y - v->rowBegin) * (size_t)v->f.width + (size_t)x;
                if (inBounds(v->f.fault, kBoundsRayPlane, (int64_t)((size_t)plane * planeSize + inBand),
                             (int64_t)planeSize * v->rays))
                    v->rayOut[(size_t)plane * planeSize + inBand] = make_float4(sum[0], sum[1], sum[2], (float)bits);
            } else if (inBounds(v->f.fault, kBoundsPixel, (int64_t)index, pixels)) {
                v->hdr[index] = make_float4(sum[0] * v->share, sum[1] * v->share, sum[2] * v->share, (float)bits);
            }
        }
        __syncwarp();
    }
    flushMixed(tally, rounds, p.counters);
}

/* The views from the table (a batch).  The kernels come in pairs: the guards chosen at run time, and all
 * of them as constants, which every trace with all guards runs (frames, bands and batches alike, so that
 * their bits agree): its dead branches fold away and its code is smaller. */
__global__ void __launch_bounds__(256, 2) traceMixedTable(const MixedParams p) { mixedTiles<false, false>(p, nullptr); }
__global__ void __launch_bounds__(256, 2) traceMixedTableAll(const MixedParams p) { mixedTiles<false, true>(p, nullptr); }
__global__ void __launch_bounds__(256, 2) traceMixedTableSplit(const MixedParams p) { mixedTiles<false, true, true>(p, nullptr); }

/* A single view (a frame) as a kernel parameter: its fields are then read from the constant bank where
 * they are used, not loaded from the view table in global memory at every step. */
__global__ void __launch_bounds__(256, 2) traceMixedOne(const MixedParams p, const __grid_constant__ MixedView view) {
    mixedTiles<true, false>(p, &view);
}
__global__ void __launch_bounds__(256, 2) traceMixedOneAll(const MixedParams p, const __grid_constant__ MixedView view) {
    mixedTiles<true, true>(p, &view);
}
__global__ void __launch_bounds__(256, 2) traceMixedOneSplit(const MixedParams p, const __grid_constant__ MixedView view) {
    mixedTiles<true, true, true>(p, &view);
}

/* Each pixel of the views with ray planes: its rays' radiance summed in ray order and scaled by
 * 1 / rays, and their class bits; the same operations, in the same order, as the per-pixel path. */
__device__ __forceinline__ void combinePlanes(const MixedView& v) {
    chained();
    if (!v.rayOut) return;
    const size_t pixels = (size_t)v.f.width * (size_t)v.rows; /* the band's */
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= pixels) return;
    float sum[3] = {0.f, 0.f, 0.f};
    unsigned bits = 0;
    for (int k = 0; k < v.rays; ++k) {
        const float4 q = v.rayOut[(size_t)k * pixels + i];
        sum[0] = sum[0] + q.x, sum[1] = sum[1] + q.y, sum[2] = sum[2] + q.z;
        bits |= (unsigned)q.w;
    }
    const size_t at = (size_t)v.rowBegin * (size_t)v.f.width + i;
    if (inBounds(v.f.fault, kBoundsPixel, (int64_t)at, (int64_t)v.f.width * v.f.height))
        v.hdr[at] = make_float4(sum[0] * v.share, sum[1] * v.share, sum[2] * v.share, (float)bits);
}

__global__ void __launch_bounds__(256) combineTable(const MixedView* views) { combinePlanes(views[blockIdx.y]); }
__global__ void __launch_bounds__(256) combineOne(const __grid_constant__ MixedView view) { combinePlanes(view); }

/* The per-ray entry point: rays at given image positions in a view. */
__global__ void __launch_bounds__(128) traceMixedList(const MixedParams p,
                                                      const __grid_constant__ MixedView view, const int count,
                                                      const float* nx, const float* ny, const float* time, float* rgb) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    __shared__ unsigned tally[kMixedCount][256];
    unsigned rounds = 0;
    clearMixed(tally);
    if (i < count) {
        float sum[3] = {0.f, 0.f, 0.f};
        traceRayMixed<false>(p, view, nx[i], ny[i], time[i], sum, view.ends ? view.ends + i : nullptr, tally, rounds);
        for (int k = 0; k < 3; ++k) rgb[3 * i + k] = sum[k];
    }
    __syncwarp();
    flushMixed(tally, rounds, p.counters);
}

MixedParams paramsOf(const TraceLaunch& l, const void* deviceTable, int viewCount, int totalUnits) {
    MixedParams p;
    p.views = (const MixedView*)deviceTable;
    p.viewCount = viewCount;
    p.totalUnits = totalUnits;
    p.counters = l.counters;
    p.stepScale = l.stepScale;
    p.maxSteps = l.stepScale < .75f ? 384 : 192;
    p.guards = l.guards ? l.guards : ARTF_CUDA_GUARD_ALL;
    p.order = nullptr;
    p.classes = nullptr;
    p.cornersLog2 = p.mostHeavy = 0;
    return p;
}

}  // namespace

namespace {

/* widen against the hardware's float-to-double conversion, on every float bit pattern (256 a thread);
 * bad[0] counts differing results (two NaNs agree), bad[2] keeps the least differing input. */
__global__ void __launch_bounds__(256) checkWiden(unsigned long long* bad) {
    const uint32_t first = (blockIdx.x * 256u + threadIdx.x) << 8;
    for (uint32_t k = 0; k < 256u; ++k) {
        const float f = __uint_as_float(first | k);
        const double want = (double)f, got = widen(f);
        const bool same = (want != want && got != got) || __double_as_longlong(want) == __double_as_longlong(got);
        if (!same) {
            atomicAdd(bad, 1ull);
            atomicMin(bad + 2, (unsigned long long)(first | k));
        }
    }
}

__device__ __forceinline__ unsigned long long mixBits(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

/* narrow against the hardware's double-to-float conversion, on `perThread` doubles a thread: exponents
 * around float's range and random fractions, a quarter of them with the 29 bits rounding looks at set
 * to a tie or next to one, an eighth with the kept bits all ones; one in sixteen a random bit pattern.
 * bad[1] counts differing results, bad[3] keeps the least differing input. */
__global__ void __launch_bounds__(256) checkNarrow(unsigned long long* bad, uint32_t perThread) {
    const unsigned long long id = blockIdx.x * 256ull + threadIdx.x;
    for (uint32_t k = 0; k < perThread; ++k) {
        const unsigned long long r = mixBits(id * perThread + k), s = mixBits(r);
        unsigned long long bits;
        if ((r & 15u) == 0u) {
            bits = s;
        } else {
            const unsigned long long e = 880u + (r >> 8) % 290u;
            unsigned long long fraction = s & 0xFFFFFFFFFFFFFull;
            const uint32_t rests[4] = {0x10000000u, 0x0FFFFFFFu, 0x10000001u, 0u};
            if (((r >> 4) & 3u) == 0u) fraction = (fraction & ~0x1FFFFFFFull) | rests[(r >> 6) & 3u];
            if (((r >> 20) & 7u) == 0u) fraction |= 0x7FFFFFull << 29;
            bits = ((r >> 63) << 63) | (e << 52) | fraction;
        }
        const double d = __longlong_as_double((long long)bits);
        const float want = (float)d, got = narrow(d);
        const bool same = (want != want && got != got) || __float_as_uint(want) == __float_as_uint(got);
        if (!same) {
            atomicAdd(bad + 1, 1ull);
            atomicMin(bad + 3, bits);
        }
    }
}

}  // namespace

size_t mixedViewBytes() { return sizeof(MixedView); }

int mixedFillView(const TraceLaunch& l, const ArtfCudaHoleFrame& frame, const ArtfCudaHoleFrame64& frame64,
                  const float* map, const float* fluid, float4* hdr, ArtfCudaRayEnd* ends, float4* rayOut, int unitBase,
                  int tileBase, void* slot, int* tiles) {
    MixedView v;
    memset(&v, 0, sizeof v);
    v.f.load(frame64, frame);
    v.d.load(frame64, frame);
    v.f.fault = v.d.fault = l.counters + CBoundsKind;
    v.h = frame;
    v.map = map;
    v.fluid = fluid;
    v.hdr = hdr;
    v.ends = ends;
    v.wideA2 = v.d.a * v.d.a;
    v.start64 = startTerms(v.d, (double)l.stepScale);
    for (int k = 0; k < 3; ++k) v.startNarrow[k] = (float)v.d.er[k];
    v.startNarrow[3] = (float)v.d.place[2];
    v.wScaleNarrow = (float)v.start64.wScale;
    v.stepBaseNarrow = (float)v.start64.stepBase;
    auto split = [](double x) {
        const float hi = (float)x;
        return Ff{hi, (float)(x - (double)hi)};
    };
    for (int k = 0; k < 3; ++k) {
        v.motion.forward[k] = split(v.d.forward[k]);
        v.motion.right[k] = split(v.d.right[k]);
        v.motion.up[k] = split(v.d.up[k]);
    }
    for (int k = 0; k < 4; ++k) v.motion.metric[k] = split(v.d.metric[k]);
    v.motion.rho = split(v.d.place[0]), v.motion.a = split(v.d.a), v.motion.a2 = split(v.start64.a2);
    v.motion.mu0Squared = split(v.start64.mu0Squared), v.motion.minusTwoA2 = split(v.start64.minusTwoA2);
    v.rhoScale = 1.f / (1.f - v.f.inner / v.f.outer);
    v.uGuard = (float)((double)(l.horizonBand > 0.f ? l.horizonBand : .95f) * frame64.spin[1]);
    v.rays = l.jitter ? l.jitter : (int)(frame.size[2] * frame.size[2]);
    v.share = l.jitter ? 1.f / (float)l.jitter : frame.image[3];
    v.jitter = l.jitter;
    v.seed = l.seed;
    v.tilesX = ((int)frame.size[0] + 7) / 8;
    const int tileRows = ((int)frame.size[1] + 3) / 4;
    const int bandBegin = l.tileRows > 0 ? l.tileRowBegin : 0, bandRows = l.tileRows > 0 ? l.tileRows : tileRows;
    v.rowBegin = bandBegin * 4;
    v.rows = (bandBegin + bandRows) * 4 < (int)frame.size[1] ? bandRows * 4 : (int)frame.size[1] - v.rowBegin;
    v.pixelUnits = v.tilesX * bandRows * 32;
    v.rayOut = v.rays > 1 ? rayOut : nullptr; /* (one ray a pixel: the pixel is the ray) */
    v.units = v.pixelUnits * (v.rayOut ? v.rays : 1);
    v.unitBase = unitBase;
    v.tileBase = tileBase;
    memcpy(slot, &v, sizeof v);
    *tiles = v.tilesX * bandRows;
    return v.units;
}

/* The heavy-first scratch: the weight classes' counts and cursors, a weight a tile, a slot a 32 units. */
constexpr size_t kOrderHead = 2 * 32 * sizeof(unsigned);

size_t mixedOrderBytes(int totalTiles, int totalUnits) {
    const size_t weights = ((size_t)totalTiles * sizeof(int) + 15) & ~(size_t)15;
    return kOrderHead + weights + (size_t)(totalUnits / 32) * sizeof(uint2);
}

static MixedGrid mixedGrid(const TraceLaunch& l, int totalUnits, const void* kernel) {
    const int block = l.blockSize > 0 ? l.blockSize : 128;
    int perSm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, block, 0);
    return mixedGridOf(totalUnits, block, perSm, l.smCount, l.refillBatch);
}

/* A launch that may start while the stream's work before it drains: kernels that wait in chained(). */
template <typename... P, typename... A>
static cudaError_t follow(cudaStream_t stream, void (*kernel)(P...), dim3 grid, int block, const A&... args) {
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid, c.blockDim = dim3((unsigned)block), c.stream = stream, c.attrs = &early, c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, P(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError(); /* (or the next launch's check would report it) */
    return e;
}

cudaError_t launchMixedTable(const TraceLaunch& l, const void* deviceTable, int viewCount, int totalUnits,
                             size_t combinePixels, int totalTiles, void* orderScratch, const void* hostView) {
    MixedParams p = paramsOf(l, deviceTable, viewCount, totalUnits);
    const int block = l.blockSize > 0 ? l.blockSize : 128;
    const bool single = hostView && viewCount == 1, all = p.guards == ARTF_CUDA_GUARD_ALL;
    MixedView one;
    if (single) memcpy(&one, hostView, sizeof one);
    if (l.rayCount > 0) {
        if (!single) return cudaErrorInvalidValue;
        traceMixedList<<<(l.rayCount + 127) / 128, 128, 0, l.stream>>>(p, one, l.rayCount, l.rayX, l.rayY, l.rayTime,
                                                                       l.rayRgb);
        return cudaGetLastError();
    }
    const void* kernel = single ? (all ? (const void*)traceMixedOneAll : (const void*)traceMixedOne)
                                : (all ? (const void*)traceMixedTableAll : (const void*)traceMixedTable);
    MixedGrid grid = mixedGrid(l, totalUnits, kernel);
    p.lanesLog2 = grid.lanesLog2;
    const bool ordered = orderScratch && l.order == ARTF_CUDA_ORDER_HEAVY_FIRST && totalTiles > 0;
    const bool split = ordered && all && grid.mostHeavy > 0;
    cudaError_t e = cudaSuccess;
    if (ordered && (split || !grid.resident)) {
        unsigned* classes = (unsigned*)orderScratch;
        unsigned* cursors = classes + 32;
        int* weights = (int*)((char*)orderScratch + kOrderHead);
        uint2* order = (uint2*)((char*)weights + (((size_t)totalTiles * sizeof(int) + 15) & ~(size_t)15));
        e = cudaMemsetAsync(orderScratch, 0, kOrderHead, l.stream);
        if (e != cudaSuccess) return e;
        const unsigned tiles = (unsigned)((totalTiles + 127) / 128);
        if (split) {
            p.classes = classes;
            p.mostHeavy = grid.mostHeavy;
            p.cornersLog2 = kCornersLog2;
            grid.blocks = grid.most;
        }
        const unsigned probes = (unsigned)((((long long)totalTiles << p.cornersLog2) + 127) / 128);
        if (single) {
            probeOne<<<probes, 128, 0, l.stream>>>(p, one, totalTiles, weights, classes);
            e = follow(l.stream, placeOne, dim3(tiles), 128, p, one, totalTiles, weights, classes, cursors, order);
        } else {
            probeTable<<<probes, 128, 0, l.stream>>>(p, totalTiles, weights, classes);
            e = follow(l.stream, placeTable, dim3(tiles), 128, p, totalTiles, weights, classes, cursors, order);
        }
        p.order = order;
    }
    const dim3 blocks((unsigned)grid.blocks);
    if (e == cudaSuccess && single)
        e = follow(l.stream, split ? traceMixedOneSplit : all ? traceMixedOneAll : traceMixedOne, blocks, block, p, one);
    else if (e == cudaSuccess)
        e = follow(l.stream, split ? traceMixedTableSplit : all ? traceMixedTableAll : traceMixedTable, blocks, block, p);
    if (e == cudaSuccess && combinePixels > 0) {
        const unsigned sums = (unsigned)((combinePixels + 255) / 256);
        if (single) e = follow(l.stream, combineOne, dim3(sums), 256, one);
        else e = follow(l.stream, combineTable, dim3(sums, (unsigned)viewCount), 256, p.views);
    }
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace artf

namespace artf {
int failWith(int status, const char* message);

namespace {
/* The pair arithmetic the wide sub-steps use, one record a thread: (a.hi, a.lo, b.hi, b.lo) in,
 * a + b, a b, 1 / a and 1 / sqrt(|a|) out, each as (hi, lo). */
__global__ void checkPairs(const float4* in, float* out, int count) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= count) return;
    const float4 r = in[i];
    const Ff a{r.x, r.y}, b{r.z, r.w};
    const Ff sum = ffAdd(a, b), product = ffMul(a, b), recip = ffRecip(a);
    const Ff root = ffRsqrt(Ff{fabsf(a.hi), a.hi < 0.f ? -a.lo : a.lo});
    float* o = out + (size_t)i * 8;
    o[0] = sum.hi, o[1] = sum.lo, o[2] = product.hi, o[3] = product.lo;
    o[4] = recip.hi, o[5] = recip.lo, o[6] = root.hi, o[7] = root.lo;
}
}  // namespace
}  // namespace artf

extern "C" int artfCudaCheckPairs(void* stream, const float* hostIn, int count, float* hostOut) {
    if (!hostIn || !hostOut || count < 1 || count > (1 << 24))
        return artf::failWith(ARTF_CUDA_EINVAL, "pairs check: inputs, outputs and 1 .. 2^24 records");
    const cudaStream_t s = (cudaStream_t)stream;
    void* buffer = nullptr;
    const size_t inBytes = sizeof(float) * 4 * (size_t)count, outBytes = sizeof(float) * 8 * (size_t)count;
    cudaError_t e = cudaMalloc(&buffer, inBytes + outBytes);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return artf::failWith(ARTF_CUDA_ENOMEM, "pairs check: device allocation");
    }
    float4* in = (float4*)buffer;
    float* out = (float*)((char*)buffer + inBytes);
    e = cudaMemcpyAsync(in, hostIn, inBytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        artf::checkPairs<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(in, out, count);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(hostOut, out, outBytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(buffer);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    return ARTF_CUDA_OK;
}

extern "C" int artfCudaCheckConversions(void* stream, uint64_t narrowCount, uint64_t* mismatches) {
    if (!mismatches) return artf::failWith(ARTF_CUDA_EINVAL, "mismatches is NULL");
    const cudaStream_t s = (cudaStream_t)stream;
    unsigned long long* bad = nullptr;
    cudaError_t e = cudaMalloc(&bad, sizeof(unsigned long long) * 4);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ENOMEM, "conversion check: device allocation");
    const unsigned long long init[4] = {0ull, 0ull, ~0ull, ~0ull};
    e = cudaMemcpyAsync(bad, init, sizeof init, cudaMemcpyHostToDevice, s);
    const uint32_t threads = 1u << 20;
    const uint32_t perThread = (uint32_t)((narrowCount + threads - 1) / threads);
    if (e == cudaSuccess) {
        artf::checkWiden<<<1u << 16, 256, 0, s>>>(bad); /* 2^24 threads x 256: every float */
        if (perThread > 0) artf::checkNarrow<<<threads / 256, 256, 0, s>>>(bad, perThread);
        e = cudaGetLastError();
    }
    unsigned long long out[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, bad, sizeof out, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(bad);
    if (e != cudaSuccess) return artf::failWith(ARTF_CUDA_ELAUNCH, cudaGetErrorString(e));
    for (int k = 0; k < 4; ++k) mismatches[k] = out[k];
    return ARTF_CUDA_OK;
}
