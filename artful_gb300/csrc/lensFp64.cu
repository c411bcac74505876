/* artful_cuda — the plain FP64 trace: the reference's integrator with every operation in double,
 * from the frame computed in double.  The FP64 GPU oracle the mixed-precision trace is measured against
 * (and, at half step, the discretisation reference). */
#define ARTF_FAST_FP64 1 /* FP64 division and square roots by refined hardware estimates (lensCore.cuh) */
#include "lensKernel.cuh"

namespace artf {
namespace {

/* 1 / x from the hardware's 20-bit estimate y by one iteration of third order, y (1 + e + e^2) with
 * e = 1 - x y: past 53 bits in three operations, where two of second order take four. */
__device__ __forceinline__ double recipCubic(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

/* The greater of x and a positive bound, compared as integers (a positive double's bits rise with it): a
 * double comparison takes the FP64 pipe. */
__device__ __forceinline__ double atLeast(double x, double bound) {
    return __double_as_longlong(x) > __double_as_longlong(bound) ? x : bound;
}

/* One ray in double.  What bounds it is the FP64 pipe, two lanes a cycle an SM: an instruction holds it 16
 * cycles whatever it does, so the step is arranged for the fewest of them, 79 where the shared integrator's
 * expressions take 106.  Rates carry the step (h w, h v) and the coefficients its square, so that the
 * stages' factors are constants; n_x and n_y go through the stages by the same linear map, formed once
 * (n' = A n + B v, v' = D v - C n); the drag rates' polynomials are factored, their reciprocals of third
 * order; and every test a step makes is on integers, the double test behind it.  The differences from the
 * expressions as written are in the last bits of double, and the image is rounded to float.
 * 960 x 540: 2877 -> 2381 us, the pipe 87 % busy. */
template <>
__device__ __forceinline__ unsigned traceRay(const KernelParams<double>& p, double nx, double ny, double time,
                                             double* sum, ArtfCudaRayEnd* end, Tallies& t) {
    const Frame<double>& f = p.f;
    constexpr double S = (double)(1.f / 6.f); /* (the reference's sixth: a float) */
    RayConst<double> c;
    RayState<double> s;
    rayStart(f, nx, ny, time, p.stepScale, c, s);
    const double a = f.a, a2 = a * a, h = c.step, h2 = h * h;
    const double uA = h2 * c.uA, uB = h2 * c.uB, uC = h2 * c.uC;
    const double big = h2 * c.big, twoA2 = 2.0 * (h2 * a2), bigZ = big - h2 * a2;
    const double dragOne = -2.0 * a, dragTwo = a * c.xiA, sixth = h * S;
    const double rhoScale = recipR(1.0 - divR(f.inner, f.outer));
    const long long horizon = __double_as_longlong(f.uHorizon);
    double u = s.u, w = h * s.w, n0 = s.n[0], n1 = s.n[1], z = s.n[2];
    double v0 = h * s.v[0], v1 = h * s.v[1], vz = h * s.v[2], psi = 0.0;
    auto dragOf = [&](double x) {
        const double den = atLeast(fma(x, fma(a2, x, -2.0), 1.0), (double)1e-3f);
        return x * fma(dragTwo, x, dragOne) * recipCubic(den);
    };
    double drag = dragOf(u);

    double raySum[3] = {0.0, 0.0, 0.0}, through = 1.0;
    unsigned kind = ARTF_CUDA_END_CAP, crossings = 0;
    if (end) {
        end->hitR = end->hitPhi = NAN;
        for (int k = 0; k < 3; ++k) end->dir[k] = 0.f;
        end->mino = (float)((double)p.maxSteps * h);
    }
    int i = 0;
    while (i < p.maxSteps) {
        /* the radial part */
        const double k1 = u * fma(u, fma(u, uC, uB), uA);
        const double midU = fma(.125, k1, fma(.5, w, u));
        const double k2 = midU * fma(midU, fma(midU, uC, uB), uA);
        const double uw = u + w, endU = fma(.5, k2, uw);
        const double k3 = endU * fma(endU, fma(endU, uC, uB), uA);
        const double nextU = fma(S, fma(2.0, k2, k1), uw), nextW = fma(S, fma(4.0, k2, k1 + k3), w);
        const double nextDrag = dragOf(nextU);
        const double nextPsi = fma(sixth, fma(4.0, dragOf(midU), drag + nextDrag), psi);
        /* the axis component: z'' = -(K - a^2 + 2 a^2 z^2) z */
        const double z1 = z * z, b1 = -(z * fma(twoA2, z1, bigZ));
        const double midZ = fma(.125, b1, fma(.5, vz, z)), z2 = midZ * midZ, b2 = -(midZ * fma(twoA2, z2, bigZ));
        const double zv = z + vz, endZ = fma(.5, b2, zv), z3 = endZ * endZ, b3 = -(endZ * fma(twoA2, z3, bigZ));
        const double nextZ = fma(S, fma(2.0, b2, b1), zv), nextVz = fma(S, fma(4.0, b2, b1 + b3), vz);
        /* the components about the axis */
        const double c1 = fma(twoA2, z1, big), c2 = fma(twoA2, z2, big), c3 = fma(twoA2, z3, big);
        const double q = c2 * fma(-.125, c1, 1.0);
        const double A = fma(-S, fma(2.0, q, c1), 1.0), B = fma(-S, c2, 1.0);
        const double C = S * fma(4.0, q, fma(c3, fma(-.5, q, 1.0), c1));
        const double D = fma(-S, fma(c3, fma(-.25, c2, 1.0), c2 + c2), 1.0);
        const double next0 = fma(B, v0, A * n0), next1 = fma(B, v1, A * n1);
        const double nextV0 = fma(D, v0, -(C * n0)), nextV1 = fma(D, v1, -(C * n1));
        ++i;
        bool opaque = false;
        if ((__double2hiint(z) ^ __double2hiint(nextZ)) < 0) {
            const double inv = recipCubic(h), inv2 = inv * inv;
            RayState<double> from;
            StepOut<double> o;
            from.u = u, from.w = w * inv, from.n[0] = n0, from.n[1] = n1, from.n[2] = z, from.psi = psi, from.drag = drag;
            from.v[0] = v0 * inv, from.v[1] = v1 * inv, from.v[2] = vz * inv;
            o.next.n[2] = nextZ, o.next.psi = nextPsi, o.next.drag = nextDrag;
            o.k1 = k1 * inv2, o.a1[0] = -c1 * n0 * inv2, o.a1[1] = -c1 * n1 * inv2, o.a1[2] = b1 * inv2;
            Crossing<double> x;
            if (crossingOf(f, rhoScale, c, from, o, x)) {
                ++crossings;
                double turn;
                const double light = shadeCrossing(f, rhoScale, p.map, p.fluid, c, x, through, raySum, &turn);
                if (light > 0.0 && !(kind & ARTF_CUDA_END_LIT)) {
                    kind |= ARTF_CUDA_END_LIT;
                    if (end) end->hitR = (float)recipR(x.uc), end->hitPhi = (float)(turn - floor(turn));
                }
                opaque = !(through > (double).004f);
            }
        }
        if (__double2hiint(nextU) < 0 && 0.0 > nextU) {
            const double part = divR(u, u - nextU), away[3] = {fma(part, next0 - n0, n0), fma(part, next1 - n1, n1),
                                                               fma(part, nextZ - z, z)};
            double dir[3];
            skyDirection(away, fma(part, nextPsi - psi, psi), dir);
            if (f.stars > 0.0) shadeSky(f, p.map, c, dir, through, raySum);
            kind ^= ARTF_CUDA_END_CAP ^ ARTF_CUDA_END_SKY;
            if (end) {
                for (int k = 0; k < 3; ++k) end->dir[k] = (float)dir[k];
                end->mino = (float)(((double)(i - 1) + part) * h);
            }
            break;
        }
        const bool fell = __double_as_longlong(nextU) > horizon && nextU > f.uHorizon;
        if (fell || opaque) {
            kind ^= ARTF_CUDA_END_CAP ^ (fell ? ARTF_CUDA_END_HORIZON : ARTF_CUDA_END_OPAQUE);
            if (end) end->mino = (float)((double)i * h);
            break;
        }
        u = nextU, w = nextW, drag = nextDrag, psi = nextPsi;
        n0 = next0, n1 = next1, z = nextZ, v0 = nextV0, v1 = nextV1, vz = nextVz;
    }
    for (int k = 0; k < 3; ++k) sum[k] = sum[k] + raySum[k];
    finishRay(i, crossings, kind, i, end, t);
    return kind;
}

}  // namespace

cudaError_t launchFp64(const TraceLaunch& l) { return launchUniform<double>(l, &l.frame64); }
}  // namespace artf
