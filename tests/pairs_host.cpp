/* The mixed trace's double-float arithmetic (lensPairs.cuh) on the host: how far a ray's constants of motion and a
 * coordinate's step at a turning point are from their exact values (long double), beside the same in pairs that are
 * renormalised at every operation, over rays of eyes spread over the scenes' range.  Prints "name value" lines: an
 * error's median, 99 and 99.9 % quantiles as multiples of the renormalised pairs', and its median's base-2
 * logarithm. */
#include "artful_cuda.h"
#include "lensCore.cuh"
#include "lensPairs.cuh"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

using namespace artf;
typedef long double L;

static uint64_t state = 1;
static double uniform(double lo, double hi) {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return lo + (hi - lo) * (double)(state >> 11) * 0x1p-53;
}
static L value(Ff a) { return (L)a.hi + (L)a.lo; }
static Ff split(double x) {
    const float hi = (float)x;
    return Ff{hi, (float)(x - (double)hi)};
}

/* ---- the yardstick: Dekker's pairs, every result renormalised ------------------------------------- */

namespace full {
static Ff add(Ff a, Ff b) {
    const Ff s = ffSum(a.hi, b.hi);
    return ffNorm(s.hi, s.lo + (a.lo + b.lo));
}
static Ff sub(Ff a, Ff b) { return add(a, ffNeg(b)); }
static Ff mul(Ff a, Ff b) {
    const Ff p = ffProd(a.hi, b.hi);
    return ffNorm(p.hi, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo)));
}
static Ff mul(Ff a, float b) { return mul(a, Ff{b, 0.f}); }
static Ff recip(Ff x) {
    const float y = 1.f / x.hi;
    return ffNorm(y, y * sub(Ff{1.f, 0.f}, mul(x, y)).hi);
}
static Ff rsqrt(Ff x) {
    const float y = 1.f / sqrtf(x.hi);
    return ffNorm(y, .5f * y * sub(Ff{1.f, 0.f}, mul(mul(x, y), y)).hi);
}
static Ff cubic(const Cubic& f, Ff x) { return mul(x, add(f.A, mul(x, add(f.B, mul(x, f.C))))); }
static Motion motion(const Cubic& f, float step, float x, float v) {
    const Ff h2 = ffProd(step, step), sixth = ffProd(step, 1.f / 6.f), at{x, 0.f}, rate{v, 0.f};
    const Ff k1 = cubic(f, at), k2 = cubic(f, add(add(at, ffProd(step * .5f, v)), mul(mul(h2, .125f), k1)));
    const Ff xv = add(at, ffProd(step, v)), k3 = cubic(f, add(xv, mul(mul(h2, .5f), k2)));
    return Motion{add(xv, mul(mul(h2, 1.f / 6.f), add(k1, add(k2, k2)))),
                  add(rate, mul(sixth, add(add(k1, k3), mul(k2, 4.f)))), k1};
}
static MotionFf constants(const MotionTermsFf& t, float nx, float ny) {
    MotionFf m;
    Ff d[3];
    for (int k = 0; k < 3; ++k) d[k] = add(add(t.forward[k], mul(t.right[k], nx)), mul(t.up[k], ny));
    const Ff inv = rsqrt(add(add(mul(d[0], d[0]), mul(d[1], d[1])), mul(d[2], d[2]))), dz = mul(d[2], inv);
    m.invEnergy = recip(sub(t.metric[0], mul(t.metric[1], dz)));
    m.dx = d[0], m.over = mul(inv, m.invEnergy);
    m.xi = ffNeg(mul(mul(t.metric[2], dz), m.invEnergy));
    m.xiAxis = mul(mul(t.metric[3], d[2]), m.over), m.across = mul(mul(t.rho, d[1]), m.over);
    const Ff eta = add(mul(m.across, m.across), mul(t.mu0Squared, sub(mul(m.xiAxis, m.xiAxis), t.a2)));
    const Ff off = sub(m.xi, t.a);
    m.big = add(eta, mul(m.xi, m.xi)), m.uA = sub(t.a2, m.big), m.uB = mul(add(eta, mul(off, off)), 3.f);
    m.uC = mul(t.minusTwoA2, eta), m.xiA = mul(m.xi, t.a);
    return m;
}
}  // namespace full

/* ---- errors -------------------------------------------------------------------------------------- */

struct Errors {
    const char* name;
    std::vector<double> ours, yard;
    void add(Ff a, Ff b, L want, L scale) {
        ours.push_back((double)(fabsl(value(a) - want) / scale)), yard.push_back((double)(fabsl(value(b) - want) / scale));
    }
    static double at(std::vector<double>& e, double q) {
        const size_t k = (size_t)(q * (double)e.size());
        std::nth_element(e.begin(), e.begin() + (ptrdiff_t)k, e.end());
        return e[k];
    }
    void print() {
        printf("%s_count %zu\n%s_log2 %.2f\n", name, ours.size(), name, log2(at(ours, .5)));
        printf("%s_median %.5f\n%s_99 %.5f\n%s_999 %.5f\n", name, at(ours, .5) / at(yard, .5), name,
               at(ours, .99) / at(yard, .99), name, at(ours, .999) / at(yard, .999));
    }
};
static Errors invEnergy{"invEnergy"}, xi{"xi"}, big{"big"}, uA{"uA"}, uB{"uB"}, uC{"uC"}, xiA{"xiA"};
static Errors step[2][3] = {{{"radial_x"}, {"radial_v"}, {"radial_first"}}, {{"polar_x"}, {"polar_v"}, {"polar_first"}}};
static long loose = 0;
static L axis = 0; /* the worst error of n_z's cubic */

static void kept(Ff a) { loose += (float)((double)a.hi + (double)a.lo) != a.hi; }

/* A coordinate's step where its rate turns, errors against the size of the terms. */
static void turn(Errors* e, const Cubic& f, float h, float x, float v) {
    const Motion a = motionFf(f, h, x, v), b = full::motion(f, h, x, v);
    const L A = value(f.A), B = value(f.B), C = value(f.C), h2 = (L)h * h, sixth = (L)(1.f / 6.f);
    auto cubic = [&](L y) { return y * (A + y * (B + y * C)); };
    const L k1 = cubic(x), k2 = cubic(x + .5L * h * v + h2 / 8 * k1), xv = x + (L)h * v, k3 = cubic(xv + h2 / 2 * k2);
    const L wantX = xv + h2 * sixth * (k1 + 2 * k2), wantV = v + h * sixth * (k1 + k3 + 4 * k2);
    const L size = fabsl(x) * (fabsl(A) + fabsl(x) * (fabsl(B) + fabsl(x * C)));
    kept(a.x), kept(a.v), kept(a.first);
    e[0].add(a.x, b.x, wantX, fabsl(wantX));
    e[1].add(a.v, b.v, wantV, fabsl(v) + h * size);
    e[2].add(a.first, b.first, k1, size);
}

/* Doubles from the float they round to and their rest, every exponent a step can have. */
static long lostBits() {
    long lost = 0;
    for (int k = 0; k < 1000000; ++k) {
        const double x = std::ldexp(uniform(1, 2), (int)uniform(-60, 20));
        const float f = (float)x;
        lost += withRest((double)f, restOf(x, (double)f)) != x;
    }
    return lost;
}

int main() {
    printf("lost %ld\n", lostBits());
    for (int eye = 0; eye < 96; ++eye) {
        ArtfCudaHoleParams p = {};
        p.spin = uniform(-.5, .998), p.inclination = uniform(5, 89) * 3.14159265358979 / 180, p.innerScale = 1;
        p.emissivity = 3, p.distance = uniform(20, 80), p.fovY = .6, p.outer = 12, p.height = 1e-3, p.thickness = 1;
        p.gain = p.doppler = p.stars = 1;
        ArtfCudaHoleFrame f32;
        ArtfCudaHoleFrame64 f;
        if (artfCudaHoleParamsFrames(&p, 1920, 1080, &f32, &f, nullptr) != ARTF_CUDA_OK) return 1;
        const double a = f.spin[0], a2 = a * a;
        MotionTermsFf t;
        for (int k = 0; k < 3; ++k) t.forward[k] = split(f.forward[k]), t.right[k] = split(f.right[k]), t.up[k] = split(f.up[k]);
        for (int k = 0; k < 4; ++k) t.metric[k] = split(f.metric[k]);
        t.rho = split(f.place[0]), t.a = split(a), t.a2 = split(a2);
        t.mu0Squared = split(f.place[3] * f.place[3]), t.minusTwoA2 = split(-2 * a2);
        Frame<float> frame;
        frame.load(f, f32);
        for (int ray = 0; ray < 2000; ++ray) {
            const float nx = (float)uniform(-1, 1), ny = (float)uniform(-1, 1);
            const MotionFf m = motionConstantsFf(t, nx, ny), y = full::constants(t, nx, ny);
            for (Ff v : {m.invEnergy, m.xi, m.big, m.uA, m.uB, m.uC, m.xiA, m.dx, m.over, m.across, m.xiAxis}) kept(v);
            L d[3], length2 = 0;
            for (int k = 0; k < 3; ++k)
                d[k] = value(t.forward[k]) + value(t.right[k]) * nx + value(t.up[k]) * ny, length2 += d[k] * d[k];
            const L inv = 1 / sqrtl(length2), dz = d[2] * inv, e = 1 / (value(t.metric[0]) - value(t.metric[1]) * dz);
            const L x = -value(t.metric[2]) * dz * e, xiAxis = value(t.metric[3]) * dz * e, across = value(t.rho) * d[1] * inv * e;
            const L eta = across * across + value(t.mu0Squared) * (xiAxis * xiAxis - value(t.a2)), K = eta + x * x;
            const L off = x - value(t.a), A = value(t.a2) - K, B = 3 * (eta + off * off), C = value(t.minusTwoA2) * eta;
            invEnergy.add(m.invEnergy, y.invEnergy, e, fabsl(e)), xi.add(m.xi, y.xi, x, fabsl(x));
            big.add(m.big, y.big, K, fabsl(K)), uA.add(m.uA, y.uA, A, fabsl(A)), uB.add(m.uB, y.uB, B, fabsl(B));
            uC.add(m.uC, y.uC, C, fabsl(C)), xiA.add(m.xiA, y.xiA, x * value(t.a), fabsl(x * value(t.a)));
            /* n_z's cubic with constants in pairs, and with float ones, as the ray has them without that guard */
            const float floatK = m.big.hi, floatA = (float)(a2 - (double)floatK);
            const Cubic paired = axisCubic(t.a2, m.uA, m.big.hi, true), plain = axisCubic(t.a2, Ff{floatA, 0.f}, floatK, false);
            axis = fmaxl(axis, fabsl(value(paired.A) - value(m.uA)) / fabsl(A));
            axis = fmaxl(axis, fabsl(value(plain.A) - (value(t.a2) - floatK)) / (value(t.a2) + fabsl((L)floatK)));
            axis = fmaxl(axis, fabsl(value(paired.C) + 2 * value(t.a2)) + fabsl(value(paired.B)));
            /* the ray in float, to where its rates turn */
            RayConst<float> c;
            RayState<float> s;
            rayStart(frame, nx, ny, 0.f, 1.f, c, s);
            for (int i = 0; i < 192; ++i) {
                StepOut<float> o;
                nystromStep((float)a, c, s, o);
                if ((s.w > 0) != (o.next.w > 0)) turn(step[0], Cubic{m.uA, m.uB, m.uC}, c.step, s.u, s.w);
                if ((s.v[2] > 0) != (o.next.v[2] > 0))
                    turn(step[1], paired, c.step, s.n[2], s.v[2]);
                if (o.next.u < 0 || o.next.u > frame.uHorizon) break;
                s = o.next;
            }
        }
    }
    for (Errors* e : {&invEnergy, &xi, &big, &uA, &uB, &uC, &xiA}) e->print();
    for (auto& kind : step)
        for (Errors& e : kind) e.print();
    printf("loose %ld\naxis_log2 %.2f\n", loose, axis > 0 ? (double)log2l(axis) : -99.);
    return 0;
}
