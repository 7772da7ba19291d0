// Andersen's QE-M step in double for the pair-of-lanes kernel (qe_pair_kernel), with its own elementary functions.
//
// The step is schemes.hpp:153-186 in a form with one division on the variance's chain where the textbook form has
// three divisions and three roots. With m, s2 the conditional mean and variance, u = psi / 2 = s2 / (2 m^2):
//   quadratic (psi <= 3/2): with q = sqrt(1 - u) and p = 1 - q, Andersen's a = m p and b^2 = q / p, so
//     v' = a (b + z)^2 = m (q + z (2 sqrt(q p) + z p)),  a b^2 = m q
//     K0 = -A m q / d + 1/2 ln d,  d = 1 - 2 A m p
//   exponential: 1 - p_0 = 1 / (u + 1/2), 1 / beta = m (u + 1/2), so with the tail T = 1 - U = Phi(-z)
//     v' = -ln((u + 1/2) T) m (u + 1/2) where (u + 1/2) T < 1, else 0
//     K0 = -ln(1 + A m / d),  d = 1 - A m (u + 1/2)
// p = 1 - sqrt(1 - u) is taken to a relative rounding by one Newton step on p^2 - 2 p + u = 0 (for small psi the
// difference alone would lose digits). Every lane computes both branches and keeps its own: the warps of a Heston
// book mix them at nearly every step, and straight-line code lets the log-spot's part (the division, logarithm and
// root that v' does not wait for) and the next draws overlap the variance's chain, which bounds small quotes: a
// 2^12-path ladder is less than a warp an SM.
//
// Functions: reciprocals and roots start from the hardware approximations (rcp and rsqrt.approx.ftz.f64) and take one
// third-order step of the binomial series; the logarithm takes x = 2^k z with z in [3/4, 3/2), the tabulated reciprocal
// c of the nearest of 129 centres, and ln x = k ln 2 - ln c + ln(1 + r) with r = c z - 1 by one multiply-add (the
// reduction of Story and Tang, New algorithms for improved transcendental functions on IA-64, ARITH 14, 1999); the
// angle's cosine and sine rotate a table of 256 directions by the remainder's Taylor sums; Phi(-z) is a Taylor sum of
// degree 11 about the nearest sixteenth (its derivatives are Hermite polynomials times the density). All are within about
// an ulp (the tables in 80-bit arithmetic on the host).
//
// Measured (a 252-step ladder): 650 -> 270 warp instructions a step and leg (132 FP64); 2^16 paths 0.40 -> 0.24 ms of
// kernel, 2^12 paths a call 323 -> 183 us. Against 80-bit arithmetic, over 60 ladders of 2^11 to 2^17 paths and 12 to 504
// steps, the prices are off by 1.1e-15 (rms), those of the textbook form by 2.4e-15. Of the 2^16 paths' gain the last 37 us
// (306 -> 270 a call) came from the tails: taken once a pair (a leg's tail is one minus the other's) from a table whose
// couples of coefficients lie cell by cell, they cost 26 shared-memory wavefronts a step and warp where they took 79, more
// than a third of the SM's time at 14 warps.
#pragma once

#include <cmath>

#include "model.cuh"

namespace ob {

constexpr int kTailCells = 110, kTailTerms = 12;  // |z| <= 6.77 for 32-bit uniforms
constexpr int kLogCells = 129, kTurnCells = 256;

struct alignas(16) Qe64Tables {
    // Taylor coefficients of Phi(-z) about cell / 16, two of a cell side by side and the cells of a couple in a row: the
    // lanes' cells spread over all the banks (12 in a row a cell, 96 bytes, they meet in half of them: 13.2 wavefronts a
    // 16-byte load of 32 lanes instead of 8.7)
    double tail[kTailTerms / 2][kTailCells][2];
    double log[kLogCells][2];             // c and -ln c at the centres: seven fractional bits of a binade, 3/4 to 3/2
    double turn[kTurnCells][2];           // cos and sin of 2 pi k / 256
};

// Built once a process (constants of the method).
inline const Qe64Tables& qe64_tables() {
    static const Qe64Tables* tables = [] {
        auto* t = new Qe64Tables();
        const long double pi = 3.14159265358979323846264338327950288L;
        for (int k = 0; k < kTailCells; ++k) {
            const long double c = static_cast<long double>(k) / 16;
            const long double density = std::exp(-c * c / 2) / std::sqrt(2 * pi);
            t->tail[0][k][0] = static_cast<double>(std::erfc(c / std::sqrt(2.0L)) / 2);
            long double he0 = 1, he1 = c, sign = -1, fact = 1;  // He_0, He_1; d^n Phi(-z) = -(-1)^(n-1) He_(n-1) density
            for (int n = 1; n < kTailTerms; ++n) {
                fact *= n;
                t->tail[n / 2][k][n % 2] = static_cast<double>(sign * he0 * density / fact);
                const long double next = c * he1 - n * he0;
                he0 = he1, he1 = next, sign = -sign;
            }
        }
        for (int j = 0; j < kLogCells; ++j) {
            // c = 1 from 1 - 3/512, a cell below one's own: the sum would cancel there
            const double centre = j < 64 ? (192 + j) / 256.0 : (64 + j) / 128.0;
            const double c = j == 63 || j == 64 ? 1.0 : 1 / centre;
            t->log[j][0] = c, t->log[j][1] = static_cast<double>(-std::log(static_cast<long double>(c)));
        }
        for (int k = 0; k < kTurnCells; ++k) {
            t->turn[k][0] = static_cast<double>(std::cos(2 * pi * k / kTurnCells));
            t->turn[k][1] = static_cast<double>(std::sin(2 * pi * k / kTurnCells));
        }
        return t;
    }();
    return *tables;
}

__device__ __forceinline__ double rcp64(double d) {  // a normal d
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.0);  // 1/d = r (1 + e + e^2 + ...)
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double div64(double n, double d) {
    const double r = rcp64(d), q = n * r;
    return fma(fma(-d, q, n), r, q);
}
// sqrt(x) of a normal x > 0; inv: the hardware's 1 / sqrt(x), to about 20 bits.
__device__ __forceinline__ double sqrt64(double x, double& inv) {
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(inv) : "d"(x));
    const double g = x * inv, e = fma(-g, inv, 1.0);  // sqrt(x) = g (1 - e)^(-1/2)
    return fma(g * e, fma(0.375, e, 0.5), g);
}
// 2^-127 < x < 1.5: within 2.2 2^-53 of ln x below one (the draws and the tails; 20 million of each).
__device__ __forceinline__ double log64(const Qe64Tables& t, double x) {
    const int hi = __double2hiint(x);
    const int up = (hi + 0x80000) & 0x7FF00000;              // 2^k in place: a mantissa from 3/2 counts up
    const int zh = hi - up + 0x3FF00000;                     // z, its high word
    const int cell = (zh + 0x1000 - 0x3FE80000) >> 13;       // its nearest centre
    const double2 c = *reinterpret_cast<const double2*>(t.log[cell]);
    const double r = fma(__hiloint2double(zh, __double2loint(x)), c.x, -1.0);  // |r| < 1/160
    double s = fma(r, 1.0 / 7, -1.0 / 6);
    s = fma(s, r, 1.0 / 5), s = fma(s, r, -1.0 / 4), s = fma(s, r, 1.0 / 3), s = fma(s, r, -0.5);
    const double kd = static_cast<double>((up >> 20) - 1023);
    // ln 2 as a sum, the first part (46 bits) exact times k
    const double low = fma(kd, -1.8641886737243033e-15, fma(r * r, s, r));
    return fma(kd, 0.6931471805599472, c.y) + low;
}
// ln(1 + x), |x| <= 1/16.
__device__ __forceinline__ double log1p64_small(double x) {
    const double x2 = x * x, x4 = x2 * x2;
    const double a = fma(x, 1.0 / 3, -0.5), b = fma(x, 1.0 / 5, -0.25), c = fma(x, 1.0 / 7, -1.0 / 6);
    const double d = fma(x, 1.0 / 9, -0.125), e = fma(x, 1.0 / 11, -0.1), f = fma(x, 1.0 / 13, -1.0 / 12);
    const double low = fma(x2, b, a), mid = fma(x2, d, c), top = fma(x2, f, e);
    return fma(x2, fma(x4, fma(x4, top, mid), low), x);
}
__device__ __forceinline__ double tail64(const Qe64Tables& t, double z) {  // Phi(-z), 0 <= z < 6.84
    constexpr double kMagic = 6755399441055744.0;                            // 1.5 2^52: rounds to an integer
    const double w = fma(z, 16.0, kMagic);
    const int cell = __double2loint(w);
    const double d = fma(w - kMagic, -0.0625, z);
    double2 k = *reinterpret_cast<const double2*>(t.tail[kTailTerms / 2 - 1][cell]);
    double s = fma(k.y, d, k.x);
#pragma unroll
    for (int n = kTailTerms / 2 - 2; n >= 0; --n) {
        k = *reinterpret_cast<const double2*>(t.tail[n][cell]);
        s = fma(fma(s, d, k.y), d, k.x);
    }
    return s;
}
// Box-Muller on two 32-bit draws (common.cuh's, in these functions).
__device__ __forceinline__ void box_muller64(const Qe64Tables& t, uint32_t a, uint32_t b, double& z0, double& z1) {
    double inv;
    const double r = sqrt64(-2.0 * log64(t, to_unit<double>(a)), inv);
    const uint32_t near = b + 0x800000u;  // 2 pi (b + 1/2) 2^-32: the nearest of the 256 directions and the rest
    const double2 dir = *reinterpret_cast<const double2*>(t.turn[near >> 24]);
    const double d = (static_cast<double>(static_cast<int>(near & 0xFFFFFFu) - 0x800000) + 0.5) * 1.4629180792671596e-09;
    const double d2 = d * d;
    const double sn = d * fma(d2, fma(d2, fma(d2, -1.0 / 5040, 1.0 / 120), -1.0 / 6), 1.0);
    const double cm = d2 * fma(d2, fma(d2, -1.0 / 720, 1.0 / 24), -0.5);  // cos - 1
    z0 = r * (dir.x + fma(dir.x, cm, -dir.y * sn)), z1 = r * (dir.y + fma(dir.y, cm, dir.x * sn));
}

// One step of (y, v) with normals zv, zx and tail = Phi(-zv).
__device__ __forceinline__ void qe64_step(const QeConsts<double>& c, const Qe64Tables& t, double& y, double& v,
                                          double zv, double zx, double tail) {
    const double m = fma(v - c.theta, c.E, c.theta), s2 = fma(v, c.c1, c.c2);
    const bool quad = s2 <= 1.5 * (m * m);
    const double im = rcp64(m), u = 0.5 * s2 * (im * im);
    double inv;
    const double q = sqrt64(quad ? 1.0 - u : 1.0, inv), p0 = 1.0 - q;
    const double p = fma(fma(-2.0, p0, fma(p0, p0, u)), 0.5 * inv, p0);
    double unused;
    const double g = sqrt64(quad ? q * p : 1.0, unused);
    const double vq = m * fma(zv, fma(zv, p, 2.0 * g), q);
    const double ub = u + 0.5, ib = m * ub, pr = ub * tail;
    const double ve = pr < 1.0 ? -log64(t, pr) * ib : 0.0;
    const double vn = quad ? fmax(vq, 0.0) : ve;
    const double Am = c.A * m, x = -2.0 * Am * p;
    const double den = quad ? 1.0 + x : fma(-c.A, ib, 1.0);
    const double r3 = div64(quad ? -Am * q : Am, den);
    const double lx = quad ? x : r3;
    double lg = log1p64_small(lx);
    if (fabs(lx) > 0.0625) lg = log(1.0 + lx);  // (rare: a large kappa rho / xi)
    const bool finite = den > 0.0;
    const double K0 = finite ? (quad ? fma(0.5, lg, r3) : -lg) : c.K0p;
    const double kv = finite ? -0.5 * c.K3 : c.K1;
    const double var = fma(c.K3, v, c.K4 * vn);
    const double sd = sqrt64(fmax(var, 1e-300), unused);
    y += fma(sd, zx, fma(c.K2, vn, fma(kv, v, c.mu_dt + K0)));
    v = vn;
}

}  // namespace ob
