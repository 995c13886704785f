// pdm1_fp64.cuh -- the double-precision face path without branches.
//
// The IEEE quotient and square root that the compiler emits handle every
// operand: each ends in a branch to a routine for subnormal, huge and special
// ones, so the ~130 quotients of a face run one after the other, each a chain
// of dependent FP64 instructions (measured: 3464 warp instructions per 32 faces,
// FP64 pipe 46 % busy, 3.8 of 6.9 stall cycles per issue on that latency).  Here the
// operands' ranges are checked once per tile (the state in shared memory) and
// once per face (the projected states), and inside them a quotient is a
// reciprocal by Newton's third-order iteration and Markstein's residual
// correction (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34 (1990) 111): straight-line
// code, shared reciprocals where quotients share a divisor, and the compiler
// interleaves the independent chains.  Outside the ranges the IEEE path runs.
//
// Rounding: the corrected value is off the exact quotient by at most 2^-51 of
// its last place before the final rounding, so it is the IEEE quotient but
// where that lies within 2^-51 last places of a midpoint between two doubles
// (about one pair of operands in 10^15; then the neighbouring double).
#pragma once

#include "pdm1_math.cuh"

namespace pdm1 {

// ---------------------------------------------------------------------------
// Range checks on the exponent field.  Exponents: the high word of 2^k is
// (k + 1023) << 20.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr unsigned exp_word(int k) { return (unsigned)(k + 1023) << 20; }

__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// |x| in [2^lo, 2^hi), or x = 0
template <int LO, int HI>
__device__ __forceinline__ bool zero_or_within(double x) {
    const unsigned h = abs_hi(x);
    return h - exp_word(LO) < exp_word(HI) - exp_word(LO) || (h | (unsigned)__double2loint(x)) == 0u;
}

// The state's range: a reconstruction's ratio of smoothness indicators stays
// below 2^888 and its quotients' residuals above the subnormal range.
__device__ __forceinline__ bool weno_range(double v) { return zero_or_within<-940, 200>(v); }

// ---------------------------------------------------------------------------
// Quotients and square roots of operands in range
// ---------------------------------------------------------------------------
// 1/b to within one last place: rcp.approx.ftz.f64 (about 20 bits) and one
// third-order step y (1 + e + e^2), e = 1 - b y.
__device__ __forceinline__ double rcp_near(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return fma(fma(e, e, e), y, y);
}

// a/b given y = rcp_near(b): the product and its residual correction
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// x/3 and x/6: x times the 106-bit reciprocal (N. Brisebarre, J.-M. Muller,
// S. K. Raina, "Accelerating correctly rounded floating-point division when the
// divisor is known in advance", IEEE Trans. Comput. 53 (2004) 1069).  x/3 is never
// within a sixth of a last place of a midpoint, so the result is the IEEE one.
constexpr double kThirdHi = 1.0 / 3.0;                              // 1/3 (1 - 2^-54)
constexpr double kThirdLo = kThirdHi * 0x1p-54;                     // 1/3 - kThirdHi = 1/3 2^-54
__device__ __forceinline__ double third(double x) { return fma(x, kThirdHi, x * kThirdLo); }
__device__ __forceinline__ double sixth(double x) { return fma(x, 0.5 * kThirdHi, x * (0.5 * kThirdLo)); }

// sqrt(x) for x in [2^-960, 2^900) or 0: rsqrt.approx.ftz.f64, one third-order
// step (Goldschmidt's form), one residual correction (Markstein).
__device__ __forceinline__ double sqrt_near(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double g = x * y, h = 0.5 * y;
    const double e = fma(-g, y, 1.0);
    const double p = e * fma(0.375, e, 0.5);
    const double g1 = fma(g, p, g), h1 = fma(h, p, h);
    const double s = fma(fma(-g1, g1, x), h1, g1);
    return x == 0.0 ? x : s;
}

// ---------------------------------------------------------------------------
// Reconstructions of both states of a face from the cells w[0..5] = i-3 .. i+2
// ---------------------------------------------------------------------------

// The nonlinear part of weno_left: the weighted sum of the candidate values p
// with the indicators' weights, each operation as there (2 v and 4 v are
// exact, so their difference with another value is one fused operation).
__device__ __forceinline__ double weno_weigh(double v0, double v1, double v2, double v3, double v4, double p0,
                                             double p1, double p2) {
    const double k1312 = 13.0 / 12.0;
    double a, b;
    a = fma(-2.0, v1, v0) + v2; b = fma(-4.0, v1, v0) + 3.0 * v2;
    const double beta0 = fma(0.25, b * b, k1312 * (a * a));
    a = fma(-2.0, v2, v1) + v3; b = v1 - v3;
    const double beta1 = fma(0.25, b * b, k1312 * (a * a));
    a = fma(-2.0, v3, v2) + v4; b = fma(-4.0, v3, 3.0 * v2) + v4;
    const double beta2 = fma(0.25, b * b, k1312 * (a * a));
    const double tau5 = fabs(beta2 - beta0);
    const double d0 = beta0 + kWenoEps, d1 = beta1 + kWenoEps, d2 = beta2 + kWenoEps;
    const double r0 = quotient(tau5, d0, rcp_near(d0));
    const double r1 = quotient(tau5, d1, rcp_near(d1));
    const double r2 = quotient(tau5, d2, rcp_near(d2));
    const double al0 = 0.1 * (1.0 + r0 * r0);
    const double al1 = 0.6 * (1.0 + r1 * r1);
    const double al2 = 0.3 * (1.0 + r2 * r2);
    const double s = al0 + al1 + al2, y = rcp_near(s);
    return quotient(al0, s, y) * p0 + quotient(al1, s, y) * p1 + quotient(al2, s, y) * p2;
}

// weno_left of both sides; the quotients by 3 and 6 that both use, once.
__device__ __forceinline__ void weno_pair(const double w[6], double &L, double &R) {
    const double t1 = sixth(w[1]), t4 = sixth(w[4]), c2 = third(w[2]), c3 = third(w[3]);
    const double f2 = sixth(5.0 * w[2]), f3 = sixth(5.0 * w[3]);
    L = weno_weigh(w[0], w[1], w[2], w[3], w[4], third(w[0]) - sixth(7.0 * w[1]) + sixth(11.0 * w[2]),
                   -t1 + f2 + c3, c2 + f3 - t4);
    R = weno_weigh(w[5], w[4], w[3], w[2], w[1], third(w[5]) - sixth(7.0 * w[4]) + sixth(11.0 * w[3]),
                   -t4 + f3 + c2, c3 + f2 - t1);
}

// weno3_left
__device__ __forceinline__ double weno3_near(double v0, double v1, double v2) {
    const double p0 = -0.5 * v0 + 1.5 * v1, p1 = 0.5 * v1 + 0.5 * v2;
    const double beta0 = (v1 - v0) * (v1 - v0), beta1 = (v2 - v1) * (v2 - v1);
    const double tau3 = fabs(beta1 - beta0);
    const double d0 = beta0 + kWenoEps, d1 = beta1 + kWenoEps;
    const double r0 = quotient(tau3, d0, rcp_near(d0)), r1 = quotient(tau3, d1, rcp_near(d1));
    const double al0 = (1.0 / 3.0) * (1.0 + r0 * r0), al1 = (2.0 / 3.0) * (1.0 + r1 * r1);
    const double s = al0 + al1, y = rcp_near(s);
    return quotient(al0, s, y) * p0 + quotient(al1, s, y) * p1;
}

// The IEEE path of a tile whose state leaves weno_range
static __device__ __noinline__ double weno_left_ieee(double v0, double v1, double v2, double v3, double v4) {
    return weno_left(v0, v1, v2, v3, v4);
}
static __device__ __noinline__ double weno3_left_ieee(double v0, double v1, double v2) { return weno3_left(v0, v1, v2); }

// ---------------------------------------------------------------------------
// Interface flux
// ---------------------------------------------------------------------------

// One side of a face after the realizability projection.
struct Side64 {
    double phi, jx, jy, jz, jn;
    bool ok;   // the operands that the flux divides are in range
};

// project() of the reconstructed state.  |J|^2 below 2^-900 (but not 0) is out
// of range, as is phi below 2^-450: |J| and its quotients keep every bit.
__device__ __forceinline__ Side64 side64(const double u[4]) {
    Side64 s;
    s.phi = u[0] < 0.0 ? 0.0 : u[0];
    s.jx = u[1]; s.jy = u[2]; s.jz = u[3];
    double x2 = s.jx * s.jx + s.jy * s.jy + s.jz * s.jz;
    s.ok = zero_or_within<-900, 400>(x2) && zero_or_within<-450, 200>(s.phi);
    s.jn = sqrt_near(x2);
    const double jmax = (1.0 - kRealEps) * s.phi;
    if (s.jn > jmax) {
        const double sc = quotient(jmax, s.jn, rcp_near(s.jn));
        s.jx *= sc; s.jy *= sc; s.jz *= sc;
        x2 = s.jx * s.jx + s.jy * s.jy + s.jz * s.jz;
        s.ok = s.ok && zero_or_within<-920, 400>(x2);
        s.jn = sqrt_near(x2);
    }
    // the components that are divided by |J|
    s.ok = s.ok && (x2 == 0.0 || (zero_or_within<-900, 200>(s.jx) && zero_or_within<-900, 200>(s.jy) &&
                                  zero_or_within<-900, 200>(s.jz)));
    return s;
}

// closure, physical_flux and eigen of one side.  After the projection |J| < phi,
// so below the eigenvalue floor of phi the speeds are those of a state at rest; at
// or above it the speeds' f is the closure's, held at 1 - 1e-10: one quotient and
// one square root serve both, and mu is the unit vector's normal component.
__device__ __forceinline__ void side_flux64(const Side64 &s, int axis, bool unit, double F[4], double &lmin,
                                            double &lmax) {
    const bool moving = s.jn > 0.0;
    double f = s.phi > 0.0 ? quotient(s.jn, s.phi, rcp_near(s.phi)) : 0.0;
    f = f > 1.0 ? 1.0 : f;
    const double y = rcp_near(s.jn);
    const double nx = moving ? quotient(s.jx, s.jn, y) : 0.0;
    const double ny = moving ? quotient(s.jy, s.jn, y) : 0.0;
    const double nz = moving ? quotient(s.jz, s.jn, y) : 0.0;
    const double na = axis == 0 ? nx : (axis == 1 ? ny : nz);
    double chi = third(fma(-2.0, sqrt_near(4.0 - 3.0 * f * f), 5.0));
    {
        const double iso = 0.5 * (1.0 - chi), dir = 0.5 * (3.0 * chi - 1.0);
        const double pd = s.phi * dir, pdx = pd * nx, pdy = pd * ny;
        const double diag = s.phi * (iso + dir * na * na);
        const double xy = pdx * ny, xz = pdx * nz, yz = pdy * nz;
        F[0] = axis == 0 ? s.jx : (axis == 1 ? s.jy : s.jz);
        F[1] = axis == 0 ? diag : (axis == 1 ? xy : xz);
        F[2] = axis == 0 ? xy : (axis == 1 ? diag : yz);
        F[3] = axis == 0 ? xz : (axis == 1 ? yz : diag);
    }
    if (unit) {
        lmin = -1.0;
        lmax = 1.0;
        return;
    }
    const double iso3 = 1.0 / 1.7320508075688772;   // 1/sqrt(3), as T(1) / sqrt(T(3))
    constexpr double fmax_ = 1.0 - kEigEps;
    if (f > fmax_) {
        f = fmax_;
        chi = third(fma(-2.0, sqrt_near(4.0 - 3.0 * f * f), 5.0));
    }
    const double c3 = 3.0 * chi, den = 5.0 - c3;
    const double disc = 4.0 * f * f * na * na - den * fma(-2.0, 1.0 - chi, na * na * (c3 - 1.0));
    const double root = sqrt_near(disc < 0.0 ? 0.0 : disc);
    const double c = 2.0 * f * na, yd = rcp_near(den);
    const bool rest = s.jn < kEigEps;
    lmin = rest ? -iso3 : quotient(c - root, den, yd);
    lmax = rest ? iso3 : quotient(c + root, den, yd);
}

// The IEEE path of one face: project both states, hll_flux.
static __device__ __noinline__ void face_flux_ieee(double l0, double l1, double l2, double l3, double r0, double r1,
                                                   double r2, double r3, int axis, bool unit, double *F, int stride) {
    double L[4] = {l0, l1, l2, l3}, R[4] = {r0, r1, r2, r3}, out[4];
    project(L[0], L[1], L[2], L[3]);
    project(R[0], R[1], R[2], R[3]);
    hll_flux(L, R, axis, unit, out);
#pragma unroll
    for (int c = 0; c < 4; ++c) F[c * stride] = out[c];
}

// Projection of both reconstructed states and their HLL flux into F[c * stride].
__device__ __forceinline__ void face_flux64(const double L[4], const double R[4], int axis, bool unit, double *F,
                                            int stride) {
    const Side64 a = side64(L), b = side64(R);
    double FL[4], FR[4], la, ha, lb, hb;
    side_flux64(a, axis, unit, FL, la, ha);
    side_flux64(b, axis, unit, FR, lb, hb);
    double sl = lb < la ? lb : la, sr = hb > ha ? hb : ha;
    if (sl > 0.0) sl = 0.0;
    if (sr < 0.0) sr = 0.0;
    const double den = sr - sl, sp = sl * sr, y = rcp_near(den);
    bool ok = a.ok && b.ok && abs_hi(den) - exp_word(-100) < exp_word(2) - exp_word(-100);
    const double d[4] = {b.phi - a.phi, b.jx - a.jx, b.jy - a.jy, b.jz - a.jz};
    double q[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double n = sr * FL[c] - sl * FR[c] + sp * d[c];
        ok = ok && zero_or_within<-900, 600>(n);
        q[c] = quotient(n, den, y);
    }
    if (ok) {
#pragma unroll
        for (int c = 0; c < 4; ++c) F[c * stride] = q[c];
    } else {
        face_flux_ieee(L[0], L[1], L[2], L[3], R[0], R[1], R[2], R[3], axis, unit, F, stride);
    }
}

// ---------------------------------------------------------------------------
// The stage update and the CFL bound of one cell
// ---------------------------------------------------------------------------
struct State64 { double phi, jx, jy, jz; };
static __device__ __noinline__ State64 project_ieee(double phi, double jx, double jy, double jz) {
    project(phi, jx, jy, jz);
    return {phi, jx, jy, jz};
}

// project()
__device__ __forceinline__ void project64(double u[4]) {
    const double phi = u[0] < 0.0 ? 0.0 : u[0];
    const double x2 = u[1] * u[1] + u[2] * u[2] + u[3] * u[3];
    if (zero_or_within<-900, 400>(x2) && zero_or_within<-450, 200>(phi)) {
        const double jn = sqrt_near(x2), jmax = (1.0 - kRealEps) * phi;
        if (jn > jmax) {
            const double s = quotient(jmax, jn, rcp_near(jn));
            u[1] *= s; u[2] *= s; u[3] *= s;
        }
        u[0] = phi;
    } else {
        const State64 q = project_ieee(u[0], u[1], u[2], u[3]);
        u[0] = q.phi; u[1] = q.jx; u[2] = q.jy; u[3] = q.jz;
    }
}

static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }

// a[c] / b of the four components
__device__ __forceinline__ void div4(double a[4], double b) {
    const double y = rcp_near(b);
    bool ok = abs_hi(b) - exp_word(-200) < exp_word(200) - exp_word(-200);
#pragma unroll
    for (int c = 0; c < 4; ++c) ok = ok && zero_or_within<-700, 700>(a[c]);
    if (ok) {
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = quotient(a[c], b, y);
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = div_ieee(a[c], b);
    }
}

static __device__ __noinline__ void speeds3_ieee(double phi, double jx, double jy, double jz, double *a) {
    max_abs_speeds3(phi, jx, jy, jz, a);
}

// max_abs_speeds3
__device__ __forceinline__ void speeds3_64(const double u[4], double a[3]) {
    const double x2 = u[1] * u[1] + u[2] * u[2] + u[3] * u[3];
    const double phi = u[0] < kEigEps ? kEigEps : u[0];
    const double jn = sqrt_near(x2);
    bool ok = zero_or_within<-900, 400>(x2) && abs_hi(phi) < exp_word(200);
#pragma unroll
    for (int c = 1; c < 4; ++c) ok = ok && zero_or_within<-900, 200>(u[c]);
    if (!ok) {
        double t[3];
        speeds3_ieee(u[0], u[1], u[2], u[3], t);
        a[0] = t[0]; a[1] = t[1]; a[2] = t[2];
        return;
    }
    double f = quotient(jn, phi, rcp_near(phi));
    f = f > 1.0 - kEigEps ? 1.0 - kEigEps : f;
    const double chi = third(fma(-2.0, sqrt_near(4.0 - 3.0 * f * f), 5.0));
    const double c3 = 3.0 * chi, den = 5.0 - c3, yd = rcp_near(den), yj = rcp_near(jn);
    const bool rest = jn < kEigEps;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const double mu = quotient(u[1 + ax], jn, yj);
        const double disc = 4.0 * f * f * mu * mu - den * fma(-2.0, 1.0 - chi, mu * mu * (c3 - 1.0));
        const double root = sqrt_near(disc < 0.0 ? 0.0 : disc), c = 2.0 * f * mu;
        const double lo = fabs(quotient(c - root, den, yd)), hi = fabs(quotient(c + root, den, yd));
        a[ax] = rest ? 1.0 / 1.7320508075688772 : (lo > hi ? lo : hi);
    }
}

}  // namespace pdm1
