// Elementary functions and kinetic states of the FP64 flux pass, without
// branches.
//
// The library's division, rsqrt, exp and erf each carry a rarely taken
// branch, and every branch ends a basic block: the point's and the
// neighbour's kinetic states, two directions each, then run as one long
// dependent chain.  The forms here are straight-line code over the range the
// flux pass meets, so the compiler interleaves the four chains; arguments
// outside it (and NaN) are found once per slot and take the library
// functions.  A value depends on its own argument only, never on which path
// the rest of the warp took.
#pragma once

#include "lskum_device.cuh"

namespace lskum {

// 1/x: the hardware's approximation and one third-order (Householder) step,
// y (1 + e + e^2) with e = 1 - x y: the error of the step is e^3.
__device__ __forceinline__ double rcp_h3(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1/sqrt(x): as above, y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2.
__device__ __forceinline__ double rsqrt_h3(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// exp(x) for |x| <= EXP_MAX.  Cody and Waite's reduction (x = n ln 2 + r,
// ln 2 in two parts) and 1 + r + r^2 P(r), P the degree-9 Chebyshev
// interpolant of (e^r - 1 - r) / r^2 over |r| <= ln 2 / 2 (its error times
// r^2 is at most 1.3e-17, coefficients rounded).
constexpr double EXP_MAX = 700.0;
// The polynomials' coefficients sit in constant memory: as literals each cost
// two moves into registers at every use.
static __constant__ double c_exp[14] = {
    0x1.71547652b82fep+0, 6755399441055744.0 /* 1.5 2^52 */, -0x1.62e42fefa39efp-1,
    -0x1.abc9e3b39803fp-56,
    0x1.af38a9b0ec855p-26, 0x1.289185613a3d6p-22, 0x1.71de0dae63bb3p-19, 0x1.a019b90d2ae7ap-16,
    0x1.a01a01a7c41d5p-13, 0x1.6c16c1788bd90p-10, 0x1.11111111109b3p-7, 0x1.5555555553d63p-5,
    0x1.5555555555556p-3, 0x1.0000000000001p-1};
__device__ __forceinline__ double exp_mid(double x) {
    const double t = fma(x, c_exp[0], c_exp[1]);  // n in the low word
    const int n = __double2loint(t);
    const double nd = t - c_exp[1];
    double r = fma(nd, c_exp[2], x);
    r = fma(nd, c_exp[3], r);
    double p = c_exp[4];
#pragma unroll
    for (int i = 5; i < 14; ++i) p = fma(p, r, c_exp[i]);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    return __hiloint2double(__double2hiint(p) + (int)((unsigned)n << 20), __double2loint(p));
}

// erf(x) for |x| <= ERF_MAX, z = x*x: x Q(z), Q the degree-13 Chebyshev
// interpolant of erf(sqrt z) / sqrt z over [0, ERF_MAX^2] (absolute error of
// x Q at most 2.5e-17).  1.25 covers |u| sqrt(beta) up to Mach 1.49 along a
// direction; beyond it the library's erf is taken.
constexpr double ERF_MAX = 1.25;
static __constant__ double c_erf[14] = {
    -0x1.cd03490bc5835p-39, 0x1.5daf7ab4a9346p-34, -0x1.46f41e3907e41p-30,
    0x1.fa4fba2e1e1b8p-27, -0x1.5f42a98f93ce9p-23, 0x1.b9e1480408c3dp-20,
    -0x1.f4d1ed44b13b7p-17, 0x1.f9a320de78f7ap-14, -0x1.c02db3c5bcce0p-11,
    0x1.565bcd0cfe771p-8, -0x1.b82ce3127e1adp-6, 0x1.ce2f21a04294dp-4,
    -0x1.812746b0379e3p-2, 0x1.20dd750429b6dp+0};
__device__ __forceinline__ double erf_mid(double x, double z) {
    double p = c_erf[0];
#pragma unroll
    for (int i = 1; i < 14; ++i) p = fma(p, z, c_erf[i]);
    return x * p;
}

static __device__ __noinline__ double exp_any(double x) { return exp(x); }
static __device__ __noinline__ double erf_any(double x) { return erf(x); }

__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }

// venkat_limiter and the limited qtilde of one component (limiters.F90:64-110,
// the qtilde lines of *_fluxes.F90), t = d.dq of the component: del_neg is
// -t/2, and its factor common to the quotient's numerator and denominator is
// cancelled.
__device__ __forceinline__ double limited_qtilde(double t, double q, double qmax, double qmin,
                                                 double eps2) {
    const double del_neg = -0.5 * t;
    const double del_pos = (__double2hiint(t) < 0 ? qmax : qmin) - q;
    const double a = fma(del_pos, del_pos, eps2);
    const double num = fma(-t, del_pos, a);
    const double den = fma(del_neg, del_pos - t, a);
    const double f = num * rcp_h3(den);
    const double phi = f < 1.0 && fabs(del_neg) > MFCFD_VENKAT_THR ? f : 1.0;
    return fma(phi, del_neg, q);
}

// qtilde -> the state before its exponentials (q_variables.F90:230-256).  beta
// and p/rho come from qtilde itself (beta = -qtilde_4/2, p/rho = 1/(2 beta)),
// and rho = exp(texp - log(beta)/(gamma-1)) with gamma = 1.4, a constant of
// the reference (parameter.F90:10), as exp(texp) beta^(-5/2) = exp(texp)
// (1/beta)^2 / sqrt(beta): no log.
struct KPre {
    double u1, u2, texp, rb5, sb;
};
__device__ __forceinline__ KPre kstate_pre(const double qt[4], KState &s) {
    KPre p;
    const double beta = -0.5 * qt[3];
    s.pbr = rcp_h3(-qt[3]);
    p.u1 = qt[1] * s.pbr;
    p.u2 = qt[2] * s.pbr;
    s.usq = fma(p.u1, p.u1, p.u2 * p.u2);
    p.texp = fma(beta, s.usq, qt[0]);
    const double rb = rsqrt_h3(beta);
    p.sb = beta * rb;
    p.rb5 = (4.0 * s.pbr * s.pbr) * rb;
    return p;
}

// The point's and the neighbour's kinetic states from their limited qtilde.
__device__ __forceinline__ void kstate_pair(const double qi[4], const double qk[4], double nx,
                                            double ny, double inv_sqrt_pi, KState &si, KState &sk,
                                            double ui[2], double uk[2]) {
    KState *s[2] = {&si, &sk};
    double S[2][2], E[2][3], X[2];
    KPre p[2] = {kstate_pre(qi, si), kstate_pre(qk, sk)};
    int big = 0, far = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        s[h]->ut = fma(p[h].u1, ny, -(p[h].u2 * nx));
        s[h]->un = fma(p[h].u1, nx, p[h].u2 * ny);
        S[h][0] = s[h]->ut * p[h].sb;
        S[h][1] = s[h]->un * p[h].sb;
        X[h] = p[h].texp;
        big = max(big, max(abs_hi(S[h][0]), abs_hi(S[h][1])));
        far = max(far, abs_hi(X[h]));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const double z0 = S[h][0] * S[h][0], z1 = S[h][1] * S[h][1];
        E[h][0] = exp_mid(-z0);
        E[h][1] = exp_mid(-z1);
        E[h][2] = exp_mid(X[h]);
        s[h]->e1 = erf_mid(S[h][0], z0);
        s[h]->e2 = erf_mid(S[h][1], z1);
    }
    // 1.25 = 0x3ff40000'00000000, 26^2 < 700, 700 = 0x4085e000'00000000
    if (big >= 0x3ff40000 || far >= 0x4085e000) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (abs_hi(S[h][0]) >= 0x3ff40000) s[h]->e1 = erf_any(S[h][0]);
            if (abs_hi(S[h][1]) >= 0x3ff40000) s[h]->e2 = erf_any(S[h][1]);
            if (abs_hi(S[h][0]) >= 0x403a0000) E[h][0] = exp_any(-S[h][0] * S[h][0]);
            if (abs_hi(S[h][1]) >= 0x403a0000) E[h][1] = exp_any(-S[h][1] * S[h][1]);
            if (abs_hi(X[h]) >= 0x4085e000) E[h][2] = exp_any(X[h]);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const double hb = s[h]->pbr * p[h].sb * inv_sqrt_pi;  // 0.5 / sqrt(pi beta)
        s[h]->rho = E[h][2] * p[h].rb5;
        s[h]->B1 = E[h][0] * hb;
        s[h]->B2 = E[h][1] * hb;
    }
    ui[0] = p[0].u1; ui[1] = p[0].u2;
    uk[0] = p[1].u1; uk[1] = p[1].u2;
}

// split_fluxes.F90 flux_Gxp/Gxn (u = ut, o = un) and flux_Gyp/Gyn (u = un,
// o = ut), sg = +-1 with hs = sg/2: mass, momentum along u, momentum along o
// and energy.  With a = u A + sg B the reference's expressions are rho a,
// rho (u a + p/rho A), o rho a and rho/2 ((6 p/rho + |u|^2) a + u p/rho A):
// 11 operations instead of 20.
__device__ __forceinline__ void flux_split(const KState &s, double u, double o, double B, double e,
                                           double sg, double hs, double w6, double G[4]) {
    const double A = fma(hs, e, 0.5);
    const double a = fma(u, A, sg * B);
    const double pA = s.pbr * A;
    G[0] = s.rho * a;
    G[1] = s.rho * fma(u, a, pA);
    G[2] = o * G[0];
    G[3] = (0.5 * s.rho) * fma(w6, a, u * pA);
}

}  // namespace lskum
