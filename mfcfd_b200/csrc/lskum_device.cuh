// Device-side building blocks of the LSKUM pseudo-time loop (FP64).
//
// Every function restates one reference routine of src_mpi_primal with the
// same expression association as the Fortran source (which evaluates
// a*b*c as (a*b)*c and a+b+c as (a+b)+c).  The split-flux routines are
// written once with sign arguments: a - b == a + (-1)*b exactly in IEEE
// arithmetic, so Gxp/Gxn (and GxI..GxIV) share one body.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lskum {

enum PointKind { KIND_WALL = 0, KIND_INTERIOR = 1, KIND_OUTER = 2 };

// Limiter threshold: the literal 10e-6 in limiters.F90:78,81 is a
// default-real (single precision) constant promoted to double.
#define MFCFD_VENKAT_THR 9.99999974737875163555145263671875e-06

struct __align__(32) R4 {
    double a, b, c, d;
};

__device__ __forceinline__ R4 ld4(const R4 *p) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    double2 u = __ldg(q), v = __ldg(q + 1);
    return R4{u.x, u.y, v.x, v.y};
}
// Four doubles in one 256-bit read-only load (ld.global.nc.v4.f64, sm_100);
// p is 32-byte aligned and not written by the kernel that reads it.
__device__ __forceinline__ void ld4nc(const double *p, double v[4]) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
        : "l"(p));
}
__device__ __forceinline__ R4 ld4w(const R4 *p) {
    double v[4];
    ld4nc(reinterpret_cast<const double *>(p), v);
    return R4{v[0], v[1], v[2], v[3]};
}
__device__ __forceinline__ void st4(R4 *p, double a, double b, double c, double d) {
    double2 *q = reinterpret_cast<double2 *>(p);
    q[0] = make_double2(a, b);
    q[1] = make_double2(c, d);
}

// Constant, renumbered geometry.  Wall points occupy [0, nw), outer points
// [nw, nw + no), interior points [nw + no, n).
struct Geom {
    int n, kp, nw, no;
    const double2 *xy;             // (x, y)
    const double2 *nrm;            // (nx, ny) as the reference sets them
    const double *eps2;            // (vl_const*min_dist)**3 squared
    const int *conn;               // [kp][n], 0-based renumbered indices
    const int *nbhs;               // [n]
    const unsigned long long *mx;  // bit r: slot r in xpos; bit 32+r: in xneg
    const unsigned long long *my;  // bit r: slot r in ypos; bit 32+r: in yneg
    const double *obc;             // outer points: u1_inf_rot, u2_inf_rot, e_inf, A2n_inf, B2_inf, 0,0,0
    // Tile halos of the D and I passes (nullptr: no halo, every row is
    // gathered directly).  The halo of a TILE-point tile is the sorted set of
    // rows its points read (the points themselves and their neighbours);
    // hoff[tile] .. hoff[tile + 1] index its rows in hrow (an empty range: the
    // tile's halo exceeds the grid's cap and its rows are gathered directly).
    // hloc[p * hkp + r] is slot r's row within the tile's halo, hloc[p * hkp
    // + hkp - 1] the point's own; hmost = the largest halo, hc = the staging
    // stride (hmost padded: it does not tell how many rows a tile has).
    const int *hoff = nullptr;
    const int *hrow = nullptr;
    const unsigned char *hloc = nullptr;
    int hkp = 0, hc = 0, hmost = 0;
    // FP64 flux pass, fixed per grid: per point and split list the two
    // coefficients of the list's least-squares solve ([n][8], launch_flux_coef),
    // and with power != 0 the weight of every slot ([kp][n]; else nullptr: 1).
    const double *fco = nullptr;
    const double *wsl = nullptr;
    // reverse flux pass: the third entry of each list's inverse matrix ([n][4])
    const double *fcg = nullptr;
    // FP64 D and I passes: the inverse of the full stencil's normal matrix, [n][4]
    // (xx, xy, yy, unused)
    const double *minv = nullptr;
};
// Rows a tile halo stages at most (its local row indices are bytes): an O-grid's
// tiles have some 54, those of a renumbered cloud of points about 58 and a few
// over 64.  HALO_CAP, or HALO_CAP_WIDE and the passes' wide forms where that pays
// (wide_halos_pay): gathered directly, the few large tiles (4% of a cloud of
// 40,000 points) can set the passes' time (an iteration with one inner iteration
// FP64 195.7 us, 169.6 with the wide forms; FP32 113.3 and 98.1).
constexpr int HALO_CAP = 64, HALO_CAP_WIDE = 96;
// whether a grid's staged tiles need the wide forms
inline bool wide_halos(const Geom &g) { return g.hmost > HALO_CAP; }

struct Consts {
    double cfl, power, euler, pi, gm1;  // gm1 = gamma - 1
    int power_zero;                     // power == 0: weights are exactly 1
    int rks;
};

// ---------------------------------------------------------------------------
// q_variables.F90:8-37 eval_q_variables
template <class T>
__device__ __forceinline__ void q_from_prim_t(T rho, T u1, T u2, T pr, T q[4]) {
    T beta = T(0.5) * rho / pr;
    q[0] = (log(rho) + (log(beta) * T(2.5))) - beta * (u1 * u1 + u2 * u2);
    T two_times_beta = T(2.0) * beta;
    q[1] = two_times_beta * u1;
    q[2] = two_times_beta * u2;
    q[3] = -two_times_beta;
}
__device__ __forceinline__ void q_from_prim(double rho, double u1, double u2, double pr,
                                            double q[4]) {
    q_from_prim_t<double>(rho, u1, u2, pr, q);
}

// The per-state part shared by split_fluxes.F90 and quadrant_fluxes.F90: the
// state in the point's (t, n) frame and the two Maxwellian half-moments.
template <class T>
struct KStateT {
    T rho, ut, un, pbr, usq, B1, B2, e1, e2;
};
using KState = KStateT<double>;

// erf(x) given exp(-x*x), the scalar statement of what the FP32 flux pass
// evaluates on pairs (kstate2 of primal_fp32.cu): Abramowitz & Stegun 7.1.26
// (after Hastings), erf(|x|) = 1 - t (a1 + t (a2 + t (a3 + t (a4 + t a5))))
// exp(-x^2), t = 1 / (1 + p |x|), absolute error below 1.5e-7 (5.3e-7 evaluated in
// FP32; tests/test_erf32.py reads the coefficients here, tests/test_erf32_pairs.py
// holds kstate2's to them) -- the split fluxes use erf only in 1 +- erf, so the
// absolute error is what counts -- reusing the exponential the Maxwellian moments
// take anyway (1.024M points: FP32 flux pass 0.316 -> 0.304 ms; |dCl| against the
// FP64 loop after 50 iterations 1.0e-7 with the library erff, 6e-9 with this).
template <class T>
__device__ T erf_with_exp(T x, T e);
template <>
__device__ __forceinline__ float erf_with_exp<float>(float x, float e) {
    const float ax = fabsf(x);
    const float t = 1.0f / (1.0f + 0.3275911f * ax);
    float p = 1.061405429f;
    p = p * t - 1.453152027f;
    p = p * t + 1.421413741f;
    p = p * t - 0.284496736f;
    p = p * t + 0.254829592f;
    return copysignf(1.0f - (p * t) * e, x);
}

// quadrant_fluxes.F90:12-248: GxI (s1=-1,s2=-1), GxII (+1,-1), GxIII (+1,+1),
// GxIV (-1,+1).
template <class T>
__device__ __forceinline__ void flux_quad(const KStateT<T> &s, T s1, T s2, T G[4]) {
    T A1 = T(0.5) * (T(1.0) + s1 * s.e1);
    T A2 = T(0.5) * (T(1.0) + s2 * s.e2);
    T rA2 = s.rho * A2;
    T a1b = s.ut * A1 + s1 * s.B1;
    G[0] = rA2 * a1b;
    T temp1 = s.pbr + s.ut * s.ut;
    T temp2 = temp1 * A1 + s1 * (s.ut * s.B1);
    G[1] = rA2 * temp2;
    temp2 = s.un * A2 + s2 * s.B2;
    G[2] = s.rho * a1b * temp2;
    temp1 = (T(7.0) * s.pbr) + s.usq;
    temp2 = T(0.5) * s.ut * temp1 * A1;
    temp1 = (T(6.0) * s.pbr) + s.usq;
    T temp3 = T(0.5) * s.B1 * temp1;
    T temp4 = T(0.5) * s.rho * s.un * s.B2 * a1b;
    G[3] = rA2 * (temp2 + s1 * temp3) + s2 * temp4;
}

// state_update.F90:144-163 primitive_to_conserved
template <class T>
__device__ __forceinline__ void prim_to_conserved_t(T rho, T u1, T u2, T pr, T nx, T ny, T U[4]) {
    U[0] = rho;
    T temp1 = rho * u1;
    T temp2 = rho * u2;
    U[3] = T(2.5) * pr + T(0.5) * (temp1 * temp1 + temp2 * temp2) / rho;
    U[1] = temp1 * ny - temp2 * nx;
    U[2] = temp1 * nx + temp2 * ny;
}
__device__ __forceinline__ void prim_to_conserved(double rho, double u1, double u2, double pr,
                                                  double nx, double ny, double U[4]) {
    prim_to_conserved_t<double>(rho, u1, u2, pr, nx, ny, U);
}

// state_update.F90:239-294 conserved_vector_Ubar.  The freestream half
// (inf[0..4] = u1_inf_rot, u2_inf_rot, e_inf, A2n_inf, B2_inf) depends only on
// the geometry and is computed once on the host.
template <class T>
__device__ __forceinline__ void conserved_ubar_t(T rho, T u1, T u2, T pr, T nx, T ny,
                                                 const T *inf, T pi, T gm1, T Ubar[4]) {
    const T rho_inf = T(1.0);
    T u1_inf_rot = inf[0], u2_inf_rot = inf[1], e_inf = inf[2], A2n_inf = inf[3],
      B2_inf = inf[4];
    T tx = ny, ty = -nx;
    T u1_rot = u1 * tx + u2 * ty;
    T u2_rot = u1 * nx + u2 * ny;
    T temp1 = (u1_rot * u1_rot + u2_rot * u2_rot);
    T e = pr / (rho * gm1) + T(0.5) * (temp1);
    T beta = (rho) / (T(2.0) * pr);
    T S2 = u2_rot * sqrt(beta);
    T B2 = exp(-S2 * S2) / (T(2.0) * sqrt(pi * beta));
    T A2p = T(0.5) * (T(1.0) + erf(S2));
    Ubar[0] = (rho_inf * A2n_inf) + (rho * A2p);
    Ubar[1] = (rho_inf * u1_inf_rot * A2n_inf) + (rho * u1_rot * A2p);
    temp1 = rho_inf * (u2_inf_rot * A2n_inf - B2_inf);
    T temp2 = rho * (u2_rot * A2p + B2);
    Ubar[2] = temp1 + temp2;
    temp1 = (rho_inf * A2n_inf * e_inf - T(0.5) * rho_inf * u2_inf_rot * B2_inf);
    temp2 = (rho * A2p * e + T(0.5) * rho * u2_rot * B2);
    Ubar[3] = temp1 + temp2;
}
__device__ __forceinline__ void conserved_ubar(double rho, double u1, double u2, double pr,
                                               double nx, double ny, const double *inf,
                                               double pi, double gm1, double Ubar[4]) {
    conserved_ubar_t<double>(rho, u1, u2, pr, nx, ny, inf, pi, gm1, Ubar);
}

}  // namespace lskum
