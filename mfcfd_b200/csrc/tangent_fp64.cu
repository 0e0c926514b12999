// mfcfd_tangent: forward-mode (tangent) derivative of the pseudo-time loop.
//
// The reference's tangent driver Q_LSKUM_D (src_mpi_forward/sensitivity_files/
// q_lskum_d.F90:28-89) seeds pointd%x(1) = 1, differentiates
// COMPUTE_NORMALS_D and every FPI_SOLVER_D iteration and returns the
// derivative of the objective.  Here the seed is any direction (dx, dy) over
// all points: the loop runs n iterations from the handle's state (held
// fixed) with every quantity carried as a Dual (value, derivative), and the
// result is J = sum over shapes of Cl or Cd of the final state and dJ/de in
// that direction.  For the reverse-mode gradient g of mfcfd_adjoint,
// dJ/de = <g, (dx, dy)> (the dot-product test).
//
// The D, I and flux passes have the primal's split of the work (eight lanes a
// point, a slot a lane) and its forms (flux_math.cuh), differentiated; the state
// update is a thread-per-point pass over the primal's device templates
// (q_from_prim, prim_to_conserved, conserved_ubar) instantiated on Dual.  min_dist is data, as in the
// reference.
#include <cuda_runtime.h>

#include <algorithm>
#include <new>
#include <type_traits>
#include <vector>

// handle.h (and through it the primal device templates) comes before
// dual.cuh: the templates' double instantiations must see only the libm
// overloads, and the Dual ones are found by argument-dependent lookup.
#include "handle.h"
#include "flux_math.cuh"
#include "flux_tile.cuh"
#include "dual.cuh"
#include "objective.h"

using namespace lskum;
using lskum_host::cuda_fail;
using lskum_host::fail;

namespace {

constexpr int TB = 128;
constexpr double OBT = 1.0 / 3.0;
constexpr double TBT = 2.0 / 3.0;

// value / derivative arrays of the tangent state
struct TanState {
    const double2 *xy_t, *nrm_t;  // derivatives of (x, y) and (nx, ny)
    const Dual *obc;              // outer points: 8 Duals per point
    R4 *pv[2], *pt[2];            // prim
    R4 *qv[2], *qt[2];            // q
    double *dqv[3], *dqt[3];      // dq [n][8]: the D pass's, then the inner iterations' in turn
    double *mt;                   // derivative of the stencil's normal matrix [n][4]
    double *qmv, *qmt;            // qm [n][8]
    double *dlv, *dlt;            // delta
    double *spv, *spt;            // spd
};

__device__ __forceinline__ void ld_dual4(const R4 *v, const R4 *t, int i, Dual out[4]) {
    const R4 a = v[i], b = t[i];
    out[0] = Dual(a.a, b.a);
    out[1] = Dual(a.b, b.b);
    out[2] = Dual(a.c, b.c);
    out[3] = Dual(a.d, b.d);
}
__device__ __forceinline__ void st_dual4(R4 *v, R4 *t, int i, const Dual x[4]) {
    v[i] = R4{x[0].v, x[1].v, x[2].v, x[3].v};
    t[i] = R4{x[0].d, x[1].d, x[2].d, x[3].d};
}
__device__ __forceinline__ void xy_dual(const Geom &g, const TanState &s, int i, Dual &x,
                                        Dual &y) {
    const double2 p = g.xy[i], d = s.xy_t[i];
    x = Dual(p.x, d.x);
    y = Dual(p.y, d.y);
}

// q and spd of the initial state (its derivative is zero: prim_0 is held fixed)
__global__ void k_t_init(int n, TanState s, int cur, int qc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Dual P[4], q[4];
    ld_dual4(s.pv[cur], s.pt[cur], i, P);
    q_from_prim_t<Dual>(P[0], P[1], P[2], P[3], q);
    st_dual4(s.qv[qc], s.qt[qc], i, q);
    const Dual spd = sqrt(P[1] * P[1] + P[2] * P[2]) + Dual(3.0) * sqrt(P[3] / P[0]);
    s.spv[i] = spd.v;
    s.spt[i] = spd.d;
}

// The tangents of the D and I passes by slots, as kb_grad_s and kb_inner_s of the
// primal: eight lanes a point, a slot's lane leaves its fields in shared memory
// (T_F doubles a field, T_P a point: distinct banks) and lane l sums component l
// and its derivative.  The solve's derivative comes from the stored inverse L of
// the normal matrix M: o = L s, do = L (ds - dM o).
// At 64,000 points 21 and 24 us; a thread a point, summing and solving on Duals,
// 28 and 35.
constexpr int T_PTS = TB / LPP, T_F = 9, T_P = 116;

// L s of both components, value and derivative, on each lane: the lane holds the
// sum of component l & 3 along x (l < 4) or y.
struct TSolve {
    double ox, oy, tx, ty;
    __device__ __forceinline__ TSolve(const Geom &g, const TanState &s, int i, int l, Dual sum) {
        const unsigned full = 0xffffffffu;
        const Dual o(__shfl_xor_sync(full, sum.v, 4), __shfl_xor_sync(full, sum.d, 4));
        ox = oy = tx = ty = 0.0;
        if (i < 0) return;
        const Dual sx = l < 4 ? sum : o, sy = l < 4 ? o : sum;
        double L[4], M[4];
        ld4nc(g.minv + 4 * (size_t)i, L);
        ld4nc(s.mt + 4 * (size_t)i, M);
        ox = L[0] * sx.v + L[1] * sy.v;
        oy = L[1] * sx.v + L[2] * sy.v;
        const double dx = sx.d - (M[0] * ox + M[2] * oy), dy = sy.d - (M[2] * ox + M[1] * oy);
        tx = L[0] * dx + L[1] * dy;
        ty = L[1] * dx + L[2] * dy;
    }
};

// eval_q_derivatives_d + func_delta_d (q_variables_d.F90, state_update_d.F90)
__global__ void __launch_bounds__(TB)
k_t_grad(Geom g, Consts c, TanState s, int qc, int with_delta) {
    __shared__ double sm[T_PTS * T_P];
    const unsigned full = 0xffffffffu;
    const int l = threadIdx.x % LPP, m = l & 3;
    int i = blockIdx.x * T_PTS + threadIdx.x / LPP;
    double *row = sm + threadIdx.x / LPP * T_P;
    if (i >= g.n) i = -1;
    int nb = 0;
    Dual xi, yi, qi;
    if (i >= 0) {
        nb = g.nbhs[i];
        xy_dual(g, s, i, xi, yi);
        qi = Dual(reinterpret_cast<const double *>(s.qv[qc] + i)[m],
                  reinterpret_cast<const double *>(s.qt[qc] + i)[m]);
    }
    Dual sum, ext = qi, dmin(1.0);
    int dslot = -1;  // of the smallest time step: the first, as in slot order
    const int nbw = __reduce_max_sync(full, nb);
    for (int r0 = 0; r0 < nbw; r0 += LPP) {
        const int r = r0 + l;
        if (r < nb) {
            const int k = g.conn[(size_t)r * g.n + i];
            double qv[4], qt[4];
            ld4nc(reinterpret_cast<const double *>(s.qv[qc] + k), qv);
            ld4nc(reinterpret_cast<const double *>(s.qt[qc] + k), qt);
            Dual xk, yk;
            xy_dual(g, s, k, xk, yk);
            const Dual delx = xk - xi, dely = yk - yi;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                row[f * T_F + l] = qv[f];
                row[(4 + f) * T_F + l] = qt[f];
            }
            row[8 * T_F + l] = delx.v;
            row[9 * T_F + l] = dely.v;
            row[10 * T_F + l] = delx.d;
            row[11 * T_F + l] = dely.d;
            if (with_delta) {
                Dual delta_t = sqrt(delx * delx + dely * dely) / Dual(s.spv[k], s.spt[k]);
                delta_t = Dual(c.cfl) * delta_t;
                if (dmin > delta_t) {
                    dmin = delta_t;
                    dslot = r;
                }
            }
        }
        __syncwarp();
        const double *qf = row + m * T_F, *wf = row + (8 + l / 4) * T_F;
#pragma unroll
        for (int j = 0; j < LPP; ++j) {
            if (r0 + j >= nb) break;
            const Dual qk(qf[j], qf[4 * T_F + j]), d(wf[j], wf[2 * T_F + j]);
            if (l < 4 ? qk > ext : qk < ext) ext = qk;
            sum += d * (qk - qi);
        }
        __syncwarp();
    }
    if (with_delta) {
#pragma unroll
        for (int o = 4; o; o >>= 1) {
            const Dual d(__shfl_xor_sync(full, dmin.v, o), __shfl_xor_sync(full, dmin.d, o));
            const int ds = __shfl_xor_sync(full, dslot, o);
            if (dmin > d || (dmin.v == d.v && ds < dslot)) {
                dmin = d;
                dslot = ds;
            }
        }
    }
    const TSolve o(g, s, i, l, sum);
    if (i < 0) return;
    const size_t at = 8 * (size_t)i + l;
    s.dqv[0][at] = l < 4 ? o.ox : o.oy;
    s.dqt[0][at] = l < 4 ? o.tx : o.ty;
    s.qmv[at] = ext.v;
    s.qmt[at] = ext.d;
    if (with_delta && l == 0) {
        s.dlv[i] = dmin.v;
        s.dlt[i] = dmin.d;
    }
}

// eval_q_inner_loop_d + eval_update_innerloop_d, dq buffer a -> b, in the
// primal's form dq0 + dq_i / 2 - L s / 2, s = sum of d (d . dq_k)
__global__ void __launch_bounds__(TB)
k_t_inner(Geom g, TanState s, int a, int b) {
    __shared__ double sm[T_PTS * T_P];
    const unsigned full = 0xffffffffu;
    const int l = threadIdx.x % LPP, m = l & 3;
    int i = blockIdx.x * T_PTS + threadIdx.x / LPP;
    double *row = sm + threadIdx.x / LPP * T_P;
    if (i >= g.n) i = -1;
    int nb = 0;
    Dual xi, yi;
    if (i >= 0) {
        nb = g.nbhs[i];
        xy_dual(g, s, i, xi, yi);
    }
    Dual sum;
    const int nbw = __reduce_max_sync(full, nb);
    for (int r0 = 0; r0 < nbw; r0 += LPP) {
        const int r = r0 + l;
        if (r < nb) {
            const int k = g.conn[(size_t)r * g.n + i];
            double xv[4], yv[4], xt[4], yt[4];
            ld4nc(s.dqv[a] + 8 * (size_t)k, xv);
            ld4nc(s.dqv[a] + 8 * (size_t)k + 4, yv);
            ld4nc(s.dqt[a] + 8 * (size_t)k, xt);
            ld4nc(s.dqt[a] + 8 * (size_t)k + 4, yt);
            Dual xk, yk;
            xy_dual(g, s, k, xk, yk);
            const Dual delx = xk - xi, dely = yk - yi;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const Dual t = delx * Dual(xv[f], xt[f]) + dely * Dual(yv[f], yt[f]);
                row[f * T_F + l] = t.v;
                row[(4 + f) * T_F + l] = t.d;
            }
            row[8 * T_F + l] = delx.v;
            row[9 * T_F + l] = dely.v;
            row[10 * T_F + l] = delx.d;
            row[11 * T_F + l] = dely.d;
        }
        __syncwarp();
        const double *tf = row + m * T_F, *wf = row + (8 + l / 4) * T_F;
#pragma unroll
        for (int j = 0; j < LPP; ++j) {
            if (r0 + j >= nb) break;
            sum += Dual(wf[j], wf[2 * T_F + j]) * Dual(tf[j], tf[4 * T_F + j]);
        }
        __syncwarp();
    }
    const TSolve o(g, s, i, l, sum);
    if (i < 0) return;
    const size_t at = 8 * (size_t)i + l;
    s.dqv[b][at] = s.dqv[0][at] + 0.5 * s.dqv[a][at] - 0.5 * (l < 4 ? o.ox : o.oy);
    s.dqt[b][at] = s.dqt[0][at] + 0.5 * s.dqt[a][at] - 0.5 * (l < 4 ? o.tx : o.ty);
}

// The split lists' solve coefficients (k_flux_coef of the primal) as Duals:
// per point and list a, b of the slot weight c = a dels + b deln (y lists: the
// roles swapped); and the derivative of the whole stencil's normal matrix.
// Geometry: once per call.
__global__ void __launch_bounds__(TB)
k_t_coef(Geom g, TanState s, Dual *__restrict__ co) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const int kind = i < g.nw ? KIND_WALL : (i < g.nw + g.no ? KIND_OUTER : KIND_INTERIOR);
    Dual xi, yi;
    xy_dual(g, s, i, xi, yi);
    const Dual nx(g.nrm[i].x, s.nrm_t[i].x), ny(g.nrm[i].y, s.nrm_t[i].y);
    const unsigned long long bits[2] = {g.mx[i], g.my[i]};
    Dual sxx[4], syy[4], sxy[4];
    double mxx = 0.0, myy = 0.0, mxy = 0.0;
    for (int r = 0; r < g.nbhs[i]; ++r) {
        Dual xk, yk;
        xy_dual(g, s, g.conn[(size_t)r * g.n + i], xk, yk);
        const Dual delx = xk - xi, dely = yk - yi;
        mxx += 2.0 * delx.v * delx.d;
        myy += 2.0 * dely.v * dely.d;
        mxy += delx.v * dely.d + delx.d * dely.v;
        const Dual dels = delx * ny - dely * nx, deln = delx * nx + dely * ny;
        const Dual a = dels * dels, b = deln * deln, c = dels * deln;
#pragma unroll
        for (int L = 0; L < 4; ++L) {
            if (!((bits[L >> 1] >> (r + ((L & 1) ? 32 : 0))) & 1ull)) continue;
            sxx[L] += a;
            syy[L] += b;
            sxy[L] += c;
        }
    }
#pragma unroll
    for (int L = 0; L < 4; ++L) {
        const bool none = (kind == KIND_WALL && L == 2) || (kind == KIND_OUTER && L == 3);
        const Dual ob = Dual(1.0) / (sxx[L] * syy[L] - sxy[L] * sxy[L]);
        co[8 * (size_t)i + 2 * L] = none ? Dual() : (L < 2 ? syy[L] : sxx[L]) * ob;
        co[8 * (size_t)i + 2 * L + 1] = none ? Dual() : -(sxy[L] * ob);
    }
    s.mt[4 * (size_t)i] = mxx;
    s.mt[4 * (size_t)i + 1] = myy;
    s.mt[4 * (size_t)i + 2] = mxy;
    s.mt[4 * (size_t)i + 3] = 0.0;
}

// limited_qtilde (flux_math.cuh) on Duals.
__device__ __forceinline__ Dual limited_dual(Dual t, Dual q, Dual qmax, Dual qmin, double eps2) {
    const Dual dn(-0.5 * t.v, -0.5 * t.d);
    const Dual dp = (dn.v > 0.0 ? qmax : qmin) - q;
    const Dual a = dp * dp + Dual(eps2);
    const Dual num = a - t * dp, den = a + dn * (dp - t);
    const double id = rcp_h3(den.v), f = num.v * id;
    const bool act = f < 1.0 && ::fabs(dn.v) > MFCFD_VENKAT_THR;
    const Dual phi(act ? f : 1.0, act ? (num.d - f * den.d) * id : 0.0);
    return q + phi * dn;
}

// The derivative of a kinetic state (values s, velocity u) from its limited
// qtilde's (kstate_pre / kstate_pair of flux_math.cuh, differentiated).
__device__ __forceinline__ KStateT<Dual> kstate_dual(const KState &s, const double u[2],
                                                     const Dual qt[4], Dual nx, Dual ny) {
    const double beta = -0.5 * qt[3].v, dbeta = -0.5 * qt[3].d;
    const double sb = beta * rsqrt_h3(beta), dsb = sb * s.pbr * dbeta;
    const double dpbr = s.pbr * s.pbr * qt[3].d;
    const double du1 = qt[1].d * s.pbr + qt[1].v * dpbr, du2 = qt[2].d * s.pbr + qt[2].v * dpbr;
    KStateT<Dual> k;
    k.pbr = Dual(s.pbr, dpbr);
    k.usq = Dual(s.usq, 2.0 * (u[0] * du1 + u[1] * du2));
    const double dtexp = qt[0].d + dbeta * s.usq + beta * k.usq.d;
    k.rho = Dual(s.rho, s.rho * (dtexp - 5.0 * s.pbr * dbeta));  // 2.5 / beta = 5 p/rho
    k.ut = Dual(s.ut, du1 * ny.v + u[0] * ny.d - (du2 * nx.v + u[1] * nx.d));
    k.un = Dual(s.un, du1 * nx.v + u[0] * nx.d + (du2 * ny.v + u[1] * ny.d));
    const double S1 = s.ut * sb, S2 = s.un * sb;
    const double dS1 = k.ut.d * sb + s.ut * dsb, dS2 = k.un.d * sb + s.un * dsb;
    // B = E h with h = 1 / (2 sqrt(pi beta)), so E = 2 sqrt(pi) sb B and dh = -h p/rho dbeta;
    // d erf(S) = 2/sqrt(pi) E dS = 4 sb B dS
    k.B1 = Dual(s.B1, -s.B1 * (2.0 * S1 * dS1 + s.pbr * dbeta));
    k.B2 = Dual(s.B2, -s.B2 * (2.0 * S2 * dS2 + s.pbr * dbeta));
    k.e1 = Dual(s.e1, 4.0 * sb * s.B1 * dS1);
    k.e2 = Dual(s.e2, 4.0 * sb * s.B2 * dS2);
    return k;
}

// flux_split (flux_math.cuh) on Duals.
__device__ __forceinline__ void flux_split_dual(const KStateT<Dual> &s, Dual u, Dual o, Dual B,
                                                Dual e, double sg, Dual G[4]) {
    const Dual A(0.5 + 0.5 * sg * e.v, 0.5 * sg * e.d);
    const Dual a = u * A + Dual(sg * B.v, sg * B.d);
    const Dual pA = s.pbr * A;
    const Dual w6(6.0 * s.pbr.v + s.usq.v, 6.0 * s.pbr.d + s.usq.d);
    G[0] = s.rho * a;
    G[1] = s.rho * (u * a + pA);
    G[2] = o * G[0];
    G[3] = Dual(0.5 * s.rho.v, 0.5 * s.rho.d) * (w6 * a + u * pA);
}

// cal_flux_residual_d: eight lanes a point, one slot a lane, and the pooled
// slot weights of the primal flux pass; the sum of the list derivatives as
// four values, then four derivatives, into fs [n][8].  67 us at 64,000 points
// with one state at a time and the neighbour's own list of each direction (3
// blocks of 168 registers; 77 at 2 blocks, 73 at 4, which spill); 95 with both
// states live and a loop over the lists, which a warp ran for both; 354 as a
// thread a point with list sums of Duals.  Bound by latency at 12 warps an SM.
__global__ void __launch_bounds__(TB, 3)
k_t_flux(Geom g, TanState s, int qc, int dqa, const Dual *__restrict__ coef,
         double *__restrict__ fs) {
    const int lane = threadIdx.x % LPP;
    const int i = (blockIdx.x * TB + threadIdx.x) / LPP;
    const bool valid = i < g.n;
    const int nb = valid ? g.nbhs[i] : 0;
    Dual v[4];
    for (int r = lane; r < nb; r += LPP) {
        const int kind = i < g.nw ? KIND_WALL : (i < g.nw + g.no ? KIND_OUTER : KIND_INTERIOR);
        const int k = g.conn[(size_t)r * g.n + i];
        Dual xi, yi, xk, yk;
        xy_dual(g, s, i, xi, yi);
        xy_dual(g, s, k, xk, yk);
        const Dual nx(g.nrm[i].x, s.nrm_t[i].x), ny(g.nrm[i].y, s.nrm_t[i].y);
        const Dual delx = xk - xi, dely = yk - yi;
        const Dual dels = delx * ny - dely * nx, deln = delx * nx + dely * ny;
        const Dual *co = coef + 8 * (size_t)i;
        // the lists holding the neighbour: one of each direction (lx, ly), in
        // both only when its projection is exactly 0 (tx, ty)
        const unsigned long long mx = g.mx[i] >> r, my = g.my[i] >> r;
        const int lx = mx & 1ull ? 0 : 1, ly = my & 1ull ? 0 : 1;
        const bool tx = (mx & (mx >> 32)) & 1ull, ty = (my & (my >> 32)) & 1ull;
        Dual Dt[4], Dn[4];  // differences of the fluxes along t and n
        // the point's state (h = 0), then the neighbour's, one at a time: both at
        // once take 255 registers
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const int p = h ? k : i;
            const double sgn = h ? 1.0 : -1.0;
            Dual qt[4];
            {
                double qv[4], qd[4], xv[4], yv[4], xd[4], yd[4], hv[4], lv[4], hd[4], ld[4];
                ld4nc(reinterpret_cast<const double *>(s.qv[qc] + p), qv);
                ld4nc(reinterpret_cast<const double *>(s.qt[qc] + p), qd);
                ld4nc(s.dqv[dqa] + 8 * (size_t)p, xv);
                ld4nc(s.dqv[dqa] + 8 * (size_t)p + 4, yv);
                ld4nc(s.dqt[dqa] + 8 * (size_t)p, xd);
                ld4nc(s.dqt[dqa] + 8 * (size_t)p + 4, yd);
                ld4nc(s.qmv + 8 * (size_t)p, hv);
                ld4nc(s.qmv + 8 * (size_t)p + 4, lv);
                ld4nc(s.qmt + 8 * (size_t)p, hd);
                ld4nc(s.qmt + 8 * (size_t)p + 4, ld);
                const double eps2 = g.eps2[p];
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    qt[m] = limited_dual(delx * Dual(xv[m], xd[m]) + dely * Dual(yv[m], yd[m]),
                                         Dual(qv[m], qd[m]), Dual(hv[m], hd[m]),
                                         Dual(lv[m], ld[m]), eps2);
            }
            KStateT<Dual> st;
            {
                const double q[4] = {qt[0].v, qt[1].v, qt[2].v, qt[3].v};
                KState vs, same;
                double u[2], w[2];
                kstate_pair(q, q, nx.v, ny.v, 0.56418958354775628695, vs, same, u, w);
                st = kstate_dual(vs, u, qt, nx, ny);
            }
            auto along_t = [&](int l, Dual G[4]) {
                const double sg = l ? -1.0 : 1.0;
                if (kind == KIND_INTERIOR)
                    flux_split_dual(st, st.ut, st.un, st.B1, st.e1, sg, G);
                else
                    flux_quad<Dual>(st, Dual(sg), Dual(kind == KIND_WALL ? -1.0 : 1.0), G);
            };
            auto along_n = [&](int l, Dual G[4]) {
                flux_split_dual(st, st.un, st.ut, st.B2, st.e2, l ? -1.0 : 1.0, G);
            };
            Dual G[4];
            along_t(lx, G);
#pragma unroll
            for (int m = 0; m < 4; ++m) Dt[m] = h ? G[m] - Dt[m] : G[m];
            along_n(ly, G);
#pragma unroll
            for (int m = 0; m < 4; ++m) Dn[m] = h ? G[m] - Dn[m] : G[m];
            if (tx) {
                const Dual w = Dual(sgn) * (co[2] * dels + co[3] * deln);
                along_t(1, G);
#pragma unroll
                for (int m = 0; m < 4; ++m) v[m] += w * G[m];
            }
            if (ty) {
                const Dual w = Dual(sgn) * (co[6] * deln + co[7] * dels);
                along_n(1, G);
                v[0] += w * G[0];
                v[1] += w * G[2];
                v[2] += w * G[1];
                v[3] += w * G[3];
            }
        }
        const Dual wx = co[2 * lx] * dels + co[2 * lx + 1] * deln;
        const Dual wy = co[4 + 2 * ly] * deln + co[5 + 2 * ly] * dels;
        v[0] += wx * Dt[0] + wy * Dn[0];
        v[1] += wx * Dt[1] + wy * Dn[2];
        v[2] += wx * Dt[2] + wy * Dn[1];
        v[3] += wx * Dt[3] + wy * Dn[3];
    }
    __syncwarp();
    // lane t of a point gets entry t of (four values, four derivatives)
    const unsigned full = 0xffffffffu;
    const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
    double a[4], b[2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
        a[m] = (h4 ? v[m].d : v[m].v) + __shfl_xor_sync(full, h4 ? v[m].v : v[m].d, 4);
#pragma unroll
    for (int m = 0; m < 2; ++m)
        b[m] = (h2 ? a[2 + m] : a[m]) + __shfl_xor_sync(full, h2 ? a[m] : a[2 + m], 2);
    const double sum = (h1 ? b[1] : b[0]) + __shfl_xor_sync(full, h1 ? b[0] : b[1], 1);
    if (valid) fs[8 * (size_t)i + lane] = sum;
}

// state_update_d (state_update_d.F90) + eval_q_variables_d of the new state.
__global__ void __launch_bounds__(TB)
k_t_update(Geom g, Consts c, TanState s, const double *__restrict__ fs, int A, int B, int qc,
           int rk, int last) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const int kind = i < g.nw ? KIND_WALL : (i < g.nw + g.no ? KIND_OUTER : KIND_INTERIOR);
    const Dual nx(g.nrm[i].x, s.nrm_t[i].x), ny(g.nrm[i].y, s.nrm_t[i].y);
    const Dual pi_c(c.pi), gm1(c.gm1);
    Dual delta(s.dlv[i], s.dlt[i]);
    if (kind == KIND_WALL) delta = Dual(2.0) * delta;
    Dual fr[4];
    for (int m = 0; m < 4; ++m)
        fr[m] = delta * Dual(fs[8 * (size_t)i + m], fs[8 * (size_t)i + 4 + m]);
    Dual P[4], U[4], Uo[4];
    ld_dual4(rk == 1 ? s.pv[A] : s.pv[B], rk == 1 ? s.pt[A] : s.pt[B], i, P);
    if (kind == KIND_OUTER) {
        const Dual *inf = s.obc + 8 * (size_t)(i - g.nw);
        conserved_ubar_t<Dual>(P[0], P[1], P[2], P[3], nx, ny, inf, pi_c, gm1, U);
        if (rk == 3) {
            Dual O[4];
            ld_dual4(s.pv[A], s.pt[A], i, O);
            conserved_ubar_t<Dual>(O[0], O[1], O[2], O[3], nx, ny, inf, pi_c, gm1, Uo);
        }
    } else {
        prim_to_conserved_t<Dual>(P[0], P[1], P[2], P[3], nx, ny, U);
        if (rk == 3) {
            Dual O[4];
            ld_dual4(s.pv[A], s.pt[A], i, O);
            prim_to_conserved_t<Dual>(O[0], O[1], O[2], O[3], nx, ny, Uo);
        }
    }
    for (int m = 0; m < 4; ++m) {
        if (rk != 3) U[m] = U[m] - (Dual(0.5 * c.euler) * fr[m]);
        else U[m] = Dual(TBT) * Uo[m] + Dual(OBT) * (U[m] - Dual(0.5) * fr[m]);
    }
    if (kind == KIND_WALL) U[2] = Dual(0.0);
    const Dual U2_rot = U[1], U3_rot = U[2];
    U[1] = U2_rot * ny + U3_rot * nx;
    U[2] = U3_rot * ny - U2_rot * nx;
    Dual out[4], qn[4];
    out[0] = U[0];
    const Dual temp = Dual(1.0) / U[0];
    out[1] = U[1] * temp;
    out[2] = U[2] * temp;
    out[3] = Dual(0.4) * (U[3] - (Dual(0.5) * temp) * (U[1] * U[1] + U[2] * U[2]));
    st_dual4(s.pv[B], s.pt[B], i, out);
    q_from_prim_t<Dual>(out[0], out[1], out[2], out[3], qn);
    st_dual4(s.qv[qc ^ 1], s.qt[qc ^ 1], i, qn);
    if (last) {
        const Dual spd = sqrt(out[1] * out[1] + out[2] * out[2]) + Dual(3.0) * sqrt(out[3] / out[0]);
        s.spv[i] = spd.v;
        s.spt[i] = spd.d;
    }
}

struct TanShape {
    int npts, shapes;
    const int *idx, *left, *right, *shape;
};

// compute_cl_cd_cm_d (compute_force_coeffs_d.F90): out[0] = J, out[1] =
// dJ/de.  One block: the points' terms in parallel, thread 0 adds them shape by
// shape in grid order (the reference's).
constexpr int TF = 512;
__global__ void __launch_bounds__(TF)
k_t_forces(Geom g, TanState s, TanShape t, int cur, double mach, double cos_t, double sin_t,
           int objective, double *out) {
    __shared__ double2 th[TF], tv[TF];  // value, derivative
    __shared__ int ts[TF];
    const double pr_inf = 1.0 / 1.4;
    const Dual temp(0.5 * 1.0 * mach * mach);
    Dual J;
    for (int sh = 0; sh < t.shapes; ++sh) {
        Dual H, V;
        for (int j0 = 0; j0 < t.npts; j0 += TF) {
            const int j = j0 + threadIdx.x;
            if (j < t.npts) {
                const int m = t.idx[j], l = t.left[j], r = t.right[j];
                Dual lx, ly, mxx, myy, rx, ry;
                xy_dual(g, s, l, lx, ly);
                xy_dual(g, s, m, mxx, myy);
                xy_dual(g, s, r, rx, ry);
                const Dual ds1 = sqrt((mxx - lx) * (mxx - lx) + (myy - ly) * (myy - ly));
                const Dual ds2 = sqrt((rx - mxx) * (rx - mxx) + (ry - myy) * (ry - myy));
                const Dual ds = Dual(0.5) * (ds1 + ds2);
                const Dual nx(g.nrm[m].x, s.nrm_t[m].x), ny(g.nrm[m].y, s.nrm_t[m].y);
                Dual cp = Dual(s.pv[cur][m].d, s.pt[cur][m].d) - Dual(pr_inf);
                cp = -cp / temp;
                const Dual h = cp * nx * ds, v = cp * ny * ds;
                th[threadIdx.x] = make_double2(h.v, h.d);
                tv[threadIdx.x] = make_double2(v.v, v.d);
                ts[threadIdx.x] = t.shape[j];
            }
            __syncthreads();
            if (threadIdx.x == 0)
                for (int q = 0; q < min(TF, t.npts - j0); ++q)
                    if (ts[q] == sh) {
                        H += Dual(th[q].x, th[q].y);
                        V += Dual(tv[q].x, tv[q].y);
                    }
            __syncthreads();
        }
        const Dual cl = V * Dual(cos_t) - H * Dual(sin_t);
        const Dual cd = H * Dual(cos_t) + V * Dual(sin_t);
        J = J + (objective == 1 ? cd : cl);
    }
    if (threadIdx.x == 0) {
        out[0] = J.v;
        out[1] = J.d;
    }
}

// The seed in the handle's point order, d the caller-order directions (dx, then
// dy; a missing one is zero).
__global__ void k_t_seed(int n, const int *__restrict__ perm, const double *__restrict__ d,
                         double2 *__restrict__ xy_t, double2 *__restrict__ nrm_t) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    xy_t[p] = make_double2(d[perm[p]], d[n + perm[p]]);
    nrm_t[p] = make_double2(0.0, 0.0);
}

// point_normals_d.F90 of the boundary points and, of the outer ones, the
// freestream half of Ubar (state_update.F90:248-263) with its derivative.
__global__ void k_t_normals(Geom g, TanState s, const int *__restrict__ left,
                            const int *__restrict__ right, double u1_inf, double u2_inf,
                            double pi, double2 *__restrict__ nrm_t, Dual *__restrict__ obc) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= g.nw + g.no) return;
    Dual lx, ly, mx, my, rx, ry;
    xy_dual(g, s, left[p], lx, ly);
    xy_dual(g, s, p, mx, my);
    xy_dual(g, s, right[p], rx, ry);
    const Dual vx = Dual(0.5) * ((my - ly) + (ry - my)), vy = Dual(0.5) * ((mx - lx) + (rx - mx));
    const Dual det = sqrt(vx * vx + vy * vy);
    const Dual dnx = -vx / det, dny = vy / det;
    nrm_t[p] = make_double2(dnx.d, dny.d);
    if (p < g.nw) return;
    const double pr_inf = 1.0 / 1.4, rho_inf = 1.0, gamma = 1.4;
    const Dual nx(g.nrm[p].x, dnx.d), ny(g.nrm[p].y, dny.d);
    const Dual u1r = Dual(u1_inf) * ny - Dual(u2_inf) * nx;
    const Dual u2r = Dual(u1_inf) * nx + Dual(u2_inf) * ny;
    const double beta = (0.5 * rho_inf) / pr_inf;
    const Dual S2 = u2r * Dual(::sqrt(beta));
    Dual *o = obc + 8 * (size_t)(p - g.nw);
    o[0] = u1r;
    o[1] = u2r;
    o[2] = Dual(pr_inf / (rho_inf * (gamma - 1.0))) + Dual(0.5) * (u1r * u1r + u2r * u2r);
    o[3] = Dual(0.5) * (Dual(1.0) - erf(S2));
    o[4] = exp(-S2 * S2) / Dual(2.0 * ::sqrt(pi * beta));
}

// Per-point terms of the secondary objectives (compute_entropy.F90:21-27,
// compute_enstrophy.F90:27-79, stagnation_values.F90:60-67), as Duals.
__global__ void k_t_obj_terms(Geom g, TanState s, int cur, int kind, double gamma_power,
                              double p0_inf, double *__restrict__ tv, double *__restrict__ td) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const Dual gamma(1.4), pr_inf(1.0 / 1.4);
    Dual P[4];
    ld_dual4(s.pv[cur], s.pt[cur], i, P);
    Dual t;
    if (kind == MFCFD_OBJ_ENTROPY) {
        // rho**gamma = exp(gamma log rho)
        Dual temp1 = exp(gamma * log(P[0]));
        temp1 = P[3] / temp1;
        temp1 = log(temp1);
        t = fabs(temp1 - log(pr_inf));
    } else if (kind == MFCFD_OBJ_STAGNATION) {
        const Dual m2 = (P[1] * P[1] + P[2] * P[2]) / (gamma * P[3] / P[0]);
        const Dual A = Dual(1.0) + Dual((1.4 - 1) / 2) * m2;
        const Dual d = Dual(p0_inf) - P[3] * exp(Dual(gamma_power) * log(A));
        t = d * d;
    } else {
        Dual xi, yi;
        xy_dual(g, s, i, xi, yi);
        Dual sxx, syy, sxy, sxu1, sxu2, syu1, syu2;
        const int nb = g.nbhs[i];
        for (int r = 0; r < nb; ++r) {
            const int k = g.conn[r * g.n + i];
            Dual xk, yk, Q[4];
            xy_dual(g, s, k, xk, yk);
            ld_dual4(s.pv[cur], s.pt[cur], k, Q);
            const Dual delx = xk - xi, dely = yk - yi;
            sxx = sxx + delx * delx;
            syy = syy + dely * dely;
            sxy = sxy + delx * dely;
            sxu1 = sxu1 + delx * (Q[1] - P[1]);
            sxu2 = sxu2 + delx * (Q[2] - P[2]);
            syu1 = syu1 + dely * (Q[1] - P[1]);
            syu2 = syu2 + dely * (Q[2] - P[2]);
        }
        const Dual one_by_det = Dual(1.0) / (sxx * syy - sxy * sxy);
        const Dual w = (sxu2 * syy - syu2 * sxy) * one_by_det - (syu1 * sxx - sxu1 * sxy) * one_by_det;
        t = w * w;
    }
    tv[i] = t.v;
    td[i] = t.d;
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

// Device workspace of mfcfd_tangent: one allocation of about 1.1 KB a point (27
// allocations and frees a call took longer than ten iterations of 64,000 points).
// Up to TAN_KEEP bytes it stays with the handle until mfcfd_destroy or until the
// handle's adjoint is set up (drop_tangent): an allocation and its release take 0.65 ms at
// best and 1.8 on average at 77 MB, of 4.4 ms for ten iterations of 64,000 points.
// A larger one (from some 120,000 points on) is released by the call itself, so
// that other handles and the caller's own allocator find the memory a call found
// (ten iterations, kept / released: 256,000 points 17.6 / 18.7 ms, 1,024,000 points
// 67.5 / 69.8).
constexpr size_t TAN_KEEP = 128u << 20;
struct TanWork {
    char *block = nullptr;
    size_t bytes = 0;
    TanState s{};
    double2 *xy_t = nullptr, *nrm_t = nullptr;
    Dual *obc = nullptr, *coef = nullptr;
    double *fs = nullptr, *dir = nullptr, *out = nullptr;
    int *left = nullptr, *right = nullptr;  // ring neighbours of the boundary points
    int *si = nullptr, *sl = nullptr, *sr = nullptr, *ss = nullptr;  // shape points, grid order
    int nshape = 0;
};

void lskum_host::drop_tangent(mfcfd_t *h) {
    if (!h->tan) return;
    if (h->tan->block) cudaFree(h->tan->block);
    delete h->tan;
    h->tan = nullptr;
}

namespace {

int tan_setup(mfcfd_t *h) {
    if (h->tan) return MFCFD_OK;
    const int n = h->n, nw = h->nw, no = h->no;
    std::vector<int> inv(n);
    for (int p = 0; p < n; ++p) inv[h->perm[p]] = p;
    std::vector<int> idx[6];  // left, right, si, sl, sr, ss
    for (int p = 0; p < nw + no; ++p) {
        idx[0].push_back(inv[h->left0[h->perm[p]] - 1]);
        idx[1].push_back(inv[h->right0[h->perm[p]] - 1]);
    }
    for (int i = 0; i < n; ++i) {
        if (h->flag2_0[i] <= 0) continue;
        idx[2].push_back(inv[i]);
        idx[3].push_back(inv[h->left0[i] - 1]);
        idx[4].push_back(inv[h->right0[i] - 1]);
        idx[5].push_back(h->flag2_0[i] - 1);
    }
    TanWork *w = new (std::nothrow) TanWork();
    if (!w) return fail(h, MFCFD_ERR_OOM, "host allocation failed");
    w->nshape = (int)idx[2].size();
    // the same walk sizes the block, then hands out its parts
    size_t bytes = 0;
    for (int pass = 0; pass < 2; ++pass) {
        size_t at = 0;
        auto take = [&](auto *&p, size_t count) {
            using T = std::remove_reference_t<decltype(*p)>;
            if (pass) p = reinterpret_cast<T *>(w->block + at);
            at += (count * sizeof(T) + 255) / 256 * 256;
        };
        TanState &s = w->s;
        for (int b = 0; b < 2; ++b) {
            take(s.pv[b], n);
            take(s.pt[b], n);
            take(s.qv[b], n);
            take(s.qt[b], n);
        }
        for (int b = 0; b < 3; ++b) {
            if (b > h->p.inner_iterations) break;
            take(s.dqv[b], (size_t)8 * n);
            take(s.dqt[b], (size_t)8 * n);
        }
        take(s.mt, (size_t)4 * n);
        take(s.qmv, (size_t)8 * n);
        take(s.qmt, (size_t)8 * n);
        take(s.dlv, n);
        take(s.dlt, n);
        take(s.spv, n);
        take(s.spt, n);
        take(w->xy_t, n);
        take(w->nrm_t, n);
        take(w->obc, (size_t)8 * std::max(no, 1));
        take(w->coef, (size_t)8 * n);
        take(w->fs, (size_t)8 * n);
        take(w->dir, (size_t)2 * n);
        take(w->out, 2);
        int **ints[6] = {&w->left, &w->right, &w->si, &w->sl, &w->sr, &w->ss};
        for (int a = 0; a < 6; ++a) take(*ints[a], std::max<size_t>(idx[a].size(), 1));
        if (pass) break;
        bytes = at;
        cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&w->block), bytes);
        if (e != cudaSuccess) {
            delete w;
            return cuda_fail(h, e, "mfcfd_tangent cudaMalloc");
        }
        w->bytes = bytes;
    }
    w->s.xy_t = w->xy_t;
    w->s.nrm_t = w->nrm_t;
    w->s.obc = w->obc;
    h->tan = w;
    int *dst[6] = {w->left, w->right, w->si, w->sl, w->sr, w->ss};
    for (int a = 0; a < 6; ++a)
        if (!idx[a].empty()) {
            cudaError_t e = cudaMemcpy(dst[a], idx[a].data(), idx[a].size() * sizeof(int),
                                       cudaMemcpyHostToDevice);
            if (e != cudaSuccess) {
                lskum_host::drop_tangent(h);
                return cuda_fail(h, e, "mfcfd_tangent cudaMemcpy");
            }
        }
    return MFCFD_OK;
}

}  // namespace

extern "C" int mfcfd_tangent(mfcfd_t *h, int objective, int n_iters, const double *dx,
                             const double *dy, double *J, double *dJ) {
    if (!h) return MFCFD_ERR_ARG;
    if (objective < MFCFD_OBJ_CL || objective > MFCFD_OBJ_STAGNATION)
        return fail(h, MFCFD_ERR_ARG, "objective must be 0..4");
    if (n_iters < 0) return fail(h, MFCFD_ERR_ARG, "n_iters < 0");
    if (h->fp32 || h->p.power != 0.0)
        return fail(h, MFCFD_ERR_ARG, "mfcfd_tangent needs an FP64 handle with power = 0");
    const int n = h->n, nw = h->nw, no = h->no, m = h->p.inner_iterations, rks = h->p.rks;
    DevGuard dg(h->dev);
    CK(dg.err);
    CK(cudaStreamSynchronize(h->stream));
    if (int st = tan_setup(h)) return st;
    // on every way out (cudaFree waits for the device)
    struct Release {
        mfcfd_t *h;
        ~Release() {
            if (h->tan && h->tan->bytes > TAN_KEEP) lskum_host::drop_tangent(h);
        }
    } release{h};
    const TanWork &w = *h->tan;
    const TanState &s = w.s;
    cudaStream_t str = h->stream;
    // the seed and the geometry's derivatives
    if (dx) CK(cudaMemcpyAsync(w.dir, dx, sizeof(double) * n, cudaMemcpyHostToDevice, str));
    else CK(cudaMemsetAsync(w.dir, 0, sizeof(double) * n, str));
    if (dy) CK(cudaMemcpyAsync(w.dir + n, dy, sizeof(double) * n, cudaMemcpyHostToDevice, str));
    else CK(cudaMemsetAsync(w.dir + n, 0, sizeof(double) * n, str));
    k_t_seed<<<nblk(n, 256), 256, 0, str>>>(n, h->d_perm, w.dir, w.xy_t, w.nrm_t);
    if (nw + no > 0)
        k_t_normals<<<nblk(nw + no, 128), 128, 0, str>>>(h->geom, s, w.left, w.right, h->q_inf[1],
                                                         h->q_inf[2], h->pi, w.nrm_t, w.obc);
    k_t_coef<<<nblk(n, TB), TB, 0, str>>>(h->geom, s, w.coef);
    // the handle's state (held fixed: derivative 0)
    CK(cudaMemcpyAsync(s.pv[0], h->d_prim[h->cur], sizeof(R4) * n, cudaMemcpyDeviceToDevice, str));
    CK(cudaMemsetAsync(s.pt[0], 0, sizeof(R4) * n, str));
    int cur = 0, qc = 0;
    k_t_init<<<nblk(n, 256), 256, 0, str>>>(n, s, cur, qc);
    h->launches += 4;
    for (int it = 0; it < n_iters; ++it) {
        const int A = cur, B = cur ^ 1;
        for (int rk = 1; rk <= rks; ++rk) {
            auto dq = [](int t) { return t == 0 ? 0 : 2 - (t & 1); };  // buffer of iteration t
            k_t_grad<<<nblk(n, T_PTS), TB, 0, str>>>(h->geom, h->consts, s, qc, rk == 1 ? 1 : 0);
            for (int t = 1; t <= m; ++t)
                k_t_inner<<<nblk(n, T_PTS), TB, 0, str>>>(h->geom, s, dq(t - 1), dq(t));
            k_t_flux<<<nblk(n, TB / LPP), TB, 0, str>>>(h->geom, s, qc, dq(m), w.coef, w.fs);
            k_t_update<<<nblk(n, TB), TB, 0, str>>>(h->geom, h->consts, s, w.fs, A, B, qc, rk,
                                                   rk == rks ? 1 : 0);
            qc ^= 1;
            h->launches += 3 + m;
        }
        cur = B;
        CK(cudaGetLastError());
    }
    if (objective >= MFCFD_OBJ_ENTROPY) {
        // secondary objectives: per-point Dual terms, summed in caller order
        double *d_tv = w.fs, *d_td = w.fs + n;  // (the flux sums are done with)
        const double gp = lskum_host::stagnation_gamma_power();
        const double p0_inf = lskum_host::stagnation_p0_inf(h->p.mach);
        k_t_obj_terms<<<nblk(n, 256), 256, 0, str>>>(h->geom, s, cur, objective, gp, p0_inf, d_tv,
                                                     d_td);
        h->launches += 1;
        CK(cudaGetLastError());
        std::vector<double> tv(n), td(n);
        CK(cudaMemcpyAsync(tv.data(), d_tv, sizeof(double) * n, cudaMemcpyDeviceToHost, str));
        CK(cudaMemcpyAsync(td.data(), d_td, sizeof(double) * n, cudaMemcpyDeviceToHost, str));
        CK(cudaStreamSynchronize(str));
        std::vector<int> inv(n);
        for (int p = 0; p < n; ++p) inv[h->perm[p]] = p;
        Dual sum;
        for (int k = 0; k < n; ++k) sum = sum + Dual(tv[inv[k]], td[inv[k]]);
        if (objective == MFCFD_OBJ_STAGNATION) sum = sum * Dual(1 / (p0_inf * p0_inf * n));
        if (J) *J = sum.v;
        if (dJ) *dJ = sum.d;
        return MFCFD_OK;
    }
    const TanShape ts{w.nshape, h->shapes, w.si, w.sl, w.sr, w.ss};
    k_t_forces<<<1, TF, 0, str>>>(h->geom, s, ts, cur, h->p.mach, h->cos_t, h->sin_t, objective,
                                  w.out);
    h->launches += 1;
    CK(cudaGetLastError());
    double o[2] = {0.0, 0.0};
    CK(cudaMemcpyAsync(o, w.out, sizeof(o), cudaMemcpyDeviceToHost, str));
    CK(cudaStreamSynchronize(str));
    if (J) *J = o[0];
    if (dJ) *dJ = o[1];
    return MFCFD_OK;
}
