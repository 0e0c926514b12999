// Reverse (adjoint) kernels of the LSKUM pseudo-time loop, FP64.
//
// One pseudo-time stage reverses in the order
//   k_update_b   state_update_b      prim_out_b -> prim_in_b, prim_old_b, flux_res_b, n_b
//   k_flux_b     cal_flux_residual_b flux_res_b -> q_b, dq_b, qm_b, x_b, y_b, n_b, delta_b
//   k_inner_b    eval_q_inner_loop_b (per inner iteration, last first)
//   k_grad_b     eval_q_derivatives_b + func_delta_b (first stage), and
//                eval_q_variables_b  q_b -> prim_in_b
// (the stage-by-stage order of the reference's FPI_SOLVER_B,
// src_mpi_adjoint/sensitivity_files/fpi_solver_b.F90:28-156).
//
// A point's adjoint flows to its neighbours without atomics: one thread per
// neighbour pulls it over the slots (i, r) naming it, in the fixed (i, r) order
// of the transposed stencil, from what the slot's point left behind -- a record
// per slot in the flux reverse, a record per point in the least-squares
// reverses.  Results are deterministic.
#include <cuda_runtime.h>

#include <algorithm>

#include "adjoint.h"
#include "flux_tile.cuh"
#include "lskum_adjoint.cuh"

namespace lskum {

namespace {

constexpr int BLK = 128;
constexpr int GROUPS = BLK / LPP;
// Lanes a point of the neighbours' sides on a small grid (slot_passes; their
// blocks are then about one wave), a transposed slot a lane in turn: adjoint of 8
// iterations with one inner iteration, 4 lanes / 1: 2.38 / 2.63 ms at 1,536
// points, 3.85 / 4.15 at 16,000, 4.81 / 4.87 at 24,000, 6.63 / 6.55 at 40,000.
constexpr int FEW_LANES = 4;
constexpr double OBT = 1.0 / 3.0;
constexpr double TBT = 2.0 / 3.0;

__device__ __forceinline__ void ld8a(const double *p, double a[4], double b[4]) {
    const double2 *v = reinterpret_cast<const double2 *>(p);
    double2 t0 = v[0], t1 = v[1], t2 = v[2], t3 = v[3];
    a[0] = t0.x; a[1] = t0.y; a[2] = t1.x; a[3] = t1.y;
    b[0] = t2.x; b[1] = t2.y; b[2] = t3.x; b[3] = t3.y;
}

// Sum of v over W neighbouring lanes (whole warps).
template <int W>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = W / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int W>
__device__ __forceinline__ void lanes_sum(double v[4]) {
#pragma unroll
    for (int m = 0; m < 4; ++m) v[m] = lane_sum<W>(v[m]);
}

// A kinetic state from its tape entry (rho, p/rho, B1, B2, e1, e2, u1, u2)
// and the point's normal, as kstate_pair forms ut, un and |u|^2.
__device__ __forceinline__ KState kst_taped(const double *v, double nx, double ny) {
    KState s;
    const double tx = ny, ty = -nx;
    s.rho = v[0];
    s.pbr = v[1];
    s.B1 = v[2];
    s.B2 = v[3];
    s.e1 = v[4];
    s.e2 = v[5];
    s.ut = v[6] * tx + v[7] * ty;
    s.un = v[6] * nx + v[7] * ny;
    s.usq = fma(v[6], v[6], v[7] * v[7]);
    return s;
}

// Stores n (even) doubles as 16-byte pairs; dst is 16-byte aligned (records
// are an even number of doubles from an aligned base).
__device__ __forceinline__ void st_pairs(double *dst, const double *v, int n) {
    double2 *d2 = reinterpret_cast<double2 *>(dst);
#pragma unroll
    for (int h = 0; h < n / 2; ++h) d2[h] = make_double2(v[2 * h], v[2 * h + 1]);
}

// dst[j] += v[j] for n (even) doubles, as 16-byte pairs (dst 16-byte aligned)
__device__ __forceinline__ void add_pairs(double *dst, const double *v, int n) {
    double2 *d2 = reinterpret_cast<double2 *>(dst);
#pragma unroll
    for (int h = 0; h < n / 2; ++h) {
        double2 t = d2[h];
        t.x = t.x + v[2 * h];
        t.y = t.y + v[2 * h + 1];
        d2[h] = t;
    }
}

// state_update_b (state_update.F90:10-141, reverse)
__global__ void __launch_bounds__(BLK, 3)
k_update_b(Geom g, Consts c, AdjConsts a, const R4 *__restrict__ prim_in,
           const R4 *__restrict__ prim_old, const R4 *__restrict__ fr,
           const double *__restrict__ pb_out, double *__restrict__ pb_in,
           double *__restrict__ pb_old, double *__restrict__ frb, double *__restrict__ nxb,
           double *__restrict__ nyb, int rk) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const int kind = i < g.nw ? KIND_WALL : (i < g.nw + g.no ? KIND_OUTER : KIND_INTERIOR);
    const double2 nn = g.nrm[i];
    const double nx = nn.x, ny = nn.y;
    const R4 P = ld4(prim_in + i);
    const R4 F = ld4(fr + i);
    const double frv[4] = {F.a, F.b, F.c, F.d};
    double U[4], Uo[4] = {0.0, 0.0, 0.0, 0.0};
    R4 O{0.0, 0.0, 0.0, 0.0};
    if (kind == KIND_OUTER) {
        const double *inf = g.obc + 8 * (size_t)(i - g.nw);
        conserved_ubar(P.a, P.b, P.c, P.d, nx, ny, inf, c.pi, c.gm1, U);
        if (rk == 3) {
            O = ld4(prim_old + i);
            conserved_ubar(O.a, O.b, O.c, O.d, nx, ny, inf, c.pi, c.gm1, Uo);
        }
    } else {
        prim_to_conserved(P.a, P.b, P.c, P.d, nx, ny, U);
        if (rk == 3) {
            O = ld4(prim_old + i);
            prim_to_conserved(O.a, O.b, O.c, O.d, nx, ny, Uo);
        }
    }
    double Up[4];
    for (int m = 0; m < 4; ++m) {
        if (rk != 3) Up[m] = U[m] - (0.5 * c.euler * frv[m]);
        else Up[m] = TBT * Uo[m] + OBT * (U[m] - 0.5 * frv[m]);
    }
    if (kind == KIND_WALL) Up[2] = 0.0;
    const double V1 = Up[1] * ny + Up[2] * nx;
    const double V2 = Up[2] * ny - Up[1] * nx;
    const double V0 = Up[0];
    const double tmp = 1.0 / V0;
    // reverse of prim_out = (V0, V1 tmp, V2 tmp, 0.4 (V3 - 0.5 tmp (V1^2 + V2^2)))
    const double *po = pb_out + 4 * (size_t)i;
    const double rb = po[0], u1b = po[1], u2b = po[2], pbv = po[3];
    const double inner = V1 * V1 + V2 * V2;
    const double V3b = 0.4 * pbv;
    double tmpb = -0.4 * 0.5 * inner * pbv;
    const double innerb = -0.4 * 0.5 * tmp * pbv;
    double V1b = 2.0 * V1 * innerb + u1b * tmp;
    double V2b = 2.0 * V2 * innerb + u2b * tmp;
    tmpb += u1b * V1 + u2b * V2;
    const double V0b = rb - tmpb * tmp * tmp;
    double Upb[4];
    Upb[0] = V0b;
    Upb[3] = V3b;
    Upb[1] = V1b * ny - V2b * nx;
    Upb[2] = V1b * nx + V2b * ny;
    double nxbv = V1b * Up[2] - V2b * Up[1];
    double nybv = V1b * Up[1] + V2b * Up[2];
    if (kind == KIND_WALL) Upb[2] = 0.0;
    double Ub[4], Uob[4], frbv[4];
    for (int m = 0; m < 4; ++m) {
        if (rk != 3) {
            Ub[m] = Upb[m];
            Uob[m] = 0.0;
            frbv[m] = -0.5 * c.euler * Upb[m];
        } else {
            Uob[m] = TBT * Upb[m];
            Ub[m] = OBT * Upb[m];
            frbv[m] = -0.5 * OBT * Upb[m];
        }
    }
    double pbi[4] = {0.0, 0.0, 0.0, 0.0}, pbo[4] = {0.0, 0.0, 0.0, 0.0};
    if (kind == KIND_OUTER) {
        conserved_ubar_b(P.a, P.b, P.c, P.d, nx, ny, a.q_inf, c.pi, c.gm1, Ub, pbi, nxbv, nybv);
        if (rk == 3)
            conserved_ubar_b(O.a, O.b, O.c, O.d, nx, ny, a.q_inf, c.pi, c.gm1, Uob, pbo, nxbv,
                             nybv);
    } else {
        prim_to_conserved_b(P.a, P.b, P.c, P.d, nx, ny, Ub, pbi, nxbv, nybv);
        if (rk == 3) prim_to_conserved_b(O.a, O.b, O.c, O.d, nx, ny, Uob, pbo, nxbv, nybv);
    }
    double *pin = pb_in + 4 * (size_t)i;
    // a middle stage's input adjoint begins here; the first stage's, which the
    // third stage has added to, is accumulated
    for (int m = 0; m < 4; ++m) pin[m] = rk == 1 ? pin[m] + pbi[m] : pbi[m];
    if (rk == 3) {
        double *pold = pb_old + 4 * (size_t)i;
        for (int m = 0; m < 4; ++m) pold[m] += pbo[m];
    }
    for (int m = 0; m < 4; ++m) frb[4 * (size_t)i + m] = frbv[m];
    nxb[i] += nxbv;
    nyb[i] += nybv;
}

// cal_flux_residual_b, eight lanes a point, one slot a lane, as in the forward
// flux pass.  With the list solves folded into slot weights (c = p . d, p the
// list's two coefficients, d = (dels, deln)), the flux residual is coef times
// the sum of c dG over slots and lists, so its reverse needs no list sums of
// the fluxes: with F = coef times the residual's adjoint, a slot's fluxes
// receive c F (the neighbour's) and -c F (the point's), and c receives F . dG.
// The time step's adjoint is the residual's dotted with the taped residual
// over the step.  The weights' own adjoint goes back through M p = e (M = sum
// d d^T over the list): with pb = sum cb d and z = M^-1 pb, each d receives
// -z c - p (z . d), two numbers a list summed over the point's lanes.
//
// Everything a warp's round reads but the neighbours' coordinates is copied to
// shared memory (cp.async) at its start, so the loads' latency is met once.
// 488 us at 256,000 points when the list sums and the reconstructions'
// primitive states went through shared-memory records, 404 with the folded
// weights, 226 with the copies, 214 with the own-point sums through shared
// memory instead of shuffles.  Bound by issue and by the one exposed load
// latency at 12 warps an SM (3 blocks of 168 registers; 4 spill: 269 us).
constexpr int FLUXB_MIN_BLOCKS = 3;
// A warp's shared memory: the taped states of its 32 slots (128 bytes padded
// to 144: a lane's pieces on distinct banks), its four points' rows, the
// slots' partial offset adjoints, z of each list.
struct FluxBSmem {
    double2 tape[32][KS_TAPE / 2 + 1];
    double2 more[80];  // (with the tape: the slots' own-point records)
    double2 q[4][2], dq[4][5], qm[4][5], co[4][4], fcg[4][2];
    double part[4][20][4];
    double z[4][8];
    // the own-point record of a slot: 20 doubles at a stride of 22, and 8 more
    // between points (a warp's stores and loads on distinct banks)
    __device__ __forceinline__ double2 *rec(int slot) {
        return &tape[0][0] + 11 * slot + 4 * (slot / LPP);
    }
};
static_assert(11 * 32 + 4 * 3 <= 32 * 9 + 80, "");
__global__ void __launch_bounds__(BLK, FLUXB_MIN_BLOCKS)
k_flux_b(Geom g, const R4 *__restrict__ q_in, const double *__restrict__ dq,
         const double *__restrict__ qm, const double *__restrict__ delta,
         const double *__restrict__ fr, const double *__restrict__ frb, double *__restrict__ qb,
         double *__restrict__ dqb, double *__restrict__ qmb, double *__restrict__ xb,
         double *__restrict__ yb, double *__restrict__ nxb, double *__restrict__ nyb,
         double *__restrict__ deltab, double *__restrict__ nbrec,
         const double *__restrict__ kst) {
    __shared__ FluxBSmem smem[BLK / 32];
    FluxBSmem &m = smem[threadIdx.x / 32];
    const int wl = threadIdx.x % 32, pg = wl / LPP, lane = wl % LPP;
    const int i0 = (blockIdx.x * BLK + threadIdx.x - wl) / LPP;  // the warp's first point
    const int i = i0 + pg;
    const bool valid = i < g.n;
    // copies
    const int part = wl % 8, sub = wl / 8;
    if (kst) {
        // piece `part` of slots 4 h + sub of points i0 + t
        const size_t row = (size_t)g.kp * KS_TAPE;
        const double *src = kst + i0 * row + sub * KS_TAPE + 2 * part;
        double2 *dst = &m.tape[sub][part];
        constexpr int TS = sizeof(m.tape[0]) / sizeof(double2);
#pragma unroll
        for (int t = 0; t < 4; ++t, src += row) {
            if (i0 + t >= g.n) break;
            if (sub < g.kp) halo_cp16(dst + (8 * t) * TS, src);
            if (4 + sub < g.kp) halo_cp16(dst + (8 * t + 4) * TS, src + 4 * KS_TAPE);
        }
    }
    if (i0 + sub < g.n) {
        const size_t o8 = 8 * (size_t)(i0 + sub);
        const int h = part & 3;
        if (part < 4) {
            halo_cp16(&m.dq[sub][h], dq + o8 + 2 * h);
            halo_cp16(&m.co[sub][h], g.fco + o8 + 2 * h);
        } else {
            halo_cp16(&m.qm[sub][h], qm + o8 + 2 * h);
            const double *q = reinterpret_cast<const double *>(q_in);
            if (h < 2) halo_cp16(&m.q[sub][h], q + o8 / 2 + 2 * h);
            else halo_cp16(&m.fcg[sub][h - 2], g.fcg + o8 / 2 + 2 * (h - 2));
        }
    }
    int nb = 0, kind = KIND_INTERIOR, k0 = 0;
    double nx = 0.0, ny = 1.0, eps2 = 0.0, geo_old = 0.0;
    double2 pi_ = make_double2(0.0, 0.0), pk0 = pi_;
    uint4 mm = make_uint4(0, 0, 0, 0);
    double F[4] = {0.0, 0.0, 0.0, 0.0};
    double *geo = (lane & 4 ? (lane & 2 ? nyb : nxb) : (lane & 2 ? yb : xb)) + i;
    if (valid) {
        nb = g.nbhs[i];
        if (lane < g.kp) k0 = g.conn[(size_t)lane * g.n + i];  // (unused slots name i)
        kind = i < g.nw ? KIND_WALL : (i < g.nw + g.no ? KIND_OUTER : KIND_INTERIOR);
        const unsigned long long mx = g.mx[i], my = g.my[i];
        mm = make_uint4((unsigned)mx, (unsigned)(mx >> 32), (unsigned)my, (unsigned)(my >> 32));
        const double2 nn = g.nrm[i];
        nx = nn.x;
        ny = nn.y;
        pi_ = g.xy[i];
        eps2 = g.eps2[i];
        if (!(lane & 1)) geo_old = *geo;
        double b4[4];
        ld4nc(frb + 4 * (size_t)i, b4);
        const double dl = delta[i];
        pk0 = g.xy[k0];
#pragma unroll
        for (int c = 0; c < 4; ++c) F[c] = (kind == KIND_WALL ? 2.0 * dl : dl) * b4[c];
        if (lane == 0) {
            double f4[4];
            ld4nc(fr + 4 * (size_t)i, f4);
            deltab[i] += (b4[0] * f4[0] + b4[1] * f4[1] + (b4[2] * f4[2] + b4[3] * f4[3])) / dl;
        }
    }
    const double2 *co = m.co[pg];
    double pb[8] = {}, nxs = 0.0, nys = 0.0, acc[3] = {};
    halo_wait();
    __syncwarp();
    const unsigned full = 0xffffffffu;
    const int nbw = __reduce_max_sync(full, nb);
    for (int r0 = 0; r0 < nbw; r0 += LPP) {
        const int r = r0 + lane;
        // a lane without a slot carries a zero adjoint through limited_b
        double delx = 0.0, dely = 0.0, delxb = 0.0, delyb = 0.0, delsb = 0.0, delnb = 0.0;
        double qtb[4] = {0.0, 0.0, 0.0, 0.0};
        if (r < nb) {
            const int k = r0 ? g.conn[(size_t)r * g.n + i] : k0;
            const double2 pk = r0 ? g.xy[k] : pk0;
            delx = pk.x - pi_.x;
            dely = pk.y - pi_.y;
            const double dels = delx * ny - dely * nx, deln = delx * nx + dely * ny;
            // the lists holding the neighbour: one of each direction (lx, ly), in
            // both only when its projection is exactly 0 (tx, ty)
            const unsigned bit = 1u << r;
            const int lx = mm.x & bit ? 0 : 1, ly = mm.z & bit ? 0 : 1;
            const bool tx = mm.x & mm.y & bit, ty = mm.z & mm.w & bit;
            const double2 px = co[lx], py = co[2 + ly];
            const double cx = fma(px.x, dels, px.y * deln), cy = fma(py.x, deln, py.y * dels);
            double cbx = 0.0, cby = 0.0, cbx1 = 0.0, cby1 = 0.0;
            // the neighbour's state (h = 0), then the point's (h = 1), one at a
            // time: both at once need more registers than three blocks leave
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const double sgn = h ? -1.0 : 1.0;
                KState s;
                double u1, u2;
                if (kst) {
                    // the forward re-run taped both reconstructions of this slot
                    double v[KS_TAPE / 2];
                    const int o = h ? 0 : KS_TAPE / 2;
                    if (r0 == 0) {
#pragma unroll
                        for (int c = 0; c < KS_TAPE / 4; ++c) {
                            const double2 t = m.tape[wl][o / 2 + c];
                            v[2 * c] = t.x;
                            v[2 * c + 1] = t.y;
                        }
                    } else {
                        const double *tp = kst + ((size_t)i * g.kp + r) * KS_TAPE + o;
                        ld4nc(tp, v);
                        ld4nc(tp + 4, v + 4);
                    }
                    s = kst_taped(v, nx, ny);
                    u1 = v[6];
                    u2 = v[7];
                } else {
                    const int p = h ? i : k;
                    const R4 v = ld4(q_in + p);
                    const double q[4] = {v.a, v.b, v.c, v.d};
                    double dx[4], dy[4], hi[4], lo[4], qt[4], u[2], w[2];
                    ld8a(dq + 8 * (size_t)p, dx, dy);
                    ld8a(qm + 8 * (size_t)p, hi, lo);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        qt[m] = limited_qtilde(delx * dx[m] + dely * dy[m], q[m], hi[m], lo[m],
                                               g.eps2[p]);
                    KState same;
                    kstate_pair(qt, qt, nx, ny, 0.56418958354775628695, s, same, u, w);
                    u1 = u[0];
                    u2 = u[1];
                }
                const double w6 = fma(6.0, s.pbr, s.usq);
                KStateB b;
                kzero(b);
                // reverse of sgn c (F . G) of list l along t; returns sgn F . G
                auto along_t = [&](int l, double c) {
                    const double sg = l ? -1.0 : 1.0;
                    if (kind == KIND_INTERIOR)
                        return sgn * flux_split_b(s, s.ut, s.un, s.B1, s.e1, sg, w6, F, c, b.ut,
                                                  b.un, b.B1, b.e1, b);
                    const double s2 = kind == KIND_WALL ? -1.0 : 1.0;
                    double G[4], cF[4], d = 0.0;
                    flux_quad(s, sg, s2, G);
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        d = fma(F[m], G[m], d);
                        cF[m] = c * F[m];
                    }
                    flux_quad_b(s, sg, s2, cF, b);
                    return sgn * d;
                };
                auto along_n = [&](int l, double c) {
                    const double sg = l ? -1.0 : 1.0;
                    const double Fn[4] = {F[0], F[2], F[1], F[3]};
                    return sgn * flux_split_b(s, s.un, s.ut, s.B2, s.e2, sg, w6, Fn, c, b.un, b.ut,
                                              b.B2, b.e2, b);
                };
                cbx += along_t(lx, sgn * cx);
                cby += along_n(ly, sgn * cy);
                if (tx) {
                    const double2 p = co[1];
                    cbx1 += along_t(1, sgn * fma(p.x, dels, p.y * deln));
                }
                if (ty) {
                    const double2 p = co[3];
                    cby1 += along_n(1, sgn * fma(p.x, deln, p.y * dels));
                }
                kstate_qt_b(s, u1, u2, nx, ny, b, qtb, nxs, nys);
                // from this k_flux_b_nbr reverses the neighbour's reconstruction
                if (h == 0) st_pairs(nbrec + ((size_t)i * g.kp + r) * NBREC, qtb, 4);
            }
            // the slot weights' adjoint: cb d to each list's pb, cb p to d
            delsb = fma(cbx, px.x, cby * py.y);
            delnb = fma(cbx, px.y, cby * py.x);
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const double wx = l == lx ? cbx : (l == 1 ? cbx1 : 0.0);
                const double wy = l == ly ? cby : (l == 1 ? cby1 : 0.0);
                pb[2 * l] = fma(wx, dels, pb[2 * l]);
                pb[2 * l + 1] = fma(wx, deln, pb[2 * l + 1]);
                pb[4 + 2 * l] = fma(wy, dels, pb[4 + 2 * l]);
                pb[5 + 2 * l] = fma(wy, deln, pb[5 + 2 * l]);
            }
            if (tx) {
                delsb = fma(cbx1, co[1].x, delsb);
                delnb = fma(cbx1, co[1].y, delnb);
            }
            if (ty) {
                delsb = fma(cby1, co[3].y, delsb);
                delnb = fma(cby1, co[3].x, delnb);
            }
        }
        double own[20] = {};
        {
            double qi[4], dxi[4], dyi[4], qmaxi[4], qmini[4];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double2 a = m.q[pg][c], x = m.dq[pg][c], y = m.dq[pg][2 + c],
                          hi = m.qm[pg][c], lo = m.qm[pg][2 + c];
                qi[2 * c] = a.x; qi[2 * c + 1] = a.y;
                dxi[2 * c] = x.x; dxi[2 * c + 1] = x.y;
                dyi[2 * c] = y.x; dyi[2 * c + 1] = y.y;
                qmaxi[2 * c] = hi.x; qmaxi[2 * c + 1] = hi.y;
                qmini[2 * c] = lo.x; qmini[2 * c + 1] = lo.y;
            }
            limited_b(qi, dxi, dyi, qmaxi, qmini, eps2, delx, dely, qtb, own, own + 4,
                      own + 8, own + 12, own + 16, delxb, delyb);
        }
        if (r < nb) {
            double2 *pt = reinterpret_cast<double2 *>(m.part[pg][r]);
            pt[0] = make_double2(delsb, delnb);
            pt[1] = make_double2(delxb, delyb);
        }
        // the round's own-point sums, in lane order: lane t adds fields t, t + 8
        // and t + 16 of its point's eight lanes
        __syncwarp();  // (the rows lie over the tape, which has been read)
        double2 *mine = m.rec(wl);
#pragma unroll
        for (int f = 0; f < 10; ++f) mine[f] = make_double2(own[2 * f], own[2 * f + 1]);
        __syncwarp();
#pragma unroll
        for (int t = 0; t < LPP; ++t) {
            const double *row = reinterpret_cast<const double *>(m.rec(LPP * pg + t)) + lane;
            acc[0] += row[0];
            acc[1] += row[8];
            if (lane < 4) acc[2] += row[16];
        }
        __syncwarp();
    }
    // pb summed over the point's lanes: lane 2 L + h holds component h of list
    // L, then z's component
    {
        const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
        double a[4], b[2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
            a[c] = (h4 ? pb[4 + c] : pb[c]) + __shfl_xor_sync(full, h4 ? pb[c] : pb[4 + c], 4);
#pragma unroll
        for (int c = 0; c < 2; ++c)
            b[c] = (h2 ? a[2 + c] : a[c]) + __shfl_xor_sync(full, h2 ? a[c] : a[2 + c], 2);
        const double v = (h1 ? b[1] : b[0]) + __shfl_xor_sync(full, h1 ? b[0] : b[1], 1);
        const double w = __shfl_xor_sync(full, v, 1);
        const int L = lane >> 1;
        const double2 p = co[L];
        const double gg = reinterpret_cast<const double *>(m.fcg[pg])[L];
        // the diagonal entry of M^-1 of this lane's component
        m.z[pg][lane] = fma((L < 2) == !h1 ? p.x : gg, v, p.y * w);
    }
    __syncwarp();
    double sums[4] = {0.0, 0.0, 0.0, 0.0};  // of x, y, nx, ny
    for (int r = lane; r < nb; r += LPP) {
        const double2 pk = r >= LPP ? g.xy[g.conn[(size_t)r * g.n + i]] : pk0;
        const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
        const double dels = delx * ny - dely * nx, deln = delx * nx + dely * ny;
        const double *pt = m.part[pg][r];
        double delsb = pt[0], delnb = pt[1];
        const unsigned bit = 1u << r;
        const unsigned in[4] = {mm.x, mm.y, mm.z, mm.w};
#pragma unroll
        for (int L = 0; L < 4; ++L) {
            if (!(in[L] & bit)) continue;
            const double2 c2 = co[L];
            const double ps = L < 2 ? c2.x : c2.y, pn = L < 2 ? c2.y : c2.x;
            const double zs = m.z[pg][2 * L], zn = m.z[pg][2 * L + 1];
            const double c = ps * dels + pn * deln, zd = zs * dels + zn * deln;
            delsb -= zs * c + ps * zd;
            delnb -= zn * c + pn * zd;
        }
        const double delxb = pt[2] + (delsb * ny + delnb * nx);
        const double delyb = pt[3] + (delnb * ny - delsb * nx);
        nxs += delnb * delx - delsb * dely;
        nys += delsb * delx + delnb * dely;
        reinterpret_cast<double2 *>(nbrec + ((size_t)i * g.kp + r) * NBREC)[2] =
            make_double2(delxb, delyb);
        sums[0] -= delxb;
        sums[1] -= delyb;
    }
    sums[2] = nxs;
    sums[3] = nys;
    __syncwarp();
    const double sum = reduce8(sums, lane);
    if (!valid) return;
    if (!(lane & 1)) *geo = geo_old + sum;
    // the stage's first contributions to q, dq and qm: stored, not added
    // (fields: q 4, dq 8, qm 8)
    if (lane < 4) {
        qb[4 * (size_t)i + lane] = acc[0];
        qmb[8 * (size_t)i + 4 + lane] = acc[2];
    } else {
        dqb[8 * (size_t)i + lane - 4] = acc[0];
    }
    if (lane < 4) dqb[8 * (size_t)i + 4 + lane] = acc[1];
    else qmb[8 * (size_t)i + lane - 4] = acc[1];
}

// The record of the least-squares solve whose result o = L s (L the inverse of
// the stencil's normal matrix M, s = sum of d times the slots' differences) has
// the adjoint ob: z = L ob, s's adjoint, and M's, -z o^T, as the sums of dx^2,
// dy^2 and dx dy receive it.  An inner iteration solves
// dq_t = dq0 + dq_(t-1) / 2 - L s / 2 (inner_sums), so its z and o carry the
// factor.  Fields: zx[4], zy[4], M's three, one left for k_grad_b.
__device__ __forceinline__ void lsq_record(const Geom &g, const LsqIn &in, int i,
                                           const double outx[4], const double outy[4],
                                           const double obx[4], const double oby[4],
                                           double *__restrict__ rec) {
    double L[4], x0[4], y0[4], xp[4], yp[4];
    ld4nc(g.minv + 4 * (size_t)i, L);
    if (in.inner()) {
        ld8a(in.dq0 + 8 * (size_t)i, x0, y0);
        ld8a(in.prev + 8 * (size_t)i, xp, yp);
    }
    const double f = in.inner() ? -0.5 : 1.0;
    double v[LREC];
    v[8] = v[9] = v[10] = v[11] = 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double zx = L[0] * obx[m] + L[1] * oby[m], zy = L[1] * obx[m] + L[2] * oby[m];
        double ox = outx[m], oy = outy[m];
        if (in.inner()) {  // the solve's own part of the result
            ox = ox - x0[m] - 0.5 * xp[m];
            oy = oy - y0[m] - 0.5 * yp[m];
        }
        v[m] = f * zx;
        v[4 + m] = f * zy;
        v[8] -= zx * ox;
        v[9] -= zy * oy;
        v[10] -= zx * oy + zy * ox;
    }
    st_pairs(rec + (size_t)i * LREC, v, LREC);
}

// The neighbour side of cal_flux_residual_b, one thread per neighbour k:
// over the slots (i, r) that name k (the transposed stencil, in (i, r)
// order) it reverses k's reconstruction of that slot from k_flux_b's record
// and adds the results to k's own adjoints in registers: no scatter and no
// gather of contribution records.  The part of delx/dely's adjoint that this
// reconstruction adds belongs to point i as well (delx = x_k - x_i): it is
// left in back[r][i] for k_grad_b.
constexpr int NBR_BLK = 128;
// 128 registers (256,000 points: 77 us with the solve's records; before those 74,
// 79 at 3 blocks, 91 with a record of the primitive state's adjoint)
constexpr int NBR_MIN_BLOCKS = 4;
template <int W>
__global__ void __launch_bounds__(NBR_BLK, NBR_MIN_BLOCKS)
k_flux_b_nbr(Geom g, const R4 *__restrict__ q_in, const double *__restrict__ dq,
             const double *__restrict__ qm, const int *__restrict__ tptr,
             const int *__restrict__ tlist, const double *__restrict__ nbrec, LsqIn in,
             double *__restrict__ qb, double *__restrict__ dqb, double *__restrict__ qmb,
             double *__restrict__ xb, double *__restrict__ yb, double2 *__restrict__ back,
             double *__restrict__ rec) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, w = t % W;
    const bool in_range = t / W < g.n;
    const int k = in_range ? t / W : g.n - 1;  // (the last block's other lanes: no slots)
    const R4 kv = ld4(q_in + k);
    const double qk[4] = {kv.a, kv.b, kv.c, kv.d};
    double dxk[4], dyk[4], qmaxk[4], qmink[4];
    ld8a(dq + 8 * (size_t)k, dxk, dyk);
    ld8a(qm + 8 * (size_t)k, qmaxk, qmink);
    const double eps2 = g.eps2[k];
    const double2 pk = g.xy[k];
    double qkb[4] = {0, 0, 0, 0}, dxkb[4] = {0, 0, 0, 0}, dykb[4] = {0, 0, 0, 0},
           qmaxkb[4] = {0, 0, 0, 0}, qminkb[4] = {0, 0, 0, 0};
    double xkb = 0.0, ykb = 0.0;
    const int e1 = in_range ? tptr[k + 1] : 0;
    for (int e = tptr[k] + w; e < e1; e += W) {
        const int slot = tlist[e];
        const int i = slot / g.kp, r = slot - i * g.kp;
        const double2 pi_ = g.xy[i];
        const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
        // the record: the adjoint of k's limited qtilde, delx/dely's so far
        const double2 *rv = reinterpret_cast<const double2 *>(nbrec + (size_t)slot * NBREC);
        const double2 v0 = __ldg(rv), v1 = __ldg(rv + 1), dd = __ldg(rv + 2);
        const double qtb[4] = {v0.x, v0.y, v1.x, v1.y};
        double dxr = 0.0, dyr = 0.0;
        limited_b(qk, dxk, dyk, qmaxk, qmink, eps2, delx, dely, qtb, qkb, dxkb, dykb, qmaxkb,
                  qminkb, dxr, dyr);
        xkb += dd.x + dxr;
        ykb += dd.y + dyr;
        back[(size_t)r * g.n + i] = make_double2(dxr, dyr);
    }
    lanes_sum<W>(qkb);
    lanes_sum<W>(dxkb);
    lanes_sum<W>(dykb);
    lanes_sum<W>(qmaxkb);
    lanes_sum<W>(qminkb);
    xkb = lane_sum<W>(xkb);
    ykb = lane_sum<W>(ykb);
    if (w > 0 || !in_range) return;
    add_pairs(qb + 4 * (size_t)k, qkb, 4);
    double v8[8];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        v8[m] = qmaxkb[m];
        v8[4 + m] = qminkb[m];
    }
    add_pairs(qmb + 8 * (size_t)k, v8, 8);
    xb[k] += xkb;
    yb[k] += ykb;
    // dq's adjoint is complete: what the last least-squares solve's reverse needs
    double dxo[4], dyo[4];
    ld8a(dqb + 8 * (size_t)k, dxo, dyo);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        dxkb[m] += dxo[m];
        dykb[m] += dyo[m];
    }
    if (in.inner()) {
        st_pairs(dqb + 8 * (size_t)k, dxkb, 4);
        st_pairs(dqb + 8 * (size_t)k + 4, dykb, 4);
    }
    lsq_record(g, in, k, dxk, dyk, dxkb, dykb, rec);
}

// eval_q_inner_loop_b: one inner iteration, dq_out = dq0 + dq_in / 2 - L s / 2,
// s = sum of d (d . dq_k) (inner_sums).  Half the warps take the points' own
// slots, of which only x and y's adjoints need the neighbours' rows; the other
// half the slots naming the points, which give dq_in's.
// Bound by the rows' gathers.  48 us at 256,000 points (6 blocks an SM; 51 at
// 5, 50 at 7); 293 as a pass that formed the sums again from q and dq and left
// a record of 14 doubles per slot, and a pass that gathered the records.
constexpr int INB_BLK = 128, INB_PTS = INB_BLK / 2;
__global__ void __launch_bounds__(INB_BLK, 6)
k_inner_b(Geom g, const double *__restrict__ dq_in, LsqIn in, int first,
          double *__restrict__ dqb, double *__restrict__ dq0b, const double *__restrict__ rec,
          double *__restrict__ rec_out, double *__restrict__ xb, double *__restrict__ yb,
          const int *__restrict__ tptr, const int *__restrict__ tlist) {
    __shared__ double2 own[INB_PTS];
    const int t = threadIdx.x % INB_PTS, i = blockIdx.x * INB_PTS + t;
    const bool pull = threadIdx.x >= INB_PTS;
    double dxb[4] = {0, 0, 0, 0}, dyb[4] = {0, 0, 0, 0}, gx = 0.0, gy = 0.0;
    double dxi[4], dyi[4];
    if (i < g.n) {
        const double2 pi_ = g.xy[i];
        if (pull) {
            ld4nc(dq_in + 8 * (size_t)i, dxi);
            ld4nc(dq_in + 8 * (size_t)i + 4, dyi);
            const int e1 = tptr[i + 1];
            for (int e = tptr[i]; e < e1; ++e) {
                const int j = tlist[e] / g.kp;  // a point whose neighbour i is
                double zx[4], zy[4], M[4];
                ld4nc(rec + (size_t)j * LREC, zx);
                ld4nc(rec + (size_t)j * LREC + 4, zy);
                ld4nc(rec + (size_t)j * LREC + 8, M);
                const double2 pj = g.xy[j];
                const double dx = pi_.x - pj.x, dy = pi_.y - pj.y;
                gx += 2.0 * dx * M[0] + dy * M[2];
                gy += 2.0 * dy * M[1] + dx * M[2];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double sb = zx[m] * dx + zy[m] * dy;  // of d . dq_i
                    const double s = dx * dxi[m] + dy * dyi[m];
                    gx += zx[m] * s + sb * dxi[m];
                    gy += zy[m] * s + sb * dyi[m];
                    dxb[m] += dx * sb;
                    dyb[m] += dy * sb;
                }
            }
        } else {
            double zx[4], zy[4], M[4], sx = 0.0, sy = 0.0;
            ld4nc(rec + (size_t)i * LREC, zx);
            ld4nc(rec + (size_t)i * LREC + 4, zy);
            ld4nc(rec + (size_t)i * LREC + 8, M);
            const int nb = g.nbhs[i];
#pragma unroll 2
            for (int r = 0; r < nb; ++r) {
                const int k = g.conn[(size_t)r * g.n + i];
                double dxk[4], dyk[4];
                ld4nc(dq_in + 8 * (size_t)k, dxk);
                ld4nc(dq_in + 8 * (size_t)k + 4, dyk);
                const double2 pk = g.xy[k];
                const double dx = pk.x - pi_.x, dy = pk.y - pi_.y;
                sx += dx;
                sy += dy;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double sb = zx[m] * dx + zy[m] * dy;
                    const double s = dx * dxk[m] + dy * dyk[m];
                    gx -= zx[m] * s + sb * dxk[m];
                    gy -= zy[m] * s + sb * dyk[m];
                }
            }
            gx -= 2.0 * sx * M[0] + sy * M[2];
            gy -= 2.0 * sy * M[1] + sx * M[2];
            own[t] = make_double2(gx, gy);
        }
    }
    __syncthreads();
    if (!pull || i >= g.n) return;
    xb[i] += gx + own[t].x;
    yb[i] += gy + own[t].y;
    double ox[4], oy[4];
    ld8a(dqb + 8 * (size_t)i, ox, oy);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        dxb[m] += 0.5 * ox[m];
        dyb[m] += 0.5 * oy[m];
    }
    // dq0's adjoint so far
    if (!first) {
        double ax[4], ay[4];
        ld8a(dq0b + 8 * (size_t)i, ax, ay);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            ox[m] += ax[m];
            oy[m] += ay[m];
        }
    }
    if (in.inner()) {
        st_pairs(dq0b + 8 * (size_t)i, ox, 4);
        st_pairs(dq0b + 8 * (size_t)i + 4, oy, 4);
        st_pairs(dqb + 8 * (size_t)i, dxb, 4);
        st_pairs(dqb + 8 * (size_t)i + 4, dyb, 4);
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            dxb[m] += ox[m];
            dyb[m] += oy[m];
        }
    }
    lsq_record(g, in, i, dxi, dyi, dxb, dyb, rec_out);
}

// eval_q_derivatives_b + func_delta_b, the point's own side: its sums over the
// neighbours (the solve's adjoint z comes in the record), the neighbours that
// gave qmax, qmin and the time step -- left packed in the record's last field,
// 5 bits each and 0 for none, for k_grad_b_nbr -- and the parts of delx/dely's
// adjoint that k_flux_b_nbr left in back.  256,000 points, without / with the time
// step: 33 / 45 us at 7 blocks an SM, 81 / 54 at 6 (measured twice: without the step
// the compiler's code at that bound is the slower), 38 / 55 at 8; 66 and a pass of 12
// for back when it summed the solve again and wrote a record of 24 doubles.
template <bool with_delta>
__global__ void __launch_bounds__(BLK, 7)
k_grad_b(Geom g, Consts c, const R4 *__restrict__ q, const double *__restrict__ spdA,
         const double *__restrict__ qmb, const double *__restrict__ deltab,
         const double2 *__restrict__ back, double *__restrict__ qb, double *__restrict__ xb,
         double *__restrict__ yb, double *__restrict__ rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const double2 pi_ = g.xy[i];
    double qi[4], qmax[4], qmin[4], sq[4] = {0, 0, 0, 0};
    ld4nc(reinterpret_cast<const double *>(q + i), qi);
    const int nb = g.nbhs[i];
    // arg-max, arg-min: slot + 1, 0 for the point itself
    int amax[4] = {0, 0, 0, 0}, amin[4] = {0, 0, 0, 0}, amd = 0;
    double min_delt = 1.0, sx = 0.0, sy = 0.0, bx = 0.0, by = 0.0;
#pragma unroll
    for (int m = 0; m < 4; ++m) qmax[m] = qmin[m] = qi[m];
#pragma unroll 2
    for (int r = 0; r < nb; ++r) {
        const int k = g.conn[(size_t)r * g.n + i];
        double qk[4];
        ld4nc(reinterpret_cast<const double *>(q + k), qk);
        const double2 pk = g.xy[k], v = back[(size_t)r * g.n + i];
        const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
        sx += delx;
        sy += dely;
        bx += v.x;
        by += v.y;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            sq[m] += qk[m] - qi[m];
            if (qk[m] > qmax[m]) { qmax[m] = qk[m]; amax[m] = r + 1; }
            if (qk[m] < qmin[m]) { qmin[m] = qk[m]; amin[m] = r + 1; }
        }
        if (with_delta) {
            // the taped spd of the stage's input state: the forward's own values
            const double dist = sqrt(delx * delx + dely * dely);
            double delta_t = dist / spdA[k];
            delta_t = c.cfl * delta_t;
            if (min_delt > delta_t) { min_delt = delta_t; amd = r + 1; }
        }
    }
    double *ri = rec + (size_t)i * LREC;
    double zx[4], zy[4], qib[4], qxb[4], qnb[4];
    ld8a(ri, zx, zy);
    ld8a(qmb + 8 * (size_t)i, qxb, qnb);
    const double s0b = ri[8], s1b = ri[9], s2b = ri[10];
    double xib = bx + 2.0 * sx * s0b + sy * s2b, yib = by + 2.0 * sy * s1b + sx * s2b;
    long long code = 0;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        xib += zx[m] * sq[m];
        yib += zy[m] * sq[m];
        qib[m] = -(zx[m] * sx + zy[m] * sy);
        if (!amax[m]) qib[m] += qxb[m];
        if (!amin[m]) qib[m] += qnb[m];
        code |= (long long)amax[m] << (5 * m) | (long long)amin[m] << (20 + 5 * m);
    }
    if (with_delta && amd) {
        const double dlb = deltab[i];
        if (dlb != 0.0) {
            const int k = g.conn[(size_t)(amd - 1) * g.n + i];
            const double2 pk = g.xy[k];
            const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
            const double dist = sqrt(delx * delx + dely * dely);
            const double distb = dlb * c.cfl / spdA[k];
            xib += distb * delx / dist;
            yib += distb * dely / dist;
            code |= (long long)amd << 40;
        }
    }
    ri[11] = __longlong_as_double(code);
    add_pairs(qb + 4 * (size_t)i, qib, 4);
    xb[i] -= xib;
    yb[i] -= yib;
}

// The neighbours' side of eval_q_derivatives_b + func_delta_b, one thread
// per neighbour k over the slots (i, r) naming it, in the transposed
// stencil's (i, r) order: q_k's adjoint from the point's least-squares sums
// and max/min, the time-step minimum's adjoint through k's state, and
// delx/dely's (the point's side takes the same value with the other sign).
// q's adjoint is complete then, and goes on to the primitive state
// (eval_q_variables_b).  40 us at 256,000 points (5 blocks an SM; 45 at 4, 49 at
// 6); 62 and a pass of 10 for the primitive state with the longer record.
template <int W>
__global__ void __launch_bounds__(BLK, 5)
k_grad_b_nbr(Geom g, Consts c, const R4 *__restrict__ q, const R4 *__restrict__ prim,
             const double *__restrict__ qmb, const double *__restrict__ deltab,
             const int *__restrict__ tptr, const int *__restrict__ tlist,
             const double *__restrict__ rec, const double *__restrict__ qb,
             double *__restrict__ pb, double *__restrict__ xb, double *__restrict__ yb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, w = t % W;
    const bool in_range = t / W < g.n;
    const int k = in_range ? t / W : g.n - 1;  // (the last block's other lanes: no slots)
    double qk[4], qkb[4] = {0, 0, 0, 0}, pkb[4] = {0, 0, 0, 0}, xkb = 0.0, ykb = 0.0;
    ld4nc(reinterpret_cast<const double *>(q + k), qk);
    if (w == 0) ld4nc(qb + 4 * (size_t)k, qkb);
    const R4 P = ld4(prim + k);
    const double2 pk = g.xy[k];
    const int e1 = in_range ? tptr[k + 1] : 0;
    for (int e = tptr[k] + w; e < e1; e += W) {
        const int slot = tlist[e];
        const int i = slot / g.kp, r = slot - i * g.kp;
        double zx[4], zy[4], M[4], qi[4];
        ld4nc(rec + (size_t)i * LREC, zx);
        ld4nc(rec + (size_t)i * LREC + 4, zy);
        ld4nc(rec + (size_t)i * LREC + 8, M);
        ld4nc(reinterpret_cast<const double *>(q + i), qi);
        const double2 pi_ = g.xy[i];
        const long long code = __double_as_longlong(M[3]);
        const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
        double delxb = 2.0 * delx * M[0] + dely * M[2];
        double delyb = 2.0 * dely * M[1] + delx * M[2];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            qkb[m] += zx[m] * delx + zy[m] * dely;
            if ((int)((code >> (5 * m)) & 31) == r + 1) qkb[m] += qmb[8 * (size_t)i + m];
            if ((int)((code >> (20 + 5 * m)) & 31) == r + 1) qkb[m] += qmb[8 * (size_t)i + 4 + m];
            delxb += zx[m] * (qk[m] - qi[m]);
            delyb += zy[m] * (qk[m] - qi[m]);
        }
        if ((int)(code >> 40) == r + 1) {
            const double dlb = deltab[i];
            const double modu = sqrt(P.b * P.b + P.c * P.c);
            const double cs = sqrt(P.d / P.a);
            const double spd = modu + 3.0 * cs;
            const double dist = sqrt(delx * delx + dely * dely);
            const double distb = dlb * c.cfl / spd;
            const double spdb = -dlb * c.cfl * dist / (spd * spd);
            delxb += distb * delx / dist;
            delyb += distb * dely / dist;
            if (modu > 0.0) {
                pkb[1] += spdb * P.b / modu;
                pkb[2] += spdb * P.c / modu;
            }
            const double csb = 3.0 * spdb;
            pkb[3] += csb * 0.5 / (cs * P.a);
            pkb[0] += -csb * 0.5 * P.d / (cs * P.a * P.a);
        }
        xkb += delxb;
        ykb += delyb;
    }
    lanes_sum<W>(qkb);
    lanes_sum<W>(pkb);
    xkb = lane_sum<W>(xkb);
    ykb = lane_sum<W>(ykb);
    if (w > 0 || !in_range) return;
    q_from_prim_b(P.a, P.b, P.c, P.d, qkb, pkb);
    add_pairs(pb + 4 * (size_t)k, pkb, 4);
    xb[k] += xkb;
    yb[k] += ykb;
}

// Adds the enstrophy objective's records (u1, u2, x, y of the neighbour) per
// point, in the transposed stencil's order.
__global__ void __launch_bounds__(256)
k_gather(int n, const int *__restrict__ tptr, const int *__restrict__ tlist,
         const double *__restrict__ contrib, double *__restrict__ pb, double *__restrict__ xb,
         double *__restrict__ yb) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const int e1 = tptr[k + 1];
    for (int e = tptr[k]; e < e1; ++e) {
        double v[4];
        ld4nc(contrib + (size_t)tlist[e] * OBJREC, v);
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[f] = acc[f] + v[f];
    }
    pb[4 * (size_t)k + 1] += acc[0];
    pb[4 * (size_t)k + 2] += acc[1];
    xb[k] += acc[2];
    yb[k] += acc[3];
}

// compute_force_coeffs_b: J = sum over shapes of Cl (objective 0) or Cd (1).
__global__ void k_forces_b(AdjShape t, const R4 *__restrict__ prim, const double2 *__restrict__ xy,
                           double mach, double cos_t, double sin_t, int objective,
                           double *__restrict__ pb, double *__restrict__ xb,
                           double *__restrict__ yb, double *__restrict__ nxb,
                           double *__restrict__ nyb) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double pr_inf = 1.0 / 1.4;
    const double temp = 0.5 * 1.0 * mach * mach;
    const double Hb = objective == 1 ? cos_t : -sin_t;
    const double Vb = objective == 1 ? sin_t : cos_t;
    for (int j = 0; j < t.npts; ++j) {
        const int m = t.idx[j], l = t.left[j], r = t.right[j];
        const double nx = t.nx[j], ny = t.ny[j];
        const double2 L = xy[l], M = xy[m], R = xy[r];
        const double ds1 = sqrt((M.x - L.x) * (M.x - L.x) + (M.y - L.y) * (M.y - L.y));
        const double ds2 = sqrt((R.x - M.x) * (R.x - M.x) + (R.y - M.y) * (R.y - M.y));
        const double ds = 0.5 * (ds1 + ds2);
        double cp = prim[m].d - pr_inf;
        cp = -cp / temp;
        const double cpb = Hb * nx * ds + Vb * ny * ds;
        nxb[m] += Hb * cp * ds;
        nyb[m] += Vb * cp * ds;
        const double dsb = Hb * cp * nx + Vb * cp * ny;
        pb[4 * (size_t)m + 3] += -cpb / temp;
        const double d1 = 0.5 * dsb / ds1, d2 = 0.5 * dsb / ds2;
        xb[m] += d1 * (M.x - L.x) - d2 * (R.x - M.x);
        yb[m] += d1 * (M.y - L.y) - d2 * (R.y - M.y);
        xb[l] -= d1 * (M.x - L.x);
        yb[l] -= d1 * (M.y - L.y);
        xb[r] += d2 * (R.x - M.x);
        yb[r] += d2 * (R.y - M.y);
    }
}

// compute_normals_b for wall and outer points (point_normals.F90:19-89).
__global__ void k_normals_b(int nbnd, const int *__restrict__ left, const int *__restrict__ right,
                            const double2 *__restrict__ xy, const double *__restrict__ nxb,
                            const double *__restrict__ nyb, double *__restrict__ xb,
                            double *__restrict__ yb) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int m = 0; m < nbnd; ++m) {
        const int l = left[m], r = right[m];
        const double2 L = xy[l], M = xy[m], R = xy[r];
        const double vx = 0.5 * ((M.y - L.y) + (R.y - M.y));
        const double vy = 0.5 * ((M.x - L.x) + (R.x - M.x));
        const double det = sqrt(vx * vx + vy * vy);
        double vxb = -nxb[m] / det;
        double vyb = nyb[m] / det;
        const double detb = nxb[m] * vx / (det * det) - nyb[m] * vy / (det * det);
        vxb += detb * vx / det;
        vyb += detb * vy / det;
        yb[r] += 0.5 * vxb;
        yb[l] -= 0.5 * vxb;
        xb[r] += 0.5 * vyb;
        xb[l] -= 0.5 * vyb;
    }
}

// The same two reverses with a thread per boundary point q.  src[ptr[q] ..
// ptr[q+1]) lists the entries j whose loop body above adds to xb[q] / yb[q],
// in the loop's order (ascending j; within one j the order of its
// statements), so that each sum is formed in the serial kernel's order and
// the results are the same bit for bit.  Normals: src = 2j + (0: q is
// right[j], 1: q is left[j]).  Forces: src = 3j + (0: q is idx[j], 1: q is
// left[j], 2: q is right[j]).
__global__ void k_normals_b_gather(int nbnd, const int *__restrict__ left,
                                   const int *__restrict__ right, const double2 *__restrict__ xy,
                                   const double *__restrict__ nxb, const double *__restrict__ nyb,
                                   const int *__restrict__ ptr, const int *__restrict__ src,
                                   double *__restrict__ xb, double *__restrict__ yb) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nbnd) return;
    double xq = xb[q], yq = yb[q];
    for (int e = ptr[q]; e < ptr[q + 1]; ++e) {
        const int m = src[e] >> 1, role = src[e] & 1;
        const int l = left[m], r = right[m];
        const double2 L = xy[l], M = xy[m], R = xy[r];
        const double vx = 0.5 * ((M.y - L.y) + (R.y - M.y));
        const double vy = 0.5 * ((M.x - L.x) + (R.x - M.x));
        const double det = sqrt(vx * vx + vy * vy);
        double vxb = -nxb[m] / det;
        double vyb = nyb[m] / det;
        const double detb = nxb[m] * vx / (det * det) - nyb[m] * vy / (det * det);
        vxb += detb * vx / det;
        vyb += detb * vy / det;
        if (role == 0) {
            yq += 0.5 * vxb;
            xq += 0.5 * vyb;
        } else {
            yq -= 0.5 * vxb;
            xq -= 0.5 * vyb;
        }
    }
    xb[q] = xq;
    yb[q] = yq;
}

__global__ void k_forces_b_gather(AdjShape t, int nbnd, const R4 *__restrict__ prim,
                                  const double2 *__restrict__ xy, double mach, double cos_t,
                                  double sin_t, int objective, const int *__restrict__ ptr,
                                  const int *__restrict__ src, double *__restrict__ pb,
                                  double *__restrict__ xb, double *__restrict__ yb,
                                  double *__restrict__ nxb, double *__restrict__ nyb) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nbnd) return;
    const double pr_inf = 1.0 / 1.4;
    const double temp = 0.5 * 1.0 * mach * mach;
    const double Hb = objective == 1 ? cos_t : -sin_t;
    const double Vb = objective == 1 ? sin_t : cos_t;
    double xq = xb[q], yq = yb[q];
    for (int e = ptr[q]; e < ptr[q + 1]; ++e) {
        const int j = src[e] / 3, role = src[e] % 3;
        const int m = t.idx[j], l = t.left[j], r = t.right[j];
        const double nx = t.nx[j], ny = t.ny[j];
        const double2 L = xy[l], M = xy[m], R = xy[r];
        const double ds1 = sqrt((M.x - L.x) * (M.x - L.x) + (M.y - L.y) * (M.y - L.y));
        const double ds2 = sqrt((R.x - M.x) * (R.x - M.x) + (R.y - M.y) * (R.y - M.y));
        const double ds = 0.5 * (ds1 + ds2);
        double cp = prim[m].d - pr_inf;
        cp = -cp / temp;
        const double dsb = Hb * cp * nx + Vb * cp * ny;
        const double d1 = 0.5 * dsb / ds1, d2 = 0.5 * dsb / ds2;
        if (role == 0) {
            const double cpb = Hb * nx * ds + Vb * ny * ds;
            nxb[m] += Hb * cp * ds;
            nyb[m] += Vb * cp * ds;
            pb[4 * (size_t)m + 3] += -cpb / temp;
            xq += d1 * (M.x - L.x) - d2 * (R.x - M.x);
            yq += d1 * (M.y - L.y) - d2 * (R.y - M.y);
        } else if (role == 1) {
            xq -= d1 * (M.x - L.x);
            yq -= d1 * (M.y - L.y);
        } else {
            xq += d2 * (R.x - M.x);
            yq += d2 * (R.y - M.y);
        }
    }
    xb[q] = xq;
    yb[q] = yq;
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

void launch_update_b(const Geom &g, const Consts &c, const AdjConsts &a, const R4 *prim_in,
                     const R4 *prim_old, const R4 *fr, const double *pb_out, double *pb_in,
                     double *pb_old, double *frb, double *nxb, double *nyb, int rk,
                     cudaStream_t s) {
    k_update_b<<<nblk(g.n, BLK), BLK, 0, s>>>(g, c, a, prim_in, prim_old, fr, pb_out, pb_in,
                                             pb_old, frb, nxb, nyb, rk);
}

void launch_flux_b(const Geom &g, const R4 *q_in, const double *dq, const double *qm,
                   const double *delta, const R4 *fr, const double *frb, LsqIn in, double *qb,
                   double *dqb, double *qmb, double *xb, double *yb, double *nxb, double *nyb,
                   double *deltab, double *nbrec, double *back, const int *tptr,
                   const int *tlist, const double *kst, double *rec, cudaStream_t s) {
    k_flux_b<<<nblk(g.n, GROUPS), BLK, 0, s>>>(g, q_in, dq, qm, delta,
                                               reinterpret_cast<const double *>(fr), frb, qb,
                                               dqb, qmb, xb, yb, nxb, nyb, deltab, nbrec, kst);
    double2 *bk = reinterpret_cast<double2 *>(back);
    const bool few = slot_passes(g.n);
    auto *nbr = few ? k_flux_b_nbr<FEW_LANES> : k_flux_b_nbr<1>;
    nbr<<<nblk(g.n, NBR_BLK / (few ? FEW_LANES : 1)), NBR_BLK, 0, s>>>(
        g, q_in, dq, qm, tptr, tlist, nbrec, in, qb, dqb, qmb, xb, yb, bk, rec);
}

void launch_inner_b(const Geom &g, const double *dq_in, LsqIn in, bool first, double *dqb,
                    double *dq0b, const double *rec, double *rec_out, double *xb, double *yb,
                    const int *tptr, const int *tlist, cudaStream_t s) {
    k_inner_b<<<nblk(g.n, INB_PTS), INB_BLK, 0, s>>>(g, dq_in, in, first ? 1 : 0, dqb, dq0b, rec,
                                                     rec_out, xb, yb, tptr, tlist);
}

void launch_grad_b(const Geom &g, const Consts &c, const R4 *q, const R4 *prim,
                   const double *spdA, const double *qmb, const double *deltab,
                   bool with_delta, const double *back, double *qb, double *pb, double *xb,
                   double *yb, double *rec, const int *tptr, const int *tlist, cudaStream_t s) {
    const double2 *bk = reinterpret_cast<const double2 *>(back);
    const int nb = nblk(g.n, BLK);
    if (with_delta)
        k_grad_b<true><<<nb, BLK, 0, s>>>(g, c, q, spdA, qmb, deltab, bk, qb, xb, yb, rec);
    else
        k_grad_b<false><<<nb, BLK, 0, s>>>(g, c, q, spdA, qmb, deltab, bk, qb, xb, yb, rec);
    const bool few = slot_passes(g.n);
    auto *nbr = few ? k_grad_b_nbr<FEW_LANES> : k_grad_b_nbr<1>;
    nbr<<<nblk(g.n, BLK / (few ? FEW_LANES : 1)), BLK, 0, s>>>(g, c, q, prim, qmb, deltab, tptr,
                                                               tlist, rec, qb, pb, xb, yb);
}

void launch_gather(int n, const int *tptr, const int *tlist, const double *contrib, double *pb,
                   double *xb, double *yb, cudaStream_t s) {
    k_gather<<<nblk(n, 256), 256, 0, s>>>(n, tptr, tlist, contrib, pb, xb, yb);
}

void launch_forces_b(const AdjShape &t, const AdjGather &gth, const R4 *prim, const double2 *xy,
                     double mach, double cos_t, double sin_t, int objective, double *pb,
                     double *xb, double *yb, double *nxb, double *nyb, cudaStream_t s) {
    if (gth.fptr)
        k_forces_b_gather<<<nblk(std::max(gth.nbnd, 1), 128), 128, 0, s>>>(
            t, gth.nbnd, prim, xy, mach, cos_t, sin_t, objective, gth.fptr, gth.fsrc, pb, xb, yb,
            nxb, nyb);
    else
        k_forces_b<<<1, 32, 0, s>>>(t, prim, xy, mach, cos_t, sin_t, objective, pb, xb, yb, nxb,
                                    nyb);
}

void launch_normals_b(int nbnd, const AdjGather &gth, const int *left, const int *right,
                      const double2 *xy, const double *nxb, const double *nyb, double *xb,
                      double *yb, cudaStream_t s) {
    if (gth.nptr)
        k_normals_b_gather<<<nblk(std::max(nbnd, 1), 128), 128, 0, s>>>(
            nbnd, left, right, xy, nxb, nyb, gth.nptr, gth.nsrc, xb, yb);
    else
        k_normals_b<<<1, 32, 0, s>>>(nbnd, left, right, xy, nxb, nyb, xb, yb);
}

}  // namespace lskum
