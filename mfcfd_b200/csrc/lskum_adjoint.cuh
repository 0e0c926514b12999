// Reverse-mode (adjoint) building blocks of the LSKUM pseudo-time loop, FP64.
//
// Each function is the hand-written reverse of the forward function of the
// same name in lskum_device.cuh: given the adjoint of the forward outputs
// (suffix _b) it accumulates the adjoints of the inputs.  Branches (limiter
// thresholds, split-list membership, max/min selection) are held at the
// forward outcome, as the reference's Tapenade-generated code does
// (e.g. src_mpi_adjoint/sensitivity_files/limiters_b.F90:43-165).
#pragma once

#include "flux_math.cuh"
#include "lskum_device.cuh"

namespace lskum {

#define MFCFD_TWO_OVER_SQRT_PI 1.12837916709551257390

struct KStateB {
    double rho, ut, un, pbr, usq, B1, B2, e1, e2;
};

__device__ __forceinline__ void kzero(KStateB &b) {
    b.rho = b.ut = b.un = b.pbr = b.usq = b.B1 = b.B2 = b.e1 = b.e2 = 0.0;
}

// split_fluxes_b in the forms of flux_split (flux_math.cuh): for a direction
// with velocity u along and o across it, moments B and e, list sign sg and w6
// = 6 p/rho + |u|^2, the reverse of c (F . G) for F over (mass, momentum along,
// momentum across, energy).  Returns F . G.
__device__ __forceinline__ double flux_split_b(const KState &s, double u, double o, double B,
                                               double e, double sg, double w6, const double F[4],
                                               double c, double &ub, double &ob, double &Bb,
                                               double &eb, KStateB &b) {
    const double A = fma(0.5 * sg, e, 0.5);
    const double a = fma(u, A, sg * B);
    const double pA = s.pbr * A;
    const double oF = fma(o, F[2], F[0]), hF = 0.5 * F[3];
    const double t = fma(F[1], fma(u, a, pA), fma(hF, fma(w6, a, u * pA), oF * a));
    b.rho = fma(c, t, b.rho);
    const double cr = c * s.rho, r1 = cr * F[1], r3 = cr * hF;
    const double ab = fma(r3, w6, fma(r1, u, cr * oF));
    const double pAb = fma(r3, u, r1);
    ub = fma(ab, A, fma(r3, pA, fma(r1, a, ub)));
    ob = fma(cr * F[2], a, ob);
    const double w6b = r3 * a;
    b.pbr = fma(6.0, w6b, fma(pAb, A, b.pbr));
    b.usq += w6b;
    Bb = fma(sg, ab, Bb);
    eb = fma(0.5 * sg, fma(ab, u, pAb * s.pbr), eb);
    return s.rho * t;
}

// quadrant_fluxes_b: GxI..GxIV
__device__ __forceinline__ void flux_quad_b(const KState &s, double s1, double s2,
                                            const double Gb[4], KStateB &b) {
    const double A1 = 0.5 * (1.0 + s1 * s.e1);
    const double A2 = 0.5 * (1.0 + s2 * s.e2);
    const double rA2 = s.rho * A2;
    const double a1b = s.ut * A1 + s1 * s.B1;
    const double t1 = s.pbr + s.ut * s.ut;
    const double t2 = t1 * A1 + s1 * (s.ut * s.B1);
    const double c2 = s.un * A2 + s2 * s.B2;
    const double t7 = (7.0 * s.pbr) + s.usq;
    const double t4 = 0.5 * s.ut * t7 * A1;
    const double t6 = (6.0 * s.pbr) + s.usq;
    const double t3 = 0.5 * s.B1 * t6;
    double A1b = 0.0, A2b = 0.0;
    const double rA2b = Gb[0] * a1b + Gb[1] * t2 + Gb[3] * (t4 + s1 * t3);
    const double a1bb = Gb[0] * rA2 + Gb[2] * s.rho * c2 + s2 * Gb[3] * (0.5 * s.rho * s.un * s.B2);
    // G1 = rA2 * t2
    const double t2b = Gb[1] * rA2;
    const double t1b = t2b * A1;
    A1b += t2b * t1;
    b.ut += t2b * s1 * s.B1 + 2.0 * s.ut * t1b;
    b.B1 += t2b * s1 * s.ut;
    b.pbr += t1b;
    // G2 = rho * a1b * c2
    b.rho += Gb[2] * a1b * c2;
    const double c2b = Gb[2] * s.rho * a1b;
    b.un += c2b * A2;
    A2b += c2b * s.un;
    b.B2 += c2b * s2;
    // G3 = rA2 * (t4 + s1 t3) + s2 * 0.5 rho un B2 a1b
    const double t4b = Gb[3] * rA2;
    const double t3b = Gb[3] * rA2 * s1;
    const double t5b = Gb[3] * s2;
    b.ut += t4b * 0.5 * t7 * A1;
    const double t7b = t4b * 0.5 * s.ut * A1;
    A1b += t4b * 0.5 * s.ut * t7;
    b.B1 += t3b * 0.5 * t6;
    const double t6b = t3b * 0.5 * s.B1;
    b.rho += t5b * 0.5 * s.un * s.B2 * a1b;
    b.un += t5b * 0.5 * s.rho * s.B2 * a1b;
    b.B2 += t5b * 0.5 * s.rho * s.un * a1b;
    b.pbr += 7.0 * t7b + 6.0 * t6b;
    b.usq += t7b + t6b;
    // a1b = ut A1 + s1 B1
    b.ut += a1bb * A1;
    A1b += a1bb * s.ut;
    b.B1 += a1bb * s1;
    // rA2 = rho A2
    b.rho += rA2b * A2;
    A2b += rA2b * s.rho;
    b.e1 += 0.5 * s1 * A1b;
    b.e2 += 0.5 * s2 * A2b;
}

// kstate_pre / kstate_pair (flux_math.cuh) reversed: the adjoint b of a kinetic
// state s with velocity (u1, u2) to that of its limited qtilde, added to the
// normal's.  exp(-S^2) comes back from the moments (B = exp(-S^2) / (2 sqrt(pi
// beta))), so one reciprocal and one reciprocal square root are all it takes.
__device__ __forceinline__ void kstate_qt_b(const KState &s, double u1, double u2, double nx,
                                            double ny, const KStateB &b, double qtb[4],
                                            double &nxb, double &nyb) {
    const double beta = 0.5 * rcp_h3(s.pbr);
    const double sb = beta * rsqrt_h3(beta);
    const double S1 = s.ut * sb, S2 = s.un * sb;
    const double S1b = s.B1 * (4.0 * sb * b.e1 - 2.0 * S1 * b.B1);
    const double S2b = s.B2 * (4.0 * sb * b.e2 - 2.0 * S2 * b.B2);
    const double utb = fma(S1b, sb, b.ut), unb = fma(S2b, sb, b.un);
    const double texpb = b.rho * s.rho;
    const double usqb = fma(texpb, beta, b.usq);
    const double u1b = fma(2.0 * u1, usqb, utb * ny + unb * nx);
    const double u2b = fma(2.0 * u2, usqb, unb * ny - utb * nx);
    nxb += unb * u1 - utb * u2;
    nyb += utb * u1 + unb * u2;
    // p/rho = 1/(2 beta), u = qtilde_2,3 p/rho
    const double pbrb = fma(2.0 * beta, u1b * u1 + u2b * u2, b.pbr);
    double betab = fma(texpb, s.usq - 5.0 * s.pbr, -2.0 * s.pbr * s.pbr * pbrb);
    betab = fma(s.pbr, sb * (S1b * s.ut + S2b * s.un) - (b.B1 * s.B1 + b.B2 * s.B2), betab);
    qtb[0] = texpb;
    qtb[1] = u1b * s.pbr;
    qtb[2] = u2b * s.pbr;
    qtb[3] = -0.5 * betab;
}

// limited_qtilde (flux_math.cuh) of a row reversed, all four components: the
// adjoint qtb of the limited qtilde towards (delx, dely), added to the row's
// adjoints and the offset's (limiters_b.F90:43-165).
__device__ __forceinline__ void limited_b(const double q[4], const double dqx[4],
                                          const double dqy[4], const double qmax[4],
                                          const double qmin[4], double eps2, double delx,
                                          double dely, const double qtb[4], double qb[4],
                                          double dqxb[4], double dqyb[4], double qmaxb[4],
                                          double qminb[4], double &delxb, double &delyb) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const double t = delx * dqx[r] + dely * dqy[r];
        const double dn = -0.5 * t;
        const bool up = dn > 0.0;
        const double dp = (up ? qmax[r] : qmin[r]) - q[r];
        const double a = fma(dp, dp, eps2);
        const double id = rcp_h3(fma(dn, dp - t, a));
        const double f = fma(-t, dp, a) * id;
        const bool act = f < 1.0 && fabs(dn) > MFCFD_VENKAT_THR;
        qb[r] += qtb[r];
        double dnb = qtb[r];
        if (act) {
            const double numb = qtb[r] * dn * id, denb = -numb * f;
            const double dpb = 2.0 * numb * (dp + dn) + denb * fma(2.0, dp, dn);
            dnb = fma(f, qtb[r], 2.0 * numb * dp + denb * fma(4.0, dn, dp));
            if (up) qmaxb[r] += dpb;
            else qminb[r] += dpb;
            qb[r] -= dpb;
        }
        const double tb = -0.5 * dnb;
        delxb = fma(tb, dqx[r], delxb);
        delyb = fma(tb, dqy[r], delyb);
        dqxb[r] = fma(tb, delx, dqxb[r]);
        dqyb[r] = fma(tb, dely, dqyb[r]);
    }
}

// primitive_to_conserved_b (state_update.F90:144-163)
__device__ __forceinline__ void prim_to_conserved_b(double rho, double u1, double u2, double pr,
                                                    double nx, double ny, const double Ub[4],
                                                    double pb[4], double &nxb, double &nyb) {
    const double t1 = rho * u1, t2 = rho * u2;
    const double t1b = Ub[1] * ny + Ub[2] * nx + Ub[3] * (t1 / rho);
    const double t2b = -Ub[1] * nx + Ub[2] * ny + Ub[3] * (t2 / rho);
    nxb += -Ub[1] * t2 + Ub[2] * t1;
    nyb += Ub[1] * t1 + Ub[2] * t2;
    pb[3] += 2.5 * Ub[3];
    pb[0] += Ub[0] - Ub[3] * 0.5 * (t1 * t1 + t2 * t2) / (rho * rho) + t1b * u1 + t2b * u2;
    pb[1] += t1b * rho;
    pb[2] += t2b * rho;
}

// conserved_vector_Ubar_b (state_update.F90:239-294): the point half w.r.t.
// prim and (nx, ny), and the freestream half w.r.t. (nx, ny).
__device__ __forceinline__ void conserved_ubar_b(double rho, double u1, double u2, double pr,
                                                 double nx, double ny, const double qinf[4],
                                                 double pi, double gm1, const double Ub[4],
                                                 double pb[4], double &nxb, double &nyb) {
    // point half
    const double u1r = u1 * ny - u2 * nx;
    const double u2r = u1 * nx + u2 * ny;
    const double e = pr / (rho * gm1) + 0.5 * (u1r * u1r + u2r * u2r);
    const double beta = rho / (2.0 * pr);
    const double sb = sqrt(beta);
    const double S2 = u2r * sb;
    const double spb = sqrt(pi * beta);
    const double E2 = exp(-S2 * S2);
    const double B2 = E2 / (2.0 * spb);
    const double A2p = 0.5 * (1.0 + erf(S2));
    double rhob = Ub[0] * A2p + Ub[1] * u1r * A2p + Ub[2] * (u2r * A2p + B2) +
                  Ub[3] * (A2p * e + 0.5 * u2r * B2);
    const double A2pb = Ub[0] * rho + Ub[1] * rho * u1r + Ub[2] * rho * u2r + Ub[3] * rho * e;
    double u1rb = Ub[1] * rho * A2p;
    double u2rb = Ub[2] * rho * A2p + Ub[3] * 0.5 * rho * B2;
    const double B2b = Ub[2] * rho + Ub[3] * 0.5 * rho * u2r;
    const double eb = Ub[3] * rho * A2p;
    double prb = eb / (rho * gm1);
    rhob += -eb * pr / (rho * rho * gm1);
    u1rb += eb * u1r;
    u2rb += eb * u2r;
    double S2b = A2pb * 0.5 * MFCFD_TWO_OVER_SQRT_PI * E2 + B2b * B2 * (-2.0 * S2);
    const double spbb = -B2b * B2 / spb;
    u2rb += S2b * sb;
    const double sbb = S2b * u2r;
    double betab = sbb / (2.0 * sb) + spbb * pi / (2.0 * spb);
    rhob += betab / (2.0 * pr);
    prb += -betab * beta / pr;
    pb[0] += rhob;
    pb[1] += u1rb * ny + u2rb * nx;
    pb[2] += -u1rb * nx + u2rb * ny;
    pb[3] += prb;
    nxb += -u1rb * u2 + u2rb * u1;
    nyb += u1rb * u1 + u2rb * u2;
    // freestream half
    const double rho_inf = qinf[0], u1i = qinf[1], u2i = qinf[2], pr_inf = qinf[3];
    const double u1ri = u1i * ny - u2i * nx;
    const double u2ri = u1i * nx + u2i * ny;
    const double e_inf = pr_inf / (rho_inf * gm1) + 0.5 * (u1ri * u1ri + u2ri * u2ri);
    const double beti = (0.5 * rho_inf) / pr_inf;
    const double sbi = sqrt(beti);
    const double S2i = u2ri * sbi;
    const double B2i = exp(-S2i * S2i) / (2.0 * sqrt(pi * beti));
    const double A2ni = 0.5 * (1.0 - erf(S2i));
    const double A2nib = rho_inf * (Ub[0] + Ub[1] * u1ri + Ub[2] * u2ri + Ub[3] * e_inf);
    const double e_infb = Ub[3] * rho_inf * A2ni;
    const double u1rib = Ub[1] * rho_inf * A2ni + e_infb * u1ri;
    double u2rib = Ub[2] * rho_inf * A2ni - Ub[3] * 0.5 * rho_inf * B2i + e_infb * u2ri;
    const double B2ib = -Ub[2] * rho_inf - Ub[3] * 0.5 * rho_inf * u2ri;
    const double S2ib = -A2nib * 0.5 * MFCFD_TWO_OVER_SQRT_PI * exp(-S2i * S2i) +
                        B2ib * B2i * (-2.0 * S2i);
    u2rib += S2ib * sbi;
    nxb += -u1rib * u2i + u2rib * u1i;
    nyb += u1rib * u1i + u2rib * u2i;
}

// q_variables_b (q_variables.F90:8-37)
__device__ __forceinline__ void q_from_prim_b(double rho, double u1, double u2, double pr,
                                              const double qb[4], double pb[4]) {
    const double beta = 0.5 * rho / pr;
    double betab = qb[0] * (2.5 / beta - (u1 * u1 + u2 * u2)) +
                   2.0 * (qb[1] * u1 + qb[2] * u2 - qb[3]);
    pb[0] += qb[0] / rho + betab * 0.5 / pr;
    pb[3] += -betab * beta / pr;
    pb[1] += -qb[0] * 2.0 * beta * u1 + qb[1] * 2.0 * beta;
    pb[2] += -qb[0] * 2.0 * beta * u2 + qb[2] * 2.0 * beta;
}

}  // namespace lskum
