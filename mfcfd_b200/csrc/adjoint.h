// Internal interface of the reverse (adjoint) kernels.
#pragma once

#include <cuda_runtime.h>

#include "primal.h"

namespace lskum {

// the enstrophy objective's record per (point, slot): the neighbour's u1, u2, x
// and y adjoints
constexpr int OBJREC = 4;
// flux pass: per (point, slot) the neighbour side's record (adjoint of its
// limited qtilde, delx/dely adjoint)
constexpr int NBREC = 6;
// doubles per (point, slot) of the buffer that holds the flux pass's records and
// back sums, or the objective's
constexpr int ADJ_CW = NBREC + 2;
// per point, of the least-squares solve being reversed: what its neighbours'
// side reads (LsqIn)
constexpr int LREC = 12;

// The rows of dq that made the solve's result: with inner iterations the
// D pass's dq0 and the previous iteration's; null for the D pass itself.
struct LsqIn {
    const double *dq0 = nullptr, *prev = nullptr;
    __host__ __device__ bool inner() const { return prev != nullptr; }
};

struct AdjConsts {
    double q_inf[4];
};

// Shape points in grid order with their renumbered ring neighbours.
struct AdjShape {
    int npts;
    const int *idx, *left, *right;
    const double *nx, *ny;
};

// Source lists of the gather forms of the force and normal reverses (one
// thread per boundary point; see k_forces_b_gather).  Null pointers select
// the single-thread kernels.
struct AdjGather {
    int nbnd;
    const int *fptr, *fsrc;  // forces: 3 j + role, per boundary point
    const int *nptr, *nsrc;  // normals: 2 j + role, per boundary point
};

void launch_update_b(const Geom &g, const Consts &c, const AdjConsts &a, const R4 *prim_in,
                     const R4 *prim_old, const R4 *fr, const double *pb_out, double *pb_in,
                     double *pb_old, double *frb, double *nxb, double *nyb, int rk,
                     cudaStream_t s);
// fr: the stage's taped flux residual; kst: its kinetic-state tape of the
// forward re-run ([n][kp][KS_TAPE], written by the flux pass with
// StageBufs::kstape), or nullptr to recompute.
// The flux pass reverses in two kernels: k_flux_b per point (its fluxes,
// kinetic states and own reconstruction; writes nbrec [n][kp][NBREC]) and
// k_flux_b_nbr per neighbour over the transposed stencil (the neighbour's
// reconstruction; writes back [n][kp] (delx, dely) adjoint parts that
// belong to the point as well; k_grad_b adds those to the point).
// nbrec and back share one buffer of n*kp*(NBREC+2) doubles.  dqb and rec
// receive dq's adjoint (with inner iterations; otherwise the record holds all
// that is needed of it) and the records of the solve that made dq.
void launch_flux_b(const Geom &g, const R4 *q_in, const double *dq, const double *qm,
                   const double *delta, const R4 *fr, const double *frb, LsqIn in, double *qb,
                   double *dqb, double *qmb, double *xb, double *yb, double *nxb, double *nyb,
                   double *deltab, double *nbrec, double *back, const int *tptr,
                   const int *tlist, const double *kst, double *rec, cudaStream_t s);
// One inner iteration, dq_in -> dq_out: dqb holds dq_out's adjoint on entry and
// dq_in's on exit; rec its records on entry, rec_out those of the solve `in`
// that made dq_in.  dq0b adds up the outputs' adjoints (dq0 enters every inner
// iteration's result): `first` (the last iteration, reversed first) stores.
// With in.inner() false dq_in is dq0 itself, and rec_out has the total.
void launch_inner_b(const Geom &g, const double *dq_in, LsqIn in, bool first, double *dqb,
                    double *dq0b, const double *rec, double *rec_out, double *xb, double *yb,
                    const int *tptr, const int *tlist, cudaStream_t s);
// spdA: |u| + 3 sqrt(p/rho) of the stage's input state prim as the forward pass
// used it (taped; read with with_delta only).  Two kernels: k_grad_b per point
// (its own side, completing rec) and k_grad_b_nbr per neighbour over the
// transposed stencil (adds to pb = prim's adjoint, xb, yb; q's adjoint qb ends
// there).
void launch_grad_b(const Geom &g, const Consts &c, const R4 *q, const R4 *prim,
                   const double *spdA, const double *qmb, const double *deltab,
                   bool with_delta, const double *back, double *qb, double *pb, double *xb,
                   double *yb, double *rec, const int *tptr, const int *tlist, cudaStream_t s);
// Adds the enstrophy objective's records to the neighbours' pb, xb, yb.
void launch_gather(int n, const int *tptr, const int *tlist, const double *contrib, double *pb,
                   double *xb, double *yb, cudaStream_t s);
void launch_forces_b(const AdjShape &t, const AdjGather &gth, const R4 *prim, const double2 *xy,
                     double mach, double cos_t, double sin_t, int objective, double *pb,
                     double *xb, double *yb, double *nxb, double *nyb, cudaStream_t s);
void launch_normals_b(int nbnd, const AdjGather &gth, const int *left, const int *right,
                      const double2 *xy, const double *nxb, const double *nyb, double *xb,
                      double *yb, cudaStream_t s);

}  // namespace lskum
