// FP64 kernels of the LSKUM pseudo-time loop on sm_100a.
//
// Per pseudo-time stage (fpi_solver.F90:27-53):
//   kb_grad_h   D pass  -- eval_q_derivatives (+ func_delta on the first stage)
//   kb_inner_h  I pass  -- eval_q_inner_loop + eval_update_innerloop, rearranged
//                          (dq buffers rotate; the D pass's result is kept)
//   kb_flux   F pass  -- cal_flux_residual + state_update + eval_q_variables of
//                        the new state (+ res_sqr partials on the last stage)
// and per iteration kb_residual (fpi_solver.F90:57-70).
//
// Every pass walks a schedule of instances (batch.cuh): a single grid is a
// schedule of one instance, a batch of independent grids one of many, and
// both run the same compiled kernels, so an instance's results do not depend
// on what it is batched with.
//
// Layout in HBM (renumbered points: wall | outer | interior): one 32-byte
// row per point for prim and q, 64-byte rows for dq and qm, 16-byte rows for
// (x, y) and (nx, ny); stencils as ELL columns conn[slot][point] so that lanes of
// neighbouring points read them coalesced.
#include <cuda_runtime.h>

#include <algorithm>

#include "batch.cuh"
#include "flux_math.cuh"
#include "flux_tile.cuh"
#include "halo.cuh"
#include "primal.h"

namespace lskum {

namespace {

constexpr int GRAD_BLOCK = 256;  // blocks of the per-point set-up kernels
// 4 blocks: 128 registers a thread and all of shared memory but 3.5 KB; at 3
// (168 registers) 0.420 ms at 1.024M points against 0.389
constexpr int FLUX_MIN_BLOCKS = 4;
constexpr double OBT = 1.0 / 3.0;        // state_update.F90:19-20
constexpr double TBT = 2.0 / 3.0;

// A 64-byte row (dq, qm; 32-byte aligned) in two 256-bit loads.
__device__ __forceinline__ void ld8w(const double *p, double a[4], double b[4]) {
    const R4 u = ld4w(reinterpret_cast<const R4 *>(p));
    const R4 v = ld4w(reinterpret_cast<const R4 *>(p + 4));
    a[0] = u.a; a[1] = u.b; a[2] = u.c; a[3] = u.d;
    b[0] = v.a; b[1] = v.b; b[2] = v.c; b[3] = v.d;
}

// Row sources of the per-point sums of the D and I passes: the rows of a
// point's stencil gathered from global memory, or from its tile's halo
// staged in shared memory (kb_grad_h, kb_inner_h).  Both give the same
// values, so the sums below do not depend on where their rows come from.
struct GlobalRows {
    const Geom &g;
    const R4 *q;
    const double *dq;   // I pass: dq_in
    const double *spd;  // D pass
    int i;
    __device__ __forceinline__ int self() const { return i; }
    __device__ __forceinline__ unsigned long long word(int) const { return 0ull; }
    __device__ __forceinline__ int nbr(int r, unsigned long long, int) const {
        return g.conn[(size_t)r * g.n + i];
    }
    __device__ __forceinline__ double2 xy(int k) const { return g.xy[k]; }
    __device__ __forceinline__ void qrow(int k, double v[4]) const {
        const R4 a = ld4w(q + k);
        v[0] = a.a; v[1] = a.b; v[2] = a.c; v[3] = a.d;
    }
    __device__ __forceinline__ void dqrow(int k, double x[4], double y[4]) const {
        ld8w(dq + 8 * (size_t)k, x, y);
    }
    __device__ __forceinline__ double spdv(int k) const { return spd[k]; }
};

// Shared-memory arrays of a staged tile halo, HaloStride rows each (one more
// than a multiple of eight, so that the arrays of a row start on different
// banks): D pass q[0..1], q[2..3], (x, y), (spd, -);
// I pass (x, y), dq/dx[0..1], dq/dx[2..3], dq/dy[0..1], dq/dy[2..3].  One
// 16-byte array per pair keeps a warp's reads of neighbouring rows on
// distinct banks.
constexpr int HA_I = 5, HA_D = 4;
// Stride of the staged arrays.  Fixed in the D pass, so that a row's pieces are
// immediate offsets from its first (with the slots' loop unrolled 0.088 ->
// 0.076 ms at 1.024M points at 5 blocks an SM); the I pass, whose rows are
// larger, takes the grid's own: what shared memory it leaves is L1, where the
// tiles' common rows are found (0.082 ms, 0.090 with the fixed stride).
template <int nA, int CAP>
struct HaloStride {
    int hc;
    __host__ __device__ constexpr HaloStride(int h) : hc(h) {}
};
template <>
struct HaloStride<HA_D, HALO_CAP> {
    static constexpr int hc = HALO_CAP + 1;
    __host__ __device__ constexpr HaloStride(int) {}
};
constexpr int HALO_BLOCK = 128;  // four warps, a half-warp per tile
// resident blocks per SM (96 registers), measured at 1.024M points: the D pass
// 0.082 ms at 4, 0.076 at 5, 0.089 at 6; the I pass 0.089, 0.082, 0.097
constexpr int HALO_MIN_BLOCKS_D = 5, HALO_MIN_BLOCKS_I = 5;

template <int nA, int CAP>
struct HaloRows {
    static constexpr int OXY = nA == HA_I ? 0 : 2, ODQ = 1, OSPD = 3;
    const double2 *sm;
    HaloStride<nA, CAP> st;
    HaloLoc loc;
    // i < 0: no point (nothing is loaded)
    __device__ __forceinline__ HaloRows(const Geom &g, const double2 *sm_, int i)
        : sm(sm_), st(g.hc), loc(g, i) {}
    __device__ __forceinline__ int self() const { return loc.own; }
    __device__ __forceinline__ unsigned long long word(int r0) const { return loc.word(r0); }
    // slot r0 + j of word(r0)
    __device__ __forceinline__ int nbr(int, unsigned long long w, int j) const {
        return (int)((w >> (8 * j)) & 0xffull);
    }
    __device__ __forceinline__ double2 xy(int l) const { return sm[OXY * st.hc + l]; }
    __device__ __forceinline__ void qrow(int l, double v[4]) const {
        const double2 a = sm[l], b = sm[st.hc + l];
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
    __device__ __forceinline__ void dqrow(int l, double x[4], double y[4]) const {
        const double2 a = sm[ODQ * st.hc + l], b = sm[(ODQ + 1) * st.hc + l],
                      e = sm[(ODQ + 2) * st.hc + l], f = sm[(ODQ + 3) * st.hc + l];
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        y[0] = e.x; y[1] = e.y; y[2] = f.x; y[3] = f.y;
    }
    __device__ __forceinline__ double spdv(int l) const { return sm[OSPD * st.hc + l].x; }
};

// q_variables.F90:41-112 eval_q_derivatives and state_update.F90:190-236
// func_delta over the rows of R, in slot order.
template <class Rows>
__device__ __forceinline__ void grad_sums(const Consts &c, const Geom &g, int i, const Rows &R,
                                          int nb, int with_delta, double dx[4], double dy[4],
                                          double qmax[4], double qmin[4], double &min_delt) {
    const int me = R.self();
    const double2 pi_ = R.xy(me);
    double qi[4];
    R.qrow(me, qi);
    const R4 M = ld4w(reinterpret_cast<const R4 *>(g.minv) + i);
#pragma unroll
    for (int m = 0; m < 4; ++m) qmax[m] = qmin[m] = qi[m];
    double sdxq[4] = {0.0, 0.0, 0.0, 0.0}, sdyq[4] = {0.0, 0.0, 0.0, 0.0};
    min_delt = 1.0;
    for (int r0 = 0; r0 < nb; r0 += 8) {
        const unsigned long long word = R.word(r0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = r0 + j;
            if (r >= nb) break;
            const int k = R.nbr(r, word, j);
            double qk[4];
            R.qrow(k, qk);
            const double2 pk = R.xy(k);
            const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
            const double w = g.wsl ? __ldg(g.wsl + (size_t)r * g.n + i) : 1.0;
            const double wx = w * delx, wy = w * dely;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                if (qk[m] > qmax[m]) qmax[m] = qk[m];
                if (qk[m] < qmin[m]) qmin[m] = qk[m];
                sdxq[m] = fma(wx, qk[m] - qi[m], sdxq[m]);
                sdyq[m] = fma(wy, qk[m] - qi[m], sdyq[m]);
            }
            if (with_delta) {
                double delta_t = sqrt(fma(delx, delx, dely * dely)) / R.spdv(k);
                delta_t = c.cfl * delta_t;
                if (min_delt > delta_t) min_delt = delta_t;
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        dx[m] = fma(M.a, sdxq[m], M.b * sdyq[m]);
        dy[m] = fma(M.b, sdxq[m], M.c * sdyq[m]);
    }
}

// q_variables.F90:115-227 eval_q_inner_loop + eval_update_innerloop over the
// rows of R, rearranged.  q is fixed within a stage, so the reference's
// L sum_k w d (qtilde_k - qtilde_i), with qtilde = q - d.dq/2 and L the
// inverse of the stencil's normal matrix M = sum_k w d d^T, equals
//     dq0 + dq_i / 2 - L sum_k w d (d . dq_k) / 2,
// dq0 = L sum_k w d (q_k - q_i) being the D pass's result (kept through the
// stage's inner iterations) and L M dq_i = dq_i: the same value up to
// rounding, from the neighbours' dq and (x, y) alone (no q gathers).  dq0x,
// dq0y: the point's D-pass derivatives; the point's own dq_i and the
// neighbours' come through R.
template <class Rows>
__device__ __forceinline__ void inner_sums(const Geom &g, int i, const Rows &R, int nb,
                                           const double dq0x[4], const double dq0y[4],
                                           double dx[4], double dy[4]) {
    const int me = R.self();
    const double2 pi_ = R.xy(me);
    const R4 M = ld4w(reinterpret_cast<const R4 *>(g.minv) + i);
    double sA[4] = {0.0, 0.0, 0.0, 0.0}, sB[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r0 = 0; r0 < nb; r0 += 8) {
        const unsigned long long word = R.word(r0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = r0 + j;
            if (r >= nb) break;
            const int k = R.nbr(r, word, j);
            double dxk[4], dyk[4];
            R.dqrow(k, dxk, dyk);
            const double2 pk = R.xy(k);
            const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
            const double w = g.wsl ? __ldg(g.wsl + (size_t)r * g.n + i) : 1.0;
            const double wx = w * delx, wy = w * dely;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const double t = fma(delx, dxk[m], dely * dyk[m]);
                sA[m] = fma(wx, t, sA[m]);
                sB[m] = fma(wy, t, sB[m]);
            }
        }
    }
    double dxi[4], dyi[4];
    R.dqrow(me, dxi, dyi);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const double Lx = fma(M.a, sA[m], M.b * sB[m]);
        const double Ly = fma(M.b, sA[m], M.c * sB[m]);
        dx[m] = fma(-0.5, Lx, fma(0.5, dxi[m], dq0x[m]));
        dy[m] = fma(-0.5, Ly, fma(0.5, dyi[m], dq0y[m]));
    }
}

// 64-byte rows in two 256-bit stores (st.global.v4.f64, sm_100): a warp's
// store of 32 rows touches each 128-byte line once per store instead of
// once per 16-byte piece.
__device__ __forceinline__ void st8w(double *p, const double a[4], const double b[4]) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a[0]), "d"(a[1]),
                 "d"(a[2]), "d"(a[3]) : "memory");
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p + 4), "d"(b[0]), "d"(b[1]),
                 "d"(b[2]), "d"(b[3]) : "memory");
}

// Stages a chunk's halo rows (stage_array): the D pass q (two pieces a row),
// (x, y) and, with spd != nullptr, spd; the I pass (x, y) and dq (four pieces a
// row).  Consecutive lanes copy consecutive 16-byte pieces of a row array, so
// that runs of neighbouring rows come in whole 128-byte lines.
template <int nA, int CAP>
__device__ __forceinline__ void stage_halo(const Geom &g, const R4 *q, const double *dq,
                                           const double *spd, const HaloIdx<CAP> &x, int lane,
                                           double2 *sm0, double2 *sm1) {
    using H = HaloRows<nA, CAP>;
    const HaloStride<nA, CAP> st(g.hc);
    if (nA == HA_D) stage_array<2>(q, 32, x, lane, sm0, sm1, st.hc, 0);
    stage_array<1>(g.xy, 16, x, lane, sm0, sm1, st.hc, H::OXY);
    if (nA == HA_I) stage_array<4>(dq, 64, x, lane, sm0, sm1, st.hc, H::ODQ);
    else if (spd) stage_array8(spd, x, lane, sm0, sm1, st.hc, H::OSPD);
}

// The D and I passes with tile halos (halo.cuh): a warp stages two tiles'
// halo rows, waits, and computes one point per lane from shared memory; a
// tile whose halo was too large to stage reads its rows directly.  No block
// barrier but the schedule load; the lanes of a warp meet at __syncwarp
// before the rows are read and before they are overwritten.
template <int CAP>
__global__ void __launch_bounds__(HALO_BLOCK, HALO_MIN_BLOCKS_I)
kb_inner_h(Geom g, Sched s, const double *__restrict__ dq0,
           const double *__restrict__ dq_in, double *__restrict__ dq_out) {
    extern __shared__ double2 hsm[];
    __shared__ SchedSmem ss;
    int live;
    const int ntiles = sched_begin(s, ss, live);
    const int wpb = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int half = lane / TILE, stride = gridDim.x * wpb;
    double2 *sm0 = hsm + (2 * warp) * HA_I * g.hc, *sm1 = sm0 + HA_I * g.hc;
    HaloChunk<CAP> cur;
    for (int ch = blockIdx.x * wpb + warp; 2 * ch < ntiles; ch += stride) {
        halo_chunk(g, s, ss, ntiles, ch, lane, cur);
        if (!live) return;
        stage_halo<HA_I>(g, nullptr, dq_in, nullptr, cur.x, lane, sm0, sm1);
        const HaloRows<HA_I, CAP> hr(g, half ? sm1 : sm0, cur.hn > 0 ? cur.i : -1);
        double ax[4], ay[4];
        if (cur.i >= 0) ld8w(dq0 + 8 * (size_t)cur.i, ax, ay);
        halo_wait();
        __syncwarp();
        if (cur.i >= 0) {
            double dx[4], dy[4];
            if (cur.hn > 0) inner_sums(g, cur.i, hr, cur.nb, ax, ay, dx, dy);
            else
                inner_sums(g, cur.i, GlobalRows{g, nullptr, dq_in, nullptr, cur.i}, cur.nb, ax,
                           ay, dx, dy);
            st8w(dq_out + 8 * (size_t)cur.i, dx, dy);
        }
        __syncwarp();
    }
}

template <int CAP>
__global__ void __launch_bounds__(HALO_BLOCK, HALO_MIN_BLOCKS_D)
kb_grad_h(Geom g, Consts c, Sched s, const R4 *__restrict__ q, const double *__restrict__ spd,
          double *__restrict__ dq, double *__restrict__ qm, double *__restrict__ delta,
          int with_delta) {
    extern __shared__ double2 hsm[];
    __shared__ SchedSmem ss;
    int live;
    const int ntiles = sched_begin(s, ss, live);
    const int wpb = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int half = lane / TILE, stride = gridDim.x * wpb;
    const HaloStride<HA_D, CAP> st(g.hc);
    double2 *sm0 = hsm + (2 * warp) * HA_D * st.hc, *sm1 = sm0 + HA_D * st.hc;
    HaloChunk<CAP> cur;
    for (int ch = blockIdx.x * wpb + warp; 2 * ch < ntiles; ch += stride) {
        halo_chunk(g, s, ss, ntiles, ch, lane, cur);
        if (!live) return;
        stage_halo<HA_D>(g, q, nullptr, with_delta ? spd : nullptr, cur.x, lane, sm0, sm1);
        const HaloRows<HA_D, CAP> hr(g, half ? sm1 : sm0, cur.hn > 0 ? cur.i : -1);
        halo_wait();
        __syncwarp();
        if (cur.i >= 0) {
            double dx[4], dy[4], qmax[4], qmin[4], min_delt;
            if (cur.hn > 0)
                grad_sums(c, g, cur.i, hr, cur.nb, with_delta, dx, dy, qmax, qmin, min_delt);
            else
                grad_sums(c, g, cur.i, GlobalRows{g, q, nullptr, spd, cur.i}, cur.nb, with_delta,
                          dx, dy, qmax, qmin, min_delt);
            st8w(dq + 8 * (size_t)cur.i, dx, dy);
            st8w(qm + 8 * (size_t)cur.i, qmax, qmin);
            if (with_delta) delta[cur.i] = min_delt;
        }
        __syncwarp();
    }
}

// The D and I passes of a small grid (slot_passes): eight lanes a point, a
// stencil slot a lane, four points a warp.  With few points the passes wait,
// they do not compute: the halo form's chain (halo range, row indices, copies,
// then eight slots in turn) becomes index, row, eight sums.  A slot's lane
// leaves its row in shared memory and lane l sums field l over the slots in
// slot order, the halo form's own operations, so a grid gets the same values
// from either (the products' contractions are spelled out in both).
// D and I pass at 1,536 points, one inner iteration: an iteration 65.2 ->
// 48.2 us; at 16,000 points 97.0 -> 87.8.
__global__ void __launch_bounds__(SLOT_BLOCK)
kb_grad_s(Geom g, Consts c, Sched s, const R4 *__restrict__ q, const double *__restrict__ spd,
          double *__restrict__ dq, double *__restrict__ qm, double *__restrict__ delta,
          int with_delta) {
    __shared__ SchedSmem ss;
    __shared__ double sm[SLOT_PTS * SLOT_P];
    int live;
    const int total = sched_begin(s, ss, live) * TILE;
    const int p = threadIdx.x / LPP, l = threadIdx.x % LPP, m = l & 3;
    double *row = sm + p * SLOT_P;  // fields qk[4], w dx, w dy
    for (int v0 = blockIdx.x * SLOT_PTS; v0 < total; v0 += gridDim.x * SLOT_PTS) {
        const int i = slot_point(s, ss, total, v0 + p);
        int nb = 0, k = 0;
        double2 pi_ = make_double2(0.0, 0.0);
        double qi = 0.0, M0 = 0.0, M1 = 0.0;
        if (i >= 0) {
            nb = __ldg(g.nbhs + i);
            if (l < g.kp) k = __ldg(g.conn + (size_t)l * g.n + i);
            pi_ = g.xy[i];
            qi = __ldg(reinterpret_cast<const double *>(q + i) + m);
            // dx = a sx + b sy, dy = b sx + c sy: the factors of this lane's sums
            M0 = __ldg(g.minv + 4 * (size_t)i + (l < 4 ? 0 : 2));
            M1 = __ldg(g.minv + 4 * (size_t)i + 1);
        }
        if (!live) return;
        double sum = 0.0, ext = qi, dmin = 1.0;
        const int nbw = __reduce_max_sync(0xffffffffu, nb);
        for (int r0 = 0; r0 < nbw; r0 += LPP) {
            const int r = r0 + l;
            if (r0 > 0 && r < nb) k = __ldg(g.conn + (size_t)r * g.n + i);
            if (r < nb) {
                double qk[4];
                const R4 a = ld4w(q + k);
                qk[0] = a.a; qk[1] = a.b; qk[2] = a.c; qk[3] = a.d;
                const double2 pk = g.xy[k];
                const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
                const double w = g.wsl ? __ldg(g.wsl + (size_t)r * g.n + i) : 1.0;
#pragma unroll
                for (int f = 0; f < 4; ++f) row[f * SLOT_F + l] = qk[f];
                row[4 * SLOT_F + l] = w * delx;
                row[5 * SLOT_F + l] = w * dely;
                if (with_delta) {
                    double delta_t = sqrt(fma(delx, delx, dely * dely)) / spd[k];
                    delta_t = c.cfl * delta_t;
                    if (dmin > delta_t) dmin = delta_t;
                }
            }
            __syncwarp();
            const double *qf = row + m * SLOT_F, *wf = row + (4 + l / 4) * SLOT_F;
#pragma unroll
            for (int j = 0; j < LPP; ++j) {
                if (r0 + j >= nb) break;
                const double qk = qf[j], wd = wf[j];
                if (l < 4 ? qk > ext : qk < ext) ext = qk;
                sum = fma(wd, qk - qi, sum);
            }
            __syncwarp();
        }
        // lanes 0-3 hold sx and qmax, 4-7 sy and qmin
        const double other = __shfl_xor_sync(0xffffffffu, sum, 4);
        if (with_delta) {
#pragma unroll
            for (int o = 4; o; o >>= 1) {
                const double d = __shfl_xor_sync(0xffffffffu, dmin, o);
                if (dmin > d) dmin = d;
            }
        }
        if (i >= 0) {
            dq[8 * (size_t)i + l] = l < 4 ? fma(M0, sum, M1 * other) : fma(M1, other, M0 * sum);
            qm[8 * (size_t)i + l] = ext;
            if (with_delta && l == 0) delta[i] = dmin;
        }
    }
}

__global__ void __launch_bounds__(SLOT_BLOCK)
kb_inner_s(Geom g, Sched s, const double *__restrict__ dq0, const double *__restrict__ dq_in,
           double *__restrict__ dq_out) {
    __shared__ SchedSmem ss;
    __shared__ double sm[SLOT_PTS * SLOT_P];
    int live;
    const int total = sched_begin(s, ss, live) * TILE;
    const int p = threadIdx.x / LPP, l = threadIdx.x % LPP, m = l & 3;
    double *row = sm + p * SLOT_P;  // fields d . dq_k [4], w dx, w dy
    for (int v0 = blockIdx.x * SLOT_PTS; v0 < total; v0 += gridDim.x * SLOT_PTS) {
        const int i = slot_point(s, ss, total, v0 + p);
        int nb = 0, k = 0;
        double2 pi_ = make_double2(0.0, 0.0);
        double a0 = 0.0, di = 0.0, M0 = 0.0, M1 = 0.0;
        if (i >= 0) {
            nb = __ldg(g.nbhs + i);
            if (l < g.kp) k = __ldg(g.conn + (size_t)l * g.n + i);
            pi_ = g.xy[i];
            a0 = __ldg(dq0 + 8 * (size_t)i + l);
            di = __ldg(dq_in + 8 * (size_t)i + l);
            M0 = __ldg(g.minv + 4 * (size_t)i + (l < 4 ? 0 : 2));
            M1 = __ldg(g.minv + 4 * (size_t)i + 1);
        }
        if (!live) return;
        double sum = 0.0;
        const int nbw = __reduce_max_sync(0xffffffffu, nb);
        for (int r0 = 0; r0 < nbw; r0 += LPP) {
            const int r = r0 + l;
            if (r0 > 0 && r < nb) k = __ldg(g.conn + (size_t)r * g.n + i);
            if (r < nb) {
                double dxk[4], dyk[4];
                ld8w(dq_in + 8 * (size_t)k, dxk, dyk);
                const double2 pk = g.xy[k];
                const double delx = pk.x - pi_.x, dely = pk.y - pi_.y;
                const double w = g.wsl ? __ldg(g.wsl + (size_t)r * g.n + i) : 1.0;
#pragma unroll
                for (int f = 0; f < 4; ++f) row[f * SLOT_F + l] = fma(delx, dxk[f], dely * dyk[f]);
                row[4 * SLOT_F + l] = w * delx;
                row[5 * SLOT_F + l] = w * dely;
            }
            __syncwarp();
            const double *tf = row + m * SLOT_F, *wf = row + (4 + l / 4) * SLOT_F;
#pragma unroll
            for (int j = 0; j < LPP; ++j) {
                if (r0 + j >= nb) break;
                sum = fma(wf[j], tf[j], sum);
            }
            __syncwarp();
        }
        const double other = __shfl_xor_sync(0xffffffffu, sum, 4);
        const double L = l < 4 ? fma(M0, sum, M1 * other) : fma(M1, other, M0 * sum);
        if (i >= 0) dq_out[8 * (size_t)i + l] = fma(-0.5, L, fma(0.5, di, a0));
    }
}

// flux_residual.F90:14-73 cal_flux_residual + state_update.F90:10-141 +
// q_variables.F90:8-37 on the new state.
//
// Work split: eight lanes a point, one stencil slot a lane, four points a
// warp round.  A lane reconstructs both states of its slot once (limiter +
// qtilde -> kinetic state; the reference repeats this per direction list with
// identical inputs), evaluates the split fluxes of the lists the neighbour
// belongs to, and adds their differences times the slot's weight in the
// list's least-squares solve.
//
// The solve is folded into a weight per slot: list L's derivative is
// (fx sdy2 - fy sdxy) / det with fx = sum dG dels w, fy = sum dG deln w, that
// is sum dG c with c = (a dels + b deln) w, a = sdy2 / det, b = -sdxy / det (y
// lists: the roles of dels and deln swapped).  a and b are geometry, formed
// once per grid (k_flux_coef).  The flux residual is the sum of the list
// derivatives, so the lists need not be told apart: a lane adds both
// directions' terms into four sums and eight lanes add theirs by shuffles.
// Per point and split list L: a, b of the list's solve (fco[8 i + 2 L]).
// *_fluxes.F90 dG*: the sums in slot order; a list the point's kind does not
// have (wall ypos, outer yneg) gets zeros.  fcg: the third entry of the list's
// inverse normal matrix (the reverse pass); minv: the full stencil's.
__global__ void k_flux_coef(Geom g, int base, int n, int nw, int no, double power,
                            double *__restrict__ fco, double *__restrict__ wsl,
                            double *__restrict__ fcg, double *__restrict__ minv) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int i = base + j;
    const int kind = j < nw ? KIND_WALL : (j < nw + no ? KIND_OUTER : KIND_INTERIOR);
    const double2 p = g.xy[i], nn = g.nrm[i];
    const unsigned long long bits[2] = {g.mx[i], g.my[i]};
    double sxx[4] = {}, syy[4] = {}, sxy[4] = {}, mxx = 0.0, myy = 0.0, mxy = 0.0;
    for (int r = 0; r < g.nbhs[i]; ++r) {
        const double2 pk = g.xy[g.conn[(size_t)r * g.n + i]];
        const double delx = pk.x - p.x, dely = pk.y - p.y;
        const double dels = delx * nn.y - dely * nn.x, deln = delx * nn.x + dely * nn.y;
        double w = 1.0;
        if (wsl) {
            w = pow(sqrt(delx * delx + dely * dely), power);
            wsl[(size_t)r * g.n + i] = w;
        }
        mxx = mxx + delx * delx * w;
        myy = myy + dely * dely * w;
        mxy = mxy + delx * dely * w;
        const double dw = dels * w, nw_ = deln * w;
#pragma unroll
        for (int L = 0; L < 4; ++L) {
            if (!((bits[L >> 1] >> (r + ((L & 1) ? 32 : 0))) & 1ull)) continue;
            sxx[L] = sxx[L] + dels * dw;
            syy[L] = syy[L] + deln * nw_;
            sxy[L] = sxy[L] + dels * nw_;
        }
    }
    if (minv) {
        const double ob = 1.0 / (mxx * myy - mxy * mxy);
        st4(reinterpret_cast<R4 *>(minv) + i, myy * ob, -mxy * ob, mxx * ob, 0.0);
    }
#pragma unroll
    for (int L = 0; L < 4; ++L) {
        const bool none = (kind == KIND_WALL && L == 2) || (kind == KIND_OUTER && L == 3);
        const double ob = 1.0 / (sxx[L] * syy[L] - sxy[L] * sxy[L]);
        fco[8 * (size_t)i + 2 * L] = none ? 0.0 : (L < 2 ? syy[L] : sxx[L]) * ob;
        fco[8 * (size_t)i + 2 * L + 1] = none ? 0.0 : -sxy[L] * ob;
        if (fcg) fcg[4 * (size_t)i + L] = none ? 0.0 : (L < 2 ? sxx[L] : syy[L]) * ob;
    }
}

// Shared memory of the unit that computes a tile (a warp, or in the shared
// split the block): the tile's halo rows (halo.cuh) as one array per 16-byte
// piece -- q 0-1, dq 2-5, qm 6-9, (x, y) 10 -- at a fixed stride, so that a
// row's pieces are immediate offsets from its first, and an 8-byte array of
// eps2; per point of the tile (nx, ny), the membership masks, the list
// coefficients, local rows and stencil size; the chunk's flux residuals.
// ROWS is what four blocks an SM leave room for (an O-grid's tiles have 54
// rows, a point cloud's in RCM order 54 to 60); a larger tile reads its rows
// from global memory.
struct FluxSmem {
    static constexpr int ROWS = 60, HC = ROWS + 1;
    double2 halo[11][HC];
    double eps[HC + 1];
    double2 co[TILE][4];
    FluxOwn own;
    double G[CHUNK_MAX][4];  // flux residuals, then residual terms
};
constexpr int FLUX_SMEM = FLUX_WARPS * sizeof(FluxSmem);

// Copies a tile's rows (cp.async).
template <int NT>
__device__ __forceinline__ void stage_flux(const Geom &g, const StageBufs &b, const FluxTile &t,
                                           const FluxHalo &x, FluxSmem &m, int tid) {
    stage_rows<2, NT, FluxSmem::HC>(b.q_in, x, m.halo[0], tid);
    stage_rows<4, NT, FluxSmem::HC>(b.dq, x, m.halo[2], tid);
    stage_rows<4, NT, FluxSmem::HC>(b.qm, x, m.halo[6], tid);
    if (tid < HALO_CAP) {
#pragma unroll
        for (int u0 = 0; u0 < HALO_CAP; u0 += NT < HALO_CAP ? NT : HALO_CAP) {
            const int u = u0 + tid;
            const int k = x.row(u);
            if (u < x.hn) {
                halo_cp16(&m.halo[10][u], g.xy + k);
                halo_cp8(&m.eps[u], g.eps2 + k);
            }
        }
    }
    const double2 *co = reinterpret_cast<const double2 *>(g.fco + 8 * (size_t)t.i0);
#pragma unroll
    for (int q = 0; q < (NT < 64 ? 64 / NT : 1); ++q) {
        const int pc = q * NT + tid;
        if (pc < 4 * t.cnt) halo_cp16(&m.co[pc >> 2][pc & 3], co + pc);
    }
    m.own.stage<NT>(g, t, tid);
}

// A row in registers: staged (row l of the halo) or from global memory.
struct FluxRow {
    double q[4], dx[4], dy[4], qmax[4], qmin[4], eps2;
    double2 xy;
    __device__ __forceinline__ void staged(const FluxSmem &m, int l) {
        double *f[5] = {q, dx, dy, qmax, qmin};
#pragma unroll
        for (int a = 0; a < 5; ++a)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double2 v = m.halo[2 * a + h][l];
                f[a][2 * h] = v.x;
                f[a][2 * h + 1] = v.y;
            }
        xy = m.halo[10][l];
        eps2 = m.eps[l];
    }
    __device__ __forceinline__ void global(const Geom &g, const StageBufs &b, int k) {
        const R4 v = ld4w(b.q_in + k);
        q[0] = v.a; q[1] = v.b; q[2] = v.c; q[3] = v.d;
        ld8w(b.dq + 8 * (size_t)k, dx, dy);
        ld8w(b.qm + 8 * (size_t)k, qmax, qmin);
        xy = g.xy[k];
        eps2 = g.eps2[k];
    }
    __device__ __forceinline__ void qtilde(double delx, double dely, double qt[4]) const {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            qt[c] = limited_qtilde(delx * dx[c] + dely * dy[c], q[c], qmax[c], qmin[c], eps2);
    }
};

// One point group of a warp round: the flux residual of point j of tile t
// (its list-derivative sum) into Gout.  hn: the tile's staged rows (0: none).
// TAPE: also write both reconstructed kinetic states of every slot to
// b.kstape (the adjoint's taped re-run; the primal runs TAPE = false).
template <bool TAPE>
__device__ __forceinline__ void flux_group(const Geom &g, const StageBufs &b, const FluxTile &t,
                                           int j, int hn, FluxSmem &m, double *Gout) {
    const int lane = threadIdx.x % LPP;
    const double inv_sqrt_pi = 0.56418958354775628695;
    const int kind = t.kind(j), i = t.i0 + j;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const double2 nn = m.own.nrm[j];
    const double nx = nn.x, ny = nn.y;
    const int nb = j < t.cnt ? m.own.nbhs[j] : 0;
    for (int r = lane; r < nb; r += LPP) {
        KState sk, si;
        double ui[2], uk[2], delx, dely;
        {
            double qk[4], qi[4];
            if (hn > 0) {
                int lk, li;
                m.own.rows(g, i, j, r, lk, li);
                const double2 pi_ = m.halo[10][li], pk = m.halo[10][lk];
                delx = pk.x - pi_.x;
                dely = pk.y - pi_.y;
                FluxRow o;
                o.staged(m, lk);
                o.qtilde(delx, dely, qk);
                o.staged(m, li);
                o.qtilde(delx, dely, qi);
            } else {
                const int k = g.conn[(size_t)r * g.n + i];
                const double2 pi_ = g.xy[i], pk = g.xy[k];
                delx = pk.x - pi_.x;
                dely = pk.y - pi_.y;
                FluxRow o;
                o.global(g, b, k);
                o.qtilde(delx, dely, qk);
                o.global(g, b, i);
                o.qtilde(delx, dely, qi);
            }
            kstate_pair(qi, qk, nx, ny, inv_sqrt_pi, si, sk, ui, uk);
        }
        if (TAPE) {
            // per state rho, p/rho, B1, B2, e1, e2, u1, u2 (ut, un and |u|^2
            // follow from u and the point's normal)
            const double t[KS_TAPE] = {si.rho, si.pbr, si.B1, si.B2, si.e1, si.e2, ui[0], ui[1],
                                       sk.rho, sk.pbr, sk.B1, sk.B2, sk.e1, sk.e2, uk[0], uk[1]};
            double *tp = b.kstape + ((size_t)i * g.kp + r) * KS_TAPE;
            st8w(tp, t, t + 4);
            st8w(tp + 8, t + 8, t + 12);
        }
        double dels = delx * ny - dely * nx, deln = delx * nx + dely * ny;
        if (g.wsl) {
            const double w = g.wsl[(size_t)r * g.n + i];
            dels *= w;
            deln *= w;
        }
        // Per direction the neighbour is in one list of the pair, in both only
        // when its projection is exactly 0: the second list is added then.
        const uint4 mm = m.own.mask[j];
        const double w6i = fma(6.0, si.pbr, si.usq), w6k = fma(6.0, sk.pbr, sk.usq);
        auto add_x = [&](int l, double sg) {
            const double2 co = m.co[j][l];
            const double w = fma(co.x, dels, co.y * deln);
            double Gi[4], Gk[4];
            if (kind == KIND_INTERIOR) {
                flux_split(si, si.ut, si.un, si.B1, si.e1, sg, 0.5 * sg, w6i, Gi);
                flux_split(sk, sk.ut, sk.un, sk.B1, sk.e1, sg, 0.5 * sg, w6k, Gk);
            } else {
                // wall GxII/GxI (A2neg), outer GxIII/GxIV (A2pos)
                const double s2 = kind == KIND_WALL ? -1.0 : 1.0;
                flux_quad(si, sg, s2, Gi);
                flux_quad(sk, sg, s2, Gk);
            }
#pragma unroll
            for (int d = 0; d < 4; ++d) v[d] = fma(w, Gk[d] - Gi[d], v[d]);
        };
        auto add_y = [&](int l, double sg) {
            const double2 co = m.co[j][2 + l];
            const double w = fma(co.x, deln, co.y * dels);
            double Gi[4], Gk[4];
            flux_split(si, si.un, si.ut, si.B2, si.e2, sg, 0.5 * sg, w6i, Gi);
            flux_split(sk, sk.un, sk.ut, sk.B2, sk.e2, sg, 0.5 * sg, w6k, Gk);
            v[0] = fma(w, Gk[0] - Gi[0], v[0]);
            v[1] = fma(w, Gk[2] - Gi[2], v[1]);
            v[2] = fma(w, Gk[1] - Gi[1], v[2]);
            v[3] = fma(w, Gk[3] - Gi[3], v[3]);
        };
        const unsigned bit = 1u << r;
        const bool x0 = mm.x & bit, y0 = mm.z & bit;
        add_x(x0 ? 0 : 1, x0 ? 1.0 : -1.0);
        add_y(y0 ? 0 : 1, y0 ? 1.0 : -1.0);
        if (((mm.x & mm.y) | (mm.z & mm.w)) & bit) {
            if (mm.x & mm.y & bit) add_x(1, -1.0);
            if (mm.z & mm.w & bit) add_y(1, -1.0);
        }
    }
    __syncwarp();
    const double sum = reduce8(v, lane);
    if (!(lane & 1)) Gout[lane >> 1] = sum;
}

// state_update.F90:10-141 of one point from the sum of its list derivatives;
// returns its res_sqr term.
__device__ __forceinline__ double
update_point(const Geom &g, const Consts &c, const StageBufs &b, int rk, int last, int i,
             int kind, int orow, const double *Gs) {
    const double2 nn = g.nrm[i];
    const double nx = nn.x, ny = nn.y;
    double res_sqr = 0.0;
    {
        const double delta = b.delta[i];
        const R4 P = ld4(b.prim_in + i), O = rk == 3 ? ld4(b.prim_old + i) : R4{0, 0, 0, 0};
        double fr[4];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            fr[m] = (kind == KIND_WALL ? 2.0 * delta : delta) * Gs[m];
        if (b.flux_dbg) st4(reinterpret_cast<R4 *>(b.flux_dbg) + i, fr[0], fr[1], fr[2], fr[3]);
        double U[4], Uo[4] = {0.0, 0.0, 0.0, 0.0};
        if (kind == KIND_OUTER) {
            const double *inf = g.obc + 8 * (size_t)orow;
            conserved_ubar(P.a, P.b, P.c, P.d, nx, ny, inf, c.pi, c.gm1, U);
            if (rk == 3) {
                conserved_ubar(O.a, O.b, O.c, O.d, nx, ny, inf, c.pi, c.gm1, Uo);
            }
        } else {
            prim_to_conserved(P.a, P.b, P.c, P.d, nx, ny, U);
            if (rk == 3) {
                prim_to_conserved(O.a, O.b, O.c, O.d, nx, ny, Uo);
            }
        }
        double temp = U[0];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (rk != 3) U[m] = U[m] - (0.5 * c.euler * fr[m]);
            else U[m] = TBT * Uo[m] + OBT * (U[m] - 0.5 * fr[m]);
        }
        if (kind == KIND_WALL) U[2] = 0.0;
        double U2_rot = U[1], U3_rot = U[2];
        U[1] = U2_rot * ny + U3_rot * nx;
        U[2] = U3_rot * ny - U2_rot * nx;
        if (kind != KIND_OUTER) res_sqr = (U[0] - temp) * (U[0] - temp);
        double rho = U[0];
        temp = 1.0 / U[0];
        double u1 = U[1] * temp;
        double u2 = U[2] * temp;
        double pr = 0.4 * (U[3] - (0.5 * temp) * (U[1] * U[1] + U[2] * U[2]));
        st4(b.prim_out + i, rho, u1, u2, pr);
        double qn[4];
        q_from_prim(rho, u1, u2, pr, qn);
        st4(b.q_out + i, qn[0], qn[1], qn[2], qn[3]);
        if (last) b.spd[i] = sqrt(u1 * u1 + u2 * u2) + 3.0 * sqrt(pr / rho);
    }
    return res_sqr;
}

template <bool TAPE>
struct Flux64 {
    using Smem = FluxSmem;
    const Geom &g;
    const Consts &c;
    const StageBufs &b;
    int rk, last;
    template <int NT>
    __device__ __forceinline__ void stage(const FluxTile &t, const FluxHalo &x, Smem &m, int tid) {
        stage_flux<NT>(g, b, t, x, m, tid);
    }
    __device__ __forceinline__ void group(const FluxTile &t, int j, int hn, Smem &m, double *G) {
        flux_group<TAPE>(g, b, t, j, hn, m, G);
    }
    __device__ __forceinline__ double update(int i, int kind, int orow, const double *G) {
        return update_point(g, c, b, rk, last, i, kind, orow, G);
    }
};

// F pass (flux_pass).
template <bool TAPE>
__global__ void __launch_bounds__(FLUX_BLOCK, FLUX_MIN_BLOCKS)
kb_flux(Geom g, Consts c, Sched s, StageBufs b, int rk, int last, int ct, int coop) {
    extern __shared__ double2 fsm[];
    Flux64<TAPE> p{g, c, b, rk, last};
    flux_pass(p, g, s, reinterpret_cast<FluxSmem *>(fsm), b.res_part, last, ct, coop);
}

// Sum of nparts tile partials in a fixed order (deterministic, independent
// of the launch shape of the passes that wrote them): thread t of a block of
// RES_BLOCK keeps sixteen accumulators over partials t + RES_BLOCK j (j mod 16
// picks the accumulator, so the loads of one thread are independent), adds them
// pairwise, and trees over the warps and over their sums add the threads.  The
// result is returned to warp 0; s: one double a warp.  One block an instance:
// bound by the latency of its loads.
constexpr int RES_BLOCK = 512;
__device__ __forceinline__ double sum_parts_block(const double *__restrict__ part, int nparts,
                                                  double *s) {
    constexpr int U = 16, T = RES_BLOCK;
    double acc[U] = {};
    int t = threadIdx.x;
#pragma unroll 2
    for (; t + (U - 1) * T < nparts; t += U * T) {
#pragma unroll
        for (int j = 0; j < U; ++j) acc[j] = acc[j] + __ldg(part + t + j * T);
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
        if (t + j * T < nparts) acc[j] = acc[j] + __ldg(part + t + j * T);
#pragma unroll
    for (int w = U / 2; w > 0; w >>= 1)
#pragma unroll
        for (int j = 0; j < w; ++j) acc[j] = acc[j] + acc[j + w];
    double v = acc[0];
    for (int w = 16; w > 0; w >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, w);
    if (threadIdx.x % 32 == 0) s[threadIdx.x / 32] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < T / 32 ? s[threadIdx.x] : 0.0;
        for (int w = 16; w > 0; w >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, w);
    }
    return v;
}

// fpi_solver.F90:57-70: res_new = sqrt(sum res_sqr)/plen and the residue.
// Whole block of RES_BLOCK threads; the residue is returned on thread 0.
__device__ __forceinline__ double residual_block(const double *__restrict__ part, int nparts,
                                                 Ctl *ctl, double *hist, double *s) {
    const double sum = sum_parts_block(part, nparts, s);
    if (threadIdx.x == 0) {
        double res_new = sqrt(sum) / ctl->plen;
        int it = ctl->it;
        double residue;
        if (it <= 2 && ctl->restart == 0) {
            ctl->res_old = res_new;
            residue = 0.0;
        } else {
            residue = log10(res_new / ctl->res_old);
        }
        hist[it - ctl->it_first] = residue;
        ctl->it = it + 1;
        ctl->done = ctl->done + 1;
        if (isnan(residue)) ctl->halted = 1;
        return residue;
    }
    return 0.0;
}

// Sum of nparts tile partials in the fixed order of residual_block (one
// block of RES_BLOCK threads): a partitioned grid's share of the residual, which
// the host adds over the ranks before the norm.
__global__ void __launch_bounds__(RES_BLOCK)
k_sum_parts(const double *__restrict__ part, int nparts, double *out) {
    __shared__ double s[RES_BLOCK / 32];
    const double sum = sum_parts_block(part, nparts, s);
    if (threadIdx.x == 0) *out = sum;
}

// Per-instance residual (block b = instance b): the instance's tile partials
// are reduced in the order of residual_block, then the retirement rule of the
// run is applied (NaN residue, residue <= tol, max_iters iterations).  The
// last block to finish (threadfence + ticket, no waiting) rebuilds the
// schedule from Ctl::active for the next iteration's passes: a stable
// compaction of the running instances and the prefix sums of their tile
// counts (Hillis-Steele scans over MAX_BATCH slots).
__global__ void __launch_bounds__(RES_BLOCK)
kb_residual(const InstInfo *__restrict__ inst, int n_inst, const double *__restrict__ part,
            Ctl *ctl, double *hist, int hist_ld, const BatchRun *__restrict__ run,
            int *sched) {
    __shared__ double s[RES_BLOCK / 32];
    __shared__ int s_last;
    __shared__ int cnt[MAX_BATCH], til[MAX_BATCH];
    Ctl *c = ctl + blockIdx.x;
    const InstInfo in = inst[blockIdx.x];
    // (thread 0 changes it behind the barrier of the sum, which the whole block
    // meets or, if it is 0, skips)
    const int active = c->active;
    if (active) {
        const double residue =
            residual_block(part + in.tile0, in.ntiles, c, hist + (size_t)blockIdx.x * hist_ld, s);
        if (threadIdx.x == 0) {
            if (isnan(residue)) {
                c->active = 0;
                c->state = BATCH_NONFINITE;
            } else if (residue <= run->tol) {
                c->active = 0;
                c->state = BATCH_CONVERGED;
            } else if (c->done >= run->max_iters) {
                c->active = 0;
                c->state = BATCH_MAX_ITERS;
            }
        }
    }
    int *pre = sched + SCHED_PRE, *act = sched + SCHED_ACT;
    if (gridDim.x == 1) {  // one instance: its own schedule
        if (threadIdx.x == 0) {
            const int on = c->active ? 1 : 0;
            sched[SCHED_NACT] = on;
            pre[0] = 0;
            pre[on] = on ? in.ntiles : 0;
            act[0] = 0;
        }
        return;
    }
    int *counter = sched + SCHED_COUNTER;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int t = threadIdx.x;
    int a = 0, nt = 0;
    if (t < MAX_BATCH) {
        a = (t < n_inst && reinterpret_cast<volatile const int *>(&ctl[t].active)[0]) ? 1 : 0;
        nt = a ? inst[t].ntiles : 0;
        cnt[t] = a;
        til[t] = nt;
    }
    __syncthreads();
    for (int off = 1; off < MAX_BATCH; off <<= 1) {
        int x = 0, y = 0;
        if (t < MAX_BATCH && t >= off) {
            x = cnt[t - off];
            y = til[t - off];
        }
        __syncthreads();
        if (t < MAX_BATCH) {
            cnt[t] += x;
            til[t] += y;
        }
        __syncthreads();
    }
    if (a) {
        act[cnt[t] - 1] = t;
        pre[cnt[t] - 1] = til[t] - nt;
    }
    if (t == MAX_BATCH - 1) {
        sched[SCHED_NACT] = cnt[t];
        pre[cnt[t]] = til[t];
        *counter = 0;
    }
}

// q and spd of rows [i0, i1) from their prim (set_state: every row; a
// partitioned grid: the ghost rows after their exchange)
__global__ void k_init_state(Geom g, const R4 *__restrict__ prim, R4 *__restrict__ q,
                             double *__restrict__ spd, int i0, int i1) {
    int i = i0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= i1) return;
    R4 P = ld4(prim + i);
    double qn[4];
    q_from_prim(P.a, P.b, P.c, P.d, qn);
    st4(q + i, qn[0], qn[1], qn[2], qn[3]);
    spd[i] = sqrt(P.b * P.b + P.c * P.c) + 3.0 * sqrt(P.d / P.a);
}

// compute_force_coeffs.F90:11-102.  One block of FORCE_BLOCK threads, so the
// sums do not depend on the launch: a thread adds its points j, j +
// FORCE_BLOCK, ... of a shape in grid order, then a tree over the block adds
// the threads.  (Thread 0 adding every point in turn took 108 us at 1,280
// shape points, 17 at 160; now 7 and 6.)
constexpr int FORCE_BLOCK = 512;

__global__ void __launch_bounds__(FORCE_BLOCK)
k_forces(ShapeTab t, const R4 *__restrict__ prim, double mach, double cos_t, double sin_t,
         double *out) {
    __shared__ double sm[3][FORCE_BLOCK / 32];
    const double rho_inf = 1.0, pr_inf = 1.0 / 1.4;
    double *cp_out = out + 3 * t.shapes;
    const double temp = 0.5 * rho_inf * mach * mach;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    for (int s = 0; s < t.shapes; ++s) {
        double v[3] = {0.0, 0.0, 0.0};  // H, V, pitching moment
        for (int j = threadIdx.x; j < t.npts; j += FORCE_BLOCK) {
            if (t.shape[j] != s) continue;
            const double nx = t.geo[4 * j], ny = t.geo[4 * j + 1], ds = t.geo[4 * j + 2];
            const double mx = t.geo[4 * j + 3], my = t.my[j];
            double cp = prim[t.idx[j]].d - pr_inf;
            cp = -cp / temp;
            cp_out[j] = cp;
            v[0] = v[0] + cp * nx * ds;
            v[1] = v[1] + cp * ny * ds;
            v[2] = v[2] + (-cp * ny * ds * (mx - 0.25) + cp * nx * ds * (my));
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            for (int w = 16; w > 0; w >>= 1) v[c] = v[c] + __shfl_xor_sync(0xffffffffu, v[c], w);
            if (lane == 0) sm[c][warp] = v[c];
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int c = 0; c < 3; ++c) {
                v[c] = 0.0;
                for (int w = 0; w < FORCE_BLOCK / 32; ++w) v[c] = v[c] + sm[c][w];
            }
            out[s] = v[1] * cos_t - v[0] * sin_t;                // Cl
            out[t.shapes + s] = v[0] * cos_t + v[1] * sin_t;     // Cd
            out[2 * t.shapes + s] = v[2];
        }
        __syncthreads();
    }
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

int flux_blocks(int n) { return nblk(n, TILE); }

namespace {
int sm_count() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}
}  // namespace

// Split of a flux pass for `tiles` scheduled tiles (`per_sm` resident blocks).
// Up to two tiles a resident block, the block's warps share the tile (a round
// each): FP64 11.4 us against 16.4 at 4,000 points; an iteration at 10,000 points
// 60.2 against 65.8, 16,000 70.4 / 71.6, 18,500 73.4 / 73.5, 24,000 93.9 / 88.8;
// FP32 at 12,000 47.9 / 50.1, 20,000 55.0 / 57.2, 24,000 67.3 / 62.2.
// Beyond that a warp takes chunks of one tile or, for less idle lanes in the
// updates (1.15 times the rate), of two, whichever its whole number of turns
// makes cheaper: FP64, one against two tiles, 45.8 / 52.2 us at 91,000
// points, 38.6 / 37.6 at 64,000, 112 / 105 at 256,000, 417 / 389 at 1,024,000.
FluxShape flux_shape(int tiles, int per_sm) {
    const int blocks = sm_count() * per_sm, warps = blocks * FLUX_WARPS;
    if (tiles <= 2 * blocks) return FluxShape{1, 1};
    const double one = 1.15 * nblk(tiles, warps), two = 2.0 * nblk(tiles, 2 * warps);
    return FluxShape{one < two ? 1 : 2, 0};
}

// The D and I passes by slots (kb_grad_s, kb_inner_s, and FP32) while their
// blocks are one wave, nine an SM: beyond it the halo form's fewer loads win
// (an iteration with one inner iteration on 148 SMs, by slots / halos: FP64
// 20,000 points 101.6 / 108.3 us, 24,000 112.4 / 109.4; FP32 20,000 points
// 70.4 / 79.5, 24,000 76.4 / 77.6, 32,000 86.7 / 86.7).
bool slot_passes(int n) { return nblk(n, SLOT_PTS) <= 9 * sm_count(); }

// The wide halo forms for a grid with `over` tiles of more than HALO_CAP rows.
// They cost every tile a block an SM (and the D pass its fixed stride); a tile
// gathered directly costs its warp a longer chain, which sets the pass's time while
// a warp has few chunks.  An iteration with one inner iteration on 148 SMs, wide /
// narrow with the large tiles gathered, by the share of large tiles:
//   points   precision  one tile    0.1%         0.5%         1%           2%
//    90,000  FP64   us  263 / 276   260 / 275    277 / 284    278 / 285    302 / 309
//   256,000  FP64       583 / 587   608 / 603    623 / 631    642 / 663    656 / 685
//   256,000  FP32       349 / 340   349 / 351    365 / 377    366 / 383    360 / 379
//   520,000  FP64      1201 / 1165 1260 / 1280  1269 / 1283  1289 / 1315  1313 / 1386
//   520,000  FP32       651 / 640   670 / 666    667 / 663    671 / 689    679 / 700
//   700,000  FP64      1575 / 1519 1638 / 1578  1680 / 1669  1691 / 1679  1721 / 1759
//   700,000  FP32       865 / 836   871 / 859    883 / 900    889 / 901    902 / 942
//  1,024,000 FP64      2253 / 2174 2327 / 2221       -       2407 / 2385  2439 / 2423
//  1,024,000 FP32      1253 / 1216 1250 / 1252       -       1274 / 1294  1279 / 1332
//  4,096,000 FP64      8804 / 8504 9140 / 8617       -       9308 / 9014  9463 / 9289
//  4,096,000 FP32      4723 / 4556 4738 / 4599       -       4788 / 4743  4834 / 4869
// Hence: from 200 tiles an SM on (five chunks a resident warp), narrow up to a
// share of 0.5%.
bool wide_halos_pay(int tiles, int over) { return tiles < 200 * sm_count() || 200LL * over > tiles; }

// flux-pass blocks that give every chunk its warp (or its block)
int flux_grid_blocks(int n, bool fp32) {
    const int tiles = nblk(n, TILE);
    const FluxShape f = flux_shape(tiles, fp32 ? flux32_per_sm() : FLUX_MIN_BLOCKS);
    return nblk(nblk(tiles, f.ct), f.coop ? 1 : FLUX_WARPS);
}

void launch_flux_coef(const Geom &g, int base, int n, int nw, int no, double power, double *fco,
                      double *wsl, double *fcg, double *minv, cudaStream_t st) {
    k_flux_coef<<<nblk(n, GRAD_BLOCK), GRAD_BLOCK, 0, st>>>(g, base, n, nw, no, power, fco, wsl,
                                                            fcg, minv);
}

// staging memory of a block of the halo kernels: two tiles a warp
size_t halo_smem_bytes(int kind, int hc) {
    return kind == 0 ? halo_bytes(HALO_BLOCK / 32, HA_D, std::max(hc, HALO_CAP + 1))
                     : halo_bytes(HALO_BLOCK / 32, HA_I, hc);
}

cudaError_t init_kernels() {
    cudaError_t e = cudaSuccess;
    auto room = [&](auto *kernel, int kind, int cap) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)halo_smem_bytes(kind, cap + 1));
    };
    room(kb_grad_h<HALO_CAP>, 0, HALO_CAP);
    room(kb_grad_h<HALO_CAP_WIDE>, 0, HALO_CAP_WIDE);
    room(kb_inner_h<HALO_CAP>, 1, HALO_CAP);
    room(kb_inner_h<HALO_CAP_WIDE>, 1, HALO_CAP_WIDE);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kb_flux<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 FLUX_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kb_flux<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 FLUX_SMEM);
    return e;
}

int wave_blocks(int dev, int kind, int block, size_t smem, bool fp32) {
    // the D and I passes: their own staging memory (the halo kernels' at the
    // largest stride; the FP32 I pass none)
    if (kind == 0 || kind == 1) smem = 0;
    int sms = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1) * std::max(1, batch_occupancy(kind, fp32, block, smem));
}

namespace {
// grid of a launch: `grid` blocks, or one wave of resident blocks (grid == 0)
int wave(int kind, int block, size_t smem, int grid) {
    if (grid > 0) return grid;
    int dev = 0;
    cudaGetDevice(&dev);
    return wave_blocks(dev, kind, block, smem, false);
}
}  // namespace

// the flux pass's shared memory does not depend on the stencil size
size_t flux_smem_bytes(int) { return FLUX_SMEM; }

int batch_occupancy(int kind, bool fp32, int block, size_t smem) {
    if (fp32) return batch_occupancy32(kind, block, smem);
    int nb = 0;
    cudaError_t e = cudaErrorInvalidValue;
    // the D and I passes: their tile-halo kernels (blocks of HALO_BLOCK
    // threads, the largest staging stride), which every grid with halos runs
    if (kind == 0)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_grad_h<HALO_CAP>, HALO_BLOCK,
                                                          halo_smem_bytes(0, HALO_CAP + 1));
    else if (kind == 1)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_inner_h<HALO_CAP>, HALO_BLOCK,
                                                          halo_smem_bytes(1, HALO_CAP + 1));
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_flux<false>, block, smem);
    return e == cudaSuccess ? nb : 1;
}

// blocks of a halo kernel (kind 0: D pass, 1: I pass): `grid`, but no more than
// one wave of the wide forms, or one wave (grid == 0)
int halo_grid(int kind, const Geom &g, int grid) {
    const bool wide = wide_halos(g);
    if (grid > 0 && !wide) return grid;
    const size_t smem = halo_smem_bytes(kind, g.hc);
    int nb = 0;
    auto ask = [&](auto *kernel) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, HALO_BLOCK, smem);
    };
    const cudaError_t e =
        kind == 0 ? (wide ? ask(kb_grad_h<HALO_CAP_WIDE>) : ask(kb_grad_h<HALO_CAP>))
                  : (wide ? ask(kb_inner_h<HALO_CAP_WIDE>) : ask(kb_inner_h<HALO_CAP>));
    const int wave = sm_count() * std::max(1, e == cudaSuccess ? nb : 1);
    return grid > 0 ? std::min(grid, wave) : wave;
}

void launch_grad(const Geom &g, const Consts &c, const Sched &s, const R4 *q, const double *spd,
                 double *dq, double *qm, double *delta, bool with_delta, int block, int grid,
                 cudaStream_t st) {
    (void)block;  // the halo kernels' blocks are HALO_BLOCK threads
    if (slot_passes(g.n)) {
        kb_grad_s<<<nblk(g.n, SLOT_PTS), SLOT_BLOCK, 0, st>>>(g, c, s, q, spd, dq, qm, delta,
                                                              with_delta ? 1 : 0);
        return;
    }
    auto *kernel = wide_halos(g) ? kb_grad_h<HALO_CAP_WIDE> : kb_grad_h<HALO_CAP>;
    kernel<<<halo_grid(0, g, grid), HALO_BLOCK, halo_smem_bytes(0, g.hc), st>>>(
        g, c, s, q, spd, dq, qm, delta, with_delta ? 1 : 0);
}

void launch_inner(const Geom &g, const Consts &c, const Sched &s, const double *dq0,
                  const double *dq_in, double *dq_out, int block, int grid, cudaStream_t st) {
    (void)block;
    (void)c;
    if (slot_passes(g.n)) {
        kb_inner_s<<<nblk(g.n, SLOT_PTS), SLOT_BLOCK, 0, st>>>(g, s, dq0, dq_in, dq_out);
        return;
    }
    auto *kernel = wide_halos(g) ? kb_inner_h<HALO_CAP_WIDE> : kb_inner_h<HALO_CAP>;
    kernel<<<halo_grid(1, g, grid), HALO_BLOCK, halo_smem_bytes(1, g.hc), st>>>(
        g, s, dq0, dq_in, dq_out);
}

void launch_flux(const Geom &g, const Consts &c, const Sched &s, const StageBufs &b, int rk,
                 bool last, int grid, int tiles, cudaStream_t st) {
    const FluxShape f = flux_shape(tiles, FLUX_MIN_BLOCKS);
    const int gr = wave(2, FLUX_BLOCK, FLUX_SMEM, grid);
    constexpr int sm = FLUX_SMEM;
    if (b.kstape)
        kb_flux<true><<<gr, FLUX_BLOCK, sm, st>>>(g, c, s, b, rk, last ? 1 : 0, f.ct, f.coop);
    else kb_flux<false><<<gr, FLUX_BLOCK, sm, st>>>(g, c, s, b, rk, last ? 1 : 0, f.ct, f.coop);
}

void launch_residual(const InstInfo *inst, int n_inst, const double *res_part, Ctl *ctl,
                     double *hist, int hist_ld, const BatchRun *run, int *sched,
                     cudaStream_t st) {
    kb_residual<<<n_inst, RES_BLOCK, 0, st>>>(inst, n_inst, res_part, ctl, hist, hist_ld, run, sched);
}

void launch_init_state(const Geom &g, const R4 *prim, R4 *q, double *spd, cudaStream_t s) {
    k_init_state<<<nblk(g.n, GRAD_BLOCK), GRAD_BLOCK, 0, s>>>(g, prim, q, spd, 0, g.n);
}

void launch_init_rows(const Geom &g, const R4 *prim, R4 *q, double *spd, int i0, int i1,
                      cudaStream_t s) {
    if (i1 > i0)
        k_init_state<<<nblk(i1 - i0, GRAD_BLOCK), GRAD_BLOCK, 0, s>>>(g, prim, q, spd, i0, i1);
}

void launch_sum_parts(const double *part, int nparts, double *out, cudaStream_t s) {
    k_sum_parts<<<1, RES_BLOCK, 0, s>>>(part, nparts, out);
}

void launch_forces(const ShapeTab &t, const R4 *prim, double mach, double cos_t, double sin_t,
                   double *out, cudaStream_t s) {
    k_forces<<<1, FORCE_BLOCK, 0, s>>>(t, prim, mach, cos_t, sin_t, out);
}

}  // namespace lskum
