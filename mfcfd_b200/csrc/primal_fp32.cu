// FP32-mixed kernels of the LSKUM pseudo-time loop on sm_100a.
//
// Stored per point in FP32: prim, q, dq, qm (half the FP64 gather traffic).
// Computed in FP32: the q-derivative sums of the D and I passes, the
// per-neighbour work of the flux pass -- limiter, qtilde -> kinetic state,
// Maxwellian moments and split fluxes.  The 2x2 least-squares normal
// matrices, ill-conditioned on stretched near-wall stencils, are pure
// geometry: they are formed and inverted once per grid in FP64 (Geom32) and
// only applied per iteration.  Kept in FP64: the sums of the flux
// contributions and the flux residual, the arithmetic of the state update,
// the local time step, the residual norm and the force coefficients.
#include <cuda_runtime.h>

#include <algorithm>

#include "batch.cuh"
#include "flux_tile.cuh"
#include "halo.cuh"
#include "primal.h"

namespace lskum {

namespace {

constexpr int GRAD_BLOCK = 256;
constexpr double OBT = 1.0 / 3.0;
constexpr double TBT = 2.0 / 3.0;

// A 32-byte row (dq or qm of one point) in one 256-bit read-only load
// (ld.global.nc.v8.f32, sm_100); the rows are 32-byte aligned.
__device__ __forceinline__ void ldf8w(const float *p, float a[4], float b[4]) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(b[0]), "=f"(b[1]), "=f"(b[2]),
          "=f"(b[3])
        : "l"(p));
}

// A 32-byte row in one 256-bit store (st.global.v8.f32, sm_100).
__device__ __forceinline__ void stf8w(float *p, const float a[4], const float b[4]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p),
                 "f"(a[0]), "f"(a[1]), "f"(a[2]), "f"(a[3]), "f"(b[0]), "f"(b[1]), "f"(b[2]),
                 "f"(b[3])
                 : "memory");
}

// eval_q_inner_loop + eval_update_innerloop (q_variables.F90:115-227) with
// FP32 sums, rearranged.  The reference's new derivative is
//   L sum_k w d (qt_k - qt_i),  qt = q - (d . dq)/2,  L = M^-1,  M = sum_k w d d^T
// (d = x_k - x_i).  q is fixed within a stage, so it splits into
//   dq0 + dq_i/2 - L sum_k w d (d . dq_k) / 2,
// where dq0 = L sum_k w d (q_k - q_i) is the D pass's result of this stage
// and L M = I turns the point's own term into dq_i/2.  Equal in exact
// arithmetic; only the neighbours' derivatives are gathered (no q).
// One slot at a time, as the compiler unrolls it: asking for four slots' loads
// together is 1 - 3% slower (8 slots / 20 slots a point, an iteration with three
// inner iterations: 90,000 points 168 / 306 us, 170 / 313 with four together;
// 256,000 402 / 861, 408 / 874; a pass at 1.024M points 49.7 / 89.1, 51.5 / 94.0).
__device__ __forceinline__ void
inner32_point(const Geom &g, const Geom32 &f, const float *__restrict__ dq0,
              const float *__restrict__ dq_in, float *__restrict__ dq_out, int i) {
    float tx[4] = {0.f, 0.f, 0.f, 0.f}, ty[4] = {0.f, 0.f, 0.f, 0.f};
    const int nb = g.nbhs[i];
    for (int r = 0; r < nb; ++r) {
        const int k = g.conn[(size_t)r * g.n + i];
        const float2 d = __ldg(f.dxy + (size_t)r * g.n + i);
        const float w = f.w ? __ldg(f.w + (size_t)r * g.n + i) : 1.0f;
        float dxk[4], dyk[4];
        ldf8w(dq_in + 8 * (size_t)k, dxk, dyk);
        const float wdx = w * d.x, wdy = w * d.y;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const float pk = fmaf(d.x, dxk[m], d.y * dyk[m]);
            tx[m] = fmaf(wdx, pk, tx[m]);
            ty[m] = fmaf(wdy, pk, ty[m]);
        }
    }
    float dxi[4], dyi[4], dx0[4], dy0[4];
    ldf8w(dq_in + 8 * (size_t)i, dxi, dyi);
    ldf8w(dq0 + 8 * (size_t)i, dx0, dy0);
    const float4 L = __ldg(f.lsq + i);
    float dx[4], dy[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        dx[m] = fmaf(-0.5f, fmaf(L.x, tx[m], L.y * ty[m]), fmaf(0.5f, dxi[m], dx0[m]));
        dy[m] = fmaf(-0.5f, fmaf(L.y, tx[m], L.z * ty[m]), fmaf(0.5f, dyi[m], dy0[m]));
    }
    stf8w(dq_out + 8 * (size_t)i, dx, dy);
}

__global__ void __launch_bounds__(GRAD_BLOCK)
kb_inner32(Geom g, Geom32 f, Sched s, const float *__restrict__ dq0,
           const float *__restrict__ dq_in, float *__restrict__ dq_out) {
    __shared__ SchedSmem ss;
    int live;
    const int total = sched_begin(s, ss, live) * TILE;
    for (int vp = blockIdx.x * blockDim.x + threadIdx.x; vp < total;
         vp += gridDim.x * blockDim.x) {
        const int i = sched_point(s, ss, vp);
        if (i >= 0 && live) inner32_point(g, f, dq0, dq_in, dq_out, i);
    }
}

// The D pass with tile halos (halo.cuh).  The per-slot FP32 offsets come
// from the staged FP64 (x, y) rows, rounded as the host rounds the offsets
// it stores ((float)(x_k - x_i)), so the halo and the stored-offset forms
// see the same offsets.  Row sources: GlobalRows32 reads the stored offsets
// and the rows from global memory (tiles without a staged halo); HaloRows32
// reads the staged q (float4), (x, y) and spd.  (The I pass keeps its direct
// 256-bit gathers of the 32-byte dq rows: a halo I pass staging (x, y) and dq
// measured slower, 0.057 against 0.050 ms per C2 launch, and so did one
// staging only (x, y) and the row indices, 0.064 ms.)
constexpr int HALO32_BLOCK = 128;
constexpr int HA32 = 3;  // staged arrays
// 64 registers and 8 blocks an SM: 52.1 us at 1.024M points (54.1 at 7, 56.2 at
// 6, 59.8 at 9, which spills); 55.6 with the slot loop not unrolled
constexpr int HALO32_MIN_BLOCKS = 8;

struct GlobalRows32 {
    const Geom &g;
    const Geom32 &f;
    const float4 *q;
    const double *spd;
    int i;
    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ int self() const { return i; }
    __device__ __forceinline__ unsigned long long word(int) const { return 0ull; }
    __device__ __forceinline__ int nbr(int r, unsigned long long, int) const {
        return g.conn[(size_t)r * g.n + i];
    }
    __device__ __forceinline__ float2 off(int r, int) const {
        return __ldg(f.dxy + (size_t)r * g.n + i);
    }
    __device__ __forceinline__ float4 qrow(int k) const { return __ldg(q + k); }
    __device__ __forceinline__ double spdv(int k) const { return spd[k]; }
};

// staged arrays: q 0, (x, y) 1, spd 2
struct HaloRows32 {
    static constexpr int OQ = 0, OXY = 1, OSPD = 2;
    const double2 *sm;
    int hc;  // the grid's staging stride
    HaloLoc loc;
    double2 pi;
    __device__ __forceinline__ HaloRows32(const Geom &g, const double2 *sm_, int i)
        : sm(sm_), hc(g.hc), loc(g, i), pi(make_double2(0.0, 0.0)) {}
    __device__ __forceinline__ void begin() { pi = sm[OXY * hc + loc.own]; }
    __device__ __forceinline__ int self() const { return loc.own; }
    __device__ __forceinline__ unsigned long long word(int r0) const { return loc.word(r0); }
    // slot r0 + j of word(r0)
    __device__ __forceinline__ int nbr(int, unsigned long long w, int j) const {
        return (int)((w >> (8 * j)) & 0xffull);
    }
    __device__ __forceinline__ float2 off(int, int l) const {
        const double2 pk = sm[OXY * hc + l];
        return make_float2((float)(pk.x - pi.x), (float)(pk.y - pi.y));
    }
    __device__ __forceinline__ float4 qrow(int l) const {
        return *reinterpret_cast<const float4 *>(sm + OQ * hc + l);
    }
    __device__ __forceinline__ double spdv(int l) const { return sm[OSPD * hc + l].x; }
};

// q_variables.F90:41-112 eval_q_derivatives and state_update.F90:190-236
// func_delta over the rows of R, in slot order, with FP32 sums (the FP64 pass's
// grad_sums)
template <class Rows>
__device__ __forceinline__ void grad32_sums(const Consts &c, const Geom32 &f, int n, Rows R,
                                            int nb, int with_delta, int i, float dx[4],
                                            float dy[4], float qmax[4], float qmin[4],
                                            double &min_delt) {
    R.begin();
    const float4 qv = R.qrow(R.self());
    const float qi[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) qmax[m] = qmin[m] = qi[m];
    float sx[4] = {0.f, 0.f, 0.f, 0.f}, sy[4] = {0.f, 0.f, 0.f, 0.f};
    min_delt = 1.0;
    for (int r0 = 0; r0 < nb; r0 += 8) {
        const unsigned long long word = R.word(r0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = r0 + j;
            if (r >= nb) break;
            const int k = R.nbr(r, word, j);
            const float4 kv = R.qrow(k);
            const float2 gs = R.off(r, k);
            const float qk[4] = {kv.x, kv.y, kv.z, kv.w};
            const float w = f.w ? __ldg(f.w + (size_t)r * n + i) : 1.0f;
#pragma unroll
            for (int mm = 0; mm < 4; ++mm) {
                if (qk[mm] > qmax[mm]) qmax[mm] = qk[mm];
                if (qk[mm] < qmin[mm]) qmin[mm] = qk[mm];
            }
            const float wdx = w * gs.x, wdy = w * gs.y;
#pragma unroll
            for (int mm = 0; mm < 4; ++mm) {
                const float dqm = qk[mm] - qi[mm];
                sx[mm] = fmaf(wdx, dqm, sx[mm]);
                sy[mm] = fmaf(wdy, dqm, sy[mm]);
            }
            if (with_delta) {
                const double dist = (double)sqrtf(fmaf(gs.x, gs.x, gs.y * gs.y));
                double delta_t = dist / R.spdv(k);
                delta_t = c.cfl * delta_t;
                if (min_delt > delta_t) min_delt = delta_t;
            }
        }
    }
    const float4 L = __ldg(f.lsq + i);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        dx[m] = fmaf(L.x, sx[m], L.y * sy[m]);
        dy[m] = fmaf(L.y, sx[m], L.z * sy[m]);
    }
}

template <int CAP>
__global__ void __launch_bounds__(HALO32_BLOCK, HALO32_MIN_BLOCKS)
kb_grad32_h(Geom g, Consts c, Geom32 f, Sched s, const float4 *__restrict__ q,
            const double *__restrict__ spd, float *__restrict__ dq, float *__restrict__ qm,
            double *__restrict__ delta, int with_delta) {
    extern __shared__ double2 hsm[];
    __shared__ SchedSmem ss;
    int live;
    const int ntiles = sched_begin(s, ss, live);
    const int wpb = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int half = lane / TILE, stride = gridDim.x * wpb;
    using H = HaloRows32;
    double2 *sm0 = hsm + (2 * warp) * HA32 * g.hc, *sm1 = sm0 + HA32 * g.hc;
    HaloChunk<CAP> cur;
    for (int ch = blockIdx.x * wpb + warp; 2 * ch < ntiles; ch += stride) {
        halo_chunk(g, s, ss, ntiles, ch, lane, cur);
        if (!live) return;
        stage_array<1>(q, 16, cur.x, lane, sm0, sm1, g.hc, H::OQ);
        stage_array<1>(g.xy, 16, cur.x, lane, sm0, sm1, g.hc, H::OXY);
        if (with_delta) stage_array8(spd, cur.x, lane, sm0, sm1, g.hc, H::OSPD);
        const H hr(g, half ? sm1 : sm0, cur.hn > 0 ? cur.i : -1);
        halo_wait();
        __syncwarp();
        if (cur.i >= 0) {
            float dx[4], dy[4], qmax[4], qmin[4];
            double min_delt;
            if (cur.hn > 0)
                grad32_sums(c, f, g.n, hr, cur.nb, with_delta, cur.i, dx, dy, qmax, qmin,
                            min_delt);
            else
                grad32_sums(c, f, g.n, GlobalRows32{g, f, q, spd, cur.i}, cur.nb,
                            with_delta, cur.i, dx, dy, qmax, qmin, min_delt);
            stf8w(dq + 8 * (size_t)cur.i, dx, dy);
            stf8w(qm + 8 * (size_t)cur.i, qmax, qmin);
            if (with_delta) delta[cur.i] = min_delt;
        }
        __syncwarp();
    }
}

// The D and I passes of a small grid by slots, as kb_grad_s and kb_inner_s of
// the FP64 passes: the other forms' operations, in their order.  An iteration
// at 1,536 points, one inner iteration: 55.0 -> 41.8 us; 16,000: 76.7 -> 65.5.
__global__ void __launch_bounds__(SLOT_BLOCK)
kb_grad32_s(Geom g, Consts c, Geom32 f, Sched s, const float4 *__restrict__ q,
            const double *__restrict__ spd, float *__restrict__ dq, float *__restrict__ qm,
            double *__restrict__ delta, int with_delta) {
    __shared__ SchedSmem ss;
    __shared__ float sm[SLOT_PTS * SLOT_P];
    int live;
    const int total = sched_begin(s, ss, live) * TILE;
    const int p = threadIdx.x / LPP, l = threadIdx.x % LPP, m = l & 3;
    float *row = sm + p * SLOT_P;  // fields qk[4], w dx, w dy
    for (int v0 = blockIdx.x * SLOT_PTS; v0 < total; v0 += gridDim.x * SLOT_PTS) {
        const int i = slot_point(s, ss, total, v0 + p);
        int nb = 0, k = 0;
        float qi = 0.f;
        float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= 0) {
            nb = __ldg(g.nbhs + i);
            if (l < g.kp) k = __ldg(g.conn + (size_t)l * g.n + i);
            qi = __ldg(reinterpret_cast<const float *>(q + i) + m);
            L = __ldg(f.lsq + i);
        }
        if (!live) return;
        float sum = 0.f, ext = qi;
        double dmin = 1.0;
        const int nbw = __reduce_max_sync(0xffffffffu, nb);
        for (int r0 = 0; r0 < nbw; r0 += LPP) {
            const int r = r0 + l;
            if (r0 > 0 && r < nb) k = __ldg(g.conn + (size_t)r * g.n + i);
            if (r < nb) {
                const float4 qk = __ldg(q + k);
                const float2 gs = __ldg(f.dxy + (size_t)r * g.n + i);
                const float w = f.w ? __ldg(f.w + (size_t)r * g.n + i) : 1.0f;
                row[l] = qk.x;
                row[SLOT_F + l] = qk.y;
                row[2 * SLOT_F + l] = qk.z;
                row[3 * SLOT_F + l] = qk.w;
                row[4 * SLOT_F + l] = w * gs.x;
                row[5 * SLOT_F + l] = w * gs.y;
                if (with_delta) {
                    const double dist = (double)sqrtf(fmaf(gs.x, gs.x, gs.y * gs.y));
                    double delta_t = dist / spd[k];
                    delta_t = c.cfl * delta_t;
                    if (dmin > delta_t) dmin = delta_t;
                }
            }
            __syncwarp();
            const float *qf = row + m * SLOT_F, *wf = row + (4 + l / 4) * SLOT_F;
#pragma unroll
            for (int j = 0; j < LPP; ++j) {
                if (r0 + j >= nb) break;
                const float qk = qf[j], wd = wf[j];
                if (l < 4 ? qk > ext : qk < ext) ext = qk;
                sum = fmaf(wd, qk - qi, sum);
            }
            __syncwarp();
        }
        // lanes 0-3 hold sx and qmax, 4-7 sy and qmin
        const float other = __shfl_xor_sync(0xffffffffu, sum, 4);
        if (with_delta) {
#pragma unroll
            for (int o = 4; o; o >>= 1) {
                const double d = __shfl_xor_sync(0xffffffffu, dmin, o);
                if (dmin > d) dmin = d;
            }
        }
        if (i >= 0) {
            dq[8 * (size_t)i + l] =
                l < 4 ? fmaf(L.x, sum, L.y * other) : fmaf(L.y, other, L.z * sum);
            qm[8 * (size_t)i + l] = ext;
            if (with_delta && l == 0) delta[i] = dmin;
        }
    }
}

__global__ void __launch_bounds__(SLOT_BLOCK)
kb_inner32_s(Geom g, Geom32 f, Sched s, const float *__restrict__ dq0,
             const float *__restrict__ dq_in, float *__restrict__ dq_out) {
    __shared__ SchedSmem ss;
    __shared__ float sm[SLOT_PTS * SLOT_P];
    int live;
    const int total = sched_begin(s, ss, live) * TILE;
    const int p = threadIdx.x / LPP, l = threadIdx.x % LPP, m = l & 3;
    float *row = sm + p * SLOT_P;  // fields d . dq_k [4], w dx, w dy
    for (int v0 = blockIdx.x * SLOT_PTS; v0 < total; v0 += gridDim.x * SLOT_PTS) {
        const int i = slot_point(s, ss, total, v0 + p);
        int nb = 0, k = 0;
        float a0 = 0.f, di = 0.f;
        float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= 0) {
            nb = __ldg(g.nbhs + i);
            if (l < g.kp) k = __ldg(g.conn + (size_t)l * g.n + i);
            a0 = __ldg(dq0 + 8 * (size_t)i + l);
            di = __ldg(dq_in + 8 * (size_t)i + l);
            L = __ldg(f.lsq + i);
        }
        if (!live) return;
        float sum = 0.f;
        const int nbw = __reduce_max_sync(0xffffffffu, nb);
        for (int r0 = 0; r0 < nbw; r0 += LPP) {
            const int r = r0 + l;
            if (r0 > 0 && r < nb) k = __ldg(g.conn + (size_t)r * g.n + i);
            if (r < nb) {
                const float2 d = __ldg(f.dxy + (size_t)r * g.n + i);
                const float w = f.w ? __ldg(f.w + (size_t)r * g.n + i) : 1.0f;
                float dxk[4], dyk[4];
                ldf8w(dq_in + 8 * (size_t)k, dxk, dyk);
#pragma unroll
                for (int t = 0; t < 4; ++t) row[t * SLOT_F + l] = fmaf(d.x, dxk[t], d.y * dyk[t]);
                row[4 * SLOT_F + l] = w * d.x;
                row[5 * SLOT_F + l] = w * d.y;
            }
            __syncwarp();
            const float *tf = row + m * SLOT_F, *wf = row + (4 + l / 4) * SLOT_F;
#pragma unroll
            for (int j = 0; j < LPP; ++j) {
                if (r0 + j >= nb) break;
                sum = fmaf(wf[j], tf[j], sum);
            }
            __syncwarp();
        }
        const float other = __shfl_xor_sync(0xffffffffu, sum, 4);
        const float Ls = l < 4 ? fmaf(L.x, sum, L.y * other) : fmaf(L.y, other, L.z * sum);
        if (i >= 0) dq_out[8 * (size_t)i + l] = fmaf(-0.5f, Ls, fmaf(0.5f, di, a0));
    }
}

// ---------------------------------------------------------------------------
// F pass.
//
// Pairs of FP32 values in one 64-bit register pair: sm_100 adds, multiplies
// and fuses both in one instruction (f32x2), and this pass is bound by the
// instructions it issues.  The limiter works on pairs of components, the
// kinetic states and split fluxes on the pair of directions (t, n).
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float lo(F2 a) {
    float x;
    [[maybe_unused]] float y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return x;
}
__device__ __forceinline__ float hi(F2 a) {
    float y;
    [[maybe_unused]] float x;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
    return y;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ float rcpf(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqf(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// venkat_limiter and the limited qtilde of two components (limiters.F90:64-110),
// mt = -(d . dq): del_neg is mt/2, and its factor common to the quotient's
// numerator and denominator is cancelled.
__device__ __forceinline__ F2 limited2(F2 mt, F2 q, F2 qmax, F2 qmin, F2 eps2) {
    const F2 dn = mt * f2(0.5f);
    const F2 dp = f2(lo(mt) > 0.f ? lo(qmax) : lo(qmin), hi(mt) > 0.f ? hi(qmax) : hi(qmin)) - q;
    const F2 a = fma2(dp, dp, eps2);
    const F2 num = fma2(mt, dp, a), den = fma2(dn, dp + mt, a);
    const F2 f = num * f2(rcpf(lo(den)), rcpf(hi(den)));
    constexpr float thr = (float)MFCFD_VENKAT_THR;
    const F2 phi = f2(fabsf(lo(dn)) <= thr ? 1.0f : fminf(lo(f), 1.0f),
                      fabsf(hi(dn)) <= thr ? 1.0f : fminf(hi(f), 1.0f));
    return fma2(phi, dn, q);
}

// A row of the stage's arrays: staged (row l of the halo) or from global memory.
struct Row32 {
    F2 q[2], dx[2], dy[2], qmax[2], qmin[2];
    float eps2;
    __device__ __forceinline__ void qtilde(F2 mdx, F2 mdy, F2 qt[2]) const {
        const F2 e = f2(eps2);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            qt[h] = limited2(fma2(mdx, dx[h], mdy * dy[h]), q[h], qmax[h], qmin[h], e);
    }
};

// Kinetic state of a limited reconstruction (kstate_pre's forms): the
// velocity in the point's frame, Maxwellian half-moments and erf as (t, n)
// pairs.  erf from the exponential the moments take anyway (erf_with_exp).
struct KState2 {
    F2 U, B, e;
    float rho, pbr, usq;
};
__device__ __forceinline__ KState2 kstate2(const F2 qt[2], float nx, float ny, float inv_sqrt_pi) {
    constexpr float log2e = 1.44269504088896340736f;
    KState2 s;
    const float nq = -hi(qt[1]), beta = 0.5f * nq;
    s.pbr = rcpf(nq);
    const float u1 = hi(qt[0]) * s.pbr, u2 = lo(qt[1]) * s.pbr;
    s.usq = u1 * u1 + u2 * u2;
    const float texp = lo(qt[0]) + beta * s.usq;
    const float rb = rsqf(beta), sb = beta * rb;
    s.rho = ex2f(texp * log2e) * ((4.0f * s.pbr * s.pbr) * rb);
    s.U = fma2(f2(u1), f2(ny, nx), f2(u2) * f2(-nx, ny));
    const F2 S = s.U * f2(sb);
    const F2 x = (S * S) * f2(-log2e);
    const F2 E = f2(ex2f(lo(x)), ex2f(hi(x)));
    s.B = E * f2(s.pbr * sb * inv_sqrt_pi);
    const F2 d = fma2(f2(fabsf(lo(S)), fabsf(hi(S))), f2(0.3275911f), f2(1.0f));
    const F2 t = f2(rcpf(lo(d)), rcpf(hi(d)));
    F2 p = f2(-1.061405429f);
    p = fma2(p, t, f2(1.453152027f));
    p = fma2(p, t, f2(-1.421413741f));
    p = fma2(p, t, f2(0.284496736f));
    p = fma2(p, t, f2(-0.254829592f));
    const F2 r = fma2(p * t, E, f2(1.0f));
    s.e = f2(copysignf(lo(r), lo(S)), copysignf(hi(r), hi(S)));
    return s;
}

// split_fluxes.F90 along t (first of each pair) and along n (second), sg the
// signs of the two lists: mass, momentum along the direction, momentum across
// it, energy (flux_split of the FP64 pass).
__device__ __forceinline__ void flux_split2(const KState2 &s, F2 sg, F2 G[4]) {
    const F2 A = fma2(sg * f2(0.5f), s.e, f2(0.5f));
    const F2 a = fma2(s.U, A, sg * s.B);
    const F2 pA = f2(s.pbr) * A;
    const float w6 = 6.0f * s.pbr + s.usq;
    G[0] = f2(s.rho) * a;
    G[1] = f2(s.rho) * fma2(s.U, a, pA);
    G[2] = f2(hi(s.U), lo(s.U)) * G[0];
    G[3] = f2(0.5f * s.rho) * fma2(f2(w6), a, s.U * pA);
}

__device__ __forceinline__ KStateT<float> kstate_plain(const KState2 &s) {
    KStateT<float> k;
    k.rho = s.rho; k.ut = lo(s.U); k.un = hi(s.U); k.pbr = s.pbr; k.usq = s.usq;
    k.B1 = lo(s.B); k.B2 = hi(s.B); k.e1 = lo(s.e); k.e2 = hi(s.e);
    return k;
}

// Shared memory of a unit: the tile's halo rows as one array per 16-byte piece
// (q 0, dq 1-2, qm 3-4, (x, y) 5) and the limiter's eps2, the tile's own
// points and list coefficients, the chunk's flux residuals.
struct Flux32Smem {
    static constexpr int ROWS = HALO_CAP, HC = ROWS + 1;
    double2 halo[6][HC];
    float4 co[TILE][2];
    FluxOwn own;
    double G[CHUNK_MAX][4];  // flux residuals, then residual terms
    float eps[HC + 3];
};
constexpr int FLUX32_SMEM = FLUX_WARPS * sizeof(Flux32Smem);
// 96 registers at 5 blocks: 0.214 ms at 1.024M points; 6 blocks spill (0.258),
// 4 have too few warps (0.223)
constexpr int FLUX32_MIN_BLOCKS = 5;

// cal_flux_residual + state_update + eval_q_variables of the new state with
// the per-neighbour work in FP32: the FP64 pass's split of the work
// (flux_pass) and its pooled list weights; a slot's weighted differences are
// FP32, their sums over the slots FP64.  Bound by issue (64 % of the slots at
// 620 instructions a round, 833 with scalar FP32 arithmetic and per-list
// compensated sums): 0.283 -> 0.214 ms at 1.024M points, 77 -> 65 us at
// 256,000, 26 -> 14 us at 16,000, 26 -> 10 us at 1,536.
//
// The update runs in FP64: its conversions prim -> U -> prim, four times an
// iteration, are what moved an earlier FP32 update away from the FP64 loop
// (640x400 grid, 2,000 iterations from freestream: |dCd| 1.1e-5 with an FP32
// update, 2.2e-7 with an FP64 one), while FP64 reconstruction or fluxes
// changed nothing measurable.
struct Flux32 {
    using Smem = Flux32Smem;
    const Geom &g;
    const Consts &c;
    const StageBufs32 &b;
    int rk, last;

    template <int NT>
    __device__ __forceinline__ void stage(const FluxTile &t, const FluxHalo &x, Smem &m, int tid) {
        stage_rows<1, NT, Smem::HC>(b.q_in, x, m.halo[0], tid);
        stage_rows<2, NT, Smem::HC>(b.dq, x, m.halo[1], tid);
        stage_rows<2, NT, Smem::HC>(b.qm, x, m.halo[3], tid);
        stage_rows<1, NT, Smem::HC>(g.xy, x, m.halo[5], tid);
        if (tid < HALO_CAP) {
#pragma unroll
            for (int u0 = 0; u0 < HALO_CAP; u0 += NT < HALO_CAP ? NT : HALO_CAP) {
                const int k = x.row(u0 + tid);
                if (u0 + tid < x.hn) halo_cp4(&m.eps[u0 + tid], b.eps2f + k);
            }
        }
        if (tid < 2 * t.cnt)
            halo_cp16(&m.co[0][0] + tid, b.f.flsq + 2 * (size_t)t.i0 + tid);
        m.own.stage<NT>(g, t, tid);
    }

    __device__ __forceinline__ void row(const Smem &m, int l, Row32 &o) const {
        const float4 q = *reinterpret_cast<const float4 *>(&m.halo[0][l]);
        const float4 x = *reinterpret_cast<const float4 *>(&m.halo[1][l]);
        const float4 y = *reinterpret_cast<const float4 *>(&m.halo[2][l]);
        const float4 h = *reinterpret_cast<const float4 *>(&m.halo[3][l]);
        const float4 w = *reinterpret_cast<const float4 *>(&m.halo[4][l]);
        o.q[0] = f2(q.x, q.y); o.q[1] = f2(q.z, q.w);
        o.dx[0] = f2(x.x, x.y); o.dx[1] = f2(x.z, x.w);
        o.dy[0] = f2(y.x, y.y); o.dy[1] = f2(y.z, y.w);
        o.qmax[0] = f2(h.x, h.y); o.qmax[1] = f2(h.z, h.w);
        o.qmin[0] = f2(w.x, w.y); o.qmin[1] = f2(w.z, w.w);
        o.eps2 = m.eps[l];
    }
    __device__ __forceinline__ void row(int k, Row32 &o) const {
        const float4 q = __ldg(b.q_in + k);
        float x[4], y[4], h[4], w[4];
        ldf8w(b.dq + 8 * (size_t)k, x, y);
        ldf8w(b.qm + 8 * (size_t)k, h, w);
        o.q[0] = f2(q.x, q.y); o.q[1] = f2(q.z, q.w);
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            o.dx[a] = f2(x[2 * a], x[2 * a + 1]);
            o.dy[a] = f2(y[2 * a], y[2 * a + 1]);
            o.qmax[a] = f2(h[2 * a], h[2 * a + 1]);
            o.qmin[a] = f2(w[2 * a], w[2 * a + 1]);
        }
        o.eps2 = b.eps2f[k];
    }

    __device__ __forceinline__ void group(const FluxTile &t, int j, int hn, Smem &m, double *G) {
        const int lane = threadIdx.x % LPP;
        const float inv_sqrt_pi = 0.56418958354775628695f;
        const int kind = t.kind(j), i = t.i0 + j;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        const double2 nn = m.own.nrm[j];
        const float nx = (float)nn.x, ny = (float)nn.y;
        const int nb = j < t.cnt ? m.own.nbhs[j] : 0;
        for (int r = lane; r < nb; r += LPP) {
            KState2 sk, si;
            float dx, dy;
            {
                F2 qk[2], qi[2];
                Row32 o;
                if (hn > 0) {
                    int lk, li;
                    m.own.rows(g, i, j, r, lk, li);
                    const double2 pi_ = m.halo[5][li], pk = m.halo[5][lk];
                    // rounded as the host rounds the offsets it stores
                    dx = (float)(pk.x - pi_.x);
                    dy = (float)(pk.y - pi_.y);
                    const F2 mdx = f2(-dx), mdy = f2(-dy);
                    row(m, lk, o);
                    o.qtilde(mdx, mdy, qk);
                    row(m, li, o);
                    o.qtilde(mdx, mdy, qi);
                } else {
                    const float2 d = __ldg(b.f.dxy + (size_t)r * g.n + i);
                    dx = d.x;
                    dy = d.y;
                    const F2 mdx = f2(-dx), mdy = f2(-dy);
                    row(g.conn[(size_t)r * g.n + i], o);
                    o.qtilde(mdx, mdy, qk);
                    row(i, o);
                    o.qtilde(mdx, mdy, qi);
                }
                sk = kstate2(qk, nx, ny, inv_sqrt_pi);
                si = kstate2(qi, nx, ny, inv_sqrt_pi);
            }
            const float w = b.f.w ? __ldg(b.f.w + (size_t)r * g.n + i) : 1.0f;
            const float dels = (dx * ny - dy * nx) * w, deln = (dx * nx + dy * ny) * w;
            // Per direction the neighbour is in one list of the pair, in both
            // only when its projection is exactly 0: the second list is added
            // then.
            const uint4 mm = m.own.mask[j];
            const float2 *co = reinterpret_cast<const float2 *>(m.co[j]);
            auto add = [&](int lx, int ly, bool ux, bool uy) {
                const float2 cx = co[lx], cy = co[2 + ly];
                const float sx = lx ? -1.0f : 1.0f, sy = ly ? -1.0f : 1.0f;
                const float wx = ux ? cx.x * dels + cx.y * deln : 0.0f;
                const float wy = uy ? cy.x * deln + cy.y * dels : 0.0f;
                F2 Gi[4], Gk[4];
                flux_split2(si, f2(sx, sy), Gi);
                flux_split2(sk, f2(sx, sy), Gk);
                // differences along t and along n, as scalars: a pair built in the
                // branch below from its own half came out wrong (ptxas 12.9)
                float X[4], Y[4];
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const F2 D = Gk[d] - Gi[d];
                    X[d] = lo(D);
                    Y[d] = hi(D);
                }
                if (kind != KIND_INTERIOR) {
                    // wall GxII/GxI (A2neg), outer GxIII/GxIV (A2pos)
                    const float s2 = kind == KIND_WALL ? -1.0f : 1.0f;
                    float Qi[4], Qk[4];
                    flux_quad<float>(kstate_plain(si), sx, s2, Qi);
                    flux_quad<float>(kstate_plain(sk), sx, s2, Qk);
#pragma unroll
                    for (int d = 0; d < 4; ++d) X[d] = Qk[d] - Qi[d];
                }
                v[0] += (double)(wx * X[0] + wy * Y[0]);
                v[1] += (double)(wx * X[1] + wy * Y[2]);
                v[2] += (double)(wx * X[2] + wy * Y[1]);
                v[3] += (double)(wx * X[3] + wy * Y[3]);
            };
            const unsigned bit = 1u << r;
            add(mm.x & bit ? 0 : 1, mm.z & bit ? 0 : 1, true, true);
            const bool tx = mm.x & mm.y & bit, ty = mm.z & mm.w & bit;
            if (tx || ty) add(1, 1, tx, ty);
        }
        __syncwarp();
        const double sum = reduce8(v, lane);
        if (!(lane & 1)) G[lane >> 1] = sum;
    }

    // state_update.F90:10-141 of one point from the sum of its list
    // derivatives: FP32 state in and out, FP64 arithmetic; returns its res_sqr
    // term.
    __device__ __forceinline__ double update(int i, int kind, int orow, const double *Gs) {
        const double2 nn = g.nrm[i];
        const double nx = nn.x, ny = nn.y, delta = b.delta[i];
        const float4 Pf = b.prim_in[i], Of = rk == 3 ? b.prim_old[i] : Pf;
        double fr[4];
#pragma unroll
        for (int m = 0; m < 4; ++m)
            fr[m] = (kind == KIND_WALL ? 2.0 * delta : delta) * Gs[m];
        if (b.flux_dbg) st4(reinterpret_cast<R4 *>(b.flux_dbg) + i, fr[0], fr[1], fr[2], fr[3]);
        // the residual from the increment itself, 0.5 euler fr(1), which
        // differences of the stored FP32 state would cancel (last stage: rk != 3)
        const double he = 0.5 * c.euler;
        const double res_sqr = kind != KIND_OUTER ? (he * fr[0]) * (he * fr[0]) : 0.0;
        double U[4], Uo[4] = {0.0, 0.0, 0.0, 0.0};
        if (kind == KIND_OUTER) {
            const double *inf = g.obc + 8 * (size_t)orow;
            conserved_ubar(Pf.x, Pf.y, Pf.z, Pf.w, nx, ny, inf, c.pi, c.gm1, U);
            if (rk == 3) conserved_ubar(Of.x, Of.y, Of.z, Of.w, nx, ny, inf, c.pi, c.gm1, Uo);
        } else {
            prim_to_conserved(Pf.x, Pf.y, Pf.z, Pf.w, nx, ny, U);
            if (rk == 3) prim_to_conserved(Of.x, Of.y, Of.z, Of.w, nx, ny, Uo);
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (rk != 3) U[m] = U[m] - he * fr[m];
            else U[m] = TBT * Uo[m] + OBT * (U[m] - 0.5 * fr[m]);
        }
        if (kind == KIND_WALL) U[2] = 0.0;
        const double U2_rot = U[1], U3_rot = U[2];
        U[1] = U2_rot * ny + U3_rot * nx;
        U[2] = U3_rot * ny - U2_rot * nx;
        const double temp = 1.0 / U[0];
        const float rho = (float)U[0];
        const float u1 = (float)(U[1] * temp);
        const float u2 = (float)(U[2] * temp);
        const float pr = (float)(0.4 * (U[3] - (0.5 * temp) * (U[1] * U[1] + U[2] * U[2])));
        b.prim_out[i] = make_float4(rho, u1, u2, pr);
        float qn[4];
        q_from_prim_t<float>(rho, u1, u2, pr, qn);
        b.q_out[i] = make_float4(qn[0], qn[1], qn[2], qn[3]);
        if (last) b.spd[i] = (double)(sqrtf(u1 * u1 + u2 * u2) + 3.0f * sqrtf(pr / rho));
        return res_sqr;
    }
};

__global__ void __launch_bounds__(FLUX_BLOCK, FLUX32_MIN_BLOCKS)
kb_flux32(Geom g, Consts c, Sched s, StageBufs32 b, int rk, int last, int ct, int coop) {
    extern __shared__ double2 fsm[];
    Flux32 p{g, c, b, rk, last};
    flux_pass(p, g, s, reinterpret_cast<Flux32Smem *>(fsm), b.res_part, last, ct, coop);
}

__global__ void k_init_state32(Geom g, const float4 *__restrict__ prim, float4 *__restrict__ q,
                               double *__restrict__ spd) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    float4 P = prim[i];
    double qn[4];
    q_from_prim((double)P.x, (double)P.y, (double)P.z, (double)P.w, qn);
    q[i] = make_float4((float)qn[0], (float)qn[1], (float)qn[2], (float)qn[3]);
    double u1 = P.y, u2 = P.z, rho = P.x, pr = P.w;
    spd[i] = sqrt(u1 * u1 + u2 * u2) + 3.0 * sqrt(pr / rho);
}

__global__ void k_widen(const float4 *__restrict__ in, R4 *__restrict__ out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = in[i];
    st4(out + i, v.x, v.y, v.z, v.w);
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace


cudaError_t init_kernels32() {
    // within the default 48 KB of dynamic shared memory: nothing to set
    static_assert(FLUX32_SMEM <= 48 * 1024, "");
    return cudaSuccess;
}
int flux32_per_sm() { return FLUX32_MIN_BLOCKS; }

namespace {
// dynamic shared memory of the halo kernels at staging stride hc
size_t halo32_smem(int hc) { return halo_bytes(HALO32_BLOCK / 32, HA32, hc); }
// blocks of the D pass's halo kernel, as halo_grid of the FP64 passes
int halo32_grid(const Geom &g, int grid) {
    const bool wide = wide_halos(g);
    if (grid > 0 && !wide) return grid;
    int dev = 0, sms = 1, nb = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &nb, wide ? kb_grad32_h<HALO_CAP_WIDE> : kb_grad32_h<HALO_CAP>, HALO32_BLOCK,
        halo32_smem(g.hc));
    const int wave = std::max(sms, 1) * std::max(1, e == cudaSuccess ? nb : 1);
    return grid > 0 ? std::min(grid, wave) : wave;
}
}  // namespace

// the flux pass's shared memory does not depend on the stencil size
size_t flux32_smem_bytes(int) { return FLUX32_SMEM; }

int batch_occupancy32(int kind, int block, size_t smem) {
    int nb = 0;
    cudaError_t e = cudaErrorInvalidValue;
    // the D pass: its tile-halo kernel at the largest staging stride, which
    // every grid with halos runs
    if (kind == 0)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_grad32_h<HALO_CAP>, HALO32_BLOCK,
                                                          halo32_smem(HALO_CAP + 1));
    else if (kind == 1)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_inner32, block, smem);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kb_flux32, block, smem);
    return e == cudaSuccess ? nb : 1;
}

namespace {
int wave32(int kind, int block, size_t smem, int grid) {
    if (grid > 0) return grid;
    int dev = 0;
    cudaGetDevice(&dev);
    return wave_blocks(dev, kind, block, smem, true);
}
}  // namespace

void launch_grad32(const Geom &g, const Consts &c, const Geom32 &f, const Sched &s,
                   const float4 *q, const double *spd, float *dq, float *qm, double *delta,
                   bool with_delta, int block, int grid, cudaStream_t st) {
    (void)block;  // the halo kernel's blocks are HALO32_BLOCK threads
    if (slot_passes(g.n)) {
        kb_grad32_s<<<nblk(g.n, SLOT_PTS), SLOT_BLOCK, 0, st>>>(g, c, f, s, q, spd, dq, qm, delta,
                                                                with_delta ? 1 : 0);
        return;
    }
    auto *kernel = wide_halos(g) ? kb_grad32_h<HALO_CAP_WIDE> : kb_grad32_h<HALO_CAP>;
    kernel<<<halo32_grid(g, grid), HALO32_BLOCK, halo32_smem(g.hc), st>>>(
        g, c, f, s, q, spd, dq, qm, delta, with_delta ? 1 : 0);
}

void launch_inner32(const Geom &g, const Consts &c, const Geom32 &f, const Sched &s,
                    const float *dq0, const float *dq_in, float *dq_out, int block, int grid,
                    cudaStream_t st) {
    (void)c;
    if (slot_passes(g.n)) {
        kb_inner32_s<<<nblk(g.n, SLOT_PTS), SLOT_BLOCK, 0, st>>>(g, f, s, dq0, dq_in, dq_out);
        return;
    }
    kb_inner32<<<wave32(1, block, 0, grid), block, 0, st>>>(g, f, s, dq0, dq_in, dq_out);
}

void launch_flux32(const Geom &g, const Consts &c, const Sched &s, const StageBufs32 &b,
                         int rk, bool last, int grid, int tiles, cudaStream_t st) {
    const FluxShape f = flux_shape(tiles, FLUX32_MIN_BLOCKS);
    kb_flux32<<<wave32(2, FLUX_BLOCK, FLUX32_SMEM, grid), FLUX_BLOCK, FLUX32_SMEM, st>>>(
        g, c, s, b, rk, last ? 1 : 0, f.ct, f.coop);
}

void launch_init_state32(const Geom &g, const float4 *prim, float4 *q, double *spd,
                         cudaStream_t s) {
    k_init_state32<<<nblk(g.n, GRAD_BLOCK), GRAD_BLOCK, 0, s>>>(g, prim, q, spd);
}

void launch_widen(const float4 *in, R4 *out, int n, cudaStream_t s) {
    k_widen<<<nblk(n, GRAD_BLOCK), GRAD_BLOCK, 0, s>>>(in, out, n);
}

}  // namespace lskum
