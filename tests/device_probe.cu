// The FP64 flux pass's device functions on arrays, for tests/test_gpu_device_probe.py,
// and a handle's switch that only tests use.
#include "../mfcfd_b200/csrc/handle.h"
#include "../mfcfd_b200/csrc/flux_math.cuh"

namespace {

// out[0..3] of every x: rcp_h3, rsqrt_h3, exp_mid, erf_mid (0 where x is outside a form's
// range)
__global__ void k_forms(int n, const double *x, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    out[4 * i] = rcp_h3(v);
    out[4 * i + 1] = v > 0.0 ? rsqrt_h3(v) : 0.0;
    out[4 * i + 2] = fabs(v) <= EXP_MAX ? exp_mid(v) : 0.0;
    out[4 * i + 3] = fabs(v) <= ERF_MAX ? erf_mid(v, v * v) : 0.0;
}

// qt [n][2][4], normal (nx, ny): the two states of kstate_pair, rho pbr B1 B2 e1 e2 u1 u2 each
__global__ void k_states(int n, const double *qt, double nx, double ny, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    KState s[2];
    double u[2][2];
    kstate_pair(qt + 8 * i, qt + 8 * i + 4, nx, ny, 0.56418958354775628695, s[0], s[1], u[0], u[1]);
    for (int h = 0; h < 2; ++h) {
        const double v[8] = {s[h].rho, s[h].pbr, s[h].B1, s[h].B2,
                             s[h].e1,  s[h].e2,  u[h][0], u[h][1]};
        for (int c = 0; c < 8; ++c) out[16 * i + 8 * h + c] = v[c];
    }
}

// host arrays in and out; launch(device in, device out)
template <class F>
int on_device(const double *in, size_t n_in, double *out, size_t n_out, F launch) {
    double *d_in = nullptr, *d_out = nullptr;
    int bad = 1;
    if (cudaMalloc(&d_in, n_in * sizeof(double)) == cudaSuccess &&
        cudaMalloc(&d_out, n_out * sizeof(double)) == cudaSuccess &&
        cudaMemcpy(d_in, in, n_in * sizeof(double), cudaMemcpyHostToDevice) == cudaSuccess) {
        launch(d_in, d_out);
        bad = cudaGetLastError() != cudaSuccess ||
              cudaMemcpy(out, d_out, n_out * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    }
    cudaFree(d_in);
    cudaFree(d_out);
    return bad;
}

}  // namespace

extern "C" {

int probe_forms(int n, const double *x, double *out) {
    return on_device(x, n, out, 4 * (size_t)n, [&](const double *a, double *b) {
        k_forms<<<(n + 127) / 128, 128>>>(n, a, b);
    });
}

int probe_states(int n, const double *qt, double nx, double ny, double *out) {
    return on_device(qt, 8 * (size_t)n, out, 16 * (size_t)n, [&](const double *a, double *b) {
        k_states<<<(n + 127) / 128, 128>>>(n, a, nx, ny, b);
    });
}

// the handle's adjoint without its kinetic-state tape, as where it does not fit
void probe_no_state_tape(mfcfd_t *h) { h->state_tape = false; }

}  // extern "C"
