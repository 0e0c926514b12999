"""The FP64 flux pass's own elementary functions and kinetic states on the
device (flux_math.cuh, through tests/device_probe.cu) against 50-digit values,
on both sides of every limit beyond which the library functions take over
(1.25 for erf, 26 and 700 for exp); and the adjoint without its kinetic-state
tape (the path taken where the tape does not fit) against the adjoint with it."""
import ctypes as C
import os
import subprocess

import mpmath as mp
import numpy as np
import pytest

from mfcfd_b200 import build as B
from mfcfd_b200.grid import naca_ogrid
from mfcfd_b200.solver import Solver
from tests.test_gpu_reverse_forms import _widen

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
mp.mp.dps = 50


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    try:
        nvcc = B.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("probe") / "probe.so")
    subprocess.run([nvcc, *B.ARCH, "-O3", "-std=c++17", "-I", os.path.join(B.ROOT, "include"),
                    "-Xcompiler", "-fPIC", "-shared", "-o", out,
                    os.path.join(HERE, "device_probe.cu")], check=True, capture_output=True)
    lib = C.CDLL(out)
    lib.probe_states.argtypes = [C.c_int, C.c_void_p, C.c_double, C.c_double, C.c_void_p]
    lib.probe_no_state_tape.argtypes = [C.c_void_p]
    lib.probe_no_state_tape.restype = None
    return lib


def forms(lib, x):
    x = np.ascontiguousarray(x)
    out = np.empty((x.size, 4))
    assert lib.probe_forms(x.size, x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    return out.T


def worst(got, x, f, relative=True):
    err = 0.0
    for g, v in zip(got, x):
        ref = f(mp.mpf(float(v)))
        err = max(err, float(abs(mp.mpf(float(g)) - ref) / (abs(ref) if relative else 1)))
    return err


def test_elementary_forms(gpu, probe):
    """The reciprocals' steps leave 2^-60 (from the 2^-20 of the approximation):
    one rounding of the result for 1/x, and half of one of x y for 1/sqrt(x): 1.5
    half-ulps, below 2^-52.  exp: two roundings of values up to sqrt(2) and the
    reduction's of r: below 2^-52 relative.  erf: the sum of |c_i| z^i is at most
    2.2 of the result: below 5e-16 absolute."""
    rng = np.random.default_rng(2)
    x = np.concatenate([10.0 ** rng.uniform(-30, 30, 1500), 2.0 ** np.arange(-40.0, 41)])
    got = forms(probe, x)
    assert worst(got[0], x, lambda v: 1 / v) <= 2.0**-52
    assert worst(got[1], x, lambda v: 1 / mp.sqrt(v)) <= 2.0**-52
    x = np.concatenate([rng.uniform(-700, 700, 1000), rng.uniform(-2, 2, 500),
                        [-700.0, 700.0, 0.0, -1e-300, 0.5 * np.log(2), -0.5 * np.log(2)]])
    assert worst(forms(probe, x)[2], x, mp.exp) <= 2.0**-52
    x = np.concatenate([rng.uniform(-1.25, 1.25, 1500), [-1.25, 1.25, 0.0, 1e-9]])
    assert worst(forms(probe, x)[3], x, mp.erf, relative=False) <= 5e-16


def test_states_across_the_limits(gpu, probe):
    """Velocities along and across from rest to |S| = 30 and |texp| to 708, each
    state of a pair on its own side of a limit.  With d = 2^-53: an exponent a
    carries some 4 d |a| (beta |u|^2 itself 32 d: some ten roundings of u, S and beta^(1/2), squared), its result that and the
    roundings of a few products, 20 d; erf is within 1e-15."""
    rng = np.random.default_rng(3)
    n, th = 600, 0.7
    nx, ny = np.sin(th), np.cos(th)
    beta = rng.uniform(0.3, 3.0, (n, 2))
    lim = rng.choice([0.0, 0.4, 1.2499, 1.2501, 1.25, 3.0, 25.99, 26.01, 30.0], (2, n, 2))
    S = lim * rng.choice([-1.0, 1.0], (2, n, 2)) * (1 + 1e-13 * rng.normal(size=(2, n, 2)))
    ut, un = S / np.sqrt(beta)
    u1, u2 = ut * ny + un * nx, -ut * nx + un * ny
    texp = rng.choice([-708.0, -700.5, -699.5, -3.0, 0.2, 4.0, 699.5, 700.5, 706.0], (n, 2))
    usq = u1 * u1 + u2 * u2
    qt = np.stack([texp - beta * usq, 2 * beta * u1, 2 * beta * u2, -2 * beta], axis=-1)
    qt = np.ascontiguousarray(qt)
    out = np.empty((n, 2, 8))
    assert probe.probe_states(n, qt.ctypes.data_as(C.c_void_p), nx, ny,
                              out.ctypes.data_as(C.c_void_p)) == 0
    d = 2.0**-53
    mx, my = mp.mpf(float(nx)), mp.mpf(float(ny))
    for q, o in zip(qt.reshape(-1, 4), out.reshape(-1, 8)):
        q = [mp.mpf(float(v)) for v in q]
        b, w = -q[3] / 2, -1 / q[3]
        v1, v2 = q[1] * w, q[2] * w
        us = v1 * v1 + v2 * v2
        t = q[0] + b * us
        s1, s2 = (v1 * my - v2 * mx) * mp.sqrt(b), (v1 * mx + v2 * my) * mp.sqrt(b)
        h = w * mp.sqrt(b) / mp.sqrt(mp.pi)
        # (the exponents' size: q[0] and b |u|^2 cancel in texp; s1 and s2 each come
        # from products of the size of |u| sqrt(b))
        a, c = abs(q[0]) + 8 * b * us, 8 * b * us
        ref = [(mp.exp(t) * (4 * w * w) / mp.sqrt(b), 4 * d * a + 20 * d), (w, 4 * d),
               (mp.exp(-s1 * s1) * h, 4 * d * c + 20 * d), (mp.exp(-s2 * s2) * h, 4 * d * c + 20 * d)]
        for (r, tol), g in zip(ref, o):
            # (results below the normal range lose digits)
            assert abs(mp.mpf(float(g)) - r) <= tol * abs(r) + mp.mpf(2)**-1070
        size = mp.sqrt(b * us)
        for s, g in ((s1, o[4]), (s2, o[5])):
            assert abs(mp.mpf(float(g)) - mp.erf(s)) <= 1e-15 + 16 * d * size * mp.exp(-s * s)
        for r, g in ((v1, o[6]), (v2, o[7])):
            assert abs(mp.mpf(float(g)) - r) <= 4 * d * abs(r)


@pytest.mark.parametrize("ni,nj,inner,tscheme,jitter,wide", [
    (33, 11, 1, "ssprk43", 0.1, False),   # a last block of 43 points
    (32, 12, 0, "ssprk43", 0.0, False),   # ties
    (31, 13, 2, "first", 0.1, True),      # up to 20 slots
    (200, 108, 1, "first", 0.1, False),   # past the small grids' forms on 148 SMs
])
def test_adjoint_without_state_tape(gpu, probe, ni, nj, inner, tscheme, jitter, wide):
    """The states formed again are the taped ones' own operations, but for |u|^2 and
    the products with the normal (a rounding each): equal to some 1e2 operations'
    rounding of the sum of the terms' sizes, 1e-12 of a gradient's largest entry
    times the number of passes, below 1e-9."""
    g = naca_ogrid(ni, nj, seed=15, first_spacing=5e-3, jitter=jitter)
    if wide:
        g = _widen(g, 3)
    import torch
    grads, used = [], []
    for tape in (True, False):
        with Solver(g, cfl=0.2, vl_const=5.0, mach=0.7, aoa=2.0, inner_iterations=inner,
                    tscheme=tscheme) as s:
            if not tape:
                probe.probe_no_state_tape(s.h)
            s.run(2)
            free = torch.cuda.mem_get_info(0)[0]
            grads.append(s.adjoint(2, "cd"))
            used.append(free - torch.cuda.mem_get_info(0)[0])
    if g.n > 20000:  # (128 bytes a slot and stage; the driver allocates in 2 MB pages)
        assert used[0] - used[1] > 128 * int(g.nbhs.max()) * g.n - (4 << 20)
    (J0, x0, y0, n0), (J1, x1, y1, n1) = grads
    assert J0 == J1 and n0 == n1
    for a, b in ((x0, x1), (y0, y1)):
        assert np.max(np.abs(a)) > 0.0
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a))
