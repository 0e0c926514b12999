"""The FP64 flux pass's own elementary functions and rearrangements
(mfcfd_b200/csrc/flux_math.cuh), on the CPU: the polynomials as the source
holds them against 50-digit values, and the rearranged limiter, split fluxes
and list sums against the reference's forms to rounding."""
import os
import re

import mpmath as mp
import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(HERE, "..", "mfcfd_b200", "csrc", "flux_math.cuh")).read()
mp.mp.dps = 50


def table(name):
    body = SRC[SRC.index(f"__constant__ double {name}["):]
    body = re.sub(r"/\*.*?\*/", "", body[body.index("{") + 1: body.index("}")])
    return [float.fromhex(v) if "0x" in v else float(v)
            for v in re.split(r"[,\s]+", body.strip())]


def poly(coef, x):
    p = mp.mpf(0)
    for c in coef:
        p = p * x + mp.mpf(c)
    return p


def test_exp_polynomial():
    c = table("c_exp")
    assert c[0] == float(1 / mp.log(2)) and -c[2] == float(mp.log(2))
    assert -c[3] == float(mp.log(2) - mp.mpf(-c[2])) and c[1] == 1.5 * 2.0**52
    # half an ulp of the result is 1.1e-16 of it; the interpolant adds 1.3e-17
    for r in np.linspace(-0.34658, 0.34658, 401):
        x = mp.mpf(float(r))
        got = 1 + x + x * x * poly(c[4:], x)
        assert abs(got / mp.exp(x) - 1) < 2e-17


def test_erf_polynomial():
    c = table("c_erf")
    for v in np.linspace(0.0, 1.25, 401):
        x = mp.mpf(float(v))
        assert abs(x * poly(c, x * x) - mp.erf(x)) < 4e-17
    # evaluated in FP64 (no fused operations here): a few ulp of 1
    x = np.linspace(-1.25, 1.25, 20001)
    p = np.zeros_like(x)
    for a in c:
        p = p * (x * x) + a
    ref = np.array([float(mp.erf(mp.mpf(float(v)))) for v in x[::50]])
    assert np.max(np.abs((x * p)[::50] - ref)) < 5e-16


def test_third_order_steps():
    # y0 with relative error d: the steps leave errors of d^3 and (5/2) d^3
    for d in (2.0**-20, -(2.0**-21)):
        for x in (0.3, 1.0, 7.7):
            x = mp.mpf(x)
            y = (1 + mp.mpf(d)) / x
            e = 1 - x * y
            assert abs(y * (1 + e + e * e) * x - 1) <= abs(mp.mpf(d)) ** 3 * 1.001
            y = (1 + mp.mpf(d)) / mp.sqrt(x)
            e = 1 - x * y * y
            got = y + y * e * (mp.mpf(3) / 8 * e + mp.mpf(1) / 2)
            assert abs(got * mp.sqrt(x) - 1) <= 2.6 * abs(mp.mpf(d)) ** 3


def test_limiter_and_split_flux_forms():
    rng = np.random.default_rng(4)
    n = 4000
    t = rng.normal(size=n) * 10.0 ** rng.uniform(-3, 0, n)
    q, eps2 = rng.normal(size=n), 10.0 ** rng.uniform(-12, -2, n)
    dn = -0.5 * t
    dp = np.where(dn > 0, 1.0, -1.0) * 10.0 ** rng.uniform(-4, 0, n)
    num = (dp * dp + eps2) * dn + 2.0 * dn * dn * dp
    den = (dp * dp + 2.0 * dn * dn + dn * dp + eps2) * dn
    a = dp * dp + eps2
    assert np.allclose((a - t * dp) / (a + dn * (dp - t)), num / den, rtol=1e-14, atol=0)

    rho, pbr = rng.uniform(0.2, 2, n), rng.uniform(0.3, 1.5, n)
    u, o, e, B = (rng.uniform(-1, 1, n) for _ in range(4))
    usq = u * u + o * o
    for s in (1.0, -1.0):
        A = 0.5 * (1 + s * e)
        ref = [rho * (u * A + s * B), rho * ((pbr + u * u) * A + s * u * B),
               rho * (u * o * A + s * o * B),
               rho * (0.5 * u * (7 * pbr + usq) * A + s * 0.5 * (6 * pbr + usq) * B)]
        f, w6, pA = u * A + s * B, 6 * pbr + usq, pbr * A
        got = [rho * f, rho * (u * f + pA), o * (rho * f), 0.5 * rho * (w6 * f + u * pA)]
        for g, r in zip(got, ref):
            assert np.max(np.abs(g - r)) < 1e-14


def test_pooled_list_sums():
    """Sum over the lists of (fx syy - fy sxy) / det = sum of slot weights."""
    rng = np.random.default_rng(5)
    for _ in range(200):
        nb = int(rng.integers(4, 20))
        d, w, G = rng.normal(size=(nb, 2)), rng.uniform(0.5, 2, nb), rng.normal(size=nb)
        member = [d[:, 0] <= 0, d[:, 0] >= 0]
        ref = got = size = 0.0
        for m in member:
            if m.sum() < 2:
                continue
            sxx, syy, sxy = ((w * a * b)[m].sum() for a, b in
                             ((d[:, 0], d[:, 0]), (d[:, 1], d[:, 1]), (d[:, 0], d[:, 1])))
            det = sxx * syy - sxy * sxy
            fx, fy = ((w * d[:, a] * G)[m].sum() for a in (0, 1))
            ref += (fx * syy - fy * sxy) / det
            c = (syy / det * d[:, 0] - sxy / det * d[:, 1]) * w
            got += (c * G)[m].sum()
            size += np.sum(np.abs(c * G)[m]) * (1 + sxx * syy / abs(det))
        assert abs(got - ref) <= 1e-14 * size
