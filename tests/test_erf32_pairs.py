"""The FP32 flux pass's erf as it runs, on pairs (kstate2 in
mfcfd_b200/csrc/primal_fp32.cu): its coefficients are those of the scalar form
(negated, as 1 + p t E is formed with one fused operation), and its order of
operations, in FP32, stays within the scalar form's bound: the published 1.5e-7
and some five roundings of values up to 1.1."""
import os
import re

import numpy as np
from scipy.special import erf

from tests.test_erf32 import coefficients

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(HERE, "..", "mfcfd_b200", "csrc", "primal_fp32.cu")).read()


def pair_coefficients():
    body = SRC[SRC.index("KState2 kstate2("):]
    body = body[body.index("const F2 d = fma2("): body.index("s.e = ")]
    p = float(re.search(r"f2\(([0-9.]+)f\), f2\(1\.0f\)\)", body).group(1))
    first = float(re.search(r"F2 p = f2\((-?[0-9.]+)f\);", body).group(1))
    rest = [float(v) for v in re.findall(r"p = fma2\(p, t, f2\((-?[0-9.]+)f\)\);", body)]
    assert "fma2(p * t, E, f2(1.0f))" in body
    return p, [first] + rest


def test_coefficients_are_the_scalar_form_s():
    p, a = coefficients()
    q, b = pair_coefficients()
    assert q == p and b == [-v for v in a[::-1]]


def test_error_bound_in_the_pair_s_order():
    f = np.float32
    fma = lambda a, b, c: f(np.float64(a) * np.float64(b) + np.float64(c))
    x = np.linspace(-6.0, 6.0, 200001).astype(f)
    q, b = pair_coefficients()
    E = np.exp2((x * x * f(-1.44269504)).astype(np.float64)).astype(f)
    t = (f(1) / fma(np.abs(x), f(q), f(1))).astype(f)
    p = f(b[0])
    for c in b[1:]:
        p = fma(p, t, f(c))
    got = np.copysign(fma((p * t).astype(f), E, f(1)), x)
    assert np.max(np.abs(got - erf(x.astype(np.float64)))) <= 6e-7
