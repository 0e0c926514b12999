"""The reverse and forward derivatives against each other where their passes
change: several inner iterations (the D pass's derivatives enter every one),
neighbours exactly on an axis (a grid without jitter: in both lists of a
direction), stencils of up to 20 slots (the flux reverse's later rounds) that
are not symmetric, point counts around the blocks of 64 and 128, first-order
time stepping; the small grids' forms and, past 21,000 points, the others.  Both derivatives are exact up to rounding, which some 1e2
operations a term and a few passes keep below 1e-9 of the sum of the terms'
sizes."""
import numpy as np
import pytest

from mfcfd_b200.grid import naca_ogrid
from mfcfd_b200.solver import Solver

pytestmark = pytest.mark.gpu


def _widen(g, seed):
    """Points given up to 20 of their neighbours' neighbours."""
    rng = np.random.default_rng(seed)
    nbhs, conn = g.nbhs.copy(), g.conn.copy()
    for p in np.flatnonzero(g.flag_1 == 1)[::7]:
        have = set((conn[: nbhs[p], p] - 1).tolist()) | {int(p)}
        more = {int(k) - 1 for q in have for k in g.conn[: g.nbhs[q], q]} - have
        for k in sorted(more)[: int(rng.integers(1, 13))]:
            conn[nbhs[p], p] = k + 1
            nbhs[p] += 1
    g.nbhs, g.conn = nbhs, conn
    return g


@pytest.mark.parametrize("ni,nj,jitter,inner,tscheme,wide", [
    (32, 12, 0.1, 2, "ssprk43", False),   # 384 points: whole blocks
    (33, 11, 0.1, 3, "ssprk43", False),   # 363: a last block of 43
    (29, 10, 0.1, 1, "first", False),     # 290
    (32, 12, 0.0, 1, "ssprk43", False),   # ties
    (31, 13, 0.1, 0, "ssprk43", True),    # up to 20 slots
    (31, 13, 0.0, 3, "first", True),
    (200, 108, 0.1, 1, "first", False),   # 21,600: past the small grids' forms on 148 SMs
    (200, 108, 0.0, 2, "ssprk43", True),
])
def test_adjoint_and_tangent_agree(gpu, ni, nj, jitter, inner, tscheme, wide):
    g = naca_ogrid(ni, nj, seed=15, first_spacing=5e-3, jitter=jitter)
    if wide:
        g = _widen(g, 3)
        assert g.nbhs.max() > 16
    rng = np.random.default_rng(21)
    dx, dy = rng.standard_normal(g.n), rng.standard_normal(g.n)
    with Solver(g, cfl=0.2, vl_const=5.0, mach=0.7, aoa=2.0, inner_iterations=inner,
                tscheme=tscheme) as s:
        s.run(2)
        _, dJ = s.tangent(2, dx, dy, objective="cd")
        _, gx, gy, _ = s.adjoint(2, "cd")
    dot = float(gx @ dx + gy @ dy)
    size = float(np.abs(gx * dx).sum() + np.abs(gy * dy).sum())
    assert np.isfinite(dot) and size > 0.0
    assert abs(dJ - dot) <= 1e-9 * size, (dJ, dot, size)
