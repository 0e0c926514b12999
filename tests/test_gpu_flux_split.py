"""The FP64 flux pass against the oracle where its paths change: grids around
the sizes at which the split of the work changes (a block a tile, a warp a
tile, a warp two tiles; a last tile of one point), weighted least squares,
Mach numbers beyond the polynomial erf's range, and neighbours in both lists
of a direction (a grid without jitter has neighbours exactly on an axis).
The bound on prim is the parity contract's 1e-10 relative."""
import numpy as np
import pytest

import oracle
from mfcfd_b200.grid import naca_ogrid
from mfcfd_b200.solver import Solver
from tests.helpers import max_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,flow", [
    (16, 9, dict(mach=0.8)),                     # 9 tiles
    (33, 17, dict(mach=0.8)),                    # 561 points: a last tile of one
    (96, 98, dict(mach=0.8)),                    # 588 tiles: a block a tile on 148 SMs
    (96, 99, dict(mach=0.8)),                    # 594: a warp a tile
    (192, 197, dict(mach=0.8)),                  # 2,364: one turn
    (192, 198, dict(mach=0.8)),                  # 2,376: two turns, or two tiles a warp
    (61, 23, dict(mach=0.8, power=-2.0)),
    (61, 23, dict(mach=2.6)),                    # |u| sqrt(beta) > 1.25
    (62, 24, dict(mach=0.8, jitter=0.0)),        # ties
    (62, 24, dict(mach=0.8, jitter=0.0, tscheme="first", power=-2.0)),
])
def test_flux_pass_paths(ni, nj, flow):
    flow = dict(flow)
    g = naca_ogrid(ni, nj, seed=7, first_spacing=5e-3, jitter=flow.pop("jitter", 0.1))
    flow = dict(cfl=0.2, vl_const=5.0, aoa=1.5, inner_iterations=1, **flow)
    with Solver(g, **flow) as s:
        r = s.run(4)
        got = s.get_state()
    o = oracle.Oracle(g, **flow)
    ref = o.run(4)
    assert np.allclose(r, ref, rtol=0, atol=1e-9)
    assert max_rel(got, o.prim()) < 1e-10
    o.close()
