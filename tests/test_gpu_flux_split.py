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
    (96, 99, dict(mach=0.8)),                    # 594: two for some
    (132, 143, dict(mach=0.8)),                  # 1,180: a block two tiles
    (132, 144, dict(mach=0.8)),                  # 1,188: a warp a tile
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


@pytest.mark.parametrize("ni,nj,jitter", [
    (16, 9, 0.1),      # 9 tiles
    (33, 17, 0.1),     # a last tile of one point
    (120, 98, 0.1),    # 735 tiles: a block a tile on 148 SMs
    (120, 99, 0.1),    # 743: two for some
    (152, 155, 0.1),   # 1,473: a block two tiles
    (152, 156, 0.1),   # 1,482: a warp a tile
    (240, 197, 0.1),   # 2,955: one turn
    (240, 198, 0.1),   # 2,970: two turns, or two tiles a warp
    (62, 24, 0.0),     # ties
])
def test_fp32_flux_pass_paths(ni, nj, jitter):
    """flux_res of one stage against the FP64 pass.  Each of the up to 8 slots
    of a point adds the rounding (6e-8, about ten roundings deep) of two
    fluxes of order one times delta |c| (the time step over the spacing, at
    most about 0.1, twice that on the wall): 2e-6."""
    g = naca_ogrid(ni, nj, seed=7, first_spacing=5e-3, jitter=jitter)
    wave = 0.05 * np.sin(3 * g.x + 2 * g.y)[:, None] * np.array([1, .5, .3, 1.4])
    prim = np.array([1, 0.8, 0.01, 1 / 1.4]) * (1 + wave)
    got = {}
    for precision in ("fp64", "fp32_mixed"):
        with Solver(g, cfl=0.2, vl_const=5.0, mach=0.8, aoa=1.5, tscheme="first",
                    precision=precision) as s:
            s.keep_diagnostics(True)
            s.set_state(prim)
            s.run(1)
            got[precision] = s.get_array("flux_res")
    assert np.max(np.abs(got["fp32_mixed"] - got["fp64"])) < 2e-6
