"""Device memory that mfcfd_tangent leaves in use: at most 128 MB a handle (a
workspace up to that size stays for the next call, a larger one is released),
and nothing after the handle is gone; a call after a release gives the same
derivative.  The grid sizes lie on both sides of the bound (about 1.1 KB a
point)."""
import numpy as np
import pytest

from mfcfd_b200.grid import naca_ogrid
from mfcfd_b200.solver import Solver

pytestmark = pytest.mark.gpu
KEEP, SLACK = 128 << 20, 4 << 20  # (the driver allocates in 2 MB pages)


@pytest.mark.parametrize("ni,nj,kept", [(200, 120, True), (480, 420, False)])
def test_workspace_is_bounded(gpu, ni, nj, kept):
    import torch
    free = lambda: torch.cuda.mem_get_info(0)[0]
    g = naca_ogrid(ni, nj, seed=2, spacing="arc", first_spacing="match")
    dx = np.sin(3.0 * g.x)
    flow = dict(cfl=0.1, vl_const=5.0, mach=0.7, aoa=2.0, inner_iterations=2)
    with Solver(g, **flow) as s:  # (also loads the kernels)
        first = s.tangent(2, dx, None)
        assert np.all(np.isfinite(first)) and s.tangent(2, dx, None) == first
    with Solver(g, **flow) as s:
        before = free()
        assert s.tangent(2, dx, None) == first
        held = before - free()
        assert held <= KEEP + SLACK
        assert (held > 16 << 20) == kept
