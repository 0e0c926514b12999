"""The D and I passes by slots (small grids) against the halo form (larger
ones): the same operations in the same order, so a small grid's result is the
same to the bit whether it runs alone (by slots) or in a batch with a grid that
takes the batch past the rule's line (by halos).  Grids: a last tile of one
point, ties, weights; for the halo passes' wide form, halos of more than 64 rows
(stencils of up to 20 slots, a twentieth of the points shuffled) and, not staged
at all, of more than 96 (all points shuffled)."""
import numpy as np
import pytest

from mfcfd_b200.batch import Batch
from mfcfd_b200.grid import naca_ogrid
from mfcfd_b200.solver import Solver
from tests.test_gpu_halo import shuffled

pytestmark = pytest.mark.gpu


def _widen(g):
    nbhs, conn = g.nbhs.copy(), g.conn.copy()
    for p in np.flatnonzero(g.flag_1 == 1)[::5]:
        have = set((conn[: nbhs[p], p] - 1).tolist()) | {int(p)}
        more = {int(k) - 1 for q in have for k in g.conn[: g.nbhs[q], q]} - have
        for k in sorted(more)[: 1 + int(p) % 12]:
            conn[nbhs[p], p] = k + 1
            nbhs[p] += 1
    g.nbhs, g.conn = nbhs, conn
    return g


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("precision,power,inner", [
    ("fp64", 0.0, 2), ("fp64", -2.0, 1), ("fp32_mixed", 0.0, 2), ("fp32_mixed", -2.0, 1),
])
def test_slots_and_halos_agree_to_the_bit(gpu, precision, power, inner, wide):
    ring = naca_ogrid(64, 24, seed=5, first_spacing=5e-3)
    if wide:
        grids = [_widen(naca_ogrid(48, 16, seed=3, first_spacing=5e-3)),
                 shuffled(ring, 0.05, seed=3), shuffled(ring, 1.0, seed=3)]
    else:
        grids = [naca_ogrid(33, 17, seed=7, first_spacing=5e-3),
                 naca_ogrid(62, 24, seed=7, first_spacing=5e-3, jitter=0.0), ring]
    grids.append(naca_ogrid(300, 200, seed=1, spacing="arc", first_spacing="match"))
    flow = dict(cfl=0.2, vl_const=5.0, mach=0.8, aoa=1.5, inner_iterations=inner, power=power,
                precision=precision)
    with Batch(grids, [dict(flow) for _ in grids]) as b:
        b.run(3)
        many = [b.get_state(i) for i in range(3)]
    for g, got in zip(grids, many):
        with Solver(g, **flow) as s:
            s.run(3)
            assert np.array_equal(s.get_state(), got)
