"""The D and I passes with tile halos (grids past the by-slots rule's line)
where the size of a halo decides the path: largest halos of 64 rows (the narrow
forms' most), 65 and 66, 96 (the wide forms' most) and 97, in neighbouring
tiles (a warp's pair) and in a few or many tiles of a grid; tiles not staged at
all beside staged ones; stencils of up to 20 slots (local rows in three
words).  FP64 against the oracle (the parity contract's 1e-10 relative in prim,
1e-9 absolute in the residues), FP32-mixed against FP64."""
import numpy as np
import pytest

import oracle
from mfcfd_b200.batch import Batch
from mfcfd_b200.grid import INTERIOR, OUTER, WALL, naca_ogrid
from mfcfd_b200.solver import Solver
from tests.helpers import max_rel
from tests.test_gpu_halo import TILE, shuffled

SLOTS = 9 * TILE   # points an SM up to which the passes go by slots
FEW, MANY = (1000, 1001), tuple(t for t in range(200, 1200) if t % 8 < 2)
# name: (tiles, rows of the even ones, rows of the odd ones)
GROWN = {
    "64": (FEW, 64, 64), "65": (FEW, 65, 65), "64+65": (FEW, 64, 65), "66": (FEW, 66, 66),
    "96": (FEW, 96, 96), "97": (FEW, 97, 60),
    "many 64": (MANY, 64, 64), "many 65": (MANY, 65, 65), "many 64+65": (MANY, 64, 65),
    "many 66": (MANY, 66, 66), "many 96": (MANY, 96, 96), "many 97": (MANY, 97, 96),
}


def order_of(g):
    """The library's point order: wall, outer, interior, each in caller order."""
    return np.concatenate([np.where(g.flag_1 == k)[0] for k in (WALL, OUTER, INTERIOR)])


def halo(g, order, inv, t):
    rows = set(range(t * TILE, min(g.n, (t + 1) * TILE)))
    for c in order[t * TILE:(t + 1) * TILE]:
        rows.update(inv[g.conn[: g.nbhs[c], c] - 1].tolist())
    return rows


def halo_sizes(g):
    order = order_of(g)
    inv = np.empty(g.n, np.int64)
    inv[order] = np.arange(g.n)
    return np.array([len(halo(g, order, inv, t)) for t in range(-(-g.n // TILE))])


def grown(kind, sms=148, ni=200, nj=None):
    """A ring-ordered grid past the slots' line, the halos of some tiles grown to
    the wanted rows: their points take the nearest points outside the halo, one
    each in turn."""
    tiles, even, odd = GROWN[kind]
    g = naca_ogrid(ni, nj or max(120, SLOTS * sms // ni + 2), seed=5, spacing="arc",
                   first_spacing="match")
    order = order_of(g)
    inv = np.empty(g.n, np.int64)
    inv[order] = np.arange(g.n)
    for t in tiles:
        rows = halo(g, order, inv, t)
        want = (odd if t % 2 else even) - len(rows)
        assert want >= 0
        pts = order[t * TILE:(t + 1) * TILE]
        near = range(max(0, pts[0] - 6 * ni), min(g.n, pts[-1] + 6 * ni))
        near = np.array([k for k in near if inv[k] not in rows and g.flag_1[k] == INTERIOR])
        d2 = (g.x[near] - g.x[pts[8]]) ** 2 + (g.y[near] - g.y[pts[8]]) ** 2
        for a, k in enumerate(near[np.argsort(d2, kind="stable")[:want]]):
            p = pts[2 + a % 12]
            g.conn[g.nbhs[p], p] = k + 1
            g.nbhs[p] += 1
    return g


def sm_count():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kind", GROWN)
def test_grown_tiles_have_the_rows(kind):
    g = grown(kind)
    tiles, even, odd = GROWN[kind]
    sizes = halo_sizes(g)
    assert g.n > SLOTS * 148 and g.nbhs.max() <= 20
    for t in tiles:
        assert sizes[t] == (odd if t % 2 else even)
    assert np.delete(sizes, tiles).max() <= 60


def check(g, inner=1):
    flow = dict(cfl=0.2, vl_const=5.0, mach=0.8, aoa=1.5, inner_iterations=inner)
    with Solver(g, **flow) as s:
        res = s.run(3)
        got = s.get_state()
    o = oracle.Oracle(g, **flow)
    ref = o.run(3)
    err = max_rel(got, o.prim())
    o.close()
    assert np.allclose(res, ref, rtol=0, atol=1e-9)
    assert err < 1e-10
    # FP32-mixed: the flux residual of one stage.  Each of a point's up to 20 slots
    # adds the rounding (6e-8, some ten roundings deep) of two fluxes of order one
    # and of the derivatives they are reconstructed with, times delta |c| (at most
    # about 0.1, twice that on the wall), counted twice for the inner iteration:
    # 20 * 2 * 6e-7 * 0.2 * 2 = 1e-5.
    wave = 0.05 * np.sin(3 * g.x + 2 * g.y)[:, None] * np.array([1, .5, .3, 1.4])
    prim = np.array([1, 0.8, 0.01, 1 / 1.4]) * (1 + wave)
    flux = {}
    for precision in ("fp64", "fp32_mixed"):
        with Solver(g, tscheme="first", precision=precision, **flow) as s:
            s.keep_diagnostics(True)
            s.set_state(prim)
            s.run(1)
            flux[precision] = s.get_array("flux_res")
    assert np.max(np.abs(flux["fp32_mixed"] - flux["fp64"])) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("kind", GROWN)
def test_halo_sizes_match_the_oracle(gpu, kind):
    check(grown(kind, sm_count()))


@pytest.mark.gpu
@pytest.mark.parametrize("frac", [1.0, 0.15])
def test_shuffled_grids_past_the_slots_match_the_oracle(gpu, frac):
    ring = naca_ogrid(200, max(120, SLOTS * sm_count() // 200 + 2), seed=5, spacing="arc",
                      first_spacing="match")
    g = shuffled(ring, frac, seed=3)
    sizes = halo_sizes(g)
    share = [float(np.mean(s)) for s in (sizes <= 64, (sizes > 64) & (sizes <= 96), sizes > 96)]
    assert share[2] > 0.9 if frac == 1.0 else min(share) > 0.02, share
    check(g, inner=2)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32_mixed"])
def test_few_large_tiles_of_a_large_grid(gpu, precision):
    """Two tiles of 65 rows in a grid past the line from which the wide forms need a
    share of the tiles: gathered directly, with the same bits as in a batch whose
    other grid takes both to the wide forms."""
    sms = sm_count()
    large = grown("65", sms, ni=800, nj=200 * TILE * sms // 800 + 8)
    small = grown("many 66", sms)
    assert large.n // TILE > 200 * sms and (large.n + small.n) // TILE < 200 * (len(MANY) + 2)
    flow = dict(cfl=0.1, vl_const=5.0, mach=0.8, aoa=1.5, inner_iterations=1)
    with Batch([large, small], [dict(flow, precision=precision) for _ in range(2)]) as b:
        b.run(2)
        many = b.get_state(0)
    with Solver(large, precision=precision, **flow) as s:
        s.run(2)
        assert np.array_equal(s.get_state(), many)
    if precision == "fp64":
        o = oracle.Oracle(large, **flow)
        o.run(2)
        assert max_rel(many, o.prim()) < 1e-10
        o.close()
