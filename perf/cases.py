"""Work that users of this solver have it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` builds what a user's program
holds before the call (grid, solver handle, start state), ``run`` makes one
pass through the public Python entry points and returns everything it
computes, ``exact`` computes the same outputs with plain torch in 64 bits.

The kinds of work:

* ``primal``  -- a restart: load a flow state, run iterations of the
  pseudo-time loop, read the state, the residue history and the forces back;
* ``batch``   -- the same for many grids advanced together;
* ``adjoint`` -- dJ/dx, dJ/dy of every point through some iterations;
* ``tangent`` -- dJ along one direction of grid motion.

An FP32-mixed solver stores its state in FP32, so a pass in that precision
returns its results as FP32 arrays; everything else is FP64.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from mfcfd_b200.batch import Batch
from mfcfd_b200.grid import Grid, batch_instances, naca_ogrid
from mfcfd_b200.solver import Solver

GAMMA = 1.4
PR_INF = 1.0 / 1.4


def _case(name, work, ni, nj, iters, precision="fp64", inner=0, scheme="ssprk43", wall="arc",
          points="ring", power=0.0, objective="cd", instances=1):
    """wall "arc": wall points uniform in arc length, square first cells (the
    grids of the long runs; an even ni); "coarse": cosine chord spacing with a
    5e-3 first spacing (the 16,000-point configuration); "cosine": the same
    with 1e-3 (the headline benchmark).  points "ring": points in ring order;
    "cloud": in no order, renumbered by the solver (RCM)."""
    return dict(name=name, work=work, ni=ni, nj=nj, iters=iters, precision=precision, inner=inner,
                scheme=scheme, wall=wall, points=points, power=power, objective=objective,
                instances=instances)


def listed():
    return [
        # a coarse grid, as a first look at a new geometry: launches and latency count
        _case("primal_coarse", "primal", 64, 24, 100, inner=1, wall="coarse"),
        # the 16,000-point airfoil grid of the plain FP64 configuration
        _case("primal_16k", "primal", 160, 100, 60, wall="coarse"),
        # an odd-sized cloud from a point generator, in no particular order, with the
        # reference's inverse-distance weights
        _case("primal_cloud", "primal", 250, 161, 30, points="cloud", power=-2.0),
        # the 256,000-point grid of the sensitivity studies
        _case("primal_256k", "primal", 640, 400, 30),
        # the headline benchmark: 1,024,000 points, transonic, three inner iterations
        _case("primal_1m", "primal", 1280, 800, 20, inner=3, wall="cosine"),
        # FP32-mixed on an odd-sized mid grid, first-order time stepping
        _case("primal32_90k", "primal", 386, 235, 60, precision="fp32_mixed", inner=1,
              scheme="first"),
        # the headline benchmark in FP32-mixed
        _case("primal32_1m", "primal", 1280, 800, 20, precision="fp32_mixed", inner=3,
              wall="cosine"),
        # a parameter sweep: grids of uneven size, FP32-mixed, advanced together
        _case("batch32", "batch", 0, 0, 30, precision="fp32_mixed", instances=14),
        # shape sensitivities on the coarse configuration, with an inner iteration
        _case("adjoint_16k", "adjoint", 160, 100, 12, inner=1, wall="coarse", objective="cl"),
        # shape sensitivities on the 256,000-point grid
        _case("adjoint_256k", "adjoint", 640, 400, 8),
        # one design direction, forward mode
        _case("tangent_64k", "tangent", 320, 201, 10, inner=1),
    ]


def draw(rng):
    work = rng.choice(["primal"] * 6 + ["batch", "adjoint", "adjoint", "tangent"])
    top = {"primal": 1_000_000, "batch": 0, "adjoint": 250_000, "tangent": 120_000}[work]
    if work == "batch":
        return _drawn(_case("", work, 0, 0, rng.randint(20, 40),
                            precision=rng.choice(["fp64", "fp32_mixed"]),
                            inner=rng.randint(0, 1), instances=rng.randint(3, 10)))
    n = math.exp(rng.uniform(math.log(1_500), math.log(top)))
    nj = max(12, round(math.sqrt(n / rng.uniform(1.2, 2.4))))
    ni = max(32, round(n / nj))
    wall = "coarse" if n < 60_000 and rng.random() < 0.5 else "arc"
    if wall == "arc":
        ni += ni % 2
    # a pass costs no more than the headline benchmark's: 1M points, 20 iterations
    iters = max(4, min(rng.randint(20, 60), int(12e6 / n)))
    if work != "primal":
        iters = max(4, min(12, iters))
        return _drawn(_case("", work, ni, nj, iters, inner=rng.randint(0, 1), wall=wall,
                            objective=rng.choice(["cl", "cd"])))
    precision = rng.choice(["fp64", "fp32_mixed"])
    cloud = n < 100_000 and rng.random() < 0.2
    weighted = precision == "fp64" and wall == "arc" and n < 200_000
    power = rng.choice([0.0, -2.0]) if weighted else 0.0
    return _drawn(_case("", work, ni, nj, iters, precision=precision, inner=rng.randint(0, 3),
                        wall=wall, scheme=rng.choice(["ssprk43"] * 4 + ["first"]), power=power,
                        points="cloud" if cloud else "ring"))


def _drawn(case):
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# inputs

@functools.lru_cache(maxsize=8)
def _grid(ni, nj, wall, points):
    """The grid file of a case (the same for every start state)."""
    if wall != "arc":
        g = naca_ogrid(ni, nj, seed=2000, first_spacing=1e-3 if wall == "cosine" else 5e-3)
    else:
        g = naca_ogrid(ni, nj, seed=3000, spacing="arc", first_spacing="match")
    return g if points == "ring" else _reordered(g, np.random.default_rng(7).permutation(g.n))


@functools.lru_cache(maxsize=2)
def _batch_grids(instances):
    grids, _, _ = batch_instances(instances, n_max=128_000)
    return grids


def _reordered(g: Grid, perm):
    inv = np.empty_like(perm)
    inv[perm] = np.arange(perm.size)

    def numbers(a):  # 1-based, 0 = none
        return np.ascontiguousarray(np.where(a > 0, inv[np.maximum(a, 1) - 1] + 1, 0), np.int32)

    per_point = {f: np.ascontiguousarray(getattr(g, f)[perm]) for f in
                 ("x", "y", "nx", "ny", "min_dist", "flag_1", "flag_2", "nbhs", "original_id",
                  "qtdepth")}
    return dataclasses.replace(g, **per_point, left=numbers(g.left[perm]),
                               right=numbers(g.right[perm]), conn=numbers(g.conn[:, perm]))


def _flow(case, rng):
    """Flow conditions within the configurations' ranges."""
    mach = rng.uniform(0.6, 0.85) if case["wall"] != "cosine" else rng.uniform(0.8, 0.85)
    return dict(cfl=0.2, vl_const=5.0, power=case["power"], mach=float(mach),
                aoa=float(rng.uniform(0.5, 3.0)), tscheme=case["scheme"],
                inner_iterations=case["inner"])


def _state(g: Grid, flow, rng):
    """A flow on its way to steady state: the freestream with smooth
    disturbances around the airfoil that die out towards the far field."""
    x, y = g.x, g.y
    d = np.hypot(x - np.clip(x, 0.0, 1.0), y)
    amp = np.exp(-d / 0.6)

    def wave():
        k = rng.uniform(1.0, 4.0, size=(3, 2))
        ph = rng.uniform(0.0, 2.0 * math.pi, size=3)
        return sum(np.sin(k[m, 0] * x + k[m, 1] * y + ph[m]) for m in range(3)) / 3.0

    t = math.radians(flow["aoa"])
    s = 0.10 * amp * wave()
    prim = np.empty((g.n, 4))
    prim[:, 0] = 1.0 + s
    prim[:, 1] = flow["mach"] * (math.cos(t) + 0.25 * amp * wave())
    prim[:, 2] = flow["mach"] * (math.sin(t) + 0.20 * amp * wave())
    prim[:, 3] = PR_INF * (1.0 + s) ** GAMMA
    return prim


def _inputs(case, seed):
    """(grids, flows, states) of a case, one entry per instance."""
    rng = np.random.default_rng(seed)
    if case["work"] == "batch":
        grids = _batch_grids(case["instances"])
    else:
        grids = [_grid(case["ni"], case["nj"], case["wall"], case["points"])]
    flows = [_flow(case, rng) for _ in grids]
    states = [_state(g, f, rng) for g, f in zip(grids, flows)]
    return grids, flows, states


def _direction(g: Grid, seed):
    """A smooth displacement of the whole grid, one shape-design direction."""
    rng = np.random.default_rng(seed + 1)
    a, b = rng.uniform(1.0, 3.0, 2)
    d = np.exp(-np.hypot(g.x - np.clip(g.x, 0.0, 1.0), g.y) / 0.5)
    return d * np.sin(a * g.x + b), d * np.cos(b * g.x - a)


def prepare(case, seed):
    grids, flows, states = _inputs(case, seed)
    s = dict(case=case, states=states)
    if case["work"] == "batch":
        s["batch"] = Batch(grids, [dict(f, precision=case["precision"]) for f in flows])
        return s
    s["solver"] = Solver(grids[0], precision=case["precision"],
                         ordering="rcm" if case["points"] == "cloud" else "kind", **flows[0])
    if case["work"] == "tangent":
        s["direction"] = _direction(grids[0], seed)
    return s


def run(state):
    case, n = state["case"], state["case"]["iters"]
    f = np.float32 if case["precision"] == "fp32_mixed" else np.float64
    if case["work"] == "batch":
        b = state["batch"]
        for i, prim in enumerate(state["states"]):
            b.set_state(i, prim)
        r = b.run(n)
        coeffs = [np.concatenate(b.forces(i)).astype(f) for i in range(b.n_inst)]
        return dict(iters=r.iters_done, residue=np.stack(r.residue).astype(f),
                    prim=[b.get_state(i).astype(f) for i in range(b.n_inst)], coeffs=coeffs)
    s = state["solver"]
    s.set_state(state["states"][0])
    if case["work"] == "adjoint":
        J, dx, dy, _ = s.adjoint(n, case["objective"])
        return dict(J=J, dx=dx, dy=dy)
    if case["work"] == "tangent":
        J, dJ = s.tangent(n, *state["direction"], objective=case["objective"])
        return dict(J=J, dJ=dJ)
    residue = s.run(n, it_first=1)
    return dict(residue=residue.astype(f), prim=s.get_state().astype(f),
                coeffs=np.concatenate(s.forces()).astype(f))


def work(case):
    """Bytes: per point and stage the state is read and written, the stencil,
    coordinates, limiter length and time step are read, and the gradients (and
    their bounds) cross from the pass that forms them to the passes of the
    neighbours, once per inner iteration more.  Flops: about 900 per stencil
    slot for the two limited kinetic states and their split fluxes, 60 for
    the gradients and 45 for an inner iteration, multiply and add apart.  A
    reversed iteration costs at least the forward one, its tape and about
    twice its arithmetic; a tangent about twice the primal."""
    if case["work"] == "batch":
        _, _, specs = batch_instances(case["instances"], n_max=128_000, build=False)
        points = sum(s["ni"] * s["nj"] for s in specs)
    else:
        points = case["ni"] * case["nj"]
    word = 4 if case["precision"] == "fp32_mixed" else 8
    stages = 4 if case["scheme"] == "ssprk43" else 1
    K, m = 8, case["inner"]
    per_stage = 8 * word + 4 * K + 16 + 16 + 2 * 8 * word * (2 + m)
    flops = K * (900 + 60 + 45 * m)
    reverse = {"adjoint": 3.0, "tangent": 2.0}.get(case["work"], 1.0)
    n = points * stages * case["iters"] * reverse
    return {"bytes": n * per_stage + points * 64, "flops": n * flops}


# ---------------------------------------------------------------------------
# the same results with plain torch in 64 bits

class _Plain:
    """The pseudo-time loop on whole arrays: slot tensors are (points, slots)."""

    def __init__(self, g: Grid, flow, device):
        self.flow, self.dev = flow, device
        self.n = g.n
        kp = max(int(g.nbhs.max()), 1)
        valid = np.arange(kp)[None, :] < g.nbhs[:, None]
        k = np.where(valid, g.conn[:kp].T - 1, np.arange(g.n)[:, None]).astype(np.int64)
        t = functools.partial(torch.as_tensor, device=device)
        self.valid, self.k = t(valid), t(k)
        self.x, self.y = t(g.x), t(g.y)
        self.eps2 = t(np.power(flow["vl_const"] * g.min_dist, 3.0) ** 2)
        self.wall, self.outer = t(g.flag_1 == 0), t(g.flag_1 == 2)
        bnd = np.flatnonzero(g.flag_1 != 1)
        self.bnd, self.left, self.right = t(bnd), t(g.left[bnd] - 1), t(g.right[bnd] - 1)
        shp = np.flatnonzero(g.flag_2 > 0)
        self.shp, self.sl, self.sr = (t(a.astype(np.int64)) for a in
                                      (shp, g.left[shp] - 1, g.right[shp] - 1))
        self.left, self.right = self.left.long(), self.right.long()
        self.shape, self.shapes = t(g.flag_2[shp].astype(np.int64) - 1), g.shapes
        # list membership by the sign of the projections, rounded as written
        nx, ny = (a.cpu().numpy() for a in self.normals(self.x, self.y))
        dx, dy = g.x[k] - g.x[:, None], g.y[k] - g.y[:, None]
        tx, ty = ny[:, None], -nx[:, None]
        dels = dx * tx + dy * ty
        deln = dx * nx[:, None] + dy * ny[:, None]
        wall, outer = (g.flag_1 == 0)[:, None], (g.flag_1 == 2)[:, None]
        self.lists = [t(m & valid) for m in
                      (dels <= 0, dels >= 0, (deln <= 0) & ~wall | outer,
                       (deln >= 0) & ~outer | wall)]

    def normals(self, x, y):
        b, l, r = self.bnd, self.left, self.right
        ax = 0.5 * ((y[b] - y[l]) + (y[r] - y[b]))
        ay = 0.5 * ((x[b] - x[l]) + (x[r] - x[b]))
        det = torch.sqrt(ax * ax + ay * ay)
        nx = torch.zeros_like(x).index_put((b,), -ax / det)
        ny = torch.ones_like(x).index_put((b,), ay / det)
        return nx, ny

    @staticmethod
    def q_of(P):
        rho, u1, u2, pr = P
        beta = 0.5 * rho / pr
        return [torch.log(rho) + torch.log(beta) * 2.5 - beta * (u1 * u1 + u2 * u2),
                2 * beta * u1, 2 * beta * u2, -2 * beta]

    def geometry(self, x, y):
        k, v = self.k, self.valid
        dx = torch.where(v, x[k] - x[:, None], 1.0)
        dy = torch.where(v, y[k] - y[:, None], 1.0)
        dist = torch.sqrt(dx * dx + dy * dy)
        p = self.flow["power"]
        w = v.to(dx.dtype) if p == 0.0 else torch.where(v, dist ** p, 0.0)
        return dx, dy, dist, w

    def delta(self, P, dist):
        spd = torch.sqrt(P[1] * P[1] + P[2] * P[2]) + 3.0 * torch.sqrt(P[3] / P[0])
        dt = torch.where(self.valid, self.flow["cfl"] * dist / spd[self.k], 1.0)
        return torch.clamp(dt.min(dim=1).values, max=1.0)

    def solve(self, dx, dy, w, fs):
        """Least-squares x and y derivatives of slot differences fs."""
        wx, wy = w * dx, w * dy
        sxx, syy, sxy = (wx * dx).sum(1), (wy * dy).sum(1), (wx * dy).sum(1)
        det = sxx * syy - sxy * sxy
        out = []
        for f in fs:
            fx, fy = (wx * f).sum(1), (wy * f).sum(1)
            out.append(((fx * syy - fy * sxy) / det, (fy * sxx - fx * sxy) / det))
        return out

    def limited(self, q, gx, gy, qmax, qmin, eps2, dx, dy):
        t = dx * gx + dy * gy
        neg = -0.5 * t
        flat = neg.abs() <= float(np.float32(10e-6))
        neg_ = torch.where(flat, 1.0, neg)
        pos = torch.where(neg > 0, qmax - q, qmin - q)
        num = pos * pos + eps2 + 2.0 * neg_ * pos
        den = pos * pos + 2.0 * neg_ * neg_ + neg_ * pos + eps2
        den = torch.where(flat, 1.0, den)
        phi = torch.where(flat, 1.0, torch.clamp(num / den, max=1.0))
        return q - 0.5 * phi * t

    @staticmethod
    def maxwell(qt, nx, ny):
        beta = -0.5 * qt[3]
        pbr = 0.5 / beta
        u1, u2 = qt[1] * pbr, qt[2] * pbr
        rho = torch.exp(qt[0] + beta * (u1 * u1 + u2 * u2) - torch.log(beta) / (GAMMA - 1))
        ut, un = u1 * ny - u2 * nx, u1 * nx + u2 * ny
        sb = torch.sqrt(beta)
        c = 0.5 / torch.sqrt(math.pi * beta)
        return (rho, ut, un, pbr, ut * ut + un * un, torch.exp(-(ut * sb) ** 2) * c,
                torch.exp(-(un * sb) ** 2) * c, torch.erf(ut * sb), torch.erf(un * sb))

    @staticmethod
    def split(s, sg, along_x):
        rho, ut, un, pbr, usq, B1, B2, e1, e2 = s
        u, o, B, e = (ut, un, B1, e1) if along_x else (un, ut, B2, e2)
        A, B = 0.5 * (1.0 + sg * e), sg * B
        G = [u * A + B, (pbr + u * u) * A + u * B, u * o * A + o * B,
             0.5 * u * (7.0 * pbr + usq) * A + 0.5 * (6.0 * pbr + usq) * B]
        G = [rho * f for f in G]
        return G if along_x else [G[0], G[2], G[1], G[3]]

    @staticmethod
    def quadrant(s, s1, s2):
        rho, ut, un, pbr, usq, B1, B2, e1, e2 = s
        A1, A2, B1, B2 = 0.5 * (1.0 + s1 * e1), 0.5 * (1.0 + s2 * e2), s1 * B1, s2 * B2
        a, b = ut * A1 + B1, un * A2 + B2
        return [rho * A2 * a, rho * A2 * ((pbr + ut * ut) * A1 + ut * B1), rho * a * b,
                rho * A2 * (0.5 * ut * (7.0 * pbr + usq) * A1 + 0.5 * (6.0 * pbr + usq) * B1)
                + 0.5 * rho * un * B2 * a]

    def flux_residual(self, x, y, q, g, qmax, qmin, delta):
        k = self.k
        dx, dy, _, w = self.geometry(x, y)
        nx, ny = self.normals(x, y)
        nx, ny = nx[:, None], ny[:, None]
        own, nbr = [], []
        for c in range(4):
            own.append(self.limited(q[c][:, None], g[c][0][:, None], g[c][1][:, None],
                                    qmax[c][:, None], qmin[c][:, None], self.eps2[:, None],
                                    dx, dy))
            nbr.append(self.limited(q[c][k], g[c][0][k], g[c][1][k], qmax[c][k], qmin[c][k],
                                    self.eps2[k], dx, dy))
        si, sk = self.maxwell(own, nx, ny), self.maxwell(nbr, nx, ny)
        dels, deln = dx * ny - dy * nx, dx * nx + dy * ny
        bnd = (self.wall | self.outer)
        s2 = torch.where(self.wall, -1.0, 1.0)[bnd][:, None]
        sib, skb = ([a[bnd] for a in s] for s in (si, sk))
        skip = {2: self.wall, 3: self.outer}
        total = [0.0] * 4
        for L, member in enumerate(self.lists):
            sg = 1.0 if L % 2 == 0 else -1.0
            f = [b - a for a, b in zip(self.split(si, sg, L < 2), self.split(sk, sg, L < 2))]
            if L < 2:
                fb = [b - a for a, b in zip(self.quadrant(sib, sg, s2),
                                            self.quadrant(skb, sg, s2))]
                f = [a.index_put((bnd,), b) for a, b in zip(f, fb)]
            use = member if L < 2 else member & ~skip[L][:, None]
            wl = torch.where(use, w, 0.0)
            if L >= 2:  # a list the point does not have: any regular system
                wl = torch.where(skip[L][:, None], w, wl)
            d = self.solve(dels, deln, wl, f)
            for c in range(4):
                part = d[c][0 if L < 2 else 1]
                total[c] = total[c] + (part if L < 2 else torch.where(skip[L], 0.0, part))
        fac = delta * torch.where(self.wall, 2.0, 1.0)
        return [fac * a for a in total]

    @staticmethod
    def conserved(P, nx, ny):
        rho, u1, u2, pr = P
        return [rho, rho * (u1 * ny - u2 * nx), rho * (u1 * nx + u2 * ny),
                2.5 * pr + 0.5 * rho * (u1 * u1 + u2 * u2)]

    def far_field(self, P, nx, ny):
        def half(rho, u1, u2, pr, sg):
            ut, un = u1 * ny - u2 * nx, u1 * nx + u2 * ny
            beta = 0.5 * rho / pr
            e = pr / (rho * (GAMMA - 1)) + 0.5 * (ut * ut + un * un)
            S = un * torch.sqrt(beta)
            B = sg * torch.exp(-S * S) / (2.0 * torch.sqrt(math.pi * beta))
            A = 0.5 * (1.0 + sg * torch.erf(S))
            return [rho * A, rho * ut * A, rho * (un * A + B), rho * A * e + 0.5 * rho * un * B]
        one = torch.ones_like(P[0])
        t = math.radians(self.flow["aoa"])
        M = self.flow["mach"]
        inf = half(one, M * math.cos(t) * one, M * math.sin(t) * one, PR_INF * one, -1.0)
        return [a + b for a, b in zip(inf, half(*P, 1.0))]

    def to_state(self, P, nx, ny):
        U, V = self.conserved(P, nx, ny), self.far_field(P, nx, ny)
        return [torch.where(self.outer, b, a) for a, b in zip(U, V)]

    def stage(self, rk, euler, x, y, delta, P, O):
        dx, dy, _, w = self.geometry(x, y)
        P, O = list(P.unbind(0)), list(O.unbind(0))
        q = self.q_of(P)
        k, v = self.k, self.valid
        qk = [a[k] for a in q]
        qmax = [torch.where(v, b, a[:, None]).max(1).values.maximum(a) for a, b in zip(q, qk)]
        qmin = [torch.where(v, b, a[:, None]).min(1).values.minimum(a) for a, b in zip(q, qk)]
        g = self.solve(dx, dy, w, [b - a[:, None] for a, b in zip(q, qk)])
        for _ in range(self.flow["inner_iterations"]):
            df = [(qk[c] - 0.5 * (dx * g[c][0][k] + dy * g[c][1][k]))
                  - (q[c][:, None] - 0.5 * (dx * g[c][0][:, None] + dy * g[c][1][:, None]))
                  for c in range(4)]
            g = self.solve(dx, dy, w, df)
        fr = self.flux_residual(x, y, q, g, qmax, qmin, delta)
        nx, ny = self.normals(x, y)
        U = self.to_state(P, nx, ny)
        before = U[0]
        if rk == 3:
            Uo = self.to_state(O, nx, ny)
            U = [2.0 / 3.0 * o + 1.0 / 3.0 * (a - 0.5 * f) for a, o, f in zip(U, Uo, fr)]
        else:
            U = [a - 0.5 * euler * f for a, f in zip(U, fr)]
        U[2] = torch.where(self.wall, 0.0, U[2])
        m1, m2 = U[1] * ny + U[2] * nx, U[2] * ny - U[1] * nx
        res = torch.where(self.outer, 0.0, (U[0] - before) ** 2).sum()
        pr = 0.4 * (U[3] - 0.5 * (m1 * m1 + m2 * m2) / U[0])
        return torch.stack([U[0], m1 / U[0], m2 / U[0], pr]), res

    def loop(self, x, y, P, iters, keep=False):
        """(final state, residue history); keep: for a gradient (recomputed stages)."""
        first = self.flow["tscheme"] == "first"
        stages, euler = (1, 2.0) if first else (4, 1.0)
        hist, old = [], None
        for it in range(1, iters + 1):
            delta = self.delta(list(P.unbind(0)), self.geometry(x, y)[2])
            O = P
            for rk in range(1, stages + 1):
                if keep:
                    P, res = checkpoint(self.stage, rk, euler, x, y, delta, P, O,
                                        use_reentrant=False)
                else:
                    P, res = self.stage(rk, euler, x, y, delta, P, O)
            norm = torch.sqrt(res.detach()) / self.n
            old = norm if it <= 2 else old
            hist.append(torch.log10(norm / old))
        return P, torch.stack(hist)

    def forces(self, x, y, P):
        """(Cl, Cd, Cm) per shape and cp per shape point."""
        m, l, r = self.shp, self.sl, self.sr
        nx, ny = (a[m] for a in self.normals(x, y))
        seg = lambda a, b: torch.sqrt((x[a] - x[b]) ** 2 + (y[a] - y[b]) ** 2)  # noqa: E731
        ds = 0.5 * (seg(m, l) + seg(r, m))
        cp = -(P[3][m] - PR_INF) / (0.5 * self.flow["mach"] ** 2)
        add = lambda v: torch.zeros(self.shapes, dtype=v.dtype, device=v.device).index_add(  # noqa: E731
            0, self.shape, v)
        H, V = add(cp * nx * ds), add(cp * ny * ds)
        M = add(cp * ds * (nx * y[m] - ny * (x[m] - 0.25)))
        t = math.radians(self.flow["aoa"])
        return V * math.cos(t) - H * math.sin(t), H * math.cos(t) + V * math.sin(t), M, cp


def _exact_primal(g, flow, prim, iters, device):
    with torch.no_grad():
        p = _Plain(g, flow, device)
        P, hist = p.loop(p.x, p.y, torch.as_tensor(prim.T.copy(), device=device), iters)
        return (hist.cpu().numpy(), P.T.contiguous().cpu().numpy(),
                torch.cat(p.forces(p.x, p.y, P)).cpu().numpy())


def exact(case, seed):
    if not torch.cuda.is_available() and case["work"] != "batch" and case["ni"] * case["nj"] > 2e4:
        return None  # minutes on the host
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    grids, flows, states = _inputs(case, seed)
    if case["work"] == "batch":
        got = [_exact_primal(g, f, s, case["iters"], device)
               for g, f, s in zip(grids, flows, states)]
        return dict(iters=None, residue=np.stack([a for a, _, _ in got]),
                    prim=[b for _, b, _ in got], coeffs=[c for _, _, c in got])
    g, flow, prim = grids[0], flows[0], states[0]
    if case["work"] == "primal":
        residue, prim, coeffs = _exact_primal(g, flow, prim, case["iters"], device)
        return dict(residue=residue, prim=prim, coeffs=coeffs)
    p = _Plain(g, flow, device)
    x, y = p.x.requires_grad_(), p.y.requires_grad_()
    P, _ = p.loop(x, y, torch.as_tensor(prim.T.copy(), device=device), case["iters"], keep=True)
    cl, cd, _, _ = p.forces(x, y, P)
    J = (cl if case["objective"] == "cl" else cd).sum()
    dx, dy = (a.cpu().numpy() for a in torch.autograd.grad(J, (x, y)))
    if case["work"] == "adjoint":
        return dict(J=J.item(), dx=dx, dy=dy)
    ex, ey = _direction(g, seed)
    return dict(J=J.item(), dJ=float(np.dot(dx, ex) + np.dot(dy, ey)))
