"""Measured cases of the BSSN framework: what a program that evolves black-hole
space-times has it do, through the public entry points.

Kinds of work (``case["kind"]``):

* ``rhs``         ``BSSNSolver.rhs_dict``: one right-hand side, {field: d/dt}
* ``step``        ``BSSNEvolution.step``: one RK4 step (KO order 6 or 8, free
                  or periodic boundary)
* ``graph``       the captured RK4 step of ``BSSNEvolution.capture``, replayed
* ``msrk``        ``BSSNEvolution.msrk_step``: one 2-step / 3-stage MSRK step
* ``constraints`` ``ConstraintSolver``: H and M_i on the grid and their norms
* ``derivs``      ``fused_rhs.derivatives``: the derivative bundle with KO sums
* ``ozaki``       ``OzakiDerivatives.rhs``: the RHS on INT8 tensor-core derivatives
* ``amr``         ``BatchedEvolution``: the captured RK4 step of a block list
* ``amr_ozaki``   ``BatchedOzakiEvolution``: the same through the INT8 path

Inputs are states in the middle of an evolution: two punctures whose chi and
lapse carry smooth waves, a metric of unit determinant near delta_ij, and
waves of about 2 % in K, shift, A~, Gamma~ and B, all made on the GPU from the
seed. Periodic cases have waves of whole periods and no punctures.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import torch

_ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(_ROOT / "integer-schemes_b200"))

from bssn3d_b200 import amr  # noqa: E402
from bssn3d_b200.constraints import ConstraintSolver  # noqa: E402
from bssn3d_b200.evolve import BSSNEvolution  # noqa: E402
from bssn3d_b200.fused_rhs import derivatives, device_scalars, pack_S  # noqa: E402
from bssn3d_b200.grid import Grid  # noqa: E402
from bssn3d_b200.ozaki import BatchedOzakiEvolution, OzakiDerivatives  # noqa: E402
from bssn3d_b200.rhs import BSSNSolver  # noqa: E402
from bssn3d_b200.state import BSSNState, PhysicsParams  # noqa: E402

F64 = torch.float64
SIGMA = 0.1          # Kreiss-Oliger strength of the repository's workloads
T0 = 0.75            # start time of a step (the lapse damping depends on it)


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------

def _grid_case(kind, n, ng=3, **more):
    nx, ny, nz = (n, n, n) if isinstance(n, int) else n
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, ng=ng, **more)


def listed():
    named = [
        # the smallest block the AMR workloads hold (16^3 interior): one RHS call
        ("rhs_16", _grid_case("rhs", 16)),
        # a ragged box with an odd z extent (53 + 6 = 59): no aligned rows
        ("rhs_ragged", _grid_case("rhs", (37, 70, 53))),
        # the 64^3 equal-mass workload, advanced by replaying the captured step
        ("graph_64", _grid_case("graph", 64, ko=6, bc="none")),
        # the headline workload: 128^3, q = 1/10, one RK4 step with KO6
        ("step_128", _grid_case("step", 128, ko=6, bc="none")),
        # BSSNEvolution's own defaults (periodic, KO order 8) on a box with odd extents
        ("step_periodic_ko8", _grid_case("step", (41, 48, 56), ng=4, ko=8, bc="periodic")),
        # the low-storage integrator, RK4-2(2)
        ("msrk_96", _grid_case("msrk", 96, ko=6, bc="none", method="rk4_2_2")),
        # constraint monitoring of the headline grid
        ("constraints_128", _grid_case("constraints", 128)),
        # the derivative bundle with KO sums, as an analysis program takes it
        ("derivs_80", _grid_case("derivs", 80, ko=6)),
        # the INT8 workload: 192^3, the smallest digit count that meets 1e-10
        ("ozaki_192", _grid_case("ozaki", 192, k=6)),
        # 600 blocks on 3 levels with ghost exchange, on the tuner's usual tile
        ("amr_600", dict(kind="amr", workload=3, count=600, ghosts="exchange", variant=2, ko=6)),
        # a short list of blocks that evolve their own ghosts, on the default tile
        ("amr_40_evolve", dict(kind="amr", workload=3, count=40, ghosts="evolve", variant=0, ko=6)),
        # part of the 5-level q = 1/100 list through the INT8 path
        ("amr_ozaki_120", dict(kind="amr_ozaki", workload=4, count=120, ghosts="exchange", k=7, ko=6)),
    ]
    return [dict(name=name, **c) for name, c in named]


def _size(rng, lo, hi):
    """An extent, even spread over its logarithm; odd ones as often as even ones."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "step", "step", "graph", "msrk", "constraints", "derivs", "ozaki",
                       "amr", "amr", "amr_ozaki"])
    if kind == "amr":
        return dict(kind=kind, workload=rng.choice([3, 4]), count=_size(rng, 12, 500),
                    ghosts=rng.choice(["exchange", "evolve"]), variant=rng.randrange(4), ko=rng.choice([6, 6, 8]))
    if kind == "amr_ozaki":
        return dict(kind=kind, workload=rng.choice([3, 4]), count=_size(rng, 12, 110),
                    ghosts=rng.choice(["exchange", "evolve"]), k=rng.randint(5, 8), ko=rng.choice([6, 6, 8]))
    base = _size(rng, 14, 118)
    n = tuple(max(9, int(base * math.exp(rng.uniform(-0.25, 0.08)))) for _ in range(3))
    if kind in ("rhs", "constraints"):
        return _grid_case(kind, n, ng=rng.choice([3, 3, 4]))
    if kind == "derivs":
        return _grid_case(kind, n, ng=4, ko=rng.choice([6, 8]))
    if kind == "ozaki":
        return _grid_case(kind, n, k=rng.randint(5, 8))
    ko = rng.choice([6, 6, 8])
    ng = 4 if ko == 8 else 3
    bc = rng.choice(["none", "none", "periodic"])
    if kind == "msrk":
        return _grid_case(kind, n, ng=ng, ko=ko, bc=bc, method=rng.choice(["rk4_2_1", "rk4_2_2"]))
    return _grid_case(kind, n, ng=ng, ko=ko, bc=bc)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _domain(case):
    """(lo, h) per axis: the repository's [-8, 8]^3, periodic cases on [-0.5, 0.5]^3."""
    L = 1.0 if case.get("bc") == "periodic" else 16.0
    n = (case["nx"], case["ny"], case["nz"])
    return [-0.5 * L] * 3, [L / m for m in n]


def _coords(case):
    lo, h = _domain(case)
    n, ng = (case["nx"], case["ny"], case["nz"]), case["ng"]
    return [(lo[a] + torch.arange(-ng, n[a] + ng, dtype=F64, device="cuda") * h[a])[None] for a in range(3)]


class _Data:
    """Smooth fields of position, drawn from a seed; evaluated on one grid or on
    a batch of blocks (coordinates (nb, n) per axis)."""

    def __init__(self, seed, periodic):
        g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
        u = lambda *s: torch.rand(*s, generator=g, dtype=F64)  # noqa: E731
        if periodic:
            k = 2.0 * math.pi * torch.randint(-2, 3, (24, 3, 3), generator=g).to(F64)
        else:
            k = 1.6 * u(24, 3, 3) - 0.8
        self.k, self.phase, self.amp = k.tolist(), (2 * math.pi * u(24, 3)).tolist(), (0.4 + 0.6 * u(24, 3)).tolist()
        self.periodic = periodic
        s = u(8).tolist()
        self.punctures = [] if periodic else [
            (0.85 + 0.1 * s[0], (-0.6 + 0.2 * s[1], 0.2 * s[2] - 0.1, 0.2 * s[3] - 0.1)),
            (0.08 + 0.02 * s[4], (4.9 + 0.2 * s[5], 0.2 * s[6] - 0.1, 0.2 * s[7] - 0.1))]

    def wave(self, f, x):
        out = 0.0
        for m in range(3):
            e = [torch.exp(1j * (self.k[f][m][a] * x[a])) for a in range(3)]
            e[0] = e[0] * complex(math.cos(self.phase[f][m]), math.sin(self.phase[f][m]))
            p = e[0][:, :, None, None] * e[1][:, None, :, None] * e[2][:, None, None, :]
            out = out + self.amp[f][m] * p.imag
        return out

    def state(self, x, h):
        """(nb, 24, Sx, Sy, Sz) on the coordinates x; h is the smallest resolved radius x 2."""
        nb, shape = x[0].shape[0], tuple(a.shape[1] for a in x)
        U = torch.empty((nb, 24) + shape, dtype=F64, device="cuda")
        psi = torch.ones((nb,) + shape, dtype=F64, device="cuda")
        for m, c in self.punctures:
            r = torch.sqrt(((x[0] - c[0]) ** 2)[:, :, None, None] + ((x[1] - c[1]) ** 2)[:, None, :, None]
                           + ((x[2] - c[2]) ** 2)[:, None, None, :])
            psi += m / (2.0 * torch.maximum(r, torch.as_tensor(0.5 * h, dtype=F64, device="cuda")))
        U[:, 0] = psi ** -2 * (1.0 + 0.02 * self.wave(0, x))
        U[:, 1] = psi ** -4 * (1.0 + 0.02 * self.wave(1, x))
        U[:, 2] = 0.02 * self.wave(2, x)
        for p in range(6):
            U[:, 3 + p] = (1.0 if p in (0, 3, 5) else 0.0) + 0.02 * self.wave(3 + p, x)
        for f in range(9, 24):
            U[:, f] = 0.02 * self.wave(f, x)
        g, A = [U[:, 3 + p] for p in range(6)], [U[:, 12 + p] for p in range(6)]
        det = (g[0] * (g[3] * g[5] - g[4] * g[4]) - g[1] * (g[1] * g[5] - g[4] * g[2])
               + g[2] * (g[1] * g[4] - g[3] * g[2]))
        U[:, 3:9] *= (det ** (-1.0 / 3.0))[:, None]
        iu = [g[3] * g[5] - g[4] * g[4], g[2] * g[4] - g[1] * g[5], g[1] * g[4] - g[2] * g[3],
              g[0] * g[5] - g[2] * g[2], g[1] * g[2] - g[0] * g[4], g[0] * g[3] - g[1] * g[1]]
        tr = (iu[0] * A[0] + iu[3] * A[3] + iu[5] * A[5] + 2.0 * (iu[1] * A[1] + iu[2] * A[2] + iu[4] * A[4])) / 3.0
        for p in range(6):
            A[p] -= tr * g[p]
        return U


def _grid_state(case, seed):
    _, h = _domain(case)
    return _Data(seed, case.get("bc") == "periodic").state(_coords(case), max(h))[0]


def _grid(case):
    lo, h = _domain(case)
    return Grid(Nx=case["nx"], Ny=case["ny"], Nz=case["nz"], dx=h[0], dy=h[1], dz=h[2], ng=case["ng"],
                xmin=lo[0], ymin=lo[1], zmin=lo[2])


def _dt(case):
    return 0.25 * min(_domain(case)[1])


def _before(U):
    """A state as one step earlier: the dynamic fields a little smaller."""
    V = U.clone()
    V[2] *= 0.95
    V[9:] *= 0.95
    return V


def _block_state(pool, seed):
    """The pooled state of a block list: the same smooth fields at every block's points."""
    data = _Data(seed, False)
    U = torch.empty(pool.size, dtype=F64, device="cuda")
    groups = {}
    for i, b in enumerate(pool.blocks):
        groups.setdefault(b.n, []).append(i)
    for ids in groups.values():
        for at in range(0, len(ids), 16):
            part = ids[at:at + 16]
            bl = [pool.blocks[i] for i in part]
            h = torch.tensor([b.h for b in bl], dtype=F64, device="cuda")
            s = torch.arange(-bl[0].ng, bl[0].n + bl[0].ng, dtype=F64, device="cuda")
            x = [torch.tensor([b.origin[a] for b in bl], dtype=F64, device="cuda")[:, None] + s[None] * h[:, None]
                 for a in range(3)]
            V = data.state(x, h[:, None, None, None])
            for j, i in enumerate(part):
                o = int(pool.offsets[i])
                U[o:o + V[j].numel()] = V[j].reshape(-1)
    return U


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("amr", "amr_ozaki"):
        blocks, _, dt = amr.workload(case["workload"], count=case["count"], ng=4 if case["ko"] == 8 else 3)
        pool = amr.BlockPool(blocks)
        U = _block_state(pool, seed)
        if kind == "amr":
            evo = amr.BatchedEvolution(pool, ko_sigma=SIGMA, ko_order=case["ko"], variant=case["variant"],
                                       ghosts=case["ghosts"])
        else:
            evo = BatchedOzakiEvolution(pool, k=case["k"], ko_sigma=SIGMA, ko_order=case["ko"],
                                        ghosts=case["ghosts"])
        g, U_g, S_g = evo.capture(U, evo.scalars(T0, dt))
        return dict(kind="graph", graph=g, U0=U, S0=S_g.clone(), U=U_g, S=S_g, evo=evo)
    U, grid = _grid_state(case, seed), _grid(case)
    st = dict(kind=kind, U=U, grid=grid, dt=_dt(case))
    if kind == "rhs":
        st["solver"] = BSSNSolver(grid, ko_order=2 * case["ng"], dt=st["dt"])
        st["state"] = BSSNState(U)
    elif kind in ("step", "graph", "msrk"):
        evo = BSSNEvolution(grid, ko_sigma=SIGMA, ko_order=case["ko"], bc=case["bc"],
                            integrator=case.get("method", "rk4"))
        st.update(evo=evo, state=BSSNState(U))
        if kind == "graph":
            S = device_scalars(_pack(grid, st["dt"]), "cuda")
            g, U_g, S_g = evo.capture(U, S)
            st.update(graph=g, U0=U, S0=S, U=U_g, S=S_g)
        if kind == "msrk":
            st["prev"] = evo.rhs(BSSNState(_before(U)), T0, st["dt"])      # f(y_{n-1})
    elif kind == "constraints":
        st.update(solver=ConstraintSolver(grid), state=BSSNState(U))
    elif kind == "derivs":
        st.update(S=device_scalars(_pack(grid, st["dt"]), "cuda"), ko=case["ko"])
    elif kind == "ozaki":
        st.update(S=device_scalars(_pack(grid, st["dt"]), "cuda"),
                  oz=OzakiDerivatives(tuple(U.shape[1:]), case["k"]))
    return st


def _pack(grid, dt):
    p = PhysicsParams()
    return pack_S(p.eta, p.cahd_c, dt, grid.dx, p.ssl_h, p.ssl_sigma, T0, p.lmbda, p.lambda_f, grid.dy, grid.dz)


def run(st):
    kind = st["kind"]
    if kind == "rhs":
        return st["solver"].rhs_dict(st["state"], T0, st["dt"])
    if kind == "step":
        return st["evo"].step(st["state"], T0, st["dt"]).data
    if kind == "graph":          # a host program's state into the captured step, which advances it in place
        st["U"].copy_(st["U0"])
        st["S"].copy_(st["S0"])
        st["graph"].replay()
        return st["U"]
    if kind == "msrk":
        a, b = st["evo"].msrk_step(st["state"], st["prev"], T0, st["dt"])
        return a.data, b.data
    if kind == "constraints":
        return st["solver"].constraints(st["state"]), st["solver"].l2_tensor(st["state"])
    if kind == "derivs":
        return derivatives(st["U"], st["S"], ko_sigma=SIGMA, ko_order=st["ko"])
    return st["oz"].rhs(st["U"], st["S"])


# --------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# --------------------------------------------------------------------------

RHS_FLOPS = 6714     # algebra 4,278 and derivatives 2,436 per point
KO_FLOPS = 936       # 24 fields x 3 axes, 7 taps


def _points(case):
    """(points evaluated, points held) of one pass over the state."""
    if "workload" in case:
        ng = 4 if case["ko"] == 8 else 3
        blocks, _, _ = amr.workload(case["workload"], count=case["count"], ng=ng)
        held = sum(b.points for b in blocks)
        return (sum(b.interior_points for b in blocks) if case["ghosts"] == "exchange" else held), held
    n = math.prod(case[k] + 2 * case["ng"] for k in ("nx", "ny", "nz"))
    return n, n


def work(case):
    kind, (n, held) = case["kind"], _points(case)
    if kind in ("rhs", "ozaki"):
        return {"bytes": 48 * 8 * n, "flops": RHS_FLOPS * n}
    if kind == "constraints":
        return {"bytes": 28 * 8 * n, "flops": 2 * 5000 * n}
    if kind == "derivs":
        return {"bytes": (24 + 162) * 8 * n, "flops": (2436 + KO_FLOPS) * n}
    if kind == "msrk":
        return {"bytes": 96 * 8 * n, "flops": 3 * (RHS_FLOPS + KO_FLOPS) * n}
    return {"bytes": 48 * 8 * held, "flops": 4 * (RHS_FLOPS + KO_FLOPS) * n}


# (rel, max) = four times what the path was seen to differ from ``exact`` by, over
# sizes to 192^3: rounding of second derivatives (eps / h^2), times dt in a step.
# INT8 derivatives: k digits of 7 bits carry a field to 2^-7k of its largest value
# in a line, so each digit takes a factor 128 until float64 rounding is reached.
_TOL = {"rhs": (4e-12, 2e-11), "constraints": (4e-12, 2e-11), "derivs": (8e-13, 1.2e-11), "msrk": (6e-13, 8e-12),
        "step": (2e-14, 4e-13), "graph": (2e-14, 4e-13), "amr": (2e-14, 1e-12)}
_TOL_K = {5: (7e-7, 8e-6), 6: (6e-9, 6e-8), 7: (5e-11, 5e-10), 8: (2e-12, 2e-11)}


def tolerance(case):
    if case["kind"] == "ozaki":
        rel, most = _TOL_K[case["k"]]
    elif case["kind"] == "amr_ozaki":      # a step moves the state by dt x rate, dt <= 1/64
        rel, most = (max(a, b / 64.0) for a, b in zip(_TOL["amr"], _TOL_K[case["k"]]))
    else:
        rel, most = _TOL[case["kind"]]
    return {"rel": rel, "max": most}


# --------------------------------------------------------------------------
# the same in plain torch float64
# --------------------------------------------------------------------------

_SYM = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
_PAIR = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))
_W = (1.0, 2.0, 2.0, 1.0, 2.0, 1.0)


def _taps(u, axis, coef):
    """sum_k c_k u[i + k] along axis, the index clamped at the array's ends."""
    n = u.shape[axis]
    i = torch.arange(n, device=u.device)
    out = None
    for k, c in coef:
        v = c * u.index_select(axis, (i + k).clamp(0, n - 1))
        out = v if out is None else out + v
    return out


_C1 = [(-3, -1.0), (-2, 9.0), (-1, -45.0), (1, 45.0), (2, -9.0), (3, 1.0)]
_C2 = [(-3, 2.0), (-2, -27.0), (-1, 270.0), (0, -490.0), (1, 270.0), (2, -27.0), (3, 2.0)]
_K6 = [(-3, 1.0), (-2, -6.0), (-1, 15.0), (0, -20.0), (1, 15.0), (2, -6.0), (3, 1.0)]
_K8 = [(-4, -1.0), (-3, 8.0), (-2, -28.0), (-1, 56.0), (0, -70.0), (1, 56.0), (2, -28.0), (3, 8.0), (4, -1.0)]


def _d(u, a, h):
    return _taps(u, a, _C1) / (60.0 * h[a])


def _grad(u, h):
    return [_d(u, a, h) for a in range(3)]


def _hess(u, h, d=None):
    d = _grad(u, h) if d is None else d
    return [_taps(u, i, _C2) / (180.0 * h[i] * h[i]) if i == j else _d(d[i], j, h) for i, j in _PAIR]


def _diss(u, h, order):
    c, den = (_K6, 64.0) if order == 6 else (_K8, 256.0)
    return sum(_taps(u, a, c) * (SIGMA / (den * h[a])) for a in range(3))


def _geometry(U, h):
    """Inverse metric, Christoffel symbols, chi's gradient and the Ricci tensor."""
    chi, g, b3 = U[1], [U[3 + p] for p in range(6)], U[18:21]
    G = lambda i, j: g[_SYM[i][j]]  # noqa: E731
    c = [g[3] * g[5] - g[4] * g[4], g[2] * g[4] - g[1] * g[5], g[1] * g[4] - g[2] * g[3],
         g[0] * g[5] - g[2] * g[2], g[1] * g[2] - g[0] * g[4], g[0] * g[3] - g[1] * g[1]]
    det = g[0] * c[0] + g[1] * c[1] + g[2] * c[2]
    gu = [x / det for x in c]
    Gu = lambda i, j: gu[_SYM[i][j]]  # noqa: E731
    dg, R = [], []
    for p in range(6):
        d = _grad(g[p], h)
        dg.append(d)
        R.append(-0.5 * sum(_W[q] * gu[q] * x for q, x in enumerate(_hess(g[p], h, d))))
    D = lambda a, i, j: dg[_SYM[i][j]][a]  # noqa: E731
    C1 = [[0.5 * (D(i, k, j) + D(j, k, i) - D(k, i, j)) for i, j in _PAIR] for k in range(3)]
    C2 = [[sum(Gu(k, m) * C1[m][p] for m in range(3)) for p in range(6)] for k in range(3)]
    cal = [sum(_W[p] * gu[p] * C2[k][p] for p in range(6)) for k in range(3)]
    dG = [_grad(b3[k], h) for k in range(3)]
    W = [[[sum(Gu(m, n) * C1[j][_SYM[k][n]] for n in range(3)) for m in range(3)] for k in range(3)]
         for j in range(3)]
    for p, (i, j) in enumerate(_PAIR):
        R[p] = R[p] + 0.5 * sum(G(k, i) * dG[k][j] + G(k, j) * dG[k][i]
                                + cal[k] * (C1[i][_SYM[j][k]] + C1[j][_SYM[i][k]]) for k in range(3))
        for k in range(3):
            for m in range(3):
                R[p] = R[p] + (C2[k][_SYM[m][i]] * W[j][k][m] + C2[k][_SYM[m][j]] * W[i][k][m]
                               + C2[k][_SYM[i][m]] * W[k][j][m])
    del W, C1
    dchi = _grad(chi, h)
    Dchi = [x - sum(C2[k][p] * dchi[k] for k in range(3)) for p, x in enumerate(_hess(chi, h, dchi))]
    lap = sum(_W[p] * gu[p] * Dchi[p] for p in range(6))
    sq = sum(Gu(i, j) * dchi[i] * dchi[j] for i in range(3) for j in range(3))
    for p, (i, j) in enumerate(_PAIR):
        R[p] = R[p] + (Dchi[p] + g[p] * lap) / (2.0 * chi) - (dchi[i] * dchi[j] + 3.0 * g[p] * sq) / (4.0 * chi * chi)
    A = [U[12 + p] for p in range(6)]
    M = [[sum(A[_SYM[i][k]] * Gu(k, j) for k in range(3)) for j in range(3)] for i in range(3)]
    AU = [sum(Gu(i, k) * M[k][j] for k in range(3)) for i, j in _PAIR]
    AA = sum(_W[p] * A[p] * AU[p] for p in range(6))
    H = chi * sum(_W[p] * gu[p] * R[p] for p in range(6)) + (2.0 / 3.0) * U[2] * U[2] - AA
    return dict(g=g, gu=gu, C2=C2, cal=cal, dG=dG, R=R, dchi=dchi, A=A, M=M, AU=AU, AA=AA, H=H)


def _rhs(U, t, dt, h, ko=0):
    """The 24 rates (CAHD + SSL), with Kreiss-Oliger sums of order ``ko`` if given."""
    P = PhysicsParams()
    q = _geometry(U, h)
    g, gu, C2, cal, dG, R, dchi, A, M, AU, AA, H = (q[k] for k in (
        "g", "gu", "C2", "cal", "dG", "R", "dchi", "A", "M", "AU", "AA", "H"))
    Gu = lambda i, j: gu[_SYM[i][j]]  # noqa: E731
    al, chi, K, be, B = U[0], U[1], U[2], U[9:12], U[21:24]
    adv = lambda d: be[0] * d[0] + be[1] * d[1] + be[2] * d[2]  # noqa: E731
    out = torch.empty_like(U)
    dal = _grad(al, h)
    gca = sum(Gu(i, j) * dchi[i] * dal[j] for i in range(3) for j in range(3))
    dda = [x - sum(C2[k][p] * dal[k] for k in range(3))
           + (dal[i] * dchi[j] + dal[j] * dchi[i] - g[p] * gca) / (2.0 * chi)
           for (p, (i, j)), x in zip(enumerate(_PAIR), _hess(al, h, dal))]
    X = [al * R[p] - dda[p] for p in range(6)]
    trX = sum(_W[p] * gu[p] * X[p] for p in range(6))
    lapa = sum(_W[p] * gu[p] * dda[p] for p in range(6))
    del dda
    db = [_grad(be[k], h) for k in range(3)]
    div = db[0][0] + db[1][1] + db[2][2]
    ddb = [_hess(be[k], h, db[k]) for k in range(3)]
    dd = [sum(ddb[k][_SYM[j][k]] for k in range(3)) for j in range(3)]
    lapb = [sum(_W[p] * gu[p] * ddb[k][p] for p in range(6)) for k in range(3)]
    del ddb
    dK = _grad(K, h)
    sq = torch.sqrt(chi)
    out[0] = (P.lmbda[0] * adv(dal) - 2.0 * al * K
              - sq * P.ssl_h * (al - sq) * math.exp(-0.5 * t * t / P.ssl_sigma ** 2))
    dx2 = h[0] * h[0]
    out[1] = (adv(dchi) + (2.0 / 3.0) * chi * (al * K - div)
              + P.cahd_c * dx2 * chi * H / (dt * (10.0 * dx2 + 1.0)))
    out[2] = adv(dK) - chi * lapa + al * (K * K / 3.0 + AA)
    for p, (i, j) in enumerate(_PAIR):
        out[3 + p] = (adv(_grad(g[p], h)) - (2.0 / 3.0) * g[p] * div - 2.0 * al * A[p]
                      + sum(g[_SYM[i][k]] * db[k][j] + g[_SYM[j][k]] * db[k][i] for k in range(3)))
        aga = sum(M[i][k] * A[_SYM[k][j]] for k in range(3))
        out[12 + p] = (adv(_grad(A[p], h)) - (2.0 / 3.0) * A[p] * div
                       + sum(A[_SYM[i][k]] * db[k][j] + A[_SYM[j][k]] * db[k][i] for k in range(3))
                       + chi * (X[p] - g[p] * trX / 3.0) + al * (K * A[p] - 2.0 * aga))
    for i in range(3):
        out[9 + i] = P.lmbda[1] * adv(db[i]) + 0.75 * (P.lambda_f[0] + P.lambda_f[1] * al) * B[i]
        aG = adv(dG[i])
        v = (aG - sum(cal[j] * db[i][j] for j in range(3)) + (2.0 / 3.0) * cal[i] * div + lapb[i]
             + sum(Gu(i, j) * dd[j] for j in range(3)) / 3.0
             - sum(AU[_SYM[i][j]] * (2.0 * dal[j] + 3.0 * al * dchi[j] / chi) for j in range(3))
             - (4.0 / 3.0) * al * sum(Gu(i, j) * dK[j] for j in range(3))
             + 2.0 * al * sum(_W[p] * C2[i][p] * AU[p] for p in range(6)))
        out[18 + i] = v
        out[21 + i] = v - P.eta * B[i] + P.lmbda[2] * adv(_grad(B[i], h)) - P.lmbda[3] * aG
    if ko:
        for f in range(24):
            out[f] += _diss(U[f], h, ko)
    return out


def _enforce(U):
    P = PhysicsParams()
    U = U.clone()
    g, A = [U[3 + p] for p in range(6)], [U[12 + p] for p in range(6)]
    det = (g[0] * (g[3] * g[5] - g[4] * g[4]) - g[1] * (g[1] * g[5] - g[4] * g[2])
           + g[2] * (g[1] * g[4] - g[3] * g[2]))
    U[3:9] *= (det ** (-1.0 / 3.0))[None]
    iu = [g[3] * g[5] - g[4] * g[4], g[2] * g[4] - g[1] * g[5], g[1] * g[4] - g[2] * g[3],
          g[0] * g[5] - g[2] * g[2], g[1] * g[2] - g[0] * g[4], g[0] * g[3] - g[1] * g[1]]
    tr = sum(_W[p] * iu[p] * A[p] for p in range(6)) / 3.0
    for p in range(6):
        A[p] -= tr * g[p]
    U[1].clamp_(min=P.chi_floor)
    U[0].clamp_(min=P.alpha_floor)
    return U


def _synced(U, case):
    if case.get("bc") != "periodic":
        return U
    U, ng = U.clone(), case["ng"]
    for a in (1, 2, 3):
        n = U.shape[a]
        U.narrow(a, 0, ng).copy_(U.narrow(a, n - 2 * ng, ng).clone())
        U.narrow(a, n - ng, ng).copy_(U.narrow(a, ng, ng).clone())
    return U


def exact(case, seed):
    kind = case["kind"]
    if kind in ("amr", "amr_ozaki"):
        return None      # hundreds of blocks and their ghost fills: minutes in plain torch
    U, (_, h), dt = _grid_state(case, seed), _domain(case), _dt(case)
    f = lambda y, t: _rhs(_synced(y, case), t, dt, h, case["ko"])  # noqa: E731
    if kind in ("rhs", "ozaki"):
        V = _rhs(U, T0, dt, h)
        if kind == "ozaki":
            return V
        names = ["alpha", "chi", "K"] + ["gt%d" % p for p in range(6)] + ["beta%d" % i for i in range(3)] \
            + ["At%d" % p for p in range(6)] + ["Gt%d" % i for i in range(3)] + ["B%d" % i for i in range(3)]
        return {n: V[k] for k, n in enumerate(names)}
    if kind in ("step", "graph"):
        k = f(U, T0)
        acc = k
        for c, w in ((0.5, 2.0), (0.5, 2.0), (1.0, 1.0)):
            k = f(U + c * dt * k, T0 + c * dt)
            acc = acc + w * k
        return _enforce(U + (dt / 6.0) * acc)
    if kind == "msrk":
        a20, a21, a30, a31, a32, b0, b1, b2, b3 = _MSRK[case["method"]]
        k0 = f(_before(U), T0)
        k1 = f(U, T0)
        k2 = f(U + dt * (a20 * k0 + a21 * k1), T0 + (a20 + a21) * dt)
        k3 = f(U + dt * (a30 * k0 + a31 * k1 + a32 * k2), T0 + (a30 + a31 + a32) * dt)
        return _enforce(U + dt * (b0 * k0 + b1 * k1 + b2 * k2 + b3 * k3)), k1
    if kind == "constraints":
        q = _geometry(U, h)
        Gu = lambda i, j: q["gu"][_SYM[i][j]]  # noqa: E731
        A = lambda i, j: q["A"][_SYM[i][j]]  # noqa: E731
        dA, dK, m = [_grad(a, h) for a in q["A"]], _grad(U[2], h), []
        for i in range(3):
            v = -(2.0 / 3.0) * dK[i] - sum(U[18 + j] * A(i, j) for j in range(3))
            for j in range(3):
                for k in range(3):
                    v = v + Gu(j, k) * (dA[_SYM[k][i]][j] - 1.5 * A(k, i) * q["dchi"][j] / U[1]
                                        - sum(q["C2"][n][_SYM[j][i]] * A(k, n) for n in range(3)))
            m.append(v)
        g = case["ng"]
        cut = lambda x: x[g:-g, g:-g, g:-g]  # noqa: E731
        l2 = torch.stack([cut(q["H"]).square().mean().sqrt(), sum(cut(v).square() for v in m).mean().sqrt()])
        return {"H": q["H"], "M0": m[0], "M1": m[1], "M2": m[2]}, l2
    out = torch.empty((162,) + tuple(U.shape[1:]), dtype=F64, device=U.device)
    second = (0, 1, 3, 4, 5, 6, 7, 8, 9, 10, 11)
    for n in range(24):
        d = _grad(U[n], h)
        for a in range(3):
            out[3 * n + a] = d[a]
        if n in second:
            for p, x in enumerate(_hess(U[n], h, d)):
                out[72 + 6 * second.index(n) + p] = x
        out[138 + n] = _diss(U[n], h, case["ko"])
    return out


# (a20, a21, a30, a31, a32, b0..b3) of RK4-2(1) and RK4-2(2), arXiv:2603.05763, Table 1
_MSRK = {
    "rk4_2_1": (-49 / 1250, 399 / 1250, 7033 / 960000, -217633 / 210000, 5473 / 10752,
                -643 / 1536, -4237 / 1092, 38125 / 10752, 4375 / 2496),
    "rk4_2_2": (1309 / 15500, -31999 / 15500, -241289 / 5880000, 22846301 / 16170000, -936169 / 2587200,
                -191 / 882, 48241 / 59994, 193750 / 4351347, 100000 / 271791),
}
