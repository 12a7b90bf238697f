"""The work that a user of this library has it do, through its public entry
points (magudi_gb300.solver, magudi_gb300.configs), over the range of sizes
and options in use: per-call stepping of a host solver, whole gradient
evaluations (checkpointed and with the trajectory kept), forward, tangent and
batched runs, one block and several, 2D and 3D, Cartesian and curvilinear
grids, constant step size and constant CFL. Everything is FP64.

A case is a dict of plain values; `kind` names the entry points it goes
through, the rest are grid sizes, step counts and options. exact() restates
the single-block cases on far-field or periodic grids in plain torch (dense
SBP matrices, the discrete adjoint by automatic differentiation); the other
cases have no restatement here.
"""
import math

import numpy as np
import torch

from magudi_gb300 import capi, configs
from magudi_gb300.problem import quiescent_state
from magudi_gb300.solver import Batch, Solver

GAMMA = 1.4
RK = (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)


def listed():
    return [
        # a host solver's loop at the smallest grids: one RK4 step forward and
        # one adjoint step of a wall-bounded channel, one call per stage
        {"name": "percall_wall_41x33", "kind": "percall", "flow": "wall", "nx": 41, "ny": 33},
        # the same loop on the acoustic monopole grid of the benchmark
        {"name": "percall_monopole_201", "kind": "percall", "flow": "monopole", "nx": 201, "ny": 201},
        # the benchmark's gradient evaluation (201x201, checkpoints every 10
        # steps, recomputed beside the adjoint) over a quarter of its horizon
        {"name": "gradient_201", "kind": "gradient", "nx": 201, "ny": 201, "steps": 240, "save": 10,
         "resident": False, "curvilinear": False, "scheme": 0},
        # ragged sizes, trajectory kept on the device instead of recomputed
        {"name": "gradient_resident_151x113", "kind": "gradient", "nx": 151, "ny": 113, "steps": 120, "save": 12,
         "resident": True, "curvilinear": False, "scheme": 0},
        # small curvilinear grid with SBP 3-6, the scheme of the reference's examples
        {"name": "gradient_curvilinear_97x81", "kind": "gradient", "nx": 97, "ny": 81, "steps": 60, "save": 7,
         "resident": False, "curvilinear": True, "scheme": 3},
        # a larger 2D grid at constant CFL, forward only
        {"name": "forward_cfl_401x301", "kind": "forward", "nx": 401, "ny": 301, "steps": 40},
        # the gradient-check sweep: forward runs of instances of mixed grid sizes as one batch
        {"name": "sweep_16", "kind": "sweep", "instances": 16, "nmin": 65, "nmax": 201, "steps": 20},
        # two blocks across an interface
        {"name": "region_two_block", "kind": "region", "nx1": 101, "nx2": 89, "ny": 121, "steps": 40, "save": 8},
        # tangent run along a stored forward run
        {"name": "tangent_121x161", "kind": "tangent", "nx": 121, "ny": 161, "steps": 60, "save": 10},
        # 3D periodic Taylor-Green: forward and adjoint at constant CFL
        {"name": "tgv_gradient_64", "kind": "tgv", "n": 64, "steps": 6, "save": 3, "adjoint": True, "cfl": True},
        # the largest 3D grid here, forward at a constant step size
        {"name": "tgv_forward_144", "kind": "tgv", "n": 144, "steps": 4, "save": 4, "adjoint": False, "cfl": False},
        # the three-block curvilinear jet, forward and adjoint
        {"name": "jet_gradient", "kind": "jet", "nx": 96, "ny_core": 48, "ny_side": 43, "nz": 48, "steps": 4,
         "save": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["percall", "gradient", "gradient", "forward", "sweep", "region", "tangent", "tgv", "jet"])
    if kind == "percall":
        return {"kind": kind, "flow": rng.choice(["wall", "monopole"]), "nx": _log(rng, 41, 401),
                "ny": _log(rng, 33, 301)}
    if kind == "gradient":
        return {"kind": kind, "nx": _log(rng, 61, 301), "ny": _log(rng, 61, 251), "steps": rng.randint(20, 120),
                "save": rng.randint(4, 15), "resident": rng.random() < 0.4, "curvilinear": rng.random() < 0.3,
                "scheme": rng.choice([0, 0, 3])}
    if kind == "forward":
        return {"kind": kind, "nx": _log(rng, 81, 501), "ny": _log(rng, 81, 401), "steps": rng.randint(10, 40)}
    if kind == "sweep":
        return {"kind": kind, "instances": rng.randint(4, 24), "nmin": rng.randint(61, 91),
                "nmax": rng.randint(121, 201), "steps": rng.randint(6, 20)}
    if kind == "region":
        return {"kind": kind, "nx1": _log(rng, 41, 201), "nx2": _log(rng, 41, 201), "ny": _log(rng, 61, 201),
                "steps": rng.randint(10, 40), "save": rng.randint(3, 10)}
    if kind == "tangent":
        return {"kind": kind, "nx": _log(rng, 61, 201), "ny": _log(rng, 61, 201), "steps": rng.randint(20, 60),
                "save": rng.randint(5, 12)}
    if kind == "tgv":
        adjoint = rng.random() < 0.6
        return {"kind": kind, "n": _log(rng, 28, 80) if adjoint else _log(rng, 40, 128),
                "steps": rng.randint(2, 6) if adjoint else rng.randint(1, 4), "save": 3, "adjoint": adjoint,
                "cfl": rng.random() < 0.5}
    return {"kind": kind, "nx": rng.randint(40, 96), "ny_core": rng.randint(28, 48), "ny_side": rng.randint(28, 43),
            "nz": rng.randint(28, 48), "steps": rng.randint(2, 4), "save": 2}


# ---------------------------------------------------------------------------
# problems
# ---------------------------------------------------------------------------
def _monopole(nx, ny, curvilinear=False, scheme=0, cfl=None, controller=False, steps=10, save=10):
    """The acoustic monopole of configs.monopole_2d on the benchmark's domain
    (coarser grids keep the mesh width of 0.14 and cover less of it)."""
    half = 0.07 * (min(nx, ny) - 1)
    half = min(14.0, max(half, 4.2))
    P = configs.monopole_2d(n=nx, ny=ny, n_steps=steps, save_interval=save, half_width=half,
                            target_center=(0.0, 0.5 * half), mollifier_sigma=min(1.0, half / 8.0),
                            sponge_points=max(6, min(20, min(nx, ny) // 8)), dt=0.02, cfl=cfl,
                            controller_switch=controller)
    P.options.discretization_scheme = scheme
    if curvilinear:
        P.options.curvilinear = True
        x, y = P.blocks[0].coordinates
        k = math.pi / half
        a = 0.04 * half
        P.blocks[0].coordinates = np.ascontiguousarray(
            np.stack([x + a * np.sin(k * x) * np.sin(k * y), y + a * np.sin(k * y) * np.sin(0.5 * k * x)]))
    return P


def _problem(case):
    k = case["kind"]
    if k == "percall" and case["flow"] == "wall":
        return configs.wall_channel_2d(n=case["nx"], ny=case["ny"])
    if k == "percall":
        return _monopole(case["nx"], case["ny"])
    if k == "gradient":
        return _monopole(case["nx"], case["ny"], case["curvilinear"], case["scheme"], steps=case["steps"],
                         save=case["save"])
    if k == "forward":
        return _monopole(case["nx"], case["ny"], cfl=0.5, steps=case["steps"], save=case["steps"])
    if k == "tangent":
        return _monopole(case["nx"], case["ny"], controller=True, steps=case["steps"], save=case["save"])
    if k == "region":
        return configs.two_block_2d(nx1=case["nx1"], nx2=case["nx2"], ny=case["ny"], n_steps=case["steps"],
                                    functional=True, sponge_points=8)
    if k == "tgv":
        n = case["n"]
        return configs.taylor_green_3d(n=n, n_steps=case["steps"], save_interval=case["save"],
                                       dt=None if case["cfl"] else 0.5 / n)
    return configs.jet_3block_3d(nx=case["nx"], ny_core=case["ny_core"], ny_side=case["ny_side"], nz=case["nz"],
                                 n_steps=case["steps"], save_interval=case["save"])


def _sweep_sizes(case):
    m = case["instances"]
    return [case["nmin"] + ((case["nmax"] - case["nmin"]) * k) // max(1, m - 1) for k in range(m)]


def _perturbed(block, nD, rng, base, amplitude):
    """base plus a smooth disturbance: random waves in density, velocity and pressure."""
    xs = block.coordinates
    span = [float(x.max() - x.min()) for x in xs]
    periodic = block.periodicity_type[0] != 0

    def wave():
        s = np.zeros(block.n_points)
        for _ in range(2):
            arg = rng.uniform(0.0, 2.0 * np.pi)
            for d in range(nD):
                kd = rng.integers(1, 4) * (1.0 if periodic else 2.0 * np.pi / span[d])
                arg = arg + kd * xs[d]
            s += np.sin(arg)
        return 0.5 * amplitude * s

    rho0 = base[0]
    u0 = [base[1 + d] / rho0 for d in range(nD)]
    p0 = (GAMMA - 1.0) * (base[nD + 1] - 0.5 * rho0 * sum(u * u for u in u0))
    rho = rho0 * (1.0 + wave())
    u = [u0[d] + wave() for d in range(nD)]
    p = p0 * (1.0 + wave())
    q = np.empty((nD + 2, block.n_points))
    q[0] = rho
    for d in range(nD):
        q[1 + d] = rho * u[d]
    q[nD + 1] = p / (GAMMA - 1.0) + 0.5 * rho * sum(x * x for x in u)
    return q


def _states(P, seed, amplitude=1e-3):
    rng = np.random.default_rng(seed)
    nD = P.options.n_dimensions
    return [_perturbed(b, nD, rng, b.initial_state, amplitude) for b in P.blocks]


def _adjoint_state(P, seed):
    """A smooth adjoint field, as a run leaves it some steps from its end."""
    rng = np.random.default_rng(seed + 7)
    b, nD = P.blocks[0], P.options.n_dimensions
    lam = _perturbed(b, nD, rng, quiescent_state(b.n_points, nD, GAMMA), 1e-2)
    return lam - quiescent_state(b.n_points, nD, GAMMA)


def _forcing(n_rows, P, seed, amplitude=1e-3):
    """Control forcing rows: a smooth signal in time and space."""
    rng = np.random.default_rng(seed + 3)
    t = np.arange(n_rows)[:, None] / 40.0
    x = np.arange(P)[None, :] / max(1, P)
    a, b, c = rng.uniform(0.0, 2.0 * np.pi, 3)
    return amplitude * np.sin(t + a) * (1.0 + 0.5 * np.cos(6.0 * x + b)) + 0.3 * amplitude * np.cos(3.0 * t + c)


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "sweep":
        solvers, states = [], []
        for k, n in enumerate(_sweep_sizes(case)):
            P = _monopole(n, n, controller=True, steps=case["steps"], save=case["steps"])
            s = Solver(P)
            s.set_control_forcing(_forcing(4 * case["steps"], s.actuator_points(), seed + 100 * k))
            solvers.append(s)
            states.append(_states(P, seed + 100 * k)[0])
        return {"case": case, "batch": Batch(solvers), "solvers": solvers, "states": states}
    P = _problem(case)
    st = {"case": case, "problem": P, "states": _states(P, seed)}
    s = st["solver"] = Solver(P)
    if case["kind"] == "percall":
        st["adjoint"] = _adjoint_state(P, seed)
    if case["kind"] == "tangent":
        st["delta"] = _forcing(4 * case["steps"], s.actuator_points(), seed)
        st["perturbation"] = _adjoint_state(P, seed)
    if case["kind"] == "tangent" or case.get("resident"):
        s.set_trajectory_storage(True)
    return st


def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "sweep":
        for s, q in zip(st["solvers"], st["states"]):
            s.set_field(1, capi.FIELD_CONSERVED, q)
        costs = st["batch"].run_forward(case["steps"])
        return {"costs": costs, "q": [s.get_field(1, capi.FIELD_CONSERVED) for s in st["solvers"]]}
    s, P = st["solver"], st["problem"]
    for bi, q in enumerate(st["states"], start=1):
        s.set_field(bi, capi.FIELD_CONSERVED, q)
    if k == "percall":
        dt = P.options.time_step_size
        s.update_state()
        t, values = 0.0, []
        for i in range(1, 5):
            t = s.rk4_substep(capi.FORWARD, t, dt, i)
            if P.options.enable_functional:
                values.append(s.functional())
        q = s.get_field(1, capi.FIELD_CONSERVED)
        s.set_field(1, capi.FIELD_ADJOINT, st["adjoint"])
        if P.options.enable_functional:
            s.update_adjoint_forcing(False)
        for i in range(4, 0, -1):
            t = s.rk4_substep(capi.ADJOINT, t, dt, i)
        return {"q": q, "J": np.array(values), "lam": s.get_field(1, capi.FIELD_ADJOINT)}
    n = case["steps"]
    out = {"J": np.array([s.run_forward(n, case.get("save", n))])}
    if k == "forward" or (k == "tgv" and not case["adjoint"]):
        out["q"] = s.get_field(1, capi.FIELD_CONSERVED)
        return out
    if k == "tangent":
        s.set_field(1, capi.FIELD_ADJOINT, st["perturbation"])
        out["dJ"] = np.array([s.run_linearized(st["delta"])])
        out["dq"] = s.get_field(1, capi.FIELD_ADJOINT)
        return out
    out["sensitivity"] = np.array([s.run_adjoint()])
    if s.actuator_points():
        out["gradient"] = s.gradient(4 * n)
    out["lam"] = [s.get_field(bi, capi.FIELD_ADJOINT) for bi in range(1, len(P.blocks) + 1)]
    return out


def work(case):
    """Compulsory array traffic of the fused RK4 stages (200 bytes a point in
    2D, 280 in 3D forward; 232 and 320 adjoint) and the operation list of the
    RHS (407 and 700 a point forward, 1073 and 2000 adjoint), over the stages
    that a pass cannot do without (no recomputation)."""
    k = case["kind"]
    three = k in ("tgv", "jet")
    if k == "sweep":
        points, steps, adj = sum(n * n for n in _sweep_sizes(case)), case["steps"], 0
    elif k == "region":
        points, steps, adj = (case["nx1"] + case["nx2"]) * case["ny"], case["steps"], 1
    elif k == "tgv":
        points, steps, adj = case["n"] ** 3, case["steps"], int(case["adjoint"])
    elif k == "jet":
        points = case["nx"] * case["nz"] * (case["ny_core"] + 2 * case["ny_side"])
        steps, adj = case["steps"], 1
    else:
        points, steps = case["nx"] * case["ny"], case.get("steps", 1)
        adj = int(k in ("percall", "gradient", "tangent"))
    fb, ab, ff, af = (280, 320, 700, 2000) if three else (200, 232, 407, 1073)
    stages = 4 * steps * points
    return {"bytes": float(stages * (fb + adj * ab)), "flops": float(stages * (ff + adj * af))}


# ---------------------------------------------------------------------------
# restatement in plain torch
# ---------------------------------------------------------------------------
def _sbp48(n):
    """Dense SBP 4-8 first derivative on n points, its norm H, and the
    composite dissipation. Q = H D is skew but for its corners; its boundary
    block follows from exactness on 1, x, .., x^4 and the three free
    parameters Q_56, Q_57, Q_67. The dissipation is H-self-adjoint: H^-1 times
    minus the fourth differences' normal matrix over 256."""
    h = np.array([1498139 / 5080320, 1107307 / 725760, 20761 / 80640, 1304999 / 725760, 299527 / 725760,
                  103097 / 80640, 670091 / 725760, 5127739 / 5080320])
    c = [4 / 5, -1 / 5, 4 / 105, -1 / 280]
    pairs = [(i, j) for i in range(8) for j in range(i + 1, 8)]
    free = {(5, 6): 541 / 1000, (5, 7): -27 / 400, (6, 7): 187 / 250}
    unknown = [p for p in pairs if p not in free]
    rows, rhs = [], []
    for m in range(8):
        for e in range(5):
            f = lambda x: (float(x - 3.5) / 4.0) ** e  # noqa: E731
            df = 0.0 if e == 0 else e * (float(m - 3.5) / 4.0) ** (e - 1) / 4.0
            r, b = np.zeros(len(unknown)), h[m] * df
            if m == 0:
                b += 0.5 * f(0)
            for (i, j), v in free.items():
                b -= v * f(j) if m == i else (-v * f(i) if m == j else 0.0)
            for j in range(8, 12):
                if j - m <= 4:
                    b -= c[j - m - 1] * f(j)
            for u, (i, j) in enumerate(unknown):
                r[u] = f(j) if m == i else (-f(i) if m == j else 0.0)
            rows.append(r)
            rhs.append(b)
    A, b = np.array(rows), np.array(rhs)
    x = np.linalg.lstsq(A, b, rcond=None)[0]
    x += np.linalg.lstsq(A, b - A @ x, rcond=None)[0]
    Q = np.zeros((n, n))
    for k in range(1, 5):
        Q += c[k - 1] * (np.eye(n, k=k) - np.eye(n, k=-k))
    B = np.zeros((8, 8))
    B[0, 0] = -0.5
    for v, (i, j) in list(zip(x, unknown)) + [(v, p) for p, v in free.items()]:
        B[i, j], B[j, i] = v, -v
    Q[:8, :8] = B
    Q[n - 8:, n - 8:] = -B[::-1, ::-1]
    H = np.ones(n)
    H[:8], H[n - 8:] = h, h[::-1]
    d4 = np.zeros((n, n))
    for i in range(n):  # the rows next to a boundary repeat its one-sided stencil
        k = min(max(i - 2, 0), n - 5)
        d4[i, k:k + 5] = [1, -4, 6, -4, 1]
    return Q / H[:, None], H, -(d4.T @ d4) / H[:, None] / 256.0


def _periodic48(n):
    D, C = np.zeros((n, n)), np.zeros((n, n))
    i = np.arange(n)
    for k, v in zip(range(1, 5), [4 / 5, -1 / 5, 4 / 105, -1 / 280]):
        D[i, (i + k) % n] += v
        D[i, (i - k) % n] -= v
    for k, v in zip(range(-4, 5), [-1, 8, -28, 56, -70, 56, -28, 8, -1]):
        C[i, (i + k) % n] += v / 256.0
    return D, np.ones(n), C


class _Plain:
    """One block with far-field SATs, sponges, one source and Gaussian target
    and control regions (2D), or one periodic box (3D), in 64-bit torch."""

    def __init__(self, P):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.P, o, b = P, P.options, P.blocks[0]
        self.nD, self.o = o.n_dimensions, o
        self.shape = tuple(reversed(b.grid_size[: self.nD]))
        self.nU = self.nD + 2
        T = self.T = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=self.dev)
        self.F = lambda a: T(a).reshape(self.shape)
        per = [t != 0 for t in b.periodicity_type[: self.nD]]
        ops = [(_periodic48 if per[d] else _sbp48)(b.grid_size[d]) for d in range(self.nD)]
        self.D, self.C = [T(x[0]) for x in ops], [T(x[2]) for x in ops]
        self.Hn = [x[1] for x in ops]
        # coordinate derivatives; a periodic coordinate is x = L i / n
        x = [self.F(c) for c in b.coordinates]
        J = [[None] * self.nD for _ in range(self.nD)]  # J[c][d] = d x_c / d xi_d
        for c in range(self.nD):
            for d in range(self.nD):
                if per[d]:
                    J[c][d] = torch.full(self.shape, b.periodic_length[d] / b.grid_size[d] if c == d else 0.0,
                                         dtype=torch.float64, device=self.dev)
                else:
                    J[c][d] = self.app(self.D[d], x[c], d)
        if self.nD == 2:
            det = J[0][0] * J[1][1] - J[0][1] * J[1][0]
            self.m = [[J[1][1], -J[0][1]], [-J[1][0], J[0][0]]]
        else:
            det = J[0][0] * J[1][1] * J[2][2]
            z = torch.zeros_like(det)
            self.m = [[J[1][1] * J[2][2], z, z], [z, J[0][0] * J[2][2], z], [z, z, J[0][0] * J[1][1]]]
        self.jac = 1.0 / det
        norm = det
        for d in range(self.nD):
            s = [1] * self.nD
            s[self.nD - 1 - d] = -1
            norm = norm * T(self.Hn[d]).reshape(s)
        self.norm = norm
        self.sat, self.act, self.tgt = [], None, None
        self.qt = self.Q(b.target_state)
        self.sponge = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        for p in P.patches:
            e = p.resolved_extent(b.grid_size)
            sl = (slice(e[2] - 1, e[3]), slice(e[0] - 1, e[1]))
            d = abs(p.normal_direction) - 1
            if p.type == "SAT_FAR_FIELD":
                self.sat.append((sl, d, math.copysign(1.0, p.normal_direction) / self.Hn[d][0],
                                 p.normal_direction > 0))
            elif p.type == "SPONGE":
                arc = torch.sqrt(sum(J[c][d] ** 2 for c in range(self.nD)))[sl]
                ax = self.nD - 1 - d
                cum = torch.cumsum(arc, ax)
                tot = cum.narrow(ax, cum.shape[ax] - 1, 1)
                last = arc.narrow(ax, arc.shape[ax] - 1, 1)
                first = arc.narrow(ax, 0, 1)
                frac = (cum - arc) / (tot - last) if p.normal_direction > 0 else (tot - cum) / (tot - first)
                self.sponge[sl] += p.sponge_amount * (1.0 - frac) ** p.sponge_exponent
            elif p.type == "COST_TARGET":
                self.tgt = sl
            elif p.type == "ACTUATOR":
                self.act = sl
        if o.enable_functional and self.tgt is not None:
            mt = self.F(b.target_mollifier)[self.tgt]
            self.mt = mt / (self.norm[self.tgt] * mt).sum()
            mc = self.F(b.control_mollifier)[self.act]
            self.mc = mc / (self.norm[self.act] * mc).sum()
        self.src = [(s, torch.exp(-9.0 / (2.0 * s.radius ** 2) * sum((x[d] - s.location[d]) ** 2 for d in range(2))))
                    for s in P.sources]
        # incoming Jacobians of the quiescent target along each patch's metric
        # row: eigenvalues 0, 0, c, -c, so A+ = A (A + c) / (2 c) and A- = -A (A - c) / (2 c)
        for k, (sl, d, sig, positive) in enumerate(self.sat):
            mx, my = self.m[d][0][sl].reshape(-1), self.m[d][1][sl].reshape(-1)
            arc = torch.sqrt(mx * mx + my * my)  # ambient sound speed 1
            A = torch.zeros(mx.numel(), 4, 4, dtype=torch.float64, device=self.dev)
            T0 = 1.0 / (GAMMA - 1.0)
            A[:, 0, 1], A[:, 0, 2] = mx, my
            A[:, 1, 3], A[:, 2, 3] = (GAMMA - 1.0) * mx, (GAMMA - 1.0) * my
            A[:, 3, 1], A[:, 3, 2] = T0 * mx, T0 * my
            a = arc[:, None, None]
            Ain = (A @ A + a * A) / (2 * a) if positive else -(A @ A - a * A) / (2 * a)
            self.sat[k] = (sl, d, sig, Ain)

    def Q(self, q):
        return self.T(q).reshape((self.nU,) + self.shape)

    def app(self, M, f, d):
        ax = f.dim() - 1 - d
        return torch.movedim(torch.movedim(f, ax, -1) @ M.T, -1, ax)

    def prims(self, q):
        v = 1.0 / q[0]
        u = [v * q[1 + d] for d in range(self.nD)]
        p = (GAMMA - 1.0) * (q[self.nD + 1] - 0.5 * q[0] * sum(x * x for x in u))
        return v, u, p, GAMMA / (GAMMA - 1.0) * p * v

    def rhs(self, q, t, f=None):
        nD, o = self.nD, self.o
        v, u, p, T = self.prims(q)
        mu = ((GAMMA - 1.0) * T) ** o.viscosity_power_law_exponent / o.reynolds_number
        la = (o.bulk_viscosity_ratio - 2.0 / 3.0) * mu
        kd = mu / o.prandtl_number
        W = torch.stack(u + [T])
        dW = [self.app(self.D[d], W, d) for d in range(nD)]
        G = [self.jac * sum(self.m[d][x] * dW[d] for d in range(nD)) for x in range(nD)]  # G[x][c]
        div = la * sum(G[x][x] for x in range(nD))
        tau = [[mu * (G[d][c] + G[c][d]) + (div if c == d else 0.0) for d in range(nD)] for c in range(nD)]
        E = q[nD + 1]
        flux, visc = [], []
        for d in range(nD):
            flux.append(torch.stack([q[1 + d]] + [q[1 + c] * u[d] + (p if c == d else 0.0) for c in range(nD)]
                                    + [u[d] * (E + p)]))
            visc.append(torch.stack([torch.zeros_like(p)] + [tau[c][d] for c in range(nD)]
                                    + [sum(u[c] * tau[c][d] for c in range(nD)) + kd * G[d][nD]]))
        r = torch.zeros_like(q)
        for i in range(nD):
            Fh = sum(self.m[i][d] * (flux[d] - visc[d]) for d in range(nD))
            r = r - self.app(self.D[i], Fh, i)
            r = r + o.dissipation_amount * self.app(self.C[i], q, i)
        r = r * self.jac
        for sl, d, sig, Ain in self.sat:
            s = (slice(None),) + sl
            dq = (q - self.qt)[s].reshape(self.nU, -1).T[:, :, None]
            t1 = (Ain @ dq)[:, :, 0].T.reshape(q[s].shape)
            fv = sum(visc[j][s] * self.m[d][j][sl] for j in range(nD))
            add = torch.zeros_like(q)
            add[s] = sig * self.jac[sl] * (fv - t1)
            r = r + add
        r = r - self.sponge * (q - self.qt)
        extra = torch.zeros_like(p)
        for s, g in self.src:
            extra = extra + s.amplitude * math.cos(2.0 * math.pi * s.frequency * t + s.phase) * g
        if f is not None:
            e2 = torch.zeros_like(p)
            e2[self.act] = self.mc * f.reshape(self.mc.shape)
            extra = extra + e2
        return torch.cat([r[: nD + 1], (r[nD + 1] + extra)[None]])

    def J(self, q):
        if self.tgt is None:
            return (self.norm * 0.5 * sum(q[1 + d] ** 2 for d in range(self.nD)) / q[0]).sum()
        F = self.prims(q)[2][self.tgt] - 1.0 / GAMMA
        return (self.norm[self.tgt] * F * F * self.mt).sum()

    def dt(self, q):
        if not self.o.use_constant_cfl:
            return self.o.time_step_size
        with torch.no_grad():
            v, u, p, T = self.prims(q)
            m2 = sum(self.m[j][k] ** 2 for j in range(self.nD) for k in range(self.nD))
            w = torch.sqrt((GAMMA - 1.0) * T) * torch.sqrt(m2)
            for j in range(self.nD):
                w = w + sum(u[k] * self.m[j][k] for k in range(self.nD)).abs()
            mu = ((GAMMA - 1.0) * T) ** self.o.viscosity_power_law_exponent / self.o.reynolds_number
            wv = self.jac ** 2 * m2 * torch.maximum(2.0 * mu, mu / self.o.prandtl_number)
            return min(float((self.o.cfl / (self.jac * w)).min()), float((self.o.cfl / wv).min()))

    def step(self, q, t, dt, f=None, each=None):
        """One RK4 step; with a time-integrated functional also its share of J."""
        def rhs(x, i):
            return self.rhs(x, t + (0.0, 0.5, 0.5, 1.0)[i] * dt, None if f is None else f[i])
        J = 0.0
        r = rhs(q, 0)
        b2, x = q + dt * r / 6.0, q + dt * r / 2.0
        for i in (1, 2, 3):
            if self.tgt is not None:
                Ji = self.J(x)
                J = J + RK[i - 1] * dt * Ji
                if each is not None:
                    each.append(Ji)
            r = rhs(x, i)
            if i < 3:
                b2, x = b2 + dt * r / 3.0, q + dt * r / (2.0 if i == 1 else 1.0)
            else:
                x = b2 + dt * r / 6.0
        if self.tgt is not None:
            Ji = self.J(x)
            J = J + RK[3] * dt * Ji
            if each is not None:
                each.append(Ji)
        return x, J

    def forward(self, q, n, keep=False, forcing=None):
        t, J, qs, dts = 0.0, 0.0, [], []
        for k in range(n):
            if keep:
                qs.append(q)
            dts.append(self.dt(q))
            f = None if forcing is None else [forcing[4 * (n - 1 - k) + 3 - i] for i in range(4)]
            q, dJ = self.step(q, t, dts[-1], f)
            J = J + dJ
            t += dts[-1]
        return q, (J if self.tgt is not None else self.J(q)), qs, dts

    def gradient(self, q, n):
        with torch.no_grad():
            qT, J, qs, dts = self.forward(q, n, keep=True)
        starts = np.concatenate([[0.0], np.cumsum(dts)])
        if self.tgt is None:
            x = qT.clone().requires_grad_(True)
            (bar,) = torch.autograd.grad(self.J(x), x)
        else:
            bar = torch.zeros_like(qT)
        P = self.mc.numel() if self.tgt is not None else 0
        rows, sens = [], 0.0
        for k in range(n - 1, -1, -1):
            x = qs[k].clone().requires_grad_(True)
            f = [torch.zeros(P, dtype=torch.float64, device=self.dev, requires_grad=True) for _ in range(4)] if P else None
            y, dJ = self.step(x, float(starts[k]), dts[k], f)
            g = torch.autograd.grad((y * bar).sum() + dJ, [x] + (f or []))
            bar = g[0]
            for i in (3, 2, 1, 0):
                if P:
                    w = self.norm[self.act].reshape(-1)
                    row = g[1 + i] / (RK[i] * dts[k] * w)
                    rows.append(row)
                    sens += RK[i] * dts[k] * float((w * row * row).sum())
        return J, sens, rows, bar / self.norm


def _flat(q):
    return q.detach().reshape(q.shape[0], -1).cpu()


def exact(case, seed):
    k = case["kind"]
    if k in ("region", "jet") or (k == "percall" and case["flow"] == "wall") or case.get("scheme") or (
            k == "tgv" and case["n"] * (3 if case["adjoint"] else 1) > 300):
        return None
    if k == "sweep":
        costs, qs = [], []
        for j, n in enumerate(_sweep_sizes(case)):
            P = _monopole(n, n, controller=True, steps=case["steps"], save=case["steps"])
            M = _Plain(P)
            f = M.T(_forcing(4 * case["steps"], M.mc.numel(), seed + 100 * j))
            with torch.no_grad():
                q, J, _, _ = M.forward(M.Q(_states(P, seed + 100 * j)[0]), case["steps"], forcing=f)
            costs.append(float(J))
            qs.append(_flat(q))
        return {"costs": np.array(costs), "q": qs}
    P = _problem(case)
    M = _Plain(P)
    q0 = M.Q(_states(P, seed)[0])
    if k == "percall":
        dt, each = P.options.time_step_size, []
        with torch.no_grad():
            q, _ = M.step(q0, 0.0, dt, each=each)
            v, u, p, _ = M.prims(q)
            F = -2.0 * M.mt * (GAMMA - 1.0) * (p[M.tgt] - 1.0 / GAMMA)
            force = torch.zeros_like(q)
            force[(slice(None),) + M.tgt] = torch.stack(
                [0.5 * sum(x[M.tgt] ** 2 for x in u) * F] + [-x[M.tgt] * F for x in u] + [F])
        x = q.clone().requires_grad_(True)
        R = M.rhs(x, 0.0)

        def adj(lam, factor):
            (g,) = torch.autograd.grad(R, x, lam * M.norm, retain_graph=True)
            return -g / M.norm + factor * force
        lam = M.Q(_adjoint_state(P, seed))
        r = adj(lam, 2.0)
        b1, b2, y = lam, lam - dt * r / 6.0, lam - dt * r / 2.0
        r = adj(y, 1.0)
        b2, y = b2 - dt * r / 3.0, b1 - dt * r / 2.0
        r = adj(y, 0.5)
        b2, y = b2 - dt * r / 3.0, b1 - dt * r
        y = b2 - dt * adj(y, 1.0) / 6.0
        return {"q": _flat(q), "J": np.array([float(j) for j in each]), "lam": _flat(y)}
    n = case["steps"]
    if k == "forward" or (k == "tgv" and not case["adjoint"]):
        with torch.no_grad():
            q, J, _, _ = M.forward(q0, n)
        return {"J": np.array([float(J)]), "q": _flat(q)}
    if k == "tangent":
        df = M.T(_forcing(4 * n, M.mc.numel(), seed))
        dq = M.Q(_adjoint_state(P, seed))
        q, t, dt, dJ, J = q0, 0.0, P.options.time_step_size, 0.0, 0.0
        zero = [torch.zeros(M.mc.numel(), dtype=torch.float64, device=M.dev) for _ in range(4)]
        for s in range(n):
            fs = [df[4 * (n - 1 - s) + 3 - i] for i in range(4)]
            (y, j), (dy, dj) = torch.func.jvp(lambda a, *f: M.step(a, t, dt, list(f)), (q, *zero), (dq, *fs))
            q, dq, J, dJ, t = y, dy, J + float(j), dJ + float(dj), t + dt
        return {"J": np.array([J]), "dJ": np.array([dJ]), "dq": _flat(dq)}
    J, sens, rows, lam = M.gradient(q0, n)
    if k == "tgv":
        return {"J": np.array([float(J)]), "sensitivity": None, "lam": [_flat(lam)]}
    return {"J": np.array([float(J)]), "sensitivity": np.array([sens]), "gradient": torch.stack(rows).cpu(), "lam": [_flat(lam)]}
