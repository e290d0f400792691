"""Cases by which this framework's speed is measured.

Each case is one kind of work that a program gives this library through its
public entry points: a right-hand side evaluation, steps of the single
quasi-dynamic driver (linear elastic, power law, fault-response mode), one
step of an ensemble of drivers, a batch of wave-equation steps, an operator
application, an elliptic solve, a gradient.  ``listed`` holds the measured
ones, ``draw`` gives others of the same ranges.

The drivers start from a prestressed fault a little above its steady state
at the loading rate, after about 30 years of loading, and take steps of the
interseismic period whose size the settings cap, so a pass is the same work
every time.
"""
import os
import tempfile

import numpy as np
import torch

from scycle_b200 import configs
from scycle_b200.adjoint import Adjoint
from scycle_b200.batch import Batch
from scycle_b200.cycle import Cycle
from scycle_b200.qd import QD
from scycle_b200.sbp import SbpOps

MU = 32.04          # GPa
LENGTH = 30.0       # km, both directions
PRESTRESS = 26.0    # MPa
LOADED = 1.0e9      # s of loading before the drivers start
STEP = 1.0e4        # s, the cap of the drivers' steps
STAGES = {"RK32": 3, "RK43": 6}


def listed():
    return [
        # the smallest call: one right-hand side evaluation from and to host arrays, as a caller with
        # its own integrator makes it (the grid size of the tests)
        dict(name="rates_61", kind="rates", ny=61, nz=61, order=4, law="agingLaw", stretch=False),
        # a single run of the small benchmark problem, output every fourth step
        dict(name="step_101", kind="step", ny=101, nz=101, law="agingLaw", stretch=False, method="RK32", steps=4),
        # a single run of the headline problem (stretched grid, slip law)
        dict(name="step_401", kind="step", ny=401, nz=401, law="slipLaw", stretch=True, method="RK32", steps=4),
        # a single power-law viscoelastic run on a grid that is not square
        dict(name="step_pl_151x201", kind="step_pl", ny=151, nz=201, method="RK43", steps=1),
        # the quasi-dynamic phases of the cycle workload: every stage from the precomputed fault response
        dict(name="response_401", kind="response", ny=401, nz=401, law="agingLaw", stretch=False, method="RK43",
             steps=8),
        # the headline: an ensemble that fills the GPU, one step of every instance
        dict(name="ensemble_32x401", kind="ensemble", count=32, ny=401, nz=401, law="slipLaw", stretch=True,
             method="RK32", steps=1),
        # a small ensemble with odd sizes
        dict(name="ensemble_7x129x97", kind="ensemble", count=7, ny=129, nz=97, law="agingLaw", stretch=False,
             method="RK32", steps=1),
        # the power-law ensemble: three grid sizes, three operator groups in one batch
        dict(name="ensemble_pl_mixed", kind="ensemble_pl", count=3, n0=101, n1=201, n2=301, method="RK43", steps=1),
        # the wave-equation phase of the cycle workload between two looks at the fields
        dict(name="wave_801", kind="wave", ny=801, nz=801, law="agingLaw", steps=256),
        # one operator application on the largest grid a single field is used at
        dict(name="apply_2049x1537", kind="apply", ny=2049, nz=1537, order=4, stretch=True),
        # an elliptic solve with a shear modulus that varies in both directions (multigrid)
        dict(name="solve_257x385", kind="solve", ny=257, nz=385, order=4, stretch=False, precision="fp64"),
        # forward and reverse sweep of the adjoint workload's grid over a short window
        dict(name="gradient_201", kind="gradient", ny=201, nz=201, law="agingLaw", steps=12, every=6),
    ]


def _odd(rng, lo, hi):
    """A size between lo and hi, even in its logarithm; three in four are odd."""
    n = int(round(lo * (hi / lo) ** rng.random()))
    return min(hi, n + 1 - n % 2 if rng.random() < 0.75 else n)


def draw(rng):
    kind = rng.choice(["rates", "step", "step", "step_pl", "response", "ensemble", "ensemble", "ensemble_pl", "wave",
                       "apply", "solve", "solve", "gradient"])
    law = rng.choice(["agingLaw", "slipLaw"])
    stretch = rng.random() < 0.5
    method = rng.choice(["RK32", "RK43"])
    if kind == "rates":
        return dict(kind=kind, ny=_odd(rng, 33, 201), nz=_odd(rng, 33, 201), order=rng.choice([2, 4]), law=law,
                    stretch=stretch)
    if kind == "step":
        return dict(kind=kind, ny=_odd(rng, 65, 401), nz=_odd(rng, 65, 401), law=law, stretch=stretch, method=method,
                    steps=rng.randint(1, 4))
    if kind == "step_pl":
        return dict(kind=kind, ny=_odd(rng, 61, 201), nz=_odd(rng, 61, 201), method=method, steps=1)
    if kind == "response":
        return dict(kind=kind, ny=_odd(rng, 101, 401), nz=_odd(rng, 101, 401), law=law, stretch=stretch,
                    method=method, steps=rng.randint(4, 8))
    if kind == "ensemble":
        ny, nz = _odd(rng, 65, 401), _odd(rng, 65, 401)
        return dict(kind=kind, count=min(_odd(rng, 2, 32), 32 * 401 ** 2 // (ny * nz)), ny=ny, nz=nz, law=law,
                    stretch=stretch, method=method if ny * nz < 100000 else "RK32", steps=1)
    if kind == "ensemble_pl":
        return dict(kind=kind, count=rng.randint(1, 3), n0=_odd(rng, 61, 101), n1=_odd(rng, 101, 201),
                    n2=_odd(rng, 201, 301), method=method, steps=1)
    if kind == "wave":
        return dict(kind=kind, ny=_odd(rng, 101, 801), nz=_odd(rng, 101, 801), law=law, steps=rng.randint(64, 256))
    if kind == "apply":
        return dict(kind=kind, ny=_odd(rng, 129, 2049), nz=_odd(rng, 129, 1537), order=rng.choice([2, 4]),
                    stretch=stretch)
    if kind == "solve":
        # cells near square, as the multigrid preconditioner wants them
        ny = _odd(rng, 65, 321)
        return dict(kind=kind, ny=ny, nz=_odd(rng, max(65, ny * 4 // 5), ny * 5 // 4), order=rng.choice([2, 4]),
                    stretch=False, precision=rng.choice(["fp64", "mixed"]))
    return dict(kind=kind, ny=_odd(rng, 65, 201), nz=_odd(rng, 65, 201), law=law, steps=rng.randint(6, 12),
                every=rng.randint(3, 6))


# ---------------------------------------------------------------------------
# inputs
def _settings(case, loaded=LOADED):
    return {"initTime": repr(loaded), "maxDeltaT": repr(STEP), "rootTol": "1e-13"}


def _input(folder, name, case, seed, **kw):
    """An input file of the reference's format with its per-node fields; the fault's prestress and its state
    vary smoothly and by seeded noise."""
    rng = np.random.default_rng(seed)
    ny, nz = kw.pop("ny", case.get("ny")), kw.pop("nz", case.get("nz"))
    make = kw.pop("make", configs.make_qd_problem)
    args = dict(Ny=ny, Nz=nz, Ly=LENGTH, Lz=LENGTH, seed=seed, name=name, integrator=case.get("method", "RK32"),
                init_dt=STEP, years=1.0e6, guess_ss=0)
    if "order" in case:
        args["order"] = case["order"]
    if "law" in case:
        args["state_law"] = case["law"]
    if case.get("stretch"):
        args.update(grid="variableGridSpacing", stretch_beta=2.0)
    if case.get("law") == "slipLaw":
        args["dc_lognormal"] = True
    extra = _settings(case)
    extra.update(kw.pop("extra", {}))
    args.update(kw)
    path = make(folder, extra=extra, **args)
    z = np.linspace(0.0, 1.0, nz)
    level = PRESTRESS + 0.2 * np.sin(2.0 * np.pi * (z + rng.random())) + 0.02 * rng.random()
    configs.write_petsc_vec(os.path.join(folder, name + "_in_prestress"), level)
    return path


def _coordinates(case):
    """y and z of the grid's lines, clustered at the fault and the surface where the case stretches them."""
    f = configs.tanh_stretch if case["stretch"] else lambda n, length, _: np.linspace(0.0, length, n)
    return f(case["ny"], LENGTH, 2.0), f(case["nz"], LENGTH, 2.0)


def _modulus(case, seed):
    """A shear modulus that varies over both directions: layers and a damage zone at the fault."""
    rng = np.random.default_rng(seed + 1)
    y, z = (v / LENGTH for v in _coordinates(case))
    p = rng.random(3)
    layers = 1.0 + 0.3 * np.sin(2.0 * np.pi * (1.5 * z[None, :] + p[0])) * np.cos(2.0 * np.pi * (y[:, None] + p[1]))
    return MU * layers * (1.0 - (0.3 + 0.2 * p[2]) * np.exp(-10.0 * y[:, None]) * np.exp(-3.0 * z[None, :]))


def _smooth(case, seed, terms=6):
    """A displacement (m): a few smooth modes, seeded."""
    rng = np.random.default_rng(seed + 2)
    y, z = (v / LENGTH for v in _coordinates(case))
    u = np.zeros((case["ny"], case["nz"]))
    for k in range(1, terms + 1):
        a, b, c = rng.random(3)
        u += (a - 0.5) / k * np.outer(np.sin(np.pi * (k * y + b)), np.cos(np.pi * (k * z + c)))
    return u


def _slip(case, seed):
    rng = np.random.default_rng(seed + 3)
    z = np.linspace(0.0, 1.0, case["nz"])
    p = rng.random(2)
    return 0.02 * (1.0 + np.sin(2.0 * np.pi * (z + p[0]))) + 0.003 * np.sin(6.0 * np.pi * (z + p[1]))


def _psi(case, seed):
    return 0.6 + np.random.default_rng(seed).normal(0.0, 1e-4, size=case["nz"])


def prepare(case, seed):
    kind = case["kind"]
    with tempfile.TemporaryDirectory() as folder:
        if kind in ("rates", "step", "step_pl", "response"):
            make = configs.make_pl_problem if kind == "step_pl" else configs.make_qd_problem
            q = QD.from_in(_input(folder, "run", case, seed, make=make))
            if kind == "rates":
                return dict(case=case, q=q, t=LOADED, psi=_psi(case, seed), slip=_slip(case, seed))
            if kind == "response":
                q.set_mode("response")
            q.integrate_begin_from_in()
            return dict(case=case, q=q)
        if kind == "ensemble":
            paths = [_input(os.path.join(folder, str(i)), "run", case, 1000 * seed + i) for i in range(case["count"])]
            return dict(case=case, b=Batch(paths))
        if kind == "ensemble_pl":
            paths = [_input(os.path.join(folder, "%d_%d" % (n, i)), "run", case, 1000 * seed + i, ny=n, nz=n,
                            grad=20.0 + 2.0 * i, make=configs.make_pl_problem)
                     for n in (case["n0"], case["n1"], case["n2"]) for i in range(case["count"])]
            return dict(case=case, b=Batch(paths))
        if kind == "wave":
            # a pulse on its way to the fault; the switch back to the quasi-dynamic phase stays off
            c = Cycle.from_in(_input(folder, "run", case, seed, make=configs.make_qdfd_problem, integrator="RK43",
                                     extra={"initTime": "0", "limit_fd": "1e12", "maxDeltaT": "1e10"}))
            c.begin_from_in()
            rng = np.random.default_rng(seed)
            y, z = np.linspace(0.0, LENGTH, case["ny"]), np.linspace(0.0, LENGTH, case["nz"])
            at, wide = (8.0 + 8.0 * rng.random(), 8.0 + 14.0 * rng.random()), 2.0 + rng.random()
            u = 0.05 * np.exp(-((y[:, None] - at[0]) ** 2 + (z[None, :] - at[1]) ** 2) / wide ** 2).ravel()
            now = dict(psi=_psi(case, seed), slip=np.zeros(case["nz"]), u=u)
            tau = np.full(case["nz"], PRESTRESS + 0.5)
            c.set_fd_state(0.0, 0, False, now, now, np.zeros(u.size), now["slip"], tau, np.full(case["nz"], 1e-9))
            return dict(case=case, c=c)
        if kind == "gradient":
            q = QD.from_in(_input(folder, "run", case, seed, extra={"initTime": "0"}))
            q.integrate_begin_from_in()
            a = Adjoint(q, case["every"])
            a.set_steps(np.full(case["steps"], STEP))
            rng = np.random.default_rng(seed + 4)
            a.set_targets(1e-4 * rng.random((case["steps"], case["ny"])),
                          1e-9 * (0.5 + rng.random((case["steps"], case["nz"]))), 1.0, 1e12)
            return dict(case=case, a=a)
    y, z = _coordinates(case)
    full = dict(y=np.repeat(y, z.size), z=np.tile(z, y.size)) if case["stretch"] else {}
    grid = "variableGridSpacing" if case["stretch"] else "constantGridSpacing"
    mu = _modulus(case, seed) if kind == "solve" else np.full((y.size, z.size), MU)
    ops = SbpOps(case["order"], y.size, z.size, LENGTH, LENGTH, mu.ravel(), grid, **full)
    if kind == "apply":
        return dict(case=case, ops=ops, x=torch.from_numpy(_field(case, seed)).cuda().reshape(-1))
    rhs = _Operator(case, mu).apply(_smooth(case, seed))
    return dict(case=case, ops=ops, rhs=torch.from_numpy(rhs).cuda().reshape(-1))


def _field(case, seed):
    return _smooth(case, seed) + 0.01 * np.random.default_rng(seed + 5).standard_normal((case["ny"], case["nz"]))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rates":
        return state["q"].d_dt(state["t"], state["psi"], state["slip"])
    if kind in ("step", "step_pl", "response"):
        q = state["q"]
        q.integrate_steps(case["steps"])
        more = {"step": ("u",), "step_pl": ("u", "gVxy", "gVxz"), "response": ("surfDisp",)}[kind]
        return {f: q.field(f) for f in ("psi", "slip", "slipVel") + more}
    if kind in ("ensemble", "ensemble_pl"):
        b = state["b"]
        b.run(case["steps"])
        return {f: b.fault_field(f) for f in ("psi", "slip", "slipVel")}
    if kind == "wave":
        c = state["c"]
        c.run(case["steps"])
        return {f: c.field(f) for f in ("psi", "slip", "slipVel", "u")}
    if kind == "gradient":
        return state["a"].gradient()
    if kind == "apply":
        return state["ops"].apply("A", state["x"])
    return state["ops"].solve(state["rhs"], precision=case["precision"])[0]


def work(case):
    """A stage solve reads its right-hand side and its first guess and writes the displacement (24 bytes a node)
    and applies the operator twice (two 9-point lines each, multiply and add); the power law also reads and writes
    its viscous strains and their rates; a wave step reads two displacements and writes one."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "ensemble_pl":
        n = case["count"] * sum(case[k] ** 2 for k in ("n0", "n1", "n2"))
    else:
        n = case["ny"] * case["nz"] * (case["count"] if kind == "ensemble" else 1)
    solve = {"bytes": 24 * n, "flops": 72 * n}
    if kind == "apply":
        return {"bytes": 16 * n, "flops": 36 * n}
    if kind in ("rates", "solve"):
        return solve
    if kind == "wave":
        return {"bytes": 24 * n * steps, "flops": 42 * n * steps}
    if kind == "gradient":
        # forward, recomputation and reverse sweep: three stages a step each
        return {k: 9 * steps * v for k, v in solve.items()}
    if kind == "response":
        evals = steps * STAGES[case["method"]]
        return {"bytes": 8 * evals * case["nz"] ** 2, "flops": 2 * evals * case["nz"] ** 2}
    evals = steps * STAGES[case["method"]]
    if kind in ("step_pl", "ensemble_pl"):
        return {"bytes": evals * 72 * n, "flops": evals * 150 * n}
    return {k: evals * v for k, v in solve.items()}


# ---------------------------------------------------------------------------
# what run() returns, in 64 bits from numpy alone
def _line(order, n, h):
    """One direction's SBP operators: D, the diagonal of H, the boundary rows of BS, the terms (D_k, weights) of
    R = sum_k D_k^T diag(weights c_k) D_k, and the Dirichlet penalty."""
    D = np.zeros((n, n))
    H = np.ones(n)
    S = np.zeros((2, n))
    if order == 2:
        H[[0, -1]] = 0.5
        i = np.arange(1, n - 1)
        D[i, i - 1], D[i, i + 1] = -0.5, 0.5
        D[0, :2] = -1.0, 1.0
        D[-1, -2:] = -1.0, 1.0
        S[0, :2] = 1.0, -1.0
        S[1, -2:] = -1.0, 1.0
        D2 = np.zeros((n, n))
        D2[i, i - 1], D2[i, i], D2[i, i + 1] = 1.0, -2.0, 1.0
        w = np.ones(n)
        w[[0, -1]] = 0.0
        return D / h, H * h, S / h, [(D2, 0.25 / h * w, False)], -4.0 / h
    close = np.array([17.0, 59.0, 43.0, 49.0]) / 48.0
    H[:4], H[-4:] = close, close[::-1]
    i = np.arange(4, n - 4)
    for k, v in ((-2, 1.0 / 12.0), (-1, -2.0 / 3.0), (1, 2.0 / 3.0), (2, -1.0 / 12.0)):
        D[i, i + k] = v
    rows = [[-0.5, 59 / 96, -1 / 12, -1 / 32], [-59 / 96, 0, 59 / 96], [1 / 12, -59 / 96, 0, 59 / 96, -1 / 12],
            [1 / 32, 0, -59 / 96, 0, 2 / 3, -1 / 12]]
    for r, v in enumerate(rows):
        D[r, :len(v)] = v
        D[n - 1 - r, n - len(v):] = -np.array(v[::-1])
    D /= H[:, None]
    S[0, :4] = 24 / 17, -59 / 34, 4 / 17, 3 / 34
    S[1, -4:] = S[0, 3::-1]
    D3, D4 = np.zeros((n, n)), np.zeros((n, n))
    i = np.arange(3, n - 4)
    for k, v in ((-1, -1.0), (0, 3.0), (1, -3.0), (2, 1.0)):
        D3[i, i + k] = v
    for r in (0, 1, n - 2, n - 1):
        D3[r, (0 if r < 2 else n - 4):(4 if r < 2 else n)] = -1, 3, -3, 1
    q = 54642863857.0
    edge = [-185893.0 / 301051.0, 79000249461.0 / q, -33235054191.0 / q, -36887526683.0 / q, 26183621850.0 / q,
            -4386.0 / 181507.0]
    D3[2, :6] = edge
    D3[n - 3, n - 6:] = -np.array(edge[::-1])
    for r in range(n):
        c = min(max(r, 2), n - 3)
        D4[r, c - 2:c + 3] = 1, -4, 6, -4, 1
    w3, w4 = np.ones(n), np.ones(n)
    w3[[0, 1, n - 4, n - 2, n - 1]] = 0.0
    w3[[2, n - 3]] = 163928591571.0 / 53268010936.0
    w3[[3, n - 5]] = 189284.0 / 185893.0
    w4[[0, 1, n - 2, n - 1]] = 0.0
    w4[[2, n - 3]] = 1644330.0 / 301051.0
    w4[[3, n - 4]] = 156114.0 / 181507.0
    return D / h, H * h, S / h, [(D3, w3 / (18.0 * h), True), (D4, w4 / (144.0 * h), False)], -96.0 / 17.0 / h


class _Operator:
    """The assembled operator with a Dirichlet fault (y = 0) and far side (y = Ly) and free surface and bottom."""

    def __init__(self, case, mu):
        ny, nz = mu.shape
        y, z = _coordinates(case)
        hy, hz = ((1.0 / (ny - 1), 1.0 / (nz - 1)) if case["stretch"] else (LENGTH / (ny - 1), LENGTH / (nz - 1)))
        self.y, self.z = _line(case["order"], ny, hy), _line(case["order"], nz, hz)
        yq = self.y[0] @ y if case["stretch"] else np.ones(ny)
        zr = self.z[0] @ z if case["stretch"] else np.ones(nz)
        self.mu, self.qy = mu, 1.0 / yq
        self.cy, self.cz = mu / yq[:, None], mu / zr[None, :]
        self.wy, self.wz = self.z[1] * zr, self.y[1] * yq
        # the third-derivative term's coefficient is averaged with the next node of the flattened index
        f, g = self.cy.ravel(), self.cz.ravel()
        m = np.append(f[1:], f[-2])
        self.m3y = (0.5 * (f + m)).reshape(ny, nz)
        m = np.concatenate([g[1:-1], [0.0], [g[-2]]])
        m[0] += g[1]
        self.m3z = (0.5 * (g + m)).reshape(ny, nz)

    def sides(self, lo, hi, D, S, alpha, c):
        """The Dirichlet terms of two boundary rows."""
        out = np.outer(S[0], c[0] * lo) + np.outer(S[1], c[-1] * hi)
        out[0] += alpha * c[0] * lo
        out[-1] += alpha * c[-1] * hi
        return out

    def apply(self, x):
        D, H, S, terms, alpha = self.y
        out = H[:, None] * (D @ (self.cy * (D @ x)))
        for M, w, third in terms:
            out -= M.T @ (w[:, None] * (self.m3y if third else self.cy) * (M @ x))
        out += self.sides(x[0], x[-1], D, S, alpha, self.cy)
        D, H, S, terms, _ = self.z
        d = self.cz * (x @ D.T)
        res = H[None, :] * (d @ D.T)
        for M, w, third in terms:
            res -= (w[None, :] * (self.m3z if third else self.cz) * (x @ M.T)) @ M
        res[:, 0] += d[:, 0]
        res[:, -1] -= d[:, -1]
        return self.wy[None, :] * out + self.wz[:, None] * res

    def rhs(self, lo, hi):
        D, _, S, _, alpha = self.y
        return self.wy[None, :] * self.sides(lo, hi, D, S, alpha, self.cy)

    def solve(self, b):
        """A u = b for a constant modulus: the operator less its averaged corner is separable, and each pass of the
        diagonalised solve gains over ten digits."""
        ny, nz = b.shape
        mid = nz // 2
        e = np.zeros((ny, nz))
        lines = []
        for n, axis in ((ny, 0), (nz, 1)):
            D, H, S, terms, alpha = self.y if axis == 0 else self.z
            c = self.cy[:, mid] if axis == 0 else self.cz[ny // 2]
            m3 = self.m3y[:, mid] if axis == 0 else self.m3z[ny // 2]
            K = -(H[:, None] * (D @ (c[:, None] * D)))
            for M, w, third in terms:
                K += M.T @ ((w * (m3 if third else c))[:, None] * M)
            if axis == 0:
                K[:, 0] -= S[0] * c[0]
                K[:, -1] -= S[1] * c[-1]
                K[0, 0] -= alpha * c[0]
                K[-1, -1] -= alpha * c[-1]
            else:
                K[0] -= c[0] * D[0]
                K[-1] += c[-1] * D[-1]
            m = self.wz if axis == 0 else self.wy
            r = 1.0 / np.sqrt(m)
            lam, V = np.linalg.eigh(0.5 * (K + K.T) * np.outer(r, r))
            lines.append((lam, r[:, None] * V))
        (ly, Vy), (lz, Vz) = lines
        for _ in range(6):
            e -= Vy @ ((Vy.T @ (b - self.apply(e)) @ Vz) / (ly[:, None] + lz[None, :])) @ Vz.T
        return e


def _fault_rates(case, seed, stress):
    """Slip velocity and state rate of every fault node: stress - eta V = sN a asinh(V / (2 v0) e^(psi / a))."""
    nz = case["nz"]
    z = _coordinates(case)[1]
    psi = _psi(case, seed)
    a, sN, f0, v0 = 0.010, 50.0, 0.6, 1e-6
    b = np.interp(z, [0.0, 12.0, 17.0, LENGTH], [0.015, 0.015, 0.005, 0.005])
    Dc = np.full(nz, 0.008)
    if case["law"] == "slipLaw":
        noise = np.random.default_rng(seed)
        noise.normal(0.0, 1e-4, size=nz)
        Dc = np.exp(noise.normal(np.log(0.008) - 0.02, 0.2, size=nz))
    eta = np.sqrt(MU * 2.67) / 2.0
    # in the logarithm of V the residual is smooth: bisection, then Newton
    E = np.exp(psi / a) / (2.0 * v0)
    resid = lambda V: a * sN * np.arcsinh(V * E) + eta * V - stress
    lo, hi = np.full(nz, -80.0), np.full(nz, 10.0)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        up = resid(np.exp(mid)) > 0.0
        lo, hi = np.where(up, lo, mid), np.where(up, mid, hi)
    V = np.exp(0.5 * (lo + hi))
    for _ in range(4):
        V = V - resid(V) / (a * sN * E / np.sqrt(1.0 + (V * E) ** 2) + eta)
    if case["law"] == "agingLaw":
        rate = b * v0 / Dc * (np.exp((f0 - psi) / b) - V / v0)
    else:
        rate = -V / Dc * (a * np.arcsinh(V * E) - f0 - (a - b) * np.log(V / v0))
    return {"psi": rate, "slip": V}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return _smooth(case, seed).ravel()
    if kind == "apply":
        return _Operator(case, np.full((case["ny"], case["nz"]), MU)).apply(_field(case, seed)).ravel()
    if kind == "rates":
        A = _Operator(case, np.full((case["ny"], case["nz"]), MU))
        far = np.full(case["nz"], 0.5e-9 * LOADED)
        u = A.solve(A.rhs(0.5 * _slip(case, seed), far))
        rng = np.random.default_rng(seed)
        z = np.linspace(0.0, 1.0, case["nz"])
        level = PRESTRESS + 0.2 * np.sin(2.0 * np.pi * (z + rng.random())) + 0.02 * rng.random()
        return _fault_rates(case, seed, level + A.mu[0] * A.qy[0] * (A.y[0][0] @ u))
    # the integrations, the wave steps and the gradient have no values that plain numpy gives without restating the
    # whole scheme
    return None
