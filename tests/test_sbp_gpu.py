"""Device SBP-SAT operators and elliptic solve vs the oracle (GPU)."""
import itertools

import numpy as np
import pytest

from oracle.sbp2d import SbpOps as OracleSbp

pytestmark = pytest.mark.gpu

BCS = [("Dirichlet", "Neumann", "Dirichlet", "Neumann"), ("Neumann", "Dirichlet", "Neumann", "Dirichlet"),
       ("Dirichlet", "Dirichlet", "Dirichlet", "Dirichlet")]


def _case(order, grid, Ny, Nz, seed=0, compat="fullyCompatible", bcs=BCS[0]):
    rng = np.random.default_rng(seed)
    Ly, Lz = 30.0, 24.0
    q = np.repeat(np.arange(Ny) / (Ny - 1), Nz)
    r = np.tile(np.arange(Nz) / (Nz - 1), Ny)
    var = grid == "variableGridSpacing"
    y = Ly * np.sinh(2 * q) / np.sinh(2) if var else None
    z = Lz * (r + 0.2 * r * r) / 1.2 if var else None
    mu = 32.04 + 2 * rng.random(Ny * Nz)
    from scycle_b200.sbp import SbpOps
    dev = SbpOps(order, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z, compat=compat, bcs=bcs)
    ora = OracleSbp(order, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z, compat=compat, bcs=bcs)
    return dev, ora, rng


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("order,grid,bcs,shape", list(itertools.product(
    (2, 4), ("constantGridSpacing", "variableGridSpacing"), BCS, [(37, 45), (101, 67)])))
def test_apply_A_matches_oracle(order, grid, bcs, shape):
    dev, ora, rng = _case(order, grid, *shape, bcs=bcs)
    x = rng.standard_normal(dev.N)
    out = dev.apply("A", x).cpu().numpy()
    assert _rel(out, ora.A @ x) <= 1e-13


@pytest.mark.parametrize("grid,bcs", list(itertools.product(("constantGridSpacing", "variableGridSpacing"), BCS[:2])))
def test_apply_A_separable_interior(grid, bcs):
    """Constant mu: the interior tiles use the composed 9-point stencils
    built from the 1D coefficient arrays (grid large enough for such tiles)."""
    Ny, Nz = 129, 161
    Ly, Lz = 30.0, 24.0
    q = np.repeat(np.arange(Ny) / (Ny - 1), Nz)
    r = np.tile(np.arange(Nz) / (Nz - 1), Ny)
    var = grid == "variableGridSpacing"
    y = Ly * np.sinh(2 * q) / np.sinh(2) if var else None
    z = Lz * (r + 0.2 * r * r) / 1.2 if var else None
    mu = np.full(Ny * Nz, 32.04)
    from scycle_b200.sbp import SbpOps
    dev = SbpOps(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z, bcs=bcs)
    ora = OracleSbp(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z, bcs=bcs)
    x = np.random.default_rng(7).standard_normal(Ny * Nz)
    out = dev.apply("A", x).cpu().numpy()
    assert _rel(out, ora.A @ x) <= 1e-13
    # a smooth field: the operator's cancellation exposes rounding differences
    xs = np.sin(q * 3.0) * np.cos(r * 2.0) + 0.1 * q
    out = dev.apply("A", xs).cpu().numpy()
    ref = ora.A @ xs
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("order,grid", list(itertools.product((2, 4), ("constantGridSpacing", "variableGridSpacing"))))
def test_first_derivative_ops(order, grid):
    dev, ora, rng = _case(order, grid, 41, 29)
    x = rng.standard_normal(dev.N)
    checks = {"Dy": ora.Dy_Iz @ x, "Dz": ora.Iy_Dz @ x, "muxDy": ora.muxDy(x), "muxDz": ora.muxDz(x),
              "Dyxmu": ora.Dy_Iz @ (ora.mu_vec * x), "Dzxmu": ora.Iy_Dz @ (ora.mu_vec * x),
              "H": ora.H @ x, "Hinv": ora.Hinv @ x}
    for op, ref in checks.items():
        assert _rel(dev.apply(op, x).cpu().numpy(), ref) <= 1e-13, op


@pytest.mark.parametrize("order,grid,bcs", list(itertools.product((2, 4), ("constantGridSpacing", "variableGridSpacing"), BCS)))
def test_set_rhs_matches_oracle(order, grid, bcs):
    dev, ora, rng = _case(order, grid, 33, 41, bcs=bcs)
    bcL, bcR = rng.standard_normal(41), rng.standard_normal(41)
    bcT, bcB = rng.standard_normal(33), rng.standard_normal(33)
    out = dev.set_rhs(bcL, bcR, bcT, bcB).cpu().numpy()
    assert _rel(out, ora.set_rhs(bcL, bcR, bcT, bcB)) <= 1e-13


@pytest.mark.parametrize("order,grid,precision,precond", list(itertools.product(
    (2, 4), ("constantGridSpacing", "variableGridSpacing"), ("fp64", "mixed"), ("mg", "fd"))))
def test_solve_matches_direct_solve(order, grid, precision, precond):
    import scipy.sparse.linalg as spla
    dev, ora, rng = _case(order, grid, 101, 81)
    bcL = np.linspace(0, 1, 81) ** 2
    bcR = np.full(81, 0.3)
    rhs = ora.set_rhs(bcL, bcR, np.zeros(101), np.zeros(101))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    u, st = dev.solve(rhs, rtol=1e-12, max_its=300, precision=precision, precond=precond)
    assert st.converged
    assert _rel(u.cpu().numpy(), ref) <= 1e-9


@pytest.mark.parametrize("Ny,Nz,precision", [
    (45, 45, "fp64"), (46, 45, "fp64"), (17, 120, "mixed"), (33, 65, "fp64"), (129, 17, "fp64"), (89, 91, "mixed"),
    (90, 95, "fp64")])
def test_multigrid_solve_at_level_edges(Ny, Nz, precision):
    """Multigrid on a varying shear modulus where the first level, or the
    first coarse one, has just under and just over the 2048 nodes up to which
    a cycle's levels run in one cluster launch, few rows or columns for its
    eight blocks, and odd sizes.  The solve stops at 1e-12 of the rhs, the
    error may be larger by the operator's spread: the tolerance of the other
    solves against the direct one."""
    import scipy.sparse.linalg as spla
    dev, ora, rng = _case(4, "constantGridSpacing", Ny, Nz, seed=Ny)
    rhs = ora.set_rhs(rng.standard_normal(Nz), rng.standard_normal(Nz), rng.standard_normal(Ny),
                      rng.standard_normal(Ny))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    u, st = dev.solve(rhs, rtol=1e-12, max_its=400, precision=precision, precond="mg")
    assert st.converged
    assert _rel(u.cpu().numpy(), ref) <= 1e-9


@pytest.mark.parametrize("rpt,grid,mu_kind", list(itertools.product(
    (1, 2, 4), ("constantGridSpacing", "variableGridSpacing"), ("constant", "one_column"))))
def test_full_form_every_rows_per_thread(monkeypatch, rpt, grid, mu_kind):
    """The full-form operator kernels (one 17-point stencil per row and per
    column, line classes, 9-point interior tiles) at 1, 2 and 4 output rows
    per thread (SCY_FULL_RPT, read when the operator is built): A x, and a
    CG solve whose matrix-vector products and residuals run through them,
    against the oracle.  mu is constant, or constant but for one column (an
    exceptional y line)."""
    import scipy.sparse.linalg as spla
    from scycle_b200.sbp import SbpOps
    monkeypatch.setenv("SCY_FULL_RPT", str(rpt))
    Ny, Nz = 137, 163
    Ly, Lz = 30.0, 24.0
    q = np.repeat(np.arange(Ny) / (Ny - 1), Nz)
    r = np.tile(np.arange(Nz) / (Nz - 1), Ny)
    var = grid == "variableGridSpacing"
    y = Ly * np.sinh(2 * q) / np.sinh(2) if var else None
    z = Lz * (r + 0.2 * r * r) / 1.2 if var else None
    mu = np.full(Ny * Nz, 32.04)
    if mu_kind == "one_column":
        mu.reshape(Ny, Nz)[:, Nz // 3] = 27.5
    dev = SbpOps(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z)
    ora = OracleSbp(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z)
    x = np.random.default_rng(rpt).standard_normal(Ny * Nz)
    assert _rel(dev.apply("A", x).cpu().numpy(), ora.A @ x) <= 1e-13
    rhs = ora.set_rhs(np.linspace(0, 1, Nz) ** 2, np.full(Nz, 0.3), np.zeros(Ny), np.zeros(Ny))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    u, st = dev.solve(rhs, rtol=1e-12, max_its=400, precond="mg")
    assert st.converged
    assert _rel(u.cpu().numpy(), ref) <= 1e-9


@pytest.mark.parametrize("Ny,Nz,grid,mu_kind", [
    (256, 256, "constantGridSpacing", "constant"), (257, 263, "variableGridSpacing", "constant"),
    (383, 177, "constantGridSpacing", "one_column"), (1100, 61, "variableGridSpacing", "constant"),
    (33, 2001, "variableGridSpacing", "one_column"), (801, 353, "constantGridSpacing", "constant")])
def test_apply_A_in_walks(Ny, Nz, grid, mu_kind):
    """A x by warps that walk down 32 columns (grids of 65536 nodes or more
    whose operator is separable over every node): interior boxes that end
    inside tiles, no interior box at all (one exceptional column near one
    side, few rows), walks of one and of several chunks, partial last tiles.
    Both sides sum at most 34 products per node in FP64 from the same 1D
    operators; the composed coefficients' rounding leaves about 1e-14."""
    Ly, Lz = 30.0, 24.0
    q = np.repeat(np.arange(Ny) / (Ny - 1), Nz)
    r = np.tile(np.arange(Nz) / (Nz - 1), Ny)
    var = grid == "variableGridSpacing"
    y = Ly * np.sinh(2 * q) / np.sinh(2) if var else None
    z = Lz * (r + 0.2 * r * r) / 1.2 if var else None
    mu = np.full(Ny * Nz, 32.04)
    if mu_kind == "one_column":
        mu.reshape(Ny, Nz)[:, Nz // 3] = 27.5
    from scycle_b200.sbp import SbpOps
    dev = SbpOps(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z)
    ora = OracleSbp(4, Ny, Nz, Ly, Lz, mu, grid=grid, y=y, z=z)
    x = np.random.default_rng(Ny).standard_normal(Ny * Nz)
    assert _rel(dev.apply("A", x).cpu().numpy(), ora.A @ x) <= 1e-13


@pytest.mark.parametrize("Ny,Nz,mu_var", [(17, 17, False), (41, 33, True), (129, 97, False), (260, 256, False)])
def test_chained_launches_keep_stream_order(Ny, Nz, mu_var):
    """Launches whose blocks are placed before the kernel ahead of them has
    finished: chains A (A (... x)) of small and larger grids and of several
    blocks per SM, without a wait in between and between ordinary launches
    and copies of another library, on two streams at once, give bitwise what
    the same applications give one at a time."""
    import ctypes as C
    import torch
    from scycle_b200 import _lib as S
    from scycle_b200.sbp import SbpOps
    rng = np.random.default_rng(Ny)
    mu = 32.04 + (2 * rng.random(Ny * Nz) if mu_var else np.zeros(Ny * Nz))
    devs = [SbpOps(4, Ny, Nz, 30.0, 24.0, mu) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in devs]
    x = torch.from_numpy(rng.standard_normal(Ny * Nz)).cuda()
    scale, n = 1e-6, 12
    ref = x
    for _ in range(n):
        ref = devs[0].apply("A", ref) * scale
    out = []
    torch.cuda.synchronize()
    for d, st in zip(devs, streams):
        S.check(S.lib().scy_sbp_set_stream(d.h, C.c_void_p(st.cuda_stream)))
        with torch.cuda.stream(st):
            a, b, keep = x.clone(), torch.empty_like(x), torch.empty_like(x)
            for _ in range(n):
                S.check(S.lib().scy_sbp_apply(d.h, S.OPS["A"], C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr())))
                # twice more into a buffer that the next round overwrites
                S.check(S.lib().scy_sbp_apply(d.h, S.OPS["A"], C.c_void_p(b.data_ptr()), C.c_void_p(keep.data_ptr())))
                torch.mul(b, scale, out=a)
            out.append((a, b, keep))
    torch.cuda.synchronize()
    for a, _, _ in out:
        assert torch.equal(a, ref)
    for d in devs:
        S.check(S.lib().scy_sbp_set_stream(d.h, C.c_void_p(0)))


@pytest.mark.parametrize("precision", ("fp64", "mixed"))
def test_fast_diagonalisation_on_separable_stretched_grid(precision):
    """Constant mu, y(iy) and z(iz) stretched independently: the separable part
    is exact except for the mu3 column, so CG converges in a few iterations."""
    import scipy.sparse.linalg as spla
    from scycle_b200.configs import tanh_stretch
    from scycle_b200.sbp import SbpOps
    Ny, Nz = 121, 97
    y = np.repeat(tanh_stretch(Ny, 30.0, 2.0), Nz)
    z = np.tile(tanh_stretch(Nz, 24.0, 2.0), Ny)
    mu = np.full(Ny * Nz, 32.04)
    dev = SbpOps(4, Ny, Nz, 30.0, 24.0, mu, grid="variableGridSpacing", y=y, z=z)
    ora = OracleSbp(4, Ny, Nz, 30.0, 24.0, mu, grid="variableGridSpacing", y=y, z=z)
    rhs = ora.set_rhs(np.linspace(0, 1, Nz) ** 2, np.full(Nz, 0.3), np.zeros(Ny), np.zeros(Ny))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    u, st = dev.solve(rhs, rtol=1e-13, max_its=100, precision=precision, precond="fd")
    assert st.converged and st.iterations <= (12 if precision == "fp64" else 20)
    assert _rel(u.cpu().numpy(), ref) <= 1e-10


def test_fast_diagonalisation_of_a_product_shear_modulus():
    """mu = a(y) b(z) (here b spans two decades, a a factor three): the
    fast diagonalisation fits log mu as alpha(y) + beta(z) and weights the
    two directions' operators and masses by the fitted factors, which makes
    it exact for a product up to the mu3 column, so CG needs few
    iterations where the plain averages of mu would not be close."""
    import scipy.sparse.linalg as spla
    from scycle_b200.sbp import SbpOps
    Ny, Nz = 81, 73
    yy = np.linspace(0.0, 1.0, Ny)[:, None]
    zz = np.linspace(0.0, 1.0, Nz)[None, :]
    mu = (32.04 * (1.0 + 2.0 * yy) * 10.0 ** (2.0 * zz ** 2)).ravel()
    dev = SbpOps(4, Ny, Nz, 30.0, 24.0, mu)
    ora = OracleSbp(4, Ny, Nz, 30.0, 24.0, mu)
    rhs = ora.set_rhs(np.linspace(0, 1, Nz), np.full(Nz, 0.3), np.zeros(Ny), np.zeros(Ny))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    u, st = dev.solve(rhs, rtol=1e-12, max_its=200, precond="fd")
    assert st.converged and st.iterations <= 40, st.iterations
    assert _rel(u.cpu().numpy(), ref) <= 1e-9


def test_change_bc_types_rebuilds_operator():
    dev, ora, rng = _case(4, "constantGridSpacing", 45, 37)
    dev.change_bc_types("Neumann", "Neumann", "Neumann", "Neumann")
    ora.change_bc_types("Neumann", "Neumann", "Neumann", "Neumann")
    x = rng.standard_normal(dev.N)
    assert _rel(dev.apply("A", x).cpu().numpy(), ora.A @ x) <= 1e-13


def test_solve_warm_start_converges_immediately():
    dev, ora, rng = _case(4, "constantGridSpacing", 65, 65)
    rhs = ora.set_rhs(np.ones(65), np.zeros(65), np.zeros(65), np.zeros(65))
    u, st = dev.solve(rhs, rtol=1e-11)
    u2, st2 = dev.solve(rhs, u0=u, rtol=1e-11)
    # one batch of iterations runs before the first read-back; from a
    # converged start it changes nothing
    assert st2.iterations <= 1 and st2.converged
    # the extra iteration may still improve an rtol-1e-11 solution slightly
    assert np.abs(u2.cpu().numpy() - u.cpu().numpy()).max() <= 1e-9 * np.abs(u.cpu().numpy()).max()


@pytest.mark.parametrize("ratio", (1.2, 1.0 / 1.4, 1.0 / 1.6))
def test_solve_on_steep_geometric_stretching(ratio):
    """Constant mu, y spacing in geometric progression: the averaged
    coefficient of the last z column differs from the others' by
    |1/ratio - 1| / 2 (0.08, 0.2, 0.3), and 1/4 is where the FP64 fast
    diagonalisation's solve goes from defect correction to CG.  A residual of
    rtol |rhs| leaves an error of at most rtol times the condition number
    (2-norm; 3e3 to 6e5 here)."""
    import scipy.sparse.linalg as spla
    from scycle_b200.sbp import SbpOps
    Ny, Nz = 25, 21
    s = ratio ** np.arange(Ny) - 1.0
    y = np.repeat(30.0 * s / s[-1], Nz)
    z = np.tile(np.linspace(0.0, 24.0, Nz), Ny)
    mu = np.full(Ny * Nz, 32.04)
    dev = SbpOps(4, Ny, Nz, 30.0, 24.0, mu, grid="variableGridSpacing", y=y, z=z)
    ora = OracleSbp(4, Ny, Nz, 30.0, 24.0, mu, grid="variableGridSpacing", y=y, z=z)
    rhs = ora.set_rhs(np.linspace(0, 1, Nz) ** 2, np.full(Nz, 0.3), np.zeros(Ny), np.zeros(Ny))
    ref = spla.spsolve(ora.A.tocsc(), rhs)
    lam = np.linalg.eigvalsh(-0.5 * (ora.A + ora.A.T).toarray())
    u, st = dev.solve(rhs, rtol=1e-12, max_its=60, precond="fd")
    assert st.converged
    assert np.linalg.norm(u.cpu().numpy() - ref) <= 1e-12 * lam[-1] / lam[0] * np.linalg.norm(ref)


@pytest.mark.parametrize("order,Ny,Nz", [(2, 5, 9), (2, 17, 33), (4, 9, 13), (4, 15, 16), (4, 16, 17), (4, 24, 47),
                                         (4, 31, 130), (4, 130, 31), (4, 502, 18), (4, 510, 13), (4, 1010, 12),
                                         (4, 2040, 10)])
def test_fast_diagonalisation_inverts_separable_operators(order, Ny, Nz):
    """The banded sweeps in segments (one segment, a last segment of eight
    rows, four, two and one modes a block, and beyond 2000 rows whole chains)
    and the z transforms on narrow tiles: on a constant grid the
    preconditioner is the inverse up to rounding, so three corrections reach a
    residual of 1e-12 |rhs| (one gains over six digits)."""
    from scycle_b200.sbp import SbpOps
    mu = np.full(Ny * Nz, 32.04)
    dev = SbpOps(order, Ny, Nz, 30.0, 24.0, mu)
    ora = OracleSbp(order, Ny, Nz, 30.0, 24.0, mu)
    rng = np.random.default_rng(Ny)
    rhs = ora.set_rhs(rng.random(Nz), rng.random(Nz), np.zeros(Ny), np.zeros(Ny))
    u, st = dev.solve(rhs, rtol=1e-12, max_its=3, precond="fd")
    assert st.converged and st.iterations <= 3
    assert np.linalg.norm(rhs - ora.A @ u.cpu().numpy()) <= 2e-12 * np.linalg.norm(rhs)


@pytest.mark.parametrize("max_its", [8, 31, 32])
def test_solve_within_a_small_iteration_limit(max_its):
    """Where the fast diagonalisation is a few per cent from the inverse, CG
    reaches 1e-12 in 7 iterations and defect correction in 11: a limit that CG
    keeps is kept."""
    from scycle_b200.sbp import SbpOps
    n = 33
    h = (1.0 / 1.4) ** np.arange(n - 1)
    y = 30.0 * np.concatenate([[0.0], np.cumsum(h)]) / h.sum()
    z = 30.0 * (1.0 + np.tanh(2.0 * (np.linspace(0.0, 1.0, n) - 1.0)) / np.tanh(2.0))
    dev = SbpOps(4, n, n, 30.0, 30.0, np.full(n * n, 32.04), "variableGridSpacing", y=np.repeat(y, n),
                 z=np.tile(z, n))
    rhs = dev.apply("A", np.random.default_rng(1).standard_normal(n * n))
    u, st = dev.solve(rhs, rtol=1e-12, max_its=max_its)
    assert st.converged and st.iterations <= max_its
    r = dev.apply("A", u) - rhs
    assert float(r.norm()) <= 2e-12 * float(rhs.norm())


def test_first_solve_in_another_form_keeps_the_preconditioner():
    """The sweeps' tables (segments, whole chains, whole chains in FP32) are
    laid out from one factorisation when a solve first sweeps that way: the
    first solve near rounding, or in mixed precision, after one at the default
    tolerance is no second set-up (measured 1 ms against 40), and gives
    what it gives on an operator of its own."""
    import time
    import torch
    from scycle_b200.sbp import SbpOps
    n = 301
    make = lambda: SbpOps(4, n, n, 30.0, 30.0, np.full(n * n, 32.04))
    rhs = make().apply("A", np.random.default_rng(2).standard_normal(n * n))
    forms = (dict(rtol=1e-12), dict(rtol=1e-14), dict(rtol=1e-10, precision="mixed"))

    def timed(op, kw):
        torch.cuda.synchronize()
        t = time.perf_counter()
        u, _ = op.solve(rhs, **kw)
        return time.perf_counter() - t, u

    alone = [timed(make(), kw) for kw in forms]  # also loads every kernel
    op = make()
    first, _ = timed(op, forms[0])
    for (_, u), kw in zip(alone[1:], forms[1:]):
        t, v = timed(op, kw)
        assert t < 0.5 * first
        assert torch.equal(u, v)


def test_multigrid_keeps_the_finest_planes_once():
    """An operator that is not separable composes its 33 coefficient planes
    once: the FP64 multigrid's finest level uses the operator's own.  Device
    memory of an operator with its solver: planes 33 / (1 - 1/4), fields and
    vectors of all levels some 45, of the solve 6 values a node."""
    import torch
    from scycle_b200.sbp import SbpOps
    ny, nz = 257, 385
    y, z = np.linspace(0.0, 1.0, ny)[:, None], np.linspace(0.0, 1.0, nz)[None, :]
    mu = (32.0 * (1.0 + 0.3 * np.sin(6.0 * y + 4.0 * z))).ravel()

    def used():
        free = torch.cuda.mem_get_info()[0]
        op = SbpOps(4, ny, nz, 30.0, 30.0, mu)
        u, st = op.solve(rhs)
        assert st.converged
        r = op.apply("A", u) - rhs
        assert float(r.norm()) <= 2e-12 * float(rhs.norm())
        del u, r
        return free - torch.cuda.mem_get_info()[0], op

    rhs = SbpOps(4, ny, nz, 30.0, 30.0, mu).apply("A", np.random.default_rng(4).standard_normal(ny * nz))
    used()[1].close()  # kernels and workspaces of the process
    mem, op = used()
    assert mem <= 8 * ny * nz * (44 + 45 + 6)
