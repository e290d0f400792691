"""Runs at the tolerance that callers get by default (1e-12) against the
oracle, replaying the device's attempts.

At this tolerance a stage's solve is a defect correction from the previous
stage's displacement, its sweeps run in segments, and an attempt's solves are
enqueued and read back together (below 1e-13, where the other tests run, each
solve is CG with whole sweep chains).  A solve ends with a residual of at most
1e-12 |rhs|, so the bar of every comparison is ten times what residuals of that
size do to the oracle itself: its solves repeated with a smooth residual of
1e-12 |rhs| in each (a residual of low modes moves the displacement most).
"""
from types import SimpleNamespace

import numpy as np
import pytest

from oracle.powerlaw import PowerLawQD, build_pl_problem
from oracle.problem import build_qd_problem
from oracle.qd import QDLinearElastic
from oracle.qdfd import QDFDLinearElastic, build_qdfd_problem
from scycle_b200.configs import make_pl_problem, make_qd_problem, make_qdfd_problem, write_petsc_vec

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _nrel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _with_residuals(ora, seed):
    """The oracle with a residual of RTOL |rhs| in every solve."""
    rng, lu, refined = np.random.default_rng(seed), ora.lu, ora._refined
    q, r = np.linspace(0.0, 1.0, ora.Ny), np.linspace(0.0, 1.0, ora.Nz)

    def off(b):
        s = rng.choice([-1.0, 1.0]) * np.outer(np.sin(np.pi * q), np.cos(np.pi * rng.integers(0, 3) * r)).ravel()
        return b + RTOL * np.linalg.norm(b) / np.linalg.norm(s) * s

    if isinstance(ora, PowerLawQD):  # solves with its factors
        ora.lu = SimpleNamespace(solve=lambda b: lu.solve(off(b)))
    else:
        ora._refined = lambda A, f, b: refined(A, f, off(b))
    return ora


def _compare(field, make, steps, attempts, names):
    """field(name) against make()'s run; the bar from two runs with residuals."""
    ref, *off = [make() if k == 0 else _with_residuals(make(), k) for k in range(3)]
    for o in [ref] + off:
        assert o.integrate(max_steps=steps, replay=attempts).stepCount == steps
    for nm in names:
        get = lambda o: o.history[-1][nm]
        bar = 10.0 * max(_nrel(get(o), get(ref)) for o in off) + 1e-13
        assert _nrel(field(nm), get(ref)) <= bar, (nm, _nrel(field(nm), get(ref)), bar)


def _le(tmp_path, n, stretch, law, integrator, beta=2.0):
    kw = dict(grid="variableGridSpacing", stretch_beta=beta) if stretch else {}
    p = make_qd_problem(str(tmp_path), Ny=n, Nz=n, state_law=law, integrator=integrator, extra={"rootTol": "1e-14"}, **kw)
    write_petsc_vec(p[:-len(".in")] + "_in_prestress", 26.0 + np.linspace(0.0, 0.5, n))
    return p


@pytest.mark.parametrize("n,stretch,law,integrator,beta,one", [
    (41, False, "agingLaw", "RK32", 0.0, True), (61, False, "slipLaw", "RK43", 0.0, True),
    (65, True, "agingLaw", "RK32", 2.0, False), (33, True, "slipLaw", "RK43", 4.0, False)])
def test_steps_at_the_default_tolerance(tmp_path, n, stretch, law, integrator, beta, one):
    """one: one correction is enough for every solve, so every enqueued attempt
    stands; otherwise some are made again with tested solves."""
    from scycle_b200.qd import QD
    path = _le(tmp_path, n, stretch, law, integrator, beta)
    dev = QD.from_in(path)
    dev.record_attempts(True)
    dev.integrate_begin_from_in()
    first = dev.integrate_steps(0)
    st = dev.integrate_steps(60)
    assert st.step_count == 60
    more = (st.solve_its - first.solve_its) - (st.solves - first.solves)
    assert more == 0 if one else more > 0
    make = lambda: QDLinearElastic(build_qd_problem(open(path).read()), refine=1)
    _compare(dev.field, make, 60, dev.attempts(), ("slip", "psi", "slipVel", "tauP", "surfDisp"))


@pytest.mark.parametrize("stretch", [False, True])
def test_batch_steps_at_the_default_tolerance(tmp_path, stretch):
    from scycle_b200.batch import Batch
    paths = [_le(tmp_path / str(s), n, stretch, law, "RK32")
             for s, (n, law) in enumerate(((41, "agingLaw"), (41, "slipLaw"), (65, "agingLaw")))]
    b = Batch(paths)
    for i in range(b.n):
        b.instance(i).record_attempts(True)
    b.run(40)
    for i, p in enumerate(paths):
        make = lambda: QDLinearElastic(build_qd_problem(open(p).read()), refine=1)
        _compare(b.instance(i).field, make, 40, b.instance(i).attempts(), ("slip", "psi", "slipVel", "tauP", "surfDisp"))


@pytest.mark.parametrize("stretch", [False, True])
def test_power_law_at_the_default_tolerance(tmp_path, stretch):
    """The batch (defect correction) and the single driver (CG), which follow
    different rules, each within the bar, gVxz included: it starts as a
    difference of displacements that agree to rounding."""
    from scycle_b200.batch import Batch
    from scycle_b200.qd import QD
    kw = dict(grid="variableGridSpacing", stretch_beta=1.5) if stretch else {}
    paths = []
    for s, (ny, nz) in enumerate(((33, 33), (41, 37))):
        p = make_pl_problem(str(tmp_path / str(s)), Ny=ny, Nz=nz, seed=s, grad=15.0 + 5.0 * s,
                            extra={"maxDeltaT": "1e6", "rootTol": "1e-14"}, **kw)
        write_petsc_vec(p[:-len(".in")] + "_in_prestress", 26.0 + 0.3 * s + np.linspace(0.0, 0.5, nz))
        paths.append(p)
    b = Batch(paths)
    for i in range(b.n):
        b.instance(i).record_attempts(True)
    b.run(30)
    for i, p in enumerate(paths):
        att = b.instance(i).attempts()
        one = QD.from_in(p)
        one.force_attempts(att)
        one.integrate_begin_from_in()
        one.integrate_steps(30)
        make = lambda: PowerLawQD(build_pl_problem(open(p).read()), refine=1)
        for dev in (b.instance(i), one):
            _compare(dev.field, make, 30, att, ("gVxy", "gVxz", "psi", "slip", "slipVel", "tauP"))


def test_quasi_dynamic_phase_of_a_cycle_at_the_default_tolerance(tmp_path):
    from scycle_b200.cycle import Cycle
    path = make_qdfd_problem(str(tmp_path), Ny=41, Nz=41, years=1000.0, extra={"limit_fd": "0.01", "timeControlType": "P"})

    def run(seed=0, replay=None):
        m = QDFDLinearElastic(build_qdfd_problem(open(path).read()))
        if seed:
            _with_residuals(m, seed)
        rec = []
        m.integrate_cycles(record=rec, replay=replay, stop_at_step=40)
        return {h["step"]: h for h in m.history}, rec

    ref, rec = run()
    off = [run(k, rec)[0] for k in (1, 2)]
    c = Cycle.from_in(path)
    c.force_attempts(rec)
    c.begin_from_in()
    for k in (10, 40):
        c.run(k - (10 if k == 40 else 0))
        for nm in ("slip", "slipVel", "psi", "tauP", "surfDisp"):
            bar = 10.0 * max(_nrel(o[k][nm], ref[k][nm]) for o in off) + 1e-12
            assert _nrel(c.field(nm), ref[k][nm]) <= bar, (k, nm, _nrel(c.field(nm), ref[k][nm]), bar)


@pytest.mark.parametrize("law", ["agingLaw", "slipLaw"])
def test_gradient_at_the_default_tolerance(tmp_path, law):
    """The gradient at 1e-12 against that of solves near rounding (which other
    tests compare with finite differences of the oracle): a reverse sweep's
    solves carry the same relative residual as the forward ones, and the adjoint
    of the sensitive quantity, the slip velocity's logarithm, moves with the
    stress over a sN = 0.5 MPa of 26 MPa: 1e-12 x 52 x the operator's condition
    number (2e3 at 25 x 25)."""
    from scycle_b200.adjoint import Adjoint
    from scycle_b200.qd import QD
    path = _le(tmp_path, 25, False, law, "RK32")
    out = []
    for rtol in (1e-12, 1e-14):
        q = QD.from_in(path, solve_rtol=rtol)
        q.integrate_begin_from_in()
        a = Adjoint(q, 5)
        a.set_steps(np.full(15, 2.0e2))
        rng = np.random.default_rng(5)
        a.set_targets(1e-6 * rng.random((15, 25)), 1e-9 * (0.5 + rng.random((15, 25))), 1e10, 1e17)
        out.append(a.gradient())
    for x, y in zip(out[0][1:], out[1][1:]):
        assert np.linalg.norm(y) > 0 and _nrel(x, y) <= 1e-12 * 52 * 2e3
