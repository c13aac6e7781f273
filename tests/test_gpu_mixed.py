"""Mixed precision (Iarray(42) = 1, 2, 3).

The acceptance is on FP64 quantities: the true relative residual ||b - A x||/||b||
computed by the FP64 oracle must be at or below the requested tolerance, and the
error against the oracle's FP64 solution (solved to the same tolerance) is
bounded by 1e-6 relative -- CG at 1e-8 on these systems leaves a difference of
the order of cond(A) * 1e-8 between any two solutions that meet the tolerance.
"""
import numpy as np
import pytest

from frontistr_b200.mesh import box_system
from frontistr_b200.solver import GpuSolver
from oracle_ctypes import Oracle

pytestmark = pytest.mark.gpu


def mixed_solve(s, m, tol=1e-8, inner=1e-4, precond=1, mode=1):
    g = m.copy()
    g.set_iter(20000)
    g.set_resid(tol)
    g.set_precond(precond)
    g.Iarray[41] = mode
    g.Rarray[41] = inner
    info = s.solve(g)
    return g, info


@pytest.mark.parametrize("mode,bound", [(1, 1.02), (2, 6.0), (3, 6.0)])
@pytest.mark.parametrize("precond", [1, 3, 10])
def test_mixed_reaches_fp64_tolerance(precond, mode, bound):
    """mode 1: BF16-stored preconditioner inside FP64 CG -- the iteration count stays
    that of the FP64 solve (within 2 %); mode 2: restarted FP32 refinement; mode 3:
    FP32 CG with FP64 reliable updates.  Modes 2 and 3 pay extra iterations on this
    ill-conditioned cantilever (FP32 loses the Krylov recurrence's accuracy)."""
    m = box_system(16, 16, 64)
    with GpuSolver() as s:
        g, info = mixed_solve(s, m, precond=precond, mode=mode, inner=0.0)
        rec = s.last_solve_info()
    assert info["error"] == 0
    assert g.get_flag_converged() == 1
    orc = Oracle(m)
    true_res = orc.rel_resid(g.X, m.B)
    assert true_res <= 1e-8
    assert abs(rec["true_resid"] - true_res) <= 1e-3 * true_res
    ref = Oracle(m.copy()).solve(Iarray=_flags(m, precond))
    err = np.linalg.norm(g.X - ref["X"]) / np.linalg.norm(ref["X"])
    assert err <= 1e-6, err
    assert info["iter"] <= bound * ref["iter"], (info["iter"], ref["iter"])
    assert rec["outer"] >= 1


def _flags(m, precond):
    ia = m.Iarray.copy()
    ia[0] = 20000
    ia[2] = precond
    return ia


def test_mixed_heterogeneous_1e10():
    """The config-3 kind of system (jittered nodes, log-normal E, nu in [0.25, 0.40]) to 1e-10."""
    m = box_system(14, 12, 16, jitter=0.2, sigma_E=1.0, nu_range=(0.25, 0.40), seed=11)
    with GpuSolver() as s:
        g, info = mixed_solve(s, m, tol=1e-10)
    assert info["error"] == 0
    assert Oracle(m).rel_resid(g.X, m.B) <= 1e-10


def test_mixed_zero_rhs_and_maxit():
    m = box_system(6, 6, 6)
    with GpuSolver() as s:
        z = m.copy()
        z.B[:] = 0.0
        g, info = mixed_solve(s, z)
        assert info["error"] == 2002 and np.all(g.X == 0)
        t = m.copy()
        t.set_iter(3)
        t.Iarray[41] = 1
        info = s.solve(t)
        assert info["error"] == 3001
        assert t.get_flag_converged() == 0


@pytest.mark.parametrize("route", ["SSOR, SIGMA_DIAG", "SSOR, two passes", "SSOR, recycled", "ILU, two passes"])
def test_mode1_where_the_factors_are_bf16(route):
    """Precision mode 1 on the CG loops that keep BF16 factors (plain CG + SSOR and CG + block
    ILU run their FP64 one-launch kernels in mode 1 too): other bits than mode 0, the launches
    of a loop, the FP64 solve's iterations within 2 %, the tolerance on b - A x."""
    m = box_system(12, 12, 40)
    m.set_iter(20000)
    if "SIGMA" in route:
        m.set_sigma_diag(1.2)
    if "passes" in route:
        m.set_iterpremax(2)
    if "ILU" in route:
        m.set_precond(10)
    out = []
    for mode in (0, 1):
        g = m.copy()
        with GpuSolver() as s:
            if "recycled" in route:
                s.solve(g)
                for a in (g.D, g.AL, g.AU):
                    a *= 1.1
                g.X[:] = 0.0
                g.Iarray[96] = 1  # new values, recycled preconditioner
            g.Iarray[41] = mode
            rec = s.solve(g)
            out.append((rec, s.last_solve_info(), g))
    (ref, _, a), (rec, info, b) = out
    assert rec["error"] == ref["error"] == 0
    assert info["kernels"] > 4 * rec["iter"] and not np.array_equal(a.X, b.X)
    assert rec["iter"] <= 1.02 * ref["iter"] + 1
    r = b.B - b.to_scipy() @ b.X
    assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(b.B)
    assert np.linalg.norm(b.X - a.X) <= 1e-6 * np.linalg.norm(a.X)
