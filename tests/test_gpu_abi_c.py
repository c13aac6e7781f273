"""The C ABI called from C (the way the Fortran iso_c_binding shim calls it) and the
two launch modes of the CG loop (one conditional-WHILE graph vs host-driven stream)."""
import os
import subprocess

import numpy as np
import pytest

from frontistr_b200.mesh import box_system
from frontistr_b200.solver import GpuSolver
from oracle_ctypes import Oracle

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "frontistr_b200", "lib")


def test_c_driver(tmp_path):
    exe = str(tmp_path / "drop_in_driver")
    subprocess.check_call(["gcc", "-O2", "-I", os.path.join(ROOT, "include"),
                           os.path.join(ROOT, "tests", "c_driver", "drop_in_driver.c"), "-o", exe,
                           "-L", LIB, "-lhecmw33_gpu", "-lfistr_assemble", "-Wl,-rpath," + LIB])
    out = subprocess.run([exe, "8"], capture_output=True, text=True, check=True).stdout.split("\n")
    first = out[0].split()
    second = out[1].split()
    m = box_system(8, 8, 16)
    m.set_iter(20000)
    ref = Oracle(m).solve()
    assert int(first[3]) == 0 and int(first[2]) == 1
    assert abs(int(first[0]) - ref["iter"]) <= 2
    assert float(first[1]) <= 1e-8
    assert int(second[0]) == int(first[0])  # same matrix, recycled preconditioner


def test_stream_mode_matches_graph_mode(monkeypatch):
    m = box_system(12, 10, 20, jitter=0.1, seed=5)
    m.set_iter(20000)
    with GpuSolver() as s:
        a = m.copy()
        ia = s.solve(a)
        monkeypatch.setenv("HECMW33_GRAPH", "0")
        b = m.copy()
        ib = s.solve(b)
    assert ia["iter"] == ib["iter"]
    assert np.array_equal(a.X, b.X)


ROUTES = {  # what is not one launch, so that the two modes differ
    "DIAG": lambda m: m.set_precond(3),
    "SIGMA_DIAG": lambda m: m.set_sigma_diag(1.2),
    "two passes": lambda m: m.set_iterpremax(2),
    "BF16 SSOR": lambda m: (m.set_sigma_diag(1.2), m.Iarray.__setitem__(41, 1)),
    "BiCGSTAB": lambda m: m.set_method(2),
    "BiCGSTAB + ILU": lambda m: (m.set_method(2), m.set_precond(10)),
}


@pytest.mark.parametrize("route", list(ROUTES))
def test_stream_mode_matches_graph_mode_where_there_is_a_loop(route, monkeypatch):
    """test_stream_mode_matches_graph_mode's solve is one launch in either mode; these have a
    loop of launches, captured in a graph or issued kStreamChunk iterations at a time."""
    m = box_system(12, 10, 20, jitter=0.1, seed=5)
    m.set_iter(20000)
    ROUTES[route](m)
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("HECMW33_GRAPH", graph)
        g = m.copy()
        with GpuSolver() as s:
            rec = s.solve(g)
            out.append((rec["iter"], rec["error"], s.last_solve_info()["kernels"], g.X))
    assert out[0][1] == out[1][1] == 0 and out[0][0] == out[1][0]
    assert out[0][2] > out[0][0]  # a launch per iteration at least (counted in a graph only)
    assert np.array_equal(out[0][3], out[1][3])


def test_stream_mode_matches_graph_mode_load_cases(monkeypatch):
    """The load-case loop with SIGMA_DIAG != 1, which is not the one-launch kernel's."""
    m = box_system(12, 10, 20, jitter=0.1, seed=5)
    m.set_iter(20000)
    m.set_sigma_diag(1.2)
    B = np.stack([m.B, -0.5 * m.B, np.roll(m.B, 3)])
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("HECMW33_GRAPH", graph)
        X = np.zeros_like(B)
        with GpuSolver() as s:
            s.set_matrix(m)
            rec = s.solve_multi(B, X, m.Iarray.copy(), m.Rarray)
        out.append((rec["iter"], X))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
