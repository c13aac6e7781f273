"""Timed workloads of the solver, through its public Python entry points.

Each case is a dict of plain values.  ``kind`` names the call a user's program makes:

  resident   GpuSolver.solve_resident_device: one more right-hand side on the matrix and
             preconditioner that the handle already holds, B and X in device memory (a
             load step of a linear analysis, a modified-Newton or implicit-dynamic step)
  dropin     hecmw_solve: the call that fistr1 makes in every Newton iteration, the
             caller's arrays on the host, new matrix values, preconditioner rebuilt
  assemble   GpuSolver.assemble_hex8 (new values on a known mesh) and solve_assembled:
             a Newton iteration whose assembly is on the device too
  multi      GpuSolver.solve_multi_device: several load cases on one matrix
  batch      BatchSolver.solve_device: many small independent systems at once

The systems are the clamped, top-loaded HEX8 boxes of the tests and of bench.py
(structured, or with jittered nodes and log-normal moduli), solved to the tolerance
that those use.  A seed gives other loads (and other moduli where the call takes new
matrix values): a random traction direction with a random part on every loaded node.
"""
import functools

import numpy as np
import torch

from frontistr_b200.batch import BatchSolver, stack_systems
from frontistr_b200.matrix import HecMatrix
from frontistr_b200.mesh import box_system, random_box_batch
from frontistr_b200.solver import GpuSolver, hecmw_solve

SSOR, DIAG, ILU0 = 1, 3, 10
CG, BICGSTAB, GMRES = 1, 2, 3


def _case(kind, nx=0, ny=0, nz=0, **more):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, rough=False, method=CG, precond=SSOR, mode=0, learned=False,
             tol=1e-8, nrhs=1, systems=0, edge_lo=0, edge_hi=0)
    c.update(more)
    return c


def listed():
    def named(name, *a, **k):
        return dict(_case(*a, **k), name=name)

    return [
        # the smallest call: a part of a few hundred nodes, where launches and latency are all there is
        named("ssor_6x5x8", "resident", 6, 5, 8),
        # the slender cantilever that the parity tests pin: 19 thousand nodes
        named("ssor_16x16x64", "resident", 16, 16, 64),
        # the headline drop-in: 3.09 million DOF, FP64 CG + SSOR
        named("ssor_100x100x100", "resident", 100, 100, 100),
        # the same system with the learned preconditioner and BF16-stored smoother: the headline solve
        named("learned_mixed_100x100x100", "resident", 100, 100, 100, learned=True, mode=1),
        # jittered mesh, log-normal moduli, tight tolerance, BF16-stored SSOR: the mixed-precision target
        named("mixed_rough_80x80x80", "resident", 80, 80, 80, rough=True, mode=1, tol=1e-10),
        # the learned preconditioner in FP64 on an irregular mid-size box of odd sizes
        named("learned_rough_37x29x43", "resident", 37, 29, 43, rough=True, learned=True),
        # block ILU(0), the preconditioner users choose for badly conditioned models
        named("ilu0_40x40x40", "resident", 40, 40, 40, precond=ILU0),
        # BiCGSTAB, for matrices that are not symmetric positive definite
        named("bicgstab_rough_21x25x34", "resident", 21, 25, 34, rough=True, method=BICGSTAB),
        # one Newton iteration of fistr1 with host arrays
        named("dropin_48x48x48", "dropin", 48, 48, 48),
        # one Newton iteration assembled on the device
        named("assemble_32x32x40", "assemble", 32, 32, 40),
        # sixteen load cases of one model
        named("multi16_48x48x48", "multi", 48, 48, 48, nrhs=16),
        # a design study: 64 small parts of every size between 4 and 20 elements an edge
        named("batch64_edges4_20", "batch", systems=64, edge_lo=4, edge_hi=20),
    ]


def draw(rng):
    kind = rng.choice(["resident"] * 5 + ["dropin", "assemble", "multi", "batch"])
    if kind == "batch":
        lo = rng.randint(3, 8)
        return _case(kind, systems=int(round(2 ** rng.uniform(2, 7))), edge_lo=lo, edge_hi=lo + rng.randint(2, 14))
    # nodes spread over their logarithm from a few hundred to a few hundred thousand
    top = 2.0e5 if kind == "resident" else 8.0e4
    edge = (2.0e2 * (top / 2.0e2) ** rng.random()) ** (1.0 / 3.0)
    nx, ny, nz = (max(3, int(round(edge * 2 ** rng.uniform(-0.5, 0.5)))) for _ in range(3))
    rough = rng.random() < 0.5
    if kind == "dropin":
        return _case(kind, nx, ny, nz, rough=rough, precond=rng.choice([SSOR, SSOR, DIAG]))
    if kind == "assemble":
        return _case(kind, nx, ny, nz)
    if kind == "multi":
        return _case(kind, nx, ny, nz, rough=rough, nrhs=rng.randint(2, 16))
    what = rng.choice(["ssor", "ssor", "mixed", "learned", "ilu0", "diag", "bicgstab", "gmres"])
    if what == "ssor":
        return _case(kind, nx, ny, nz, rough=rough, tol=rng.choice([1e-8, 1e-10]))
    if what == "mixed":
        return _case(kind, nx, ny, nz, rough=rough, mode=1, tol=rng.choice([1e-8, 1e-10]))
    if what == "learned":
        return _case(kind, nx, ny, nz, rough=rough, learned=True, mode=rng.choice([0, 1]))
    if what == "ilu0":
        n = min(nx, 40), min(ny, 40), min(nz, 40)
        return _case(kind, *n, rough=rough, precond=ILU0)
    if what == "diag":
        return _case(kind, nx, ny, nz, rough=rough, precond=DIAG)
    n = min(nx, 32), min(ny, 32), min(nz, 32)
    return _case(kind, *n, rough=rough, method=BICGSTAB if what == "bicgstab" else GMRES)


# ---- systems -------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _box(nx, ny, nz, rough):
    if rough:
        return box_system(nx, ny, nz, jitter=0.2, sigma_E=1.0, nu_range=(0.25, 0.40), seed=3)
    return box_system(nx, ny, nz)


@functools.lru_cache(maxsize=2)
def _boxes(systems, lo, hi):
    return stack_systems(random_box_batch(systems, edge_range=(lo, hi), seed=11))


def _loads(B, count, seed):
    """count load cases on the loaded nodes of B: a traction and a random part per node."""
    rng = np.random.default_rng(seed)
    top = np.unique(np.nonzero(B)[0] // 3)
    out = np.zeros((count, B.size))
    for k in range(count):
        t = rng.standard_normal(3)
        f = t / np.linalg.norm(t) + 0.1 * rng.standard_normal((top.size, 3))
        out[k].reshape(-1, 3)[top] = f
    return out


def _inputs(case, seed):
    """(matrix, load cases): the values of a dropin matrix are the seed's own."""
    m = _box(case["nx"], case["ny"], case["nz"], case["rough"])
    if case["kind"] == "dropin":
        s = float(np.exp(np.random.default_rng([seed, 7]).uniform(-1, 1)))
        m = HecMatrix(m.N, m.NP, m.indexL, m.itemL, m.indexU, m.itemU, s * m.D, s * m.AL, s * m.AU, m.B.copy())
    return m, _loads(_box(case["nx"], case["ny"], case["nz"], case["rough"]).B, case["nrhs"], seed)


@functools.lru_cache(maxsize=2)
def _hex_box(nx, ny, nz):
    """Node grid (x fastest) and HEX8 connectivity of the box."""
    g = np.stack(np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij"), -1)
    X = g.reshape(-1, 3)[:, ::-1].astype(np.float64).copy()
    z, y, x = (a.reshape(-1) for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    at = lambda i, j, k: i + (nx + 1) * (j + (ny + 1) * k)  # noqa: E731
    corners = [(0, 0), (1, 0), (1, 1), (0, 1)]
    el = np.stack([at(x + i, y + j, z + k) for k in (0, 1) for i, j in corners], 1).astype(np.int32)
    return X, el


def _hex_inputs(case, seed):
    """Coordinates (interior nodes jittered), elements, moduli, nodal loads, clamped nodes."""
    rng = np.random.default_rng([seed, 5])
    grid, el = _hex_box(case["nx"], case["ny"], case["nz"])
    X = grid.copy()
    size = np.array([case["nx"], case["ny"], case["nz"]])
    inner = np.all((X > 0) & (X < size), axis=1)
    X[inner] += rng.uniform(-0.2, 0.2, size=(int(inner.sum()), 3))
    E = 2.1e5 * np.exp(0.5 * rng.standard_normal(len(el)))
    nu = rng.uniform(0.25, 0.40, len(el))
    F = np.zeros((len(X), 3))
    F[grid[:, 2] == case["nz"], 1] = -1.0
    return X, el, E, nu, _loads(F.reshape(-1), 1, seed)[0], np.nonzero(grid[:, 2] == 0)[0]


def _flags(case, m_ia, m_ra):
    ia, ra = m_ia.copy(), m_ra.copy()
    ia[0] = 20000  # ITER
    ia[1] = case["method"]
    ia[2] = case["precond"]
    ia[5] = 30  # NREST of GMRES
    ia[41] = case["mode"]  # precision mode
    ia[42] = 1 if case["learned"] else 0
    ra[0] = case["tol"]
    return ia, ra


# ---- the calls -----------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _network():
    """Weights of the learned preconditioner's network, trained on an earlier, smaller
    model as a program that keeps them in a file has them."""
    m = _box(12, 10, 16, False)
    ia, ra = _flags(_case("resident"), m.Iarray, m.Rarray)
    with GpuSolver() as s:
        s.set_matrix(m)
        s.learn_record(1)
        s.solve_resident(_loads(m.B, 1, 1)[0], np.zeros(3 * m.N), ia, ra)
        s.learn_record(0)
        s.learn_train(20, 5e-3)
        return s.learn_get_weights()


def _warm(ia):
    """Flags of a call that only builds the preconditioner: one iteration."""
    w = ia.copy()
    w[0] = 1
    return w


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        m, ptr = _boxes(case["systems"], case["edge_lo"], case["edge_hi"])
        ia, ra = _flags(case, m.Iarray, m.Rarray)
        s = BatchSolver()
        s.set_matrix(m, ptr, ia, ra)
        B = torch.from_numpy(_loads(m.B, 1, seed)[0]).cuda()
        return dict(kind=kind, solver=s, B=B, X=torch.empty_like(B), ia=ia, ra=ra)
    if kind == "assemble":
        X, el, E, nu, F, base = _hex_inputs(case, seed)
        fixed = [(int(n), d, 0.0) for n in base for d in (1, 2, 3)]
        s = GpuSolver()
        s.assemble_hex8(X, el, E, nu, F=F, fixed=fixed)
        ia, ra = _flags(case, *_fresh_flags())
        w = _warm(ia)
        s.solve_assembled(w, ra)
        ia[95:98] = w[95:98]
        return dict(kind=kind, solver=s, mesh=(X, el, E, nu), F=F, fixed=fixed, ia=ia, ra=ra)
    m, loads = _inputs(case, seed)
    ia, ra = _flags(case, m.Iarray, m.Rarray)
    s = GpuSolver()
    if kind == "dropin":
        m.B[:] = loads[0]
        m.Iarray[:], m.Rarray[:] = _warm(ia), ra
        hecmw_solve(m, solver=s)
        ia[95:98] = m.Iarray[95:98]
        m.Iarray[:] = ia
        return dict(kind=kind, solver=s, m=m)
    s.set_matrix(m)
    if case["learned"]:
        s.learn_set_weights(_network())
    B = torch.from_numpy(loads).cuda()
    X = torch.zeros_like(B)
    torch.cuda.current_stream().synchronize()
    w = _warm(ia)
    if kind == "multi":
        s.solve_multi_device(case["nrhs"], B.data_ptr(), X.data_ptr(), w, ra)
    else:
        s.solve_resident_device(B.data_ptr(), X.data_ptr(), w, ra)
    ia[95:98] = w[95:98]
    return dict(kind=kind, solver=s, B=B, X=X, ia=ia, ra=ra, nrhs=case["nrhs"])


def _fresh_flags():
    m = HecMatrix.empty(1, 0, 0)
    return m.Iarray, m.Rarray


def run(state):
    kind, s = state["kind"], state["solver"]
    if kind == "dropin":
        m = state["m"]
        m.X[:] = 0.0
        m.Iarray[96] = 2  # new values: rebuild the preconditioner numerically
        hecmw_solve(m, solver=s)
        return m.X
    if kind == "assemble":
        X, el, E, nu = state["mesh"]
        s.assemble_hex8(X, el, E, nu, F=state["F"], fixed=state["fixed"], symbolic=False)
        state["ia"][96] = 2
        x, _ = s.solve_assembled(state["ia"], state["ra"])
        return x
    X = state["X"]
    X.zero_()
    torch.cuda.current_stream().synchronize()  # the handle has its own stream
    if kind == "batch":
        s.solve_device(state["B"].data_ptr(), X.data_ptr(), state["ia"], state["ra"])
    elif kind == "multi":
        s.solve_multi_device(state["nrhs"], state["B"].data_ptr(), X.data_ptr(), state["ia"], state["ra"])
    else:
        s.solve_resident_device(state["B"].data_ptr(), X.data_ptr(), state["ia"], state["ra"])
    return X


# ---- work ----------------------------------------------------------------------
def _iterations(case, nx, ny, nz):
    """About the iterations to the tolerance (measured on these boxes): proportional to
    the box's edges for the one-level preconditioners, about constant for the learned
    two-level one."""
    digits = -np.log10(case["tol"]) / 8.0
    if case["learned"]:
        return (80.0 if case["rough"] else 60.0) * digits
    per = {SSOR: 2.2, DIAG: 4.4, ILU0: 1.5}[case["precond"]]
    if case["method"] != CG:
        per *= 0.6
    return per * (nx + ny + nz) * digits * (1.1 if case["rough"] else 1.0) + 5.0


def _solve_work(case, nx, ny, nz):
    """A Krylov iteration needs one product with A (each block and column index read
    once; the preconditioner's factors are A's own blocks) and x, r and p read and
    written; two operations per entry for the product and two for the preconditioner."""
    n = (nx + 1) * (ny + 1) * (nz + 1)
    nz_blocks = (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    it = _iterations(case, nx, ny, nz)
    per_vec = 6 * 24.0 * n * case["nrhs"]
    return dict(bytes=it * (76.0 * nz_blocks + per_vec), flops=it * 36.0 * nz_blocks * case["nrhs"])


def work(case):
    if case["kind"] == "batch":
        _, ptr = _boxes(case["systems"], case["edge_lo"], case["edge_hi"])
        total = dict(bytes=0.0, flops=0.0)
        for n in np.diff(ptr):
            e = float(n) ** (1.0 / 3.0) - 1.0
            w = _solve_work(case, e, e, e)
            total = {k: total[k] + w[k] for k in total}
        return total
    w = _solve_work(case, case["nx"], case["ny"], case["nz"])
    if case["kind"] == "dropin":  # the caller's values come up once
        w["bytes"] += 72.0 * (3 * case["nx"] + 1) * (3 * case["ny"] + 1) * (3 * case["nz"] + 1)
    if case["kind"] == "assemble":  # the matrix values written once
        w["bytes"] += 72.0 * (3 * case["nx"] + 1) * (3 * case["ny"] + 1) * (3 * case["nz"] + 1)
        w["flops"] += 8 * 36 * 60.0 * case["nx"] * case["ny"] * case["nz"]
    return w


def tolerance(case):
    """Two correct solves may stop an iteration or two apart with residuals at the solve's
    tolerance.  Seen against the 64-bit solution: up to 6e-10 for CG (every
    preconditioner), up to 2e-8 for BiCGSTAB, whose error is the less tightly bound to
    its residual."""
    rel = 1e-8 if case["method"] == CG else 1e-7
    return {"rel": rel, "max": 40 * rel}


# ---- the same in 64 bits -------------------------------------------------------
def _csr(m):
    """The scalar matrix in CSR on the GPU, from the block arrays."""
    N = m.N
    dev = torch.device("cuda")
    up = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(dev, t)  # noqa: E731
    iL, iU = up(m.indexL[:N + 1], torch.int64), up(m.indexU[:N + 1], torch.int64)
    ptr = iL + iU + torch.arange(N + 1, device=dev)  # blocks before each row: lower, diagonal, upper
    nb = int(ptr[-1])
    col = torch.empty(nb, dtype=torch.int32, device=dev)
    val = torch.empty((nb, 9), dtype=torch.float64, device=dev)
    rows = torch.arange(N, device=dev)
    nl, nu = iL[1:] - iL[:-1], iU[1:] - iU[:-1]
    at_l = torch.arange(m.NPL, device=dev) + torch.repeat_interleave(ptr[:-1] - iL[:-1], nl)
    at_d = ptr[:-1] + nl
    at_u = torch.arange(m.NPU, device=dev) + torch.repeat_interleave(at_d + 1 - iU[:-1], nu)
    for at, c, v in ((at_l, up(m.itemL[:m.NPL], torch.int32) - 1, m.AL[:9 * m.NPL]),
                     (at_d, rows.to(torch.int32), m.D[:9 * N]),
                     (at_u, up(m.itemU[:m.NPU], torch.int32) - 1, m.AU[:9 * m.NPU])):
        col[at] = c
        val[at] = up(v, torch.float64).view(-1, 9)
    del at_l, at_d, at_u
    # scalar rows 3i..3i+2: the block columns of row i, each expanded to three
    cnt = ptr[1:] - ptr[:-1]
    crow = torch.zeros(3 * N + 1, dtype=torch.int64, device=dev)
    crow[1:] = torch.cumsum(torch.repeat_interleave(3 * cnt, 3), 0)
    scol = torch.empty(9 * nb, dtype=torch.int32, device=dev)
    sval = torch.empty(9 * nb, dtype=torch.float64, device=dev)
    blk_row = torch.repeat_interleave(rows, cnt)
    off = torch.arange(nb, device=dev) - ptr[blk_row]
    for r in range(3):
        start = crow[3 * blk_row + r] + 3 * off
        for c in range(3):
            scol[start + c] = 3 * col + c
            sval[start + c] = val[:, 3 * r + c]
    A = torch.sparse_csr_tensor(crow.to(torch.int32), scol, sval, size=(3 * N, 3 * N))
    d = torch.from_numpy(m.D[:9 * N].reshape(-1, 9)[:, [0, 4, 8]].reshape(-1).copy()).to(dev)
    return A, d


def _cg64(apply, diag, b, tol=1e-13, most=20000):
    """Jacobi-preconditioned CG on the columns of b, restarted once on the true residual."""
    x = torch.zeros_like(b)
    inv = (1.0 / diag)[:, None]
    for rtol in (tol, 1e-2):
        r = b - apply(x)
        r0 = r.square().sum(0)
        if float(r0.max()) == 0.0:
            break
        z = inv * r
        p = z.clone()
        rho = (r * z).sum(0)
        for k in range(most):
            q = apply(p)
            alpha = rho / (p * q).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            if k % 50 == 49 and bool((r.square().sum(0) <= rtol * rtol * r0).all()):
                break
            z = inv * r
            new = (r * z).sum(0)
            p = z + (new / rho.clamp_min(1e-300)) * p
            rho = new
    return x


def _element_stiffness(X, el, E, nu):
    """(ne, 24, 24) linear-elastic HEX8 stiffness, 2x2x2 Gauss points."""
    sign = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                         [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64, device=X.device)
    xe = X[el]
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    K = torch.zeros((el.shape[0], 8, 3, 8, 3), dtype=torch.float64, device=X.device)
    eye = torch.eye(3, dtype=torch.float64, device=X.device)
    for gp in sign / np.sqrt(3.0):
        t = 1 + sign * gp
        dN = torch.stack([sign[:, 0] * t[:, 1] * t[:, 2], sign[:, 1] * t[:, 0] * t[:, 2],
                          sign[:, 2] * t[:, 0] * t[:, 1]], 1) / 8.0
        J = torch.einsum("ai,eaj->eij", dN, xe)
        w = torch.linalg.det(J)
        g = torch.einsum("ai,eji->eaj", dN, torch.linalg.inv(J))
        K += torch.einsum("eai,ebj,e->eaibj", g, g, lam * w)
        K += torch.einsum("eaj,ebi,e->eaibj", g, g, mu * w)
        K += torch.einsum("eac,ebc,ij,e->eaibj", g, g, eye, mu * w)
    return K.reshape(-1, 24, 24)


def exact(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        X, el, E, nu, F, base = _hex_inputs(case, seed)
        X, el, E, nu, F = (torch.from_numpy(a).cuda() for a in (X, el.astype(np.int64), E, nu, F))
        K = _element_stiffness(X, el, E, nu)
        dof = (3 * el[:, :, None] + torch.arange(3, device=el.device)).reshape(-1, 24)
        free = torch.ones(3 * len(X), dtype=torch.float64, device=X.device)
        free.view(-1, 3)[torch.from_numpy(base).cuda()] = 0.0

        def apply(v):
            u = (free[:, None] * v)[dof.reshape(-1)].view(-1, 24, v.shape[1])
            y = torch.zeros_like(v).index_add_(0, dof.reshape(-1), torch.bmm(K, u).reshape(-1, v.shape[1]))
            return free[:, None] * y + (1 - free)[:, None] * v

        diag = torch.zeros_like(F).index_add_(0, dof.reshape(-1), K.diagonal(dim1=1, dim2=2).reshape(-1))
        diag = free * diag + (1 - free)
        return _cg64(apply, diag, (free * F)[:, None])[:, 0].cpu().numpy()
    if kind == "batch":
        m, _ = _boxes(case["systems"], case["edge_lo"], case["edge_hi"])
        loads = _loads(m.B, 1, seed)
    else:
        m, loads = _inputs(case, seed)
    A, d = _csr(m)
    b = torch.from_numpy(loads.T.copy()).cuda()
    x = _cg64(lambda v: A @ v, d, b).T.contiguous()
    return x[0].cpu().numpy() if kind in ("batch", "dropin") else x
