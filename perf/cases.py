"""The work that users of this package have it do, as timed cases.

Every case goes through the public entry points (PETSc.Vec / Mat / PC / KSP,
MixedSolver, BatchedCG, sparse_solve) at the sizes of the package's benchmark
configurations and of the operators its tests solve, odd sizes among them.
Kinds:

  vec      the Vec updates and reductions of a hand-written Krylov loop
  mult     Mat.mult, multAdd and multTranspose of one assembled operator
  solve    KSP.solve from a host right-hand side to the host solution
  mixed    the mixed-precision solve to a true FP64 residual
  batched  CG on many independent systems with 16 right-hand sides each
  adjoint  forward solve and the gradient with respect to values and b
"""

from __future__ import annotations

import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir,
                                "mojo-petsc4py_gb300"))

from mojopetsc4py import PETSc, gallery  # noqa: E402
from mojopetsc4py.adjoint import SparseSystem, sparse_solve  # noqa: E402
from mojopetsc4py.batch import BatchedCG  # noqa: E402
from mojopetsc4py.mixed import MixedSolver  # noqa: E402

NRHS = 16  # right-hand sides of a batched system


def listed():
    return [
        # vectors far larger than L2, of a length that no vector width divides
        {"name": "vec-2^24+3", "kind": "vec", "n": 2**24 + 3},
        # the benchmark's operator, multiplied on its own: both directions
        {"name": "mult-poisson3d-128", "kind": "mult", "op": "poisson3d", "k": 128},
        # an irregular operator (random geometric graph, mean degree 8)
        {"name": "mult-graph-60001", "kind": "mult", "op": "graph", "k": 60001},
        # the smallest published problem with PETSc's default solver and
        # preconditioner: nothing but latency
        {"name": "gmres-ilu-poisson2d-32", "kind": "solve", "op": "poisson2d", "k": 32,
         "ksp": "gmres", "pc": "ilu"},
        # the small benchmark configuration
        {"name": "cg-ilu-poisson2d-128", "kind": "solve", "op": "poisson2d", "k": 128,
         "ksp": "cg", "pc": "ilu"},
        # the headline: the operator streams from HBM, the vectors sit in L2
        {"name": "cg-jacobi-poisson3d-128", "kind": "solve", "op": "poisson3d", "k": 128,
         "ksp": "cg", "pc": "jacobi"},
        # the same system with the factored preconditioner (triangular sweeps)
        {"name": "cg-icc-poisson3d-128", "kind": "solve", "op": "poisson3d", "k": 128,
         "ksp": "cg", "pc": "icc"},
        # nonsymmetric, the plain FP64 counterpart of the mixed case
        {"name": "gmres-ilu-convdiff3d-96", "kind": "solve", "op": "convdiff3d", "k": 96,
         "ksp": "gmres", "pc": "ilu"},
        # symmetric SOR on an odd grid
        {"name": "bcgs-sor-poisson3d-81", "kind": "solve", "op": "poisson3d", "k": 81,
         "ksp": "bcgs", "pc": "sor"},
        # FP32 inner solver inside FP64 refinement
        {"name": "mixed-convdiff3d-96", "kind": "mixed", "k": 96},
        # uneven independent systems, 16 right-hand sides each
        {"name": "batched-graph-24", "kind": "batched", "count": 24, "nmin": 1024,
         "nmax": 16384, "pc": "jacobi"},
        # gradient through a solve: forward and adjoint
        {"name": "adjoint-advdiff2d-256", "kind": "adjoint", "k": 256},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["vec", "mult", "mult", "solve", "solve", "solve", "solve", "mixed",
                       "batched", "adjoint"])
    if kind == "vec":
        return {"kind": kind, "n": size(1000, 2**24)}
    if kind == "mult":
        op = rng.choice(["poisson3d", "convdiff3d", "graph"])
        return {"kind": kind, "op": op, "k": size(1000, 100000) if op == "graph" else size(9, 120)}
    if kind == "solve":
        op, ksp, pc, lo, hi = rng.choice([
            ("poisson2d", "gmres", "ilu", 20, 100), ("poisson2d", "cg", "ilu", 20, 200),
            ("poisson2d", "cg", "icc", 20, 200), ("poisson2d", "fgmres", "jacobi", 20, 64),
            ("poisson3d", "cg", "jacobi", 12, 120), ("poisson3d", "cg", "icc", 12, 100),
            ("poisson3d", "gmres", "ilu", 12, 64), ("poisson3d", "bcgs", "sor", 12, 80),
            ("convdiff3d", "gmres", "ilu", 12, 90), ("graph", "cg", "icc", 1000, 60000),
        ])
        return {"kind": kind, "op": op, "k": size(lo, hi), "ksp": ksp, "pc": pc}
    if kind == "batched":
        return {"kind": kind, "count": size(4, 20), "nmin": 1024, "nmax": size(2048, 16384),
                "pc": rng.choice(["jacobi", "icc"])}
    return {"kind": kind, "k": size(24, 90) if kind == "mixed" else size(24, 160)}


# ------------------------------------------------------------------ operators
@functools.lru_cache(maxsize=8)
def _grid_operator(op, k):
    make = {"poisson2d": gallery.laplacian_2d, "poisson3d": gallery.laplacian_3d,
            "convdiff3d": gallery.convection_diffusion_3d}
    return make[op](k)


def _operator(op, k, seed):
    if op == "graph":
        return gallery.rgg_laplacian(k, np.random.default_rng(seed + 1))
    return _grid_operator(op, k)


def _mat(ip, ix, v):
    n = len(ip) - 1
    A = PETSc.Mat().createSeqAIJ((n, n))
    A.setValuesCSR(ip, ix, v)
    A.assemble()
    return A


def _rhs(n, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, n)


def _on_device(vec):
    """A Vec's device block as a tensor, without a copy."""
    return torch.as_tensor(vec._d, device="cuda")


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return {"vec": _prepare_vec, "mult": _prepare_mult, "solve": _prepare_solve,
            "mixed": _prepare_mixed, "batched": _prepare_batched,
            "adjoint": _prepare_adjoint}[case["kind"]](case, seed)


def run(state):
    return {"vec": _run_vec, "mult": _run_mult, "solve": _run_solve, "mixed": _run_mixed,
            "batched": _run_batched, "adjoint": _run_adjoint}[state["kind"]](state)


def work(case):
    return {"vec": _work_vec, "mult": _work_mult, "solve": _work_solve, "mixed": _work_mixed,
            "batched": _work_batched, "adjoint": _work_adjoint}[case["kind"]](case)


def exact(case, seed):
    return {"vec": _exact_vec, "mult": _exact_mult, "solve": _exact_solve,
            "mixed": _exact_mixed, "batched": _exact_batched,
            "adjoint": _exact_adjoint}[case["kind"]](case, seed)


# ------------------------------------------------------------------ vec
def _vec_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x, y, d = (rng.standard_normal(case["n"]) for _ in range(3))
    return x, y, d


def _prepare_vec(case, seed):
    x, y, d = (PETSc.Vec().createWithArray(a) for a in _vec_inputs(case, seed))
    s = {"kind": "vec", "x": x, "y": y, "d": d, "w": x.duplicate(), "z": x.duplicate(),
         "p": x.copy(), "s": y.copy(), "q": d.copy()}
    x.dot(d)  # the inputs are on the device
    return s


def _run_vec(st):
    x, y, d, w, z, p, s, q = (st[k] for k in "xydwzpsq")
    w.waxpy(-0.75, x, y)
    z.pointwiseMult(w, d)
    p.aypx(0.5, z)
    s.axpbypcz(0.25, -0.5, 0.5, x, p)
    q.axpy(-0.125, s)
    q.scale(0.5)
    q.maxpy([0.5, -0.25, 0.125, 0.0625], [x, y, p, s])
    dot, sq = z.dotNorm2(p)
    return {"dot": x.dot(y), "norm": q.norm(), "norm1": w.norm(PETSc.NormType.NORM_1),
            "zp": dot, "zz": sq, "w": _on_device(w), "z": _on_device(z), "p": _on_device(p),
            "s": _on_device(s), "q": _on_device(q)}


def _work_vec(case):
    # waxpy 3, mult 3, aypx 3, axpbypcz 4, axpy 3, scale 2, maxpy 6, reductions 6 operands
    n = case["n"]
    return {"bytes": 8.0 * 30 * n, "flops": 28.0 * n}


def _exact_vec(case, seed):
    x, y, d = (torch.from_numpy(a).to("cuda") for a in _vec_inputs(case, seed))
    w = y - 0.75 * x
    z = w * d
    p = z + 0.5 * x
    s = 0.25 * x - 0.5 * p + 0.5 * y
    q = 0.5 * (d - 0.125 * s) + 0.5 * x - 0.25 * y + 0.125 * p + 0.0625 * s
    return {"dot": float(x @ y), "norm": float(q.norm()), "norm1": float(w.abs().sum()),
            "zp": float(z @ p), "zz": float(z @ z), "w": w, "z": z, "p": p, "s": s, "q": q}


# ------------------------------------------------------------------ mult
def _prepare_mult(case, seed):
    A = _mat(*_operator(case["op"], case["k"], seed))
    n = A.getSize()[0]
    x = PETSc.Vec().createWithArray(_rhs(n, seed))
    v = PETSc.Vec().createWithArray(_rhs(n, seed + 1))
    st = {"kind": "mult", "A": A, "x": x, "v": v, "y": x.duplicate(), "z": x.duplicate(),
          "t": x.duplicate()}
    A.multTranspose(x, st["t"])  # A's transposed layout, made once per pattern
    A.multAdd(x, v, st["z"])
    return st


def _run_mult(st):
    A, x, v, y, z, t = (st[k] for k in ("A", "x", "v", "y", "z", "t"))
    A.mult(x, y)
    A.multAdd(x, v, z)
    A.multTranspose(x, t)
    return {"y": _on_device(y), "z": _on_device(z), "t": _on_device(t)}


def _size(op, k):
    """Rows and nonzeros (the graph's: on average)."""
    if op == "graph":
        return k, 9 * k
    n = k * k if op == "poisson2d" else k**3
    return n, (5 * n - 4 * k if op == "poisson2d" else 7 * n - 6 * k * k)


def _matrix_bytes(op, k):
    """Value and column of every nonzero and the row pointers, the columns of
    the stencils as 16-bit offsets where they fit."""
    n, nnz = _size(op, k)
    wide = op == "graph" or k * k > 32767 and op != "poisson2d"
    return (12 if wide else 10) * nnz + 4 * n


def _work_mult(case):
    n, nnz = _size(case["op"], case["k"])
    # three products, each reading the operator and one vector and writing one
    return {"bytes": 3.0 * (_matrix_bytes(case["op"], case["k"]) + 16 * n) + 8.0 * n,
            "flops": 6.0 * nnz}


def _torch_csr(ip, ix, v):
    return torch.sparse_csr_tensor(torch.from_numpy(np.asarray(ip, dtype=np.int64)),
                                   torch.from_numpy(np.asarray(ix, dtype=np.int64)),
                                   torch.from_numpy(v), size=(len(ip) - 1,) * 2).to("cuda")


def _transposed(ip, ix, v):
    n = len(ip) - 1
    rows = np.repeat(np.arange(n), np.diff(ip))
    order = np.argsort(ix, kind="stable")
    tip = np.concatenate([[0], np.cumsum(np.bincount(ix, minlength=n))])
    return tip, rows[order], v[order]


def _exact_mult(case, seed):
    ip, ix, v = _operator(case["op"], case["k"], seed)
    n = len(ip) - 1
    x, add = (torch.from_numpy(_rhs(n, seed + i)).to("cuda") for i in (0, 1))
    y = _torch_csr(ip, ix, v) @ x
    return {"y": y, "z": y + add, "t": _torch_csr(*_transposed(ip, ix, v)) @ x}


# ------------------------------------------------------------------ solve
def _rtol(case):
    # BiCGStab's stopping estimate moves by several iterations with the last
    # bit of a sum, so it is held to more digits than the others
    return 1e-12 if case["ksp"] == "bcgs" else 1e-10


def _prepare_solve(case, seed):
    A = _mat(*_operator(case["op"], case["k"], seed))
    n = A.getSize()[0]
    pc = PETSc.PC().create()
    pc.setType(case["pc"])
    if case["pc"] == "sor":
        pc.setSOROmega(1.2)
    pc.setOperators(A)
    ksp = PETSc.KSP().create()
    ksp.setPC(pc)
    ksp.setType(case["ksp"])
    ksp.setOperators(A)
    ksp.setTolerances(rtol=_rtol(case), atol=1e-50, divtol=1e30, max_it=10000)
    if case["ksp"] in ("gmres", "fgmres"):
        ksp.setGMRESRestart(30)
    ksp.setUp()
    return {"kind": "solve", "A": A, "ksp": ksp, "rhs": _rhs(n, seed),
            "b": PETSc.Vec().createSeq(n), "x": PETSc.Vec().createSeq(n)}


def _run_solve(st):
    st["b"].setArray(st["rhs"])
    st["ksp"].solve(st["b"], st["x"])
    return st["x"].getArray(readonly=True)


# iterations per grid line (per cube root, or square root, of the rows) and the
# triangular or SOR sweeps, products and vector passes of one iteration
_ITS = {("poisson2d", "gmres", "ilu"): 3.0, ("poisson2d", "cg", "ilu"): 1.2,
        ("poisson2d", "cg", "icc"): 1.2, ("poisson2d", "fgmres", "jacobi"): 14.0,
        ("poisson3d", "cg", "jacobi"): 4.2, ("poisson3d", "cg", "icc"): 1.45,
        ("poisson3d", "gmres", "ilu"): 2.6, ("poisson3d", "bcgs", "sor"): 0.95,
        ("convdiff3d", "gmres", "ilu"): 0.28, ("graph", "cg", "icc"): 0.25}


def _iterations(case):
    k = case["k"] ** 0.5 if case["op"] == "graph" else case["k"]
    return max(1.0, _ITS[case["op"], case["ksp"], case["pc"]] * k)


def _iteration_work(case):
    op, k, ksp, pc = case["op"], case["k"], case["ksp"], case["pc"]
    n, nnz = _size(op, k)
    applies = 2 if ksp == "bcgs" else 1
    # one product and one apply each, the apply reading the factor (or the
    # operator) and one vector and writing one
    precond = 24 * n if pc == "jacobi" else _matrix_bytes(op, k) + 16 * n
    # vectors read and written besides: CG's three updates and two dots, or a
    # basis of 15 on average projected and subtracted, or BiCGStab's updates
    vectors = {"cg": 11, "gmres": 34, "fgmres": 36, "bcgs": 22}[ksp]
    byts = applies * (_matrix_bytes(op, k) + 16 * n + precond) + 8 * vectors * n
    return byts, applies * 4 * nnz + 2 * vectors * n


def _work_solve(case):
    n, _ = _size(case["op"], case["k"])
    byts, flops = _iteration_work(case)
    its = _iterations(case)
    return {"bytes": its * byts + 32.0 * n, "flops": its * flops}


def _sine_solve(k, dims, b):
    """The solution of the constant-coefficient Poisson systems in 64 bits by
    their sine eigenvectors: S b S ... / eigenvalues, S = S^-1 the sine matrix."""
    i = np.arange(1, k + 1)
    S = np.sqrt(2.0 / (k + 1)) * np.sin(np.pi * np.outer(i, i) / (k + 1))
    lam = 2.0 - 2.0 * np.cos(np.pi * i / (k + 1))

    def transform(u):
        for axis in range(dims):
            u = np.moveaxis(np.tensordot(S, u, axes=(1, axis)), 0, axis)
        return u

    ev = sum(lam.reshape([-1 if a == ax else 1 for a in range(dims)]) for ax in range(dims))
    return transform(transform(b.reshape((k,) * dims)) / ev).reshape(-1)


def _bicgstab64(A, b, scale, its=4000):
    """One plain BiCGStab run in 64 bits, diagonally scaled from the right."""
    x = torch.zeros_like(b)
    r = b.clone()
    hat, p = r.clone(), r.clone()
    rho = float(hat @ r)
    stop = 1e-9 * float(b.norm())
    for _ in range(its):
        y = p * scale
        v = A @ y
        d = float(hat @ v)
        if d == 0.0:
            break
        alpha = rho / d
        s = r - alpha * v
        z = s * scale
        t = A @ z
        tt = float(t @ t)
        omega = float(t @ s) / tt if tt else 0.0
        x += alpha * y + omega * z
        r = s - omega * t
        if float(r.norm()) <= stop or omega == 0.0:
            break
        new = float(hat @ r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x


def _cg64(A, b, scale, its=20000):
    """One plain CG run in 64 bits, diagonally scaled."""
    x = torch.zeros_like(b)
    r = b.clone()
    z = r * scale
    p = z.clone()
    rz = float(r @ z)
    stop = 1e-9 * float(b.norm())
    for _ in range(its):
        w = A @ p
        alpha = rz / float(p @ w)
        x += alpha * p
        r -= alpha * w
        if float(r.norm()) <= stop:
            break
        z = r * scale
        new = float(r @ z)
        p = z + (new / rz) * p
        rz = new
    return x


def _refined(ip, ix, v, b, symmetric):
    """A^-1 b in 64 bits: runs of the iteration above on the true residual,
    until that no longer falls."""
    n = len(ip) - 1
    rows = np.repeat(np.arange(n), np.diff(ip))
    diag = np.zeros(n)
    diag[rows[rows == ix]] = v[rows == ix]
    A = _torch_csr(ip, ix, v)
    scale = torch.from_numpy(1.0 / diag).to("cuda")
    b = torch.from_numpy(b).to("cuda")
    x, best = torch.zeros_like(b), float("inf")
    for _ in range(6):
        r = b - A @ x
        norm = float(r.norm())
        if norm == 0.0 or norm > 0.5 * best:
            break
        best = norm
        x = x + (_cg64 if symmetric else _bicgstab64)(A, r, scale)
    return x.cpu().numpy()


def _exact_solve(case, seed):
    ip, ix, v = _operator(case["op"], case["k"], seed)
    b = _rhs(len(ip) - 1, seed)
    if case["op"].startswith("poisson"):
        return _sine_solve(case["k"], 2 if case["op"] == "poisson2d" else 3, b)
    return _refined(ip, ix, v, b, case["op"] == "graph")


# ------------------------------------------------------------------ mixed
def _prepare_mixed(case, seed):
    A = _mat(*_operator("convdiff3d", case["k"], seed))
    n = A.getSize()[0]
    solver = MixedSolver(A)
    solver.pc.setUp()
    return {"kind": "mixed", "A": A, "solver": solver, "rhs": _rhs(n, seed),
            "b": PETSc.Vec().createSeq(n), "x": PETSc.Vec().createSeq(n)}


def _run_mixed(st):
    st["b"].setArray(st["rhs"])
    st["solver"].solve(st["b"], st["x"], rtol=1e-10)
    return st["x"].getArray(readonly=True)


def _work_mixed(case):
    n, nnz = _size("convdiff3d", case["k"])
    its = max(8.0, 0.6 * case["k"])  # inner steps: FP32 operator, factor and basis
    return {"bytes": its * 4.0 * (3 * nnz + 36 * n) + 40.0 * nnz, "flops": its * (4.0 * nnz + 70 * n)}


def _exact_mixed(case, seed):
    ip, ix, v = _operator("convdiff3d", case["k"], seed)
    return _refined(ip, ix, v, _rhs(len(ip) - 1, seed), False)


# ------------------------------------------------------------------ batched
def _systems(case, seed):
    rng = np.random.default_rng(seed)
    # sizes log-uniform, the same for every seed: what differs is the graphs
    sizes = np.exp(np.linspace(np.log(case["nmin"]), np.log(case["nmax"]), case["count"]))
    return [gallery.rgg_laplacian(int(s), rng) for s in sizes]


def _batched_rhs(rows, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(rows, NRHS, dtype=torch.float64, device="cuda", generator=g)


def _prepare_batched(case, seed):
    systems = _systems(case, seed)
    solver = BatchedCG(systems, nrhs=NRHS)
    return {"kind": "batched", "solver": solver, "B": _batched_rhs(solver.n, seed),
            "pc": case["pc"]}


def _run_batched(st):
    X, _ = st["solver"].solve(st["B"], pc=st["pc"], rtol=1e-10)
    return X


def _work_batched(case):
    rows = float(np.exp(np.linspace(np.log(case["nmin"]), np.log(case["nmax"]),
                                    case["count"])).sum())
    its = 250.0 if case["pc"] == "jacobi" else 70.0
    per = 9 * 12 * rows + 8 * NRHS * 11 * rows
    if case["pc"] == "icc":
        per += 9 * 12 * rows + 8 * NRHS * 4 * rows
    return {"bytes": its * per, "flops": its * NRHS * rows * (18.0 + 12)}


def _exact_batched(case, seed):
    systems = _systems(case, seed)
    rows = sum(len(ip) - 1 for ip, _, _ in systems)
    B, out, at = _batched_rhs(rows, seed), [], 0
    for ip, ix, v in systems:
        n = len(ip) - 1
        A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        i = torch.from_numpy(np.repeat(np.arange(n), np.diff(ip))).to("cuda")
        A[i, torch.from_numpy(ix.astype(np.int64)).to("cuda")] = torch.from_numpy(v).to("cuda")
        b = B[at:at + n]
        L = torch.linalg.cholesky(A)
        x = torch.cholesky_solve(b, L)
        out.append(x + torch.cholesky_solve(b - A @ x, L))
        at += n
        del A, L
    return torch.cat(out)


# ------------------------------------------------------------------ adjoint
def _advection(case, seed):
    k = case["k"]
    rng = np.random.default_rng(seed)
    kappa = np.exp(gallery.gaussian_random_field(k, rng, corr=16.0))
    ip, ix, v = gallery.advection_diffusion_2d(kappa, peclet=2.0)
    observed = 0.1 * gallery.gaussian_random_field(k, rng, corr=16.0).reshape(-1)
    b = np.full(k * k, 1.0 / (k + 1) ** 2)
    return ip, ix, v, b, observed


def _prepare_adjoint(case, seed):
    ip, ix, v, b, observed = _advection(case, seed)
    dev = {"device": "cuda"}
    return {"kind": "adjoint", "system": SparseSystem(ip, ix, rtol=1e-10),
            "values": torch.tensor(v, requires_grad=True, **dev),
            "b": torch.tensor(b, requires_grad=True, **dev),
            "observed": torch.tensor(observed, **dev)}


def _run_adjoint(st):
    values, b = st["values"], st["b"]
    values.grad = b.grad = None
    u = sparse_solve(values, b, st["system"])
    ((u - st["observed"]) ** 2).sum().backward()
    return {"u": u.detach(), "values": values.grad, "b": b.grad}


def _work_adjoint(case):
    like = {"op": "poisson2d", "k": case["k"], "ksp": "gmres", "pc": "ilu"}
    byts, flops = _iteration_work(like)
    its = 2.0 * max(1.0, 0.95 * case["k"])  # forward and adjoint
    return {"bytes": its * byts, "flops": its * flops}


def _block_solve(ip, ix, v, k, b, transpose):
    """A^-1 b, or A^-T b, of a k^2 grid operator in 64 bits: block elimination
    over the grid's lines (blocks of k x k, refined once)."""
    n = k * k
    if transpose:
        ip, ix, v = _transposed(ip, ix, v)
    rows = np.repeat(np.arange(n), np.diff(ip))
    A = _torch_csr(ip, ix, v)
    D = torch.zeros(k, k, k, dtype=torch.float64)
    lo, up = torch.zeros(k, k, dtype=torch.float64), torch.zeros(k, k, dtype=torch.float64)
    same = rows // k == ix // k
    D[rows[same] // k, rows[same] % k, ix[same] % k] = torch.from_numpy(v[same])
    below, above = ix == rows - k, ix == rows + k
    lo[rows[below] // k, rows[below] % k] = torch.from_numpy(v[below])
    up[rows[above] // k, rows[above] % k] = torch.from_numpy(v[above])
    D, lo, up = D.to("cuda"), lo.to("cuda"), up.to("cuda")
    inv = []
    for j in range(k):
        M = D[j] if j == 0 else D[j] - lo[j][:, None] * inv[j - 1] * up[j - 1][None, :]
        inv.append(torch.linalg.inv(M))

    def once(r):
        r = r.reshape(k, k)
        f, x = [r[0]], [None] * k
        for j in range(1, k):
            f.append(r[j] - lo[j] * (inv[j - 1] @ f[j - 1]))
        x[k - 1] = inv[k - 1] @ f[k - 1]
        for j in range(k - 2, -1, -1):
            x[j] = inv[j] @ (f[j] - up[j] * x[j + 1])
        return torch.stack(x).reshape(-1)

    x = once(b)
    return x + once(b - A @ x)


def _exact_adjoint(case, seed):
    ip, ix, v, b, observed = _advection(case, seed)
    k = case["k"]
    u = _block_solve(ip, ix, v, k, torch.from_numpy(b).to("cuda"), False)
    g = 2.0 * (u - torch.from_numpy(observed).to("cuda"))
    lam = _block_solve(ip, ix, v, k, g, True)
    rows = torch.from_numpy(np.repeat(np.arange(k * k), np.diff(ip))).to("cuda")
    cols = torch.from_numpy(ix.astype(np.int64)).to("cuda")
    return {"u": u, "values": -lam[rows] * u[cols], "b": lam}
