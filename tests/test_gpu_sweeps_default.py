"""The sweep form that a user gets without asking, in a run of all test files too
(settings are process-wide; this file comes after those that set them): bricks on
a Cartesian grid in natural order, in solves, transposed solves and the adjoint,
with nothing allocated by a repeated apply or solve."""
import numpy as np
import pytest
import torch

from mojopetsc4py import PETSc, _lib, gallery
from mojopetsc4py.adjoint import SparseSystem, sparse_solve
from test_gpu_sweeps import _mat, _pc

pytestmark = [pytest.mark.gpu, pytest.mark.fma]


def _bricks(pc):
    got = _lib.sweep_bricks(pc._handle())
    return got["forward"]["brick"] and got["backward"]["brick"]


@pytest.mark.parametrize("pt", ["ilu", "icc", "sor"])
def test_a_grid_gets_bricks(pt):
    assert _bricks(_pc(pt, _mat(*gallery.laplacian_3d(20)), {}))
    assert _bricks(_pc(pt, _mat(*gallery.laplacian_2d(40)), {}))


def test_settings_without_arguments_are_the_default():
    _lib.set_sweep_bricks(0)
    assert not _bricks(_pc("ilu", _mat(*gallery.laplacian_3d(20)), {}))
    _lib.set_sweep_bricks()
    assert _bricks(_pc("ilu", _mat(*gallery.laplacian_3d(20)), {}))


def test_transposed_solve():
    ip, ix, v = gallery.convection_diffusion_3d(20)
    n = len(ip) - 1
    A = _mat(ip, ix, v)
    b = np.random.default_rng(0).uniform(-1.0, 1.0, n)
    x = PETSc.Vec().createSeq(n)
    ksp = PETSc.KSP().create()
    ksp.setType("gmres")
    ksp.getPC().setType("ilu")
    ksp.setOperators(A)
    ksp.setTolerances(rtol=1e-10, atol=1e-50, divtol=1e30, max_it=500)
    ksp.solveTranspose(PETSc.Vec().createWithArray(b), x)
    assert _bricks(ksp.getPC())
    rows = np.repeat(np.arange(n), np.diff(ip))
    atx = np.bincount(ix, weights=v * x.getArray()[rows], minlength=n)
    # the preconditioned residual is at 1e-10 of its start; the true one follows
    # within the preconditioner's condition number, below 1e3 here
    assert np.linalg.norm(b - atx) <= 1e-7 * np.linalg.norm(b)


def test_adjoint_equals_the_level_order():
    k = 40
    ip, ix, v = gallery.advection_diffusion_2d(np.ones((k, k)), peclet=2.0)
    out = []
    for mode in (1, 0):
        _lib.set_sweep_bricks(mode)
        _lib.set_sweep_form(mode == 1, 0)
        values = torch.tensor(v, device="cuda", requires_grad=True)
        b = torch.linspace(-1.0, 1.0, k * k, dtype=torch.float64, device="cuda",
                           requires_grad=True)
        system = SparseSystem(ip, ix, rtol=1e-10)
        sparse_solve(values, b, system).square().sum().backward()
        out.append((values.grad.cpu().numpy(), b.grad.cpu().numpy()))
    _lib.set_sweep_bricks(1)
    _lib.set_sweep_form(True, 0)
    # the same operations in the same order: bit for bit
    for a, c in zip(*out):
        np.testing.assert_array_equal(a, c)


@pytest.mark.parametrize("pt", ["ilu", "icc", "sor"])
def test_applies_and_solves_allocate_nothing(pt):
    pc = _pc(pt, _mat(*gallery.laplacian_3d(20)), {})
    assert _bricks(pc)
    b = PETSc.Vec().createWithArray(np.random.default_rng(1).normal(size=8000))
    x, y = PETSc.Vec().createSeq(8000), PETSc.Vec().createSeq(8000)
    ksp = PETSc.KSP().create()
    ksp.setPC(pc)
    ksp.setType("cg")
    ksp.setOperators(pc._pmat)
    ksp.setTolerances(rtol=1e-8, atol=1e-50, divtol=1e30, max_it=200)
    pc.apply(b, y)
    ksp.solve(b, x)
    want, sol = y.getArray().copy(), x.getArray().copy()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(3):  # the faces' two copies are used in turn
        pc.apply(b, y)
        ksp.solve(b, x)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    np.testing.assert_array_equal(y.getArray(), want)
    np.testing.assert_array_equal(x.getArray(), sol)
