"""The brick form of the triangular sweeps at the edges of its tiles: warps take
8 x 4 grid lines (32 in 2-D), CTAs up to four such tiles, steps go in groups of
8 and 16, so lines of one row, grids one line wider or narrower than a tile or a
brick, and lines around a group's length are where it can go wrong.  Every apply
must equal the oracle's bit for bit in the exact arithmetic, and the
level-ordered form's in the fused one."""
import numpy as np
import pytest

import oracle as O
from mojopetsc4py import PETSc, _lib
from test_gpu_sweeps import _apply, _laplacian_box, _mat, _pc

pytestmark = pytest.mark.gpu

BOXES = [(2, 1, 1), (33, 1, 1), (31, 33, 1), (32, 32, 1), (5, 40, 1), (130, 3, 1), (3, 129, 1),
         (2, 2, 2), (8, 4, 2), (9, 5, 3), (17, 9, 20), (16, 8, 33), (33, 17, 5), (3, 2, 40),
         (25, 26, 27)]


@pytest.fixture(autouse=True)
def _restore():
    yield
    _lib.set_sweep_form(True, 0)
    _lib.set_sweep_bricks(1)


def _operator(box):
    """The box Laplacian with unsymmetric random values, diagonally dominant."""
    ip, ix, v = _laplacian_box(*box)
    rows = np.repeat(np.arange(len(ip) - 1), np.diff(ip))
    v = -np.random.default_rng(3).uniform(0.5, 1.0, len(v))
    v[rows == ix] = 7.0
    return ip, ix, v


def _symmetric(ip, ix, v):
    rows = np.repeat(np.arange(len(ip) - 1), np.diff(ip))
    w = -(1.0 + ((rows + ix) % 5) * 0.1)
    return ip, ix, np.where(rows == ix, 9.0, w)


@pytest.mark.parametrize("ctas", [0, 2])
@pytest.mark.parametrize("pt,gopts,oopts", [
    ("ilu", {}, {}), ("icc", {}, {}), ("sor", {"setSOROmega": 1.2}, {"omega": 1.2}),
    ("sor", {"setSORSymmetric": False}, {"symmetric": False})])
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_brick_sweeps_equal_the_oracle(box, pt, gopts, oopts, ctas):
    ip, ix, v = _operator(box)
    if pt == "icc":
        ip, ix, v = _symmetric(ip, ix, v)
    n = len(ip) - 1
    _lib.set_sweep_bricks(2, 0, 0, ctas)
    pc = _pc(pt, _mat(ip, ix, v), gopts)
    got = _lib.sweep_bricks(pc._handle())
    assert got["forward"]["brick"] and got["backward"]["brick"]
    oracle = O.OraclePC(pt, ip, ix, v, **oopts)
    for seed in range(3):  # the faces' two copies are used in turn
        x = np.random.default_rng(seed).normal(size=n)
        np.testing.assert_array_equal(_apply(pc, x), oracle.apply(x))


@pytest.mark.fma
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_fused_bricks_equal_the_level_order(box):
    """ILU, its transposed apply, IC and SOR in the fused arithmetic, with an
    infinity and a NaN in the input reaching the same rows."""
    ip, ix, v = _operator(box)
    n = len(ip) - 1
    x = np.random.default_rng(4).normal(size=n)
    wild = x.copy()
    wild[n // 2], wild[n - 1] = np.inf, np.nan
    out = []
    for mode in (2, 0):
        _lib.set_sweep_bricks(mode)
        _lib.set_sweep_form(mode == 2, 0)
        res = []
        for pt, sym in (("ilu", False), ("icc", True), ("sor", False)):
            pc = _pc(pt, _mat(*(_symmetric(ip, ix, v) if sym else (ip, ix, v))), {})
            res += [_apply(pc, x), _apply(pc, wild)]
            if pt == "ilu":
                pc.setUseExactTranspose(True)
                y = PETSc.Vec().createSeq(n)
                pc.applyTranspose(PETSc.Vec().createWithArray(x), y)
                res.append(y.getArray().copy())
        out.append(res)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_an_asked_for_form_goes_before_the_brick_form():
    ip, ix, v = _operator((9, 5, 3))
    _lib.set_sweep_bricks(1)
    for tiles, rows, brick in ((True, 0, True), (False, 0, False), (True, 64, False)):
        _lib.set_sweep_form(tiles, rows)
        pc = _pc("ilu", _mat(ip, ix, v), {})
        assert _lib.sweep_bricks(pc._handle())["forward"]["brick"] == brick
