"""A backward-only SOR apply (no forward half before it: its sweep starts from the
input) on grids in the brick form: one tile, several bricks, a part of a cluster.
Bit for bit the oracle's in the exact arithmetic and the level-ordered form's in the
fused one."""
import numpy as np
import pytest

import oracle as O
from mojopetsc4py import _lib
from test_gpu_bricks import _operator, _restore  # noqa: F401
from test_gpu_mp_abi import G, both  # noqa: F401

pytestmark = pytest.mark.gpu

BOXES = [(16, 16, 1), (131, 40, 1), (8, 4, 9), (17, 9, 20), (33, 41, 34)]
ZERO_GUESS, BACKWARD, LOCAL_BACKWARD = 16, 2, 8


def _args(box, omega, fshift, flag):
    ip, ix, v = _operator(box)
    n = len(ip) - 1
    ip, ix = O.i64(ip), O.i64(ix)
    dmark = np.zeros(n, np.int64)
    O.lib().mp_mat_get_diagonal_markers(O.a(ip), O.a(ix), O.a(dmark), n)
    x = np.random.default_rng(7).normal(size=n)
    return (x, np.zeros(n), ip, ix, v, dmark, np.zeros(n), np.zeros(n), np.zeros(3 * n), omega,
            fshift, flag | ZERO_GUESS, n)


@pytest.mark.parametrize("flag", [BACKWARD, LOCAL_BACKWARD])
@pytest.mark.parametrize("omega,fshift", [(1.0, 0.0), (1.3, 0.0), (0.8, 0.1)])
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_equals_the_oracle(G, box, omega, fshift, flag):  # noqa: F811
    _lib.set_sweep_bricks(2)
    (_, g), (_, o) = both(G, "mp_pc_sor_apply", *_args(box, omega, fshift, flag))
    np.testing.assert_array_equal(g[1], o[1])


@pytest.mark.fma
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_fused_equals_the_level_order(G, box):  # noqa: F811
    out = []
    for mode in (2, 0):
        _lib.set_sweep_bricks(mode)
        _lib.set_sweep_form(mode == 2, 0)
        (_, g), _ = both(G, "mp_pc_sor_apply", *_args(box, 1.3, 0.0, LOCAL_BACKWARD))
        out.append(g[1])
    np.testing.assert_array_equal(*out)
