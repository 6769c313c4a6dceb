"""The brick sweeps with thread-block clusters of bricks (2 x 4 bricks of 16 x 8
lines in 3-D): grids of one cluster, of one and a part of one in either direction
(CTAs of a cluster with no brick, bricks with no second tile), lines shorter and
longer than a ring, one cluster at a time and all at once.  Equal to the oracle
bit for bit in the exact arithmetic, to the level-ordered form in the fused one."""
import numpy as np
import pytest

import oracle as O
from mojopetsc4py import _lib
from test_gpu_bricks import _operator, _restore, _symmetric  # noqa: F401
from test_gpu_sweeps import _apply, _mat, _pc

pytestmark = pytest.mark.gpu

BOXES = [(16, 32, 32), (32, 32, 33), (17, 9, 33), (33, 41, 5), (9, 33, 70), (48, 73, 34)]
TYPES = [("ilu", {}, {}), ("icc", {}, {}), ("sor", {"setSOROmega": 1.2}, {"omega": 1.2})]


@pytest.mark.parametrize("ctas", [0, 2])
@pytest.mark.parametrize("pt,gopts,oopts", TYPES)
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_clusters_equal_the_oracle(box, pt, gopts, oopts, ctas):
    ip, ix, v = _operator(box)
    if pt == "icc":
        ip, ix, v = _symmetric(ip, ix, v)
    _lib.set_sweep_bricks(2, 0, 0, ctas)
    pc = _pc(pt, _mat(ip, ix, v), gopts)
    assert _lib.sweep_bricks(pc._handle())["forward"]["brick"]
    oracle = O.OraclePC(pt, ip, ix, v, **oopts)
    for seed in range(3):
        x = np.random.default_rng(seed).normal(size=len(ip) - 1)
        np.testing.assert_array_equal(_apply(pc, x), oracle.apply(x))


@pytest.mark.fma
@pytest.mark.parametrize("box", BOXES, ids=lambda b: "x".join(map(str, b)))
def test_fused_clusters_equal_the_level_order(box):
    ip, ix, v = _operator(box)
    x = np.random.default_rng(4).normal(size=len(ip) - 1)
    out = []
    for mode in (2, 0):
        _lib.set_sweep_bricks(mode)
        _lib.set_sweep_form(mode == 2, 0)
        pcs = [_pc(pt, _mat(*(_symmetric(ip, ix, v) if pt == "icc" else (ip, ix, v))), g)
               for pt, g, _ in TYPES]
        out.append([_apply(pc, s * x) for s in (1.0, -2.0, 0.5) for pc in pcs])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
