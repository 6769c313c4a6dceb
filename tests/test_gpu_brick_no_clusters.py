"""Bricks on a device that cannot hold a cluster of them (asked of the device at
set-up; GPETSC_BRICK_CLUSTERS=0 stands for its no): the sweeps run without, equal to
the oracle bit for bit.  In a process of its own: the answer is read once."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CODE = """
import sys
sys.path[:0] = [{here!r}, {root!r} + "/mojo-petsc4py_gb300", {root!r} + "/oracle"]
import numpy as np
import oracle as O
from mojopetsc4py import _lib
from test_gpu_bricks import _operator, _symmetric
from test_gpu_sweeps import _apply, _mat, _pc
_lib.set_arithmetic("ordered")
_lib.set_sweep_bricks(2)
for pt, gopts, oopts in (("ilu", {{}}, {{}}), ("icc", {{}}, {{}}),
                         ("sor", {{"setSOROmega": 1.2}}, {{"omega": 1.2}})):
    ip, ix, v = _operator((33, 41, 34))
    if pt == "icc":
        ip, ix, v = _symmetric(ip, ix, v)
    pc = _pc(pt, _mat(ip, ix, v), gopts)
    oracle = O.OraclePC(pt, ip, ix, v, **oopts)
    for seed in range(3):
        x = np.random.default_rng(seed).normal(size=len(ip) - 1)
        np.testing.assert_array_equal(_apply(pc, x), oracle.apply(x))
"""


@pytest.mark.parametrize("fits", [True, False])
def test_without_room_for_a_cluster(fits):
    env = dict(os.environ, GPETSC_SWEEP_VERBOSE="1")
    env.pop("GPETSC_BRICK_CLUSTERS", None)
    if not fits:
        env["GPETSC_BRICK_CLUSTERS"] = "0"
    code = CODE.format(here=HERE, root=os.path.dirname(HERE))
    run = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    assert run.stderr.count("clusters of") == 3
    assert ("clusters of 1x1 and 1x1" in run.stderr) == (not fits)
