"""BiCGStab's fused iteration: the d2 == 0 branch (S vanishes after the first
half step), limits that fall inside a trip of several iterations, and vector
lengths around a block and a whole reduction grid."""
import numpy as np
import pytest

from mojopetsc4py import gallery
from helpers import oracle_solve
from test_gpu_ksp import solve_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.fma]

TOL = dict(rtol=1e-10, atol=1e-50, divtol=1e30, max_it=500)


def _run(ip, ix, v, b, pt="none", tol=TOL):
    return (solve_gpu("bcgs", pt, ip, ix, v, b, tol=tol),
            oracle_solve("bcgs", ip, ix, v, b, pt=pt, **tol))


def test_a_half_step_that_solves_takes_the_zero_branch():
    n = 1000
    ip = np.arange(n + 1, dtype=np.int32)
    b = np.random.default_rng(1).normal(size=n)
    g, r = _run(ip, ip[:-1].copy(), np.full(n, 2.0), b)
    assert (g["reason"], g["its"]) == (r["reason"], r["its"]) == (2, 1)
    np.testing.assert_array_equal(g["x"], r["x"])


@pytest.mark.parametrize("max_it", [0, 1, 3, 4, 5])
def test_an_iteration_limit_inside_a_trip(max_it):
    ip, ix, v = gallery.laplacian_2d(20)
    b = np.random.default_rng(2).normal(size=400)
    g, r = _run(ip, ix, v, b, "sor", dict(TOL, max_it=max_it))
    assert (g["reason"], g["its"]) == (r["reason"], r["its"])
    # at most five iterations of the same recurrence, sums in another order
    np.testing.assert_allclose(g["x"], r["x"], rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("k", [2, 15, 16, 17, 33])
def test_vector_lengths(k):
    ip, ix, v = gallery.convection_diffusion_3d(k)
    b = np.random.default_rng(3).uniform(-1.0, 1.0, k**3)
    g, r = _run(ip, ix, v, b, "jacobi")
    assert g["reason"] == r["reason"] and abs(g["its"] - r["its"]) <= 2
    # both within rtol of the solution of a well-conditioned system
    assert np.linalg.norm(g["x"] - r["x"]) <= 1e-8 * np.linalg.norm(r["x"])
