"""GMRES and FGMRES trips of several Arnoldi steps, and the step's fused
projection, norm and control: restarts that the steps of a trip divide and that
they do not, an iteration limit inside a trip, and right-hand sides at the ends
of the exponent range (where v / ||v|| leaves the corrected-quotient form)."""
import numpy as np
import pytest

from mojopetsc4py import gallery
from helpers import oracle_solve
from test_gpu_ksp import solve_gpu

pytestmark = pytest.mark.gpu

TOL = dict(rtol=1e-9, atol=1e-300, divtol=1e30, max_it=400)


def _both(kt, m, tol, scale=1.0):
    ip, ix, v = gallery.convection_diffusion_3d(7)
    n = len(ip) - 1
    b = np.random.default_rng(2).uniform(-1.0, 1.0, n) * scale
    g = solve_gpu(kt, "jacobi", ip, ix, v, b, tol=tol, ksp_opts={"setGMRESRestart": m})
    r = oracle_solve(kt, ip, ix, v, b, pt="jacobi", restart=m, **tol)
    assert (g["reason"], g["its"]) == (r["reason"], r["its"])
    return g, r


@pytest.mark.parametrize("m", [1, 2, 3, 7, 10, 13, 20, 30, 45])
@pytest.mark.parametrize("kt", ["gmres", "fgmres"])
def test_steps_of_a_trip_equal_the_oracle(kt, m):
    g, r = _both(kt, m, TOL)
    np.testing.assert_array_equal(g["x"], r["x"])


@pytest.mark.fma
@pytest.mark.parametrize("m", [1, 3, 7, 10, 30, 45])
@pytest.mark.parametrize("kt", ["gmres", "fgmres"])
def test_fused_steps_follow_the_oracle(kt, m):
    g, r = _both(kt, m, TOL)
    # the same recurrence with sums in another order: a relative 1e-16 a sum,
    # over at most 400 steps of a well-conditioned system
    assert np.linalg.norm(g["x"] - r["x"]) <= 1e-11 * np.linalg.norm(r["x"])


@pytest.mark.fma
@pytest.mark.parametrize("max_it", [0, 1, 5, 10, 11])
def test_an_iteration_limit_inside_a_trip(max_it):
    _both("gmres", 30, dict(TOL, max_it=max_it))


@pytest.mark.parametrize("scale", [1e-160, 1e-150, 1e150])
def test_normalisation_at_the_ends_of_the_range(scale):
    g, r = _both("gmres", 10, TOL, scale)
    np.testing.assert_array_equal(g["x"], r["x"])
