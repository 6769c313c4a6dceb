"""The fused BiCGStab iteration in the exact arithmetic beside the general body, which
the ordered arithmetic runs: the same operations, the sums in another order."""
import numpy as np
import pytest

from mojopetsc4py import _lib, gallery
from test_gpu_ksp import solve_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.exact]

TOL = dict(rtol=1e-10, atol=1e-50, divtol=1e30, max_it=500)


def _both(ip, ix, v, b, pt, tol):
    out = []
    for mode in ("exact", "ordered"):
        _lib.set_arithmetic(mode)
        out.append(solve_gpu("bcgs", pt, ip, ix, v, b, tol=tol))
    return out


@pytest.mark.parametrize("max_it", [1, 2, 4, 5])
@pytest.mark.parametrize("pt", ["none", "jacobi", "sor", "ilu"])
def test_first_iterations(pt, max_it):
    ip, ix, v = gallery.convection_diffusion_3d(9)
    b = np.random.default_rng(2).uniform(-1.0, 1.0, 729)
    e, o = _both(ip, ix, v, b, pt, dict(TOL, max_it=max_it))
    assert (e["reason"], e["its"]) == (o["reason"], o["its"])
    # at most five iterations of the same recurrence, sums in another order
    np.testing.assert_allclose(e["x"], o["x"], rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("pt", ["jacobi", "sor", "ilu"])
def test_whole_solves(pt):
    ip, ix, v = gallery.convection_diffusion_3d(16)
    b = np.random.default_rng(3).uniform(-1.0, 1.0, 4096)
    e, o = _both(ip, ix, v, b, pt, TOL)
    assert e["reason"] == o["reason"] and abs(e["its"] - o["its"]) <= 2
    assert np.linalg.norm(e["x"] - o["x"]) <= 1e-8 * np.linalg.norm(o["x"])
