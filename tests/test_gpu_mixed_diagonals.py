"""Mixed precision on matrices stored by diagonals: triangle passes and the FP32
multiply at the edges of their tiles (2048 rows a CTA, 512 for the multiply, four
rows a 16-byte load), one to eight diagonals a triangle, beside the forms that
other matrices keep (more than eight diagonals, a missing one in the widest row).
Lower and upper offsets start at n // 3, so a triangle's dependencies are at most
three deep and three passes are the exact triangular solve: inner iterations then
match the exact FP64 sweeps' (the multicolour test's margin of 2)."""
import numpy as np
import pytest

from mojopetsc4py import PETSc

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed, drop=None):
    """Diagonally dominant rows with entries at the given offsets (in range)."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    rows, cols, vals = [i], [i], [np.full(n, 2.0 * len(offsets))]
    for o in offsets:
        k = i[(i + o >= 0) & (i + o < n)]
        if drop:
            k = k[k % drop != abs(o) % drop]
        rows.append(k)
        cols.append(k + o)
        vals.append(rng.uniform(-1.5, 1.5, k.size))
    r, c, v = map(np.concatenate, (rows, cols, vals))
    p = np.lexsort((c, r))
    ip = np.concatenate(([0], np.cumsum(np.bincount(r, minlength=n))))
    return ip.astype(np.int32), c[p].astype(np.int32), v[p]


def solve(A, s, b, sweeps):
    x = PETSc.Vec().createSeq(len(b))
    info = s.solve(PETSc.Vec().createWithArray(b), x, rtol=1e-10, tri_sweeps=sweeps)
    return info, x.getArray()


def check(ip, ix, v, b, info, x):
    rows = np.repeat(np.arange(len(ip) - 1), np.diff(ip))
    ax = np.bincount(rows, weights=v * x[ix], minlength=len(ip) - 1)
    assert info["converged"]
    assert np.linalg.norm(b - ax) <= 1.05e-10 * np.linalg.norm(b)


CASES = [(n, w, None) for n, w in [(1, 1), (2, 1), (3, 1), (7, 1), (511, 2), (513, 3), (2047, 1),
                                   (2048, 2), (2049, 3), (4099, 3), (6001, 4), (6002, 8),
                                   (6003, 9)]] + [(4098, 3, 2), (4097, 2, 5)]


@pytest.mark.parametrize("n,w,drop", CASES)
def test_passes_by_diagonals(n, w, drop):
    from mojopetsc4py.mixed import MixedSolver

    p = max(1, n // 3)
    offsets = [o for e in range(w) for o in (-(p + e), p + e)]
    ip, ix, v = banded(n, offsets, n + w, drop)
    A = PETSc.Mat().createSeqAIJ((n, n))
    A.setValuesCSR(ip, ix, v)
    A.assemble()
    b = np.random.default_rng(5).uniform(-1, 1, n)
    s = MixedSolver(A)
    three, x3 = solve(A, s, b, 3)
    check(ip, ix, v, b, three, x3)
    exact, x0 = solve(A, s, b, 0)
    check(ip, ix, v, b, exact, x0)
    assert abs(three["inner_its"] - exact["inner_its"]) <= 2
    # new values in the same pattern: the diagonals follow
    v2 = v * np.random.default_rng(6).uniform(0.8, 1.2, v.size)
    A.setValuesCSR(ip, ix, v2)
    A.assemble()
    again, x2 = solve(A, s, b, 3)
    check(ip, ix, v2, b, again, x2)
    fresh, xf = solve(A, MixedSolver(A), b, 3)
    assert again["inner_its"] == fresh["inner_its"] and np.array_equal(x2, xf)
