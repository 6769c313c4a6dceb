"""Which of the mixed form's matrices are read by diagonals: the ones whose entries
lie on at most eight (and, for the operator, with a row that has them all), the
others as sparse rows.  The cases of test_gpu_mixed_diagonals, so that those compare
what they name."""
import ctypes

import numpy as np
import pytest

from mojopetsc4py import PETSc, _lib
from mojopetsc4py.mixed import MixedSolver
from test_gpu_mixed_diagonals import CASES, banded

pytestmark = pytest.mark.gpu


def _form(ip, ix, v, **opts):
    n = len(ip) - 1
    A = PETSc.Mat().createSeqAIJ((n, n))
    A.setValuesCSR(ip, ix, v)
    A.assemble()
    s = MixedSolver(A, **opts)
    b = PETSc.Vec().createWithArray(np.random.default_rng(5).uniform(-1, 1, n))
    s.solve(b, PETSc.Vec().createSeq(n), tri_sweeps=3)
    got = (ctypes.c_int32 * 3)()
    _lib.check(_lib.lib().gp_mixed_form(s._h, got))
    return list(got)


@pytest.mark.parametrize("n,w,drop", CASES)
def test_forms(n, w, drop):
    p = max(1, n // 3)
    ip, ix, v = banded(n, [o for e in range(w) for o in (-(p + e), p + e)], n + w, drop)
    rows = np.repeat(np.arange(n), np.diff(ip))
    off = ix - rows
    lower, upper = (len(np.unique(off[side])) for side in (off < 0, off > 0))
    total = len(np.unique(off))
    tri = [lower, upper] if 1 <= lower <= 8 and 1 <= upper <= 8 else [0, 0]
    op = total if total <= 8 and np.diff(ip).max() == total else 0
    assert _form(ip, ix, v) == [op] + tri


def test_a_reordered_factor_is_read_as_rows():
    n = 600
    ip, ix, v = banded(n, [-20, -1, 1, 20], 1)
    assert _form(ip, ix, v) == [5, 2, 2]
    assert _form(ip, ix, v, ordering="multicolor") == [5, 0, 0]
