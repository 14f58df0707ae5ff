"""Whole fronts of one warp (m <= 32) that take A's entries and their children's at the same places: the sums come out the
same bits in every repeat and reproduce the matrix (tolerance as in test_gpu_group_panel.py)."""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import EPS, bordered, dense_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [A.CHOLESKY, A.LDLT, A.LDLT_BK])
@pytest.mark.parametrize("sizes,border", [([1], 1), ([2] * 5, 6), ([7] * 40, 9), ([12, 5] * 20, 16), ([3] * 70, 29)])
def test_children_over_matrix_entries(sizes, border, kind):
    M = bordered(sizes, border, 13, indefinite=kind != A.CHOLESKY)
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(pat.n, dtype=np.int32), relax=False)
    num = A.NumericFactor(sym, kind)
    first = None
    for _ in range(20):
        assert num.factor(v)
        first = num.Lx.copy() if first is None else first
        assert np.array_equal(num.Lx, first)
    b = np.random.default_rng(1).uniform(-1, 1, (2, pat.n))
    ref = np.linalg.solve(M, b.T).T
    assert np.max(np.abs(num.solve_block(b) - ref)) <= 10 * 10 * pat.n * EPS[A.FP64] * np.max(np.abs(ref))
