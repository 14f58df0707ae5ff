"""Multi-vector sweeps over levels with more block tasks than resident CTAs, whose supernodes of one pivot block are solved
whole, and over levels just below that, at the edges of the row limit and of the vector slices, against numpy. Tolerance as
in test_gpu_group_panel.py (condition numbers below 10)."""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import EPS, bordered, dense_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision", [(A.CHOLESKY, A.FP64), (A.CHOLESKY, A.MIXED), (A.LDLT, A.FP64),
                                            (A.LDLT_BK, A.FP64)])
@pytest.mark.parametrize("sizes,border", [([10] * 100, 237), ([33] * 60, 223), ([33] * 60, 224), ([64, 7] * 45, 192),
                                          ([20] * 89, 250)])
def test_many_supernodes_in_a_level(sizes, border, kind, precision):
    M = bordered(sizes, border, 19, indefinite=kind != A.CHOLESKY)
    n = M.shape[0]
    pat, v = dense_csr(M)
    num = A.NumericFactor(A.analyze(pat, perm=np.arange(n, dtype=np.int32), relax=False), kind, precision)
    assert num.factor(v)
    B = np.random.default_rng(4).uniform(-1, 1, (64, n))
    ref = np.linalg.solve(M, B.T).T
    for q in (2, 16, 17, 33, 64, 3):
        X = num.solve_block(B[:q])
        assert np.max(np.abs(X - ref[:q])) <= 10 * 10 * n * EPS[precision] * np.max(np.abs(ref[:q]))
