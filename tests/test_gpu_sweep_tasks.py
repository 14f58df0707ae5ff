"""GPU solve sweeps at the edges of their task kinds: one-warp supernodes in tasks of more than four, whole-supernode
tasks up to and beyond their row limit, block tasks with remainders, vector counts around the slices of 16, against
numpy. Tolerance as in test_gpu_group_panel.py (condition numbers below 10)."""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import EPS, bordered, dense_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,precision", [(A.CHOLESKY, A.FP64), (A.CHOLESKY, A.MIXED), (A.LDLT, A.FP64),
                                            (A.LDLT_BK, A.FP64)])
@pytest.mark.parametrize("sizes,border", [([2] * 19, 5), ([20, 40], 193), ([20, 40], 237), ([64, 65], 192),
                                          ([3] * 9 + [30, 200], 460)])
def test_vector_counts(sizes, border, kind, precision):
    M = bordered(sizes, border, 17, indefinite=kind != A.CHOLESKY)
    n = M.shape[0]
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32), relax=False)
    num = A.NumericFactor(sym, kind, precision)
    assert num.factor(v)
    B = np.random.default_rng(4).uniform(-1, 1, (64, n))
    ref = np.linalg.solve(M, B.T).T
    for q in (1, 2, 15, 16, 17, 33, 64, 1):
        X = num.solve_block(B[:q])
        assert np.max(np.abs(X - ref[:q])) <= 10 * 10 * n * EPS[precision] * np.max(np.abs(ref[:q]))
