"""GPU whole fronts (m <= 128, one warp or one CTA each) at the edges of their classes and eight-column steps, against
numpy; tolerances as in test_gpu_group_panel.py."""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import EPS, bordered, dense_csr, dominant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 72, 100, 121, 127, 128])
def test_dense_front(n):
    M = dominant(n, n)
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32))
    assert sym.nsuper == 1
    for precision in (A.FP64, A.MIXED):
        num = A.NumericFactor(sym, A.CHOLESKY, precision)
        assert num.factor(v)
        L = np.tril(num.Lx.reshape(n, n).T)
        assert np.max(np.abs(L @ L.T - M)) <= 10 * (n + 1) * EPS[precision] * np.max(np.abs(M))
    Mi = dominant(n, n, indefinite=True)
    num = A.NumericFactor(sym, A.LDLT)
    assert num.factor(Mi.reshape(-1))
    L, D = np.tril(num.Lx.reshape(n, n).T), num.D
    assert np.max(np.abs((L * D) @ L.T - Mi)) <= 10 * (n + 1) * EPS[A.FP64] * np.max(np.abs(Mi))
    assert num.nNeg == int(np.sum(np.linalg.eigvalsh(Mi) < 0))


@pytest.mark.parametrize("kind", [A.CHOLESKY, A.LDLT, A.LDLT_BK])
@pytest.mark.parametrize("sizes,border", [([3] * 40, 20), ([3] * 40, 41), ([9, 17, 30], 70), ([64, 5], 64), ([20] * 33, 108)])
def test_fronts_with_children(sizes, border, kind):
    """Parents of more children than are fetched at once, and of every class, with update blocks and remainders."""
    M = bordered(sizes, border, 3, indefinite=kind != A.CHOLESKY)
    n = M.shape[0]
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32), relax=False)
    num = A.NumericFactor(sym, kind)
    assert num.factor(v)
    B = np.random.default_rng(1).uniform(-1, 1, (2, n))
    X = num.solve_block(B)
    ref = np.linalg.solve(M, B.T).T
    assert np.max(np.abs(X - ref)) <= 10 * 10 * n * EPS[A.FP64] * np.max(np.abs(ref))


@pytest.mark.parametrize("n,exponent", [(50, -984), (50, 970), (101, -984), (101, 970)])
def test_pivots_outside_the_reciprocal_estimate(n, exponent):
    M = dominant(n, 5)
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32))
    num = A.NumericFactor(sym)
    assert num.factor(v)
    L = num.Lx.copy()
    assert num.factor(np.ldexp(v, exponent))
    assert np.max(np.abs(np.ldexp(num.Lx, -exponent // 2) - L)) <= 10 * (n + 1) * EPS[A.FP64] * np.max(np.abs(L))


@pytest.mark.parametrize("n,bad", [(20, 0), (20, 19), (50, 0), (50, 49), (101, 8), (101, 100)])
def test_first_failing_column(n, bad):
    M = dominant(n, 9)
    M[bad, bad] = -1.0
    pat, v = dense_csr(M)
    num = A.NumericFactor(A.analyze(pat, perm=np.arange(n, dtype=np.int32)))
    assert not num.factor(v)
    assert num.failColumn == bad
