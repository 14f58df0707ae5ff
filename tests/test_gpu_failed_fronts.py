"""A factorization that fails while other fronts are being factored: the failing column is the bad front's, every time, and
the next factorization with the same object is right. Many fronts of one level, one of them with a bad pivot: small ones of
both classes (one CTA each), and fronts that take the group panel and the updates, whose CTAs start while the status changes. A first factorization with Bunch-Kaufman pivots that fails: the fronts that it does
not reach have no pivot order yet.
"""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import EPS, bordered, dense_csr

pytestmark = pytest.mark.gpu


def with_entry(pat, v, i, value):
    out = v.copy()
    out[(np.repeat(np.arange(pat.n), np.diff(pat.rowptr)) == i) & (pat.colidx == i)] = value
    return out


@pytest.mark.parametrize("kind,precision", [(A.CHOLESKY, A.FP64), (A.CHOLESKY, A.MIXED), (A.LDLT, A.FP64),
                                            (A.LDLT, A.MIXED), (A.LDLT_BK, A.FP64)])
@pytest.mark.parametrize("sizes,border,front,at", [([4] * 160, 10, 77, 3), ([40] * 50, 20, 31, 33), ([70] * 24, 40, 11, 8),
                                                   ([150, 200] * 5, 70, 4, 130)])
def test_one_bad_front(sizes, border, front, at, kind, precision):
    good = bordered(sizes, border, 5, indefinite=kind != A.CHOLESKY)
    bad = sum(sizes[:front]) + at
    pat, v = dense_csr(good)
    vb = with_entry(pat, v, bad, -1.0 if kind == A.CHOLESKY else np.nan)
    sym = A.analyze(pat, perm=np.arange(pat.n, dtype=np.int32), relax=False)
    assert np.array_equal(sym.perm, np.arange(pat.n))
    num = A.NumericFactor(sym, kind, precision)
    b = np.random.default_rng(1).uniform(-1, 1, (1, pat.n))
    ref = np.linalg.solve(good, b[0])
    first = last = bad
    if kind == A.LDLT_BK:  # other columns of the pivot block may come before the bad one, or after it in its place
        first, last = bad - at % 64, bad - at + min(at // 64 * 64 + 64, sizes[front]) - 1
    for _ in range(40):
        assert not num.factor(vb)
        assert first <= num.failColumn <= last
        assert num.factor(v)
    x = num.solve_block(b)[0]
    assert np.max(np.abs(x - ref)) <= 10 * 10 * pat.n * EPS[precision] * np.max(np.abs(ref))


@pytest.mark.parametrize("sizes,border", [([4] * 40, 10), ([40] * 20, 20), ([70] * 10, 40), ([150, 200], 70)])
def test_first_bunch_kaufman_factorization_fails(sizes, border):
    good = bordered(sizes, border, 5, indefinite=True)
    pat, v = dense_csr(good)
    sym = A.analyze(pat, perm=np.arange(pat.n, dtype=np.int32), relax=False)
    b = np.random.default_rng(1).uniform(-1, 1, (1, pat.n))
    ref = np.linalg.solve(good, b[0])
    num = A.NumericFactor(sym, A.LDLT_BK)
    assert not num.factor(with_entry(pat, v, 1, np.nan))
    assert num.factor(v)
    x = num.solve_block(b)[0]
    assert np.max(np.abs(x - ref)) <= 10 * 10 * pat.n * EPS[A.FP64] * np.max(np.abs(ref))
