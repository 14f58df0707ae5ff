"""GPU group panel at the edges of its tiles: dense fronts above the whole-front cut-off (every pivot block goes
through the group panel), with and without rows below, block widths with remainders, against numpy.

Tolerances. Cholesky and LDL^T of a diagonally dominant matrix are backward stable with |L L^T - A| <= (n + 1) eps
max |A| entrywise (n terms per entry, each at most max |A|), and condition numbers below 10 keep solutions within
10 n eps; both are given a factor of 10. FP32 factors: the same with FP32's eps.
"""
import numpy as np
import pytest

import ampsolve as A
import workloads as W

pytestmark = pytest.mark.gpu

EPS = {A.FP64: 2.0 ** -52, A.MIXED: 2.0 ** -23}


def dense_csr(M):
    n = M.shape[0]
    mask = (M != 0) | np.eye(n, dtype=bool)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(mask.sum(axis=1))
    return W.CsrPattern(n, rp, np.nonzero(mask)[1].astype(np.int32)), M[mask]


def dominant(n, seed, indefinite=False):
    """Symmetric, entries of size 1 / n, diagonal about 2 (of either sign when indefinite)."""
    rng = np.random.default_rng(seed)
    M = rng.uniform(-1, 1, (n, n)) / n
    M = (M + M.T) / 2
    d = 2.0 + rng.uniform(0, 1, n)
    if indefinite:
        d *= np.where(rng.uniform(size=n) < 0.4, -1.0, 1.0)
    M[np.diag_indices(n)] = d
    return M


def bordered(sizes, border, seed, indefinite=False):
    """Dense diagonal blocks of the given sizes, each coupled to all of `border` last rows (fronts with rows below)."""
    n = sum(sizes) + border
    M = dominant(n, seed, indefinite)
    o = 0
    for k in sizes:
        rest = np.arange(o + k, sum(sizes))
        M[np.ix_(np.arange(o, o + k), rest)] = 0.0
        M[np.ix_(rest, np.arange(o, o + k))] = 0.0
        o += k
    return M


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [129, 191, 192, 193, 256, 257, 320, 449])
def test_dense_front_reconstructs(n, group):
    M = dominant(n, n)
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32), groupBlocks=group)
    assert sym.nsuper == 1
    for precision in (A.FP64, A.MIXED):
        num = A.NumericFactor(sym, A.CHOLESKY, precision)
        assert num.factor(v)
        L = np.tril(num.Lx.reshape(n, n).T)
        assert np.max(np.abs(L @ L.T - M)) <= 10 * (n + 1) * EPS[precision] * np.max(np.abs(M))


@pytest.mark.parametrize("kind", [A.LDLT, A.LDLT_BK])
@pytest.mark.parametrize("sizes,border", [([130], 1), ([130, 200], 63), ([257], 65), ([133, 140], 130)])
def test_indefinite_fronts_with_rows_below(sizes, border, kind):
    M = bordered(sizes, border, 7, indefinite=True)
    n = M.shape[0]
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32), groupBlocks=4)
    num = A.NumericFactor(sym, kind)
    assert num.factor(v)
    assert num.nNeg == int(np.sum(np.linalg.eigvalsh(M) < 0)) and num.nPerturbed == 0
    B = np.random.default_rng(1).uniform(-1, 1, (3, n))
    X = num.solve_block(B)
    ref = np.linalg.solve(M, B.T).T
    assert np.max(np.abs(X - ref)) <= 10 * 10 * n * EPS[A.FP64] * np.max(np.abs(ref))


@pytest.mark.parametrize("exponent", [-984, 970])
def test_pivots_outside_the_reciprocal_estimate(exponent):
    """A scaled by 2^e (pivots beyond the range of the hardware estimate): L is scaled by 2^(e/2) exactly, up to the
    rounding of the exact quotient against the refined estimate."""
    n = 200
    M = dominant(n, 5)
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32))
    num = A.NumericFactor(sym)
    assert num.factor(v)
    L = num.Lx.copy()
    assert num.factor(np.ldexp(v, exponent))
    Ls = np.ldexp(num.Lx, -exponent // 2)
    assert np.max(np.abs(Ls - L)) <= 10 * (n + 1) * EPS[A.FP64] * np.max(np.abs(L))


@pytest.mark.parametrize("bad", [0, 7, 63, 64, 130, 199])
def test_first_failing_column(bad):
    n = 200
    M = dominant(n, 9)
    M[bad, bad] = -1.0
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32))
    num = A.NumericFactor(sym)
    assert not num.factor(v)
    assert num.failColumn == bad


@pytest.mark.parametrize("border", [63, 640, 2101])
def test_update_block_tiles(border):
    """Update launches of few tiles (half a task per CTA) and of more than the CTAs in flight (whole tasks)."""
    M = bordered([130, 151], border, 11)
    n = M.shape[0]
    pat, v = dense_csr(M)
    sym = A.analyze(pat, perm=np.arange(n, dtype=np.int32))
    num = A.NumericFactor(sym)
    assert num.factor(v)
    b = np.random.default_rng(2).uniform(-1, 1, n)
    x = num.solve_block(b[None, :])[0]
    ref = np.linalg.solve(M, b)
    assert np.max(np.abs(x - ref)) <= 10 * 10 * n * EPS[A.FP64] * np.max(np.abs(ref))
