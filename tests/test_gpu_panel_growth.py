"""Rows below a pivot block whose 8 x 8 diagonal blocks of L are ill conditioned: matrices made as L D L^T (L L^T) from a
chosen L, with entries of up to `size` in its 8 x 8 diagonal blocks, and real LDL^T with pivots that are tiny or perturbed
beside the edges of the eight-column steps and of the 64-column blocks.

Tolerance. Elimination and substitution are stable entry by entry whatever the multipliers: with S = |L| |D| |L|^T an entry
of L D L^T is off by at most (n + 6) eps S (up to n sums, each rounded once against partial sums of at most 2 S, and six
roundings per term), and the matrix itself is rounded to eps S; allowed is four times that. The products are formed in
80-bit arithmetic.
"""
import numpy as np
import pytest

import ampsolve as A
import workloads as W

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def dense_pattern(n):
    return W.CsrPattern(n, np.arange(0, n * n + 1, n, dtype=np.int32), np.tile(np.arange(n, dtype=np.int32), n))


def wide(M):
    return M.astype(np.clongdouble if np.iscomplexobj(M) else np.longdouble)


def chosen_factor(n, size, seed, cplx=False):
    """Unit lower triangular: entries of up to `size` inside the 8 x 8 diagonal blocks, 1 / n-sized elsewhere."""
    rng = np.random.default_rng(seed)
    L = rng.uniform(-1, 1, (n, n))
    if cplx:
        L = L + 1j * rng.uniform(-1, 1, (n, n))
    same = np.arange(n)[:, None] // 8 == np.arange(n)[None, :] // 8
    return np.tril(np.where(same, size * L, L / n), -1) + np.eye(n)


def check(L, D, M):
    n = M.shape[0]
    Lw, Dw = wide(L), wide(D)
    S = (np.abs(Lw) * np.abs(Dw)) @ np.abs(Lw).T
    off = np.tril(np.abs((Lw * Dw) @ Lw.T - wide(M)))
    assert np.all(off <= 4 * (n + 6) * EPS * S)


# (the larger ones of L L^T with size 8 are not positive definite any more when rounded to FP64)
REAL = [(k, n, s) for k in (A.CHOLESKY, A.LDLT) for n in (129, 203, 330) for s in (0.1, 1.0, 4.0, 8.0)
        if k == A.LDLT or n == 129 or s < 8.0]


@pytest.mark.parametrize("group", [1, 4])
@pytest.mark.parametrize("kind,n,size", REAL)
def test_real_fronts(kind, n, size, group):
    Lc = wide(chosen_factor(n, size, n))
    D = np.ones(n) if kind == A.CHOLESKY else np.where(np.random.default_rng(1).uniform(size=n) < 0.4, -1.0, 1.0)
    M = ((Lc * D) @ Lc.T).astype(float)
    num = A.NumericFactor(A.analyze(dense_pattern(n), perm=np.arange(n, dtype=np.int32), groupBlocks=group), kind)
    assert num.factor(M.reshape(-1))
    L = np.tril(num.Lx.reshape(n, n).T)
    check(L, np.ones(n) if kind == A.CHOLESKY else num.D, M)


@pytest.mark.parametrize("size", [0.1, 1.0, 4.0, 8.0])
@pytest.mark.parametrize("n", [72, 129, 203, 330])
def test_complex_fronts(n, size):
    Lc = wide(chosen_factor(n, size, n, True))
    D = np.exp(1j * np.random.default_rng(1).uniform(0, 6.28, n))
    M = ((Lc * D) @ Lc.T).astype(complex)
    M = np.tril(M) + np.tril(M, -1).T
    f = A.ComplexSupernodalLDLT(A.analyze(dense_pattern(n), perm=np.arange(n, dtype=np.int32)))
    r = f.factor(M.real.reshape(-1).copy(), M.imag.reshape(-1).copy())
    assert r["ok"] and r["nPerturbed"] == 0
    Lr, Li, Dr, Di = f.factors()
    check(np.tril((Lr + 1j * Li)[: n * n].reshape(n, n).T), Dr + 1j * Di, M)


@pytest.mark.parametrize("exponent", [0, -984, 970])
@pytest.mark.parametrize("n,tiny", [(50, [3, 5]), (101, [0, 7, 8]), (130, [1, 6, 63]), (203, [9, 11, 14, 64, 127]),
                                    (330, [62, 63, 192, 199, 255, 256])])
@pytest.mark.parametrize("value", [1e-4, 1e-8, 0.0])
def test_small_pivots(n, tiny, value, exponent):
    """Pivots of 1e-4 and 1e-8 of the diagonal, and of zero (perturbed to tau = 1e-8 of it), coupled to every later row."""
    rng = np.random.default_rng(n)
    M = rng.uniform(-1, 1, (n, n)) / n
    M = (M + M.T) / 2
    M[np.arange(n), np.arange(n)] = np.where(rng.uniform(size=n) < 0.4, -1.0, 1.0) * rng.uniform(1, 2, n)
    M[0, 0] = 2.0
    for z in tiny:
        M[z, :z] = M[:z, z] = 0.0
        M[z, z] = 2.0 * value
    M[n - 1, n - 1] = 2.0  # the largest diagonal entry
    tol = 1e-8 if value == 0.0 else 1e-12
    num = A.NumericFactor(A.analyze(dense_pattern(n), perm=np.arange(n, dtype=np.int32)), A.LDLT)
    assert num.factor(np.ldexp(M, exponent).reshape(-1), pivotTol=tol)
    assert num.nPerturbed == (len(tiny) if value == 0.0 else 0)
    L, D = np.tril(num.Lx.reshape(n, n).T), np.ldexp(num.D, -exponent)
    if value == 0.0:
        M[tiny, tiny] = 2.0 * tol
    check(L, D, M)
