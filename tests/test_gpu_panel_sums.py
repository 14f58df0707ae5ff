"""The group panel sums a block's products apart from the entry that they are subtracted from.

A diagonally dominant front of 449 columns, one group of eight blocks: a diagonal entry of the last full block (2 to 3, its
products of size 1 / n) is rounded at its own size once per earlier block, at most once per column of its own block, and four
times more, 75 times in all, each by an error of at most half an ulp (2^-51) and 1 / sqrt(12) of one in the mean square. So the
root mean square of L D L^T - A over the 64 entries stays below 10 ulp / sqrt(12); rounded after every product it would be 20.
Formed in 80-bit arithmetic, eight matrices.
"""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_group_panel import dominant
from test_gpu_panel_growth import dense_pattern

pytestmark = pytest.mark.gpu
N, ULP = 449, 2.0 ** -51


@pytest.mark.parametrize("kind", [A.CHOLESKY, A.LDLT, A.LDLT_BK, "complex"])
def test_diagonal_of_the_last_block(kind):
    rows = slice(384, 448)
    sym = A.analyze(dense_pattern(N), perm=np.arange(N, dtype=np.int32), groupBlocks=8)
    squares = []
    for seed in range(8):
        M = dominant(N, seed, indefinite=kind not in (A.CHOLESKY, "complex"))
        if kind == "complex":
            im = np.tril(dominant(N, 100 + seed))
            im = im + np.tril(im, -1).T
            f = A.ComplexSupernodalLDLT(sym)
            assert f.factor(M.reshape(-1), im.reshape(-1).copy())["ok"]
            Lr, Li, Dr, Di = f.factors()
            L = np.tril((Lr + 1j * Li)[: N * N].reshape(N, N).T).astype(np.clongdouble)
            d = np.sum(L * L * (Dr + 1j * Di), axis=1) - (np.diag(M) + 1j * np.diag(im))
            squares.append(np.abs(d[rows]) ** 2 / 2)  # a part of the entry's two
        else:
            num = A.NumericFactor(sym, kind)
            assert num.factor(M.reshape(-1))
            L = np.tril(num.Lx.reshape(N, N).T).astype(np.longdouble)
            D = np.ones(N) if kind == A.CHOLESKY else num.D
            squares.append((np.sum(L * L * D, axis=1) - np.diag(M))[rows] ** 2)
    assert np.sqrt(np.mean(squares)) <= 10 * ULP / np.sqrt(12)
