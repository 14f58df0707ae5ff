"""Sweeps of the complex-symmetric LDL^T at the edges of their blocks: one supernode of n columns (one block, ragged ones,
more blocks than a cluster has CTAs), and supernodes with rows of ancestors below (an arrow of dense blocks over a shared
dense border). The matrices are diagonally dominant, so x is compared with numpy's dense solve within 64 n eps."""
import numpy as np
import pytest
import scipy.sparse as sp

import ampsolve as A

pytestmark = pytest.mark.gpu


class _Pat:
    def __init__(self, S):
        S = sp.csr_matrix(S)
        S.sort_indices()
        self.n, self.rowptr, self.colidx = S.shape[0], S.indptr.astype(np.int32), S.indices.astype(np.int32)

    @property
    def nnz(self):
        return int(self.rowptr[-1])


def check(mask, seed):
    rng = np.random.default_rng(seed)
    n = mask.shape[0]
    G = np.tril(rng.uniform(-1, 1, (n, n)) + 1j * rng.uniform(-1, 1, (n, n)), -1) * mask
    G = G + G.T
    G[np.arange(n), np.arange(n)] = 2.0 * mask.sum(1) * np.exp(1j * rng.uniform(0, 6.28, n))
    pat = _Pat(mask)
    r = np.repeat(np.arange(n), np.diff(pat.rowptr))
    v = G[r, pat.colidx]
    f = A.ComplexSupernodalLDLT(A.analyze(pat, perm=np.arange(n, dtype=np.int32)))
    assert f.factor(v.real.copy(), v.imag.copy())["ok"]
    b = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    x = f.solve(b.real.copy(), b.imag.copy())
    ref = np.linalg.solve(G, b)
    assert np.linalg.norm(x["re"] + 1j * x["im"] - ref) <= 64 * n * np.finfo(float).eps * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 513, 577, 700])
def test_one_supernode(n):
    check(np.ones((n, n), bool), n)


@pytest.mark.parametrize("k,w,border", [(1, 64, 1), (3, 5, 63), (5, 33, 65), (2, 130, 200), (2, 70, 600), (300, 2, 40),
                                        (90, 9, 70)])
def test_border(k, w, border):
    n = k * w + border
    mask = np.zeros((n, n), bool)
    for i in range(k):
        mask[i * w:(i + 1) * w, i * w:(i + 1) * w] = True
    mask[k * w:, :] = True
    mask[:, k * w:] = True
    check(mask, 1000 + n)
