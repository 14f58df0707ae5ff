"""Pivot blocks of the complex-symmetric LDL^T: widths around the eight-column steps and the 64-column blocks, pivots that are
perturbed (exactly zero, their rows decoupled from the columns before) at the edges of steps and blocks. The count is exact
and L D L^T reproduces the matrix (zero pivots replaced by tau) within 64 n eps of its largest entry."""
import numpy as np
import pytest

import ampsolve as A
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,zeros", [(1, []), (7, []), (8, [7]), (9, [0]), (17, [8, 16]), (63, [62]), (64, [0, 63]),
                                     (65, [64]), (71, [63, 64]), (130, [7, 64, 129]), (200, []), (330, [5, 255, 256])])
def test_one_front(n, zeros):
    rng = np.random.default_rng(n)
    G = np.tril(rng.uniform(-1, 1, (n, n)) + 1j * rng.uniform(-1, 1, (n, n)), -1)
    G = G + G.T
    G[np.arange(n), np.arange(n)] = 2.0 * n * np.exp(1j * rng.uniform(0, 6.28, n))
    for z in zeros:
        G[z, :] = 0
        G[:, z] = 0
    tol = 1e-10
    tau = tol * np.abs(np.diag(G)).max()
    perm = np.arange(n, dtype=np.int32)
    pat = W.CsrPattern(n, np.arange(0, n * n + 1, n, dtype=np.int32), np.tile(perm, n))
    f = A.ComplexSupernodalLDLT(A.analyze(pat, perm=perm))
    r = f.factor(G.real.reshape(-1).copy(), G.imag.reshape(-1).copy(), pivotTol=tol)
    assert r["ok"] and r["nPerturbed"] == len(zeros)
    Lr, Li, Dr, Di = f.factors()
    L = np.tril((Lr + 1j * Li)[: n * n].reshape(n, n).T)
    want = G.copy()
    want[zeros, zeros] = tau
    assert np.abs((L * (Dr + 1j * Di)) @ L.T - want).max() <= 64 * n * np.finfo(float).eps * np.abs(G).max()
