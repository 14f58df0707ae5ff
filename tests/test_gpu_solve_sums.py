"""The multi-vector sweeps over FP64 factors sum in pieces of 64 columns.

LDL^T of a dense front of 1,025 columns with L(i, j) of size 2 / n, all positive, and solutions near one: the backward sum of a
first row has some 1,000 products of 0.002 and grows to 2. Summed one after another, half of them are rounded at a size
between one and two (an ulp of 2^-52) and a quarter at half that: a root mean square error of sqrt(512 + 64) 2^-52 / sqrt(12) =
6.9 2^-52. In 16 pieces, eight roundings at that size and 64 x 16 at an eighth of one or less add up to 1.1 2^-52, and the
entry's other roundings (the division, the inverse block's product) to less than another one. Allowed are 3 2^-52 over the
first block, against substitution with the computed factor in 80-bit arithmetic.
"""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_panel_growth import dense_pattern, wide

pytestmark = pytest.mark.gpu
N = 1025


@pytest.mark.parametrize("q", [2, 17])
def test_long_sums(q):
    rng = np.random.default_rng(3)
    L = np.tril(rng.uniform(0.5, 1.5, (N, N)) * 2 / N, -1) + np.eye(N)
    M = L @ L.T
    num = A.NumericFactor(A.analyze(dense_pattern(N), perm=np.arange(N, dtype=np.int32)), A.LDLT)
    assert num.factor(((M + M.T) / 2).reshape(-1))
    B = rng.uniform(0.5, 1.5, (q, N)) @ M
    X = num.solve_block(B)
    Lw, Dw = wide(np.tril(num.Lx.reshape(N, N).T)), wide(num.D)
    Y = wide(B).T.copy()
    for j in range(N):
        Y[j + 1:] -= np.outer(Lw[j + 1:, j], Y[j])
    Y /= Dw[:, None]
    for j in range(N - 1, 0, -1):
        Y[:j] -= np.outer(Lw[j, :j], Y[j])
    assert np.sqrt(np.mean((wide(X).T - Y)[:64] ** 2)) <= 3 * 2.0 ** -52
