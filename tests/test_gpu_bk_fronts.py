"""Whole fronts with Bunch-Kaufman pivots whose every step searches the row of the larger pivot (small or zero diagonals):
many of them side by side, one warp or one CTA each. The factor, the pivot orders and D are the same bits in every repeat,
and the factor reproduces the matrix (check_bk)."""
import numpy as np
import pytest

import ampsolve as A
from test_gpu_bk import check_bk, csr_from_dense

pytestmark = pytest.mark.gpu


def saddle_blocks(sizes, border, seed):
    """Dense diagonal blocks with entries of order one and a diagonal of 0.01 or zero, coupled to `border` dominant rows."""
    rng = np.random.default_rng(seed)
    n = sum(sizes) + border
    M = np.zeros((n, n))
    o = 0
    for k in sizes:
        B = rng.standard_normal((k, k))
        B = (B + B.T) / 2
        B[np.arange(k), np.arange(k)] = np.where(np.arange(k) % 3 == 0, 0.0, 0.01)
        M[o:o + k, o:o + k] = B
        o += k
    C = rng.uniform(-1, 1, (border, o)) / n
    M[o:, :o], M[:o, o:] = C, C.T
    M[np.arange(o, n), np.arange(o, n)] = 4.0
    return M


@pytest.mark.parametrize("sizes,border", [([6] * 30, 8), ([20] * 20, 10), ([40, 33, 64] * 8, 20), ([100, 77] * 4, 28)])
def test_fronts_that_search(sizes, border):
    pat, v = csr_from_dense(saddle_blocks(sizes, border, len(sizes)))
    kw = {"perm": np.arange(pat.n, dtype=np.int32), "relax": False}
    check_bk(pat, v, kw)
    f = A.SupernodalLDLT(A.analyze(pat, **kw), pivoting="bunch-kaufman")
    first = None
    for _ in range(30):
        assert f.factor(v)["ok"]
        doff, piv = f.num.pivots()
        now = (f.Lx.copy(), f.D.copy(), doff.copy(), piv.copy())
        first = first or now
        assert all(np.array_equal(a, b) for a, b in zip(first, now))
    assert np.count_nonzero(first[2]) > 0
