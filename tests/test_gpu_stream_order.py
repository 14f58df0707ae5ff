"""Host inputs reach the device before the kernels that read them: repeated applications of the shift-invert operator to
host blocks, each with new data in a pageable buffer, must be bitwise equal to the application to the same block held in
device memory (the same kernels on the same data)."""
import numpy as np
import pytest
import torch

import ampsolve as A
import eigen as E
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 6, 64])
def test_shift_invert_host_block_in_order(m):
    w0, w1 = W.maxwell3d(8, 2, 12.0, 0.0, 5, 1), W.maxwell3d(8, 2, 12.0, 1.0, 5, 1)
    K, M = w0.values, w0.values - w1.values
    num = A.NumericFactor(A.analyze(w0.pat), A.LDLT)
    assert num.factor(K - 30.0 * M)
    num.set_mass(M)
    rng = np.random.default_rng(7)
    for _ in range(20):
        X = rng.uniform(-1, 1, (m, w0.pat.n))
        dX = torch.from_numpy(X).cuda()
        dY = torch.empty_like(dX)
        torch.cuda.synchronize()
        assert A.lib().amp_shift_invert_apply(num._h, dX.data_ptr(), m, dY.data_ptr(), 1) == 0
        assert np.array_equal(num.shift_invert_apply(X.copy()), dY.cpu().numpy())


def test_eigenpairs_every_run():
    """No run is repeated: each has every explicit residual within max(1e3 tol, 1e-9)."""
    w0, w1 = W.maxwell3d(8, 2, 12.0, 0.0, 5, 1), W.maxwell3d(8, 2, 12.0, 1.0, 5, 1)
    K, M = w0.values, w0.values - w1.values
    for _ in range(12):
        r = E.shiftInvertEigen(w0.pat, K, M, sigma=30.0, nWant=6, tol=1e-12, maxBasis=48, attempts=1)
        assert r["stats"]["converged"] and float(np.max(r["residual"])) <= 1e-9
