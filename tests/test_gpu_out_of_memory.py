"""A factor object that cannot be made for want of device memory: the error is that call's alone, and what was made before,
or is made later on the same plan, works."""
import numpy as np
import pytest

import ampsolve as A
import workloads as W

pytestmark = pytest.mark.gpu


class FullDevice:
    """Holds all device memory but a rest of less than 2 MB."""

    def __enter__(self):
        import torch

        torch.cuda.init()
        torch.cuda.empty_cache()
        self.held, size = [], torch.cuda.mem_get_info()[0]
        while size >= 1 << 21:
            try:
                self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                size //= 2

    def __exit__(self, *exc):
        import torch

        self.held.clear()
        torch.cuda.empty_cache()


def test_later_calls_do_not_report_it():
    w = W.heat2d_lognormal(300, 1, 1)
    sym = A.analyze(w.pat)
    num = A.NumericFactor(sym)
    assert num.factor(w.values)
    x = num.solve_block(w.rhs)
    with FullDevice():
        with pytest.raises(A.AmpError, match="memory"):
            A.NumericFactor(sym)
        assert num.factor(w.values)
    assert np.array_equal(num.solve_block(w.rhs), x)
