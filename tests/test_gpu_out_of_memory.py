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


def test_complex_schedule_is_built_again():
    """The complex factor's schedule is uploaded by the first one made on a plan; here that upload fails halfway once."""
    w = W.heat2d_lognormal(300, 1, 1)
    im = 0.1 * w.values
    rng = np.random.default_rng(1)
    br, bi = rng.uniform(-1, 1, w.n), rng.uniform(-1, 1, w.n)
    fresh = A.ComplexSupernodalLDLT(A.analyze(w.pat))
    assert fresh.factor(w.values, im)["ok"]
    want = fresh.solve(br, bi)
    sym = A.analyze(w.pat)
    A.NumericFactor(sym)  # the plan's own tables
    with FullDevice():
        with pytest.raises(A.AmpError, match="memory"):
            A.ComplexSupernodalLDLT(sym)
    f = A.ComplexSupernodalLDLT(sym)
    assert f.factor(w.values, im)["ok"]
    got = f.solve(br, bi)
    for part in ("re", "im"):  # the sums run in any order; condition of some 4e6 (the mesh's 4e4, a contrast of 100): 1e2 eps of it
        assert np.max(np.abs(got[part] - want[part])) <= 1e-7 * np.max(np.abs(want[part]))
