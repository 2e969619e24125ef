"""Restriction of the stencils and its transpose with values that are not finite: they stay in the taps that they overlap, as in the
oracle; the finite entries agree to 1e-6 (float32) / 1e-14 (float64: sums of at most 27 products per slot)."""
import numpy as np
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-6), (torch.float64, 1e-14)])
@pytest.mark.parametrize("stencils", [1, 2])
@pytest.mark.parametrize("value", [None, np.inf, -np.inf, np.nan])
def test_non_finite_taps_stay_where_they_belong(dtype, tol, stencils, value, oracle):
    from _pyaprwrapper.aprnet import cuda as C
    L = 5
    rng = np.random.RandomState(2)
    w = rng.randn(stencils, 9, 15, 3, 3, 3)              # 135 filters: more than a block of them, one with every tap hit once
    g = rng.randn(L, 9, 15, 3, 3, 3)
    if value is not None:
        for t in range(27):
            w.reshape(stencils, -1, 27)[-1, 5 * t, t] = value
            g.reshape(L, -1, 27)[stencils + t % (L - stencils), 5 * t, t] = value
    with np.errstate(invalid="ignore"):
        for got, want in ((C.restrict_kernel333_forward(torch.from_numpy(w).to("cuda", dtype), L), oracle.restrict333_forward(w, L)),
                          (C.restrict_kernel333_backward(torch.from_numpy(g).to("cuda", dtype), stencils), oracle.restrict333_backward(g, stencils))):
            got, want = H.t2n(got).astype(np.float64), np.asarray(want)
            finite = np.isfinite(want)
            assert np.array_equal(np.isfinite(got), finite) and np.array_equal(np.isnan(got), np.isnan(want))
            assert value is None or 0 < (~finite).sum() < want.size
            assert H.rel_err(got[finite], want[finite]) <= tol
