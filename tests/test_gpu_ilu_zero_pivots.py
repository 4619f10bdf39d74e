"""ILU(0) with zero pivots: the rows that a zero pivot does not reach have the values of the
scalar factorization (1e-11 of the largest of them, as where there is no zero pivot)."""
import numpy as np
import pytest

import yafel_b200 as yb
from test_gpu_ilu_rows import device, ikj, scalar, spd, substitute

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("at", [0, 60, 119])
def test_rows_that_a_zero_pivot_does_not_reach(ctx, B, at):
    nb = 120
    ptr, col, vals = spd(nb, B, 11 + B, extra=1)
    vals = vals * (1 + 0.2 * np.random.default_rng(B).standard_normal(vals.shape))  # not symmetric
    for t in range(ptr[at], ptr[at + 1]):  # the block's first scalar row: nothing up to its diagonal
        if col[t] < at:
            vals[t][0, :] = 0.0
        elif col[t] == at:
            vals[t][0, 0] = 0.0
    A, P = scalar(ptr, col, vals)
    F, zeros = ikj(A, P)
    assert F[at * B, at * B] == 0.0
    K = device(ptr, col, vals)
    M = yb.ILUPreconditioner(K)
    assert M.zero_pivots == zeros
    z = np.random.default_rng(5).standard_normal(nb * B)
    with np.errstate(all="ignore"):
        want = substitute(F, P, z)
    got = yb.DeviceVector(z)
    M.solve(got)
    got = got.numpy()
    fine = np.isfinite(want)
    assert 0 < fine.sum() < fine.size
    assert np.array_equal(fine, np.isfinite(got))
    assert np.abs(got[fine] - want[fine]).max() <= 1e-11 * np.abs(want[fine]).max()
