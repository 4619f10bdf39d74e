"""ILU(0) by block rows against a scalar IKJ factorization and substitutions in
numpy (dense, on the same pattern): every block size, zero pivots, rows without a
diagonal, more block rows than warps; and against the oracle where rows are longer
than a warp's shared memory (updated in place).  The matrices are diagonally
dominant by 1.2, so the factors' condition is below about 10 and the tolerance is
1e-11 of the largest entry of the result (rounding of some 1e3 operations)."""
import numpy as np
import pytest

import yafel_b200 as yb
from oracle import oracle as O
from test_gpu_pcg_resident import device, spd

pytestmark = pytest.mark.gpu


def scalar(ptr, col, vals):
    """Dense matrix and pattern of the scalar expansion."""
    B, nb = vals.shape[1], ptr.size - 1
    A, P = np.zeros((nb * B, nb * B)), np.zeros((nb * B, nb * B), bool)
    for i in range(nb):
        for t in range(ptr[i], ptr[i + 1]):
            A[i * B:(i + 1) * B, col[t] * B:(col[t] + 1) * B] = vals[t]
            P[i * B:(i + 1) * B, col[t] * B:(col[t] + 1) * B] = True
    return A, P


def ikj(A, P):
    A, zeros = A.copy(), 0
    for i in range(len(A)):
        for k in np.nonzero(P[i, :i])[0]:
            if not P[k, k] or A[k, k] == 0:
                zeros += 1
                continue
            A[i, k] /= A[k, k]
            c = np.nonzero(P[i] & P[k])[0]
            c = c[c > k]
            A[i, c] -= A[i, k] * A[k, c]
    return A, zeros


def substitute(F, P, z):
    z = z.copy()
    for i in range(len(z)):
        c = np.nonzero(P[i, :i])[0]
        z[i] -= F[i, c] @ z[c]
    for i in range(len(z) - 1, -1, -1):
        c = np.nonzero(P[i])[0]
        d = i if P[i, i] else c[0]  # a row without a diagonal divides by its first entry
        c = c[c > d]
        z[i] = (z[i] - F[i, c] @ z[c]) / F[i, d]
    return z


@pytest.mark.parametrize("B", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("case", ["one", "some", "many", "zero", "no_diagonal"])
def test_against_scalar_ikj(ctx, B, case):
    nb = {"one": 1, "some": 37, "many": 1300 if B == 1 else 160, "zero": 25, "no_diagonal": 21}[case]
    ptr, col, vals = spd(nb, B, 3 * nb + B)
    vals = vals * (1 + 0.2 * np.random.default_rng(B).standard_normal(vals.shape))  # not symmetric
    row = np.repeat(np.arange(nb), np.diff(ptr))
    if case == "zero":
        for i in (0, 3):
            vals[np.nonzero((row == i) & (col == i))[0][0]][0, :] = 0.0  # scalar rows that are zero in their block
    if case == "no_diagonal":
        keep = ~((row == col) & np.isin(row, (2, 9, nb - 1)))
        ptr = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=nb))])
        col, vals = col[keep], vals[keep]
    K = device(ptr, col, vals)
    A, P = scalar(ptr, col, vals)
    F, zeros = ikj(A, P)
    M = yb.ILUPreconditioner(K)
    assert M.zero_pivots == zeros
    z = np.random.default_rng(5).standard_normal(nb * B)
    with np.errstate(all="ignore"):
        want = substitute(F, P, z)
    for _ in range(2):  # the vectors an apply polls are set up again each time
        got = yb.DeviceVector(z)
        M.solve(got)
        got = got.numpy()
        fine = np.isfinite(want)
        assert np.array_equal(fine, np.isfinite(got))
        if case != "zero":  # (a zero pivot divides by zero: what follows is not finite)
            assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()


def test_rows_longer_than_shared_memory(ctx):
    nb, B = 3400, 3
    rng = np.random.default_rng(2)
    keys = sorted({(i, i) for i in range(nb)} | {(0, j) for j in range(nb)} | {(j, 0) for j in range(nb)} |
                  {(nb - 1, j) for j in range(nb)} | {(j, nb - 1) for j in range(nb)})
    keys = np.array(keys)
    vals = rng.uniform(-1, 1, (len(keys), B, B)) / nb
    d = keys[:, 0] == keys[:, 1]
    vals[d] += 4.0 * np.eye(B)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(keys[:, 0], minlength=nb))])
    K = device(ptr, keys[:, 1], vals)
    r, c, v = K.copy_triplets()
    o = np.lexsort((c, r))
    sp = np.concatenate([[0], np.cumsum(np.bincount(r[o], minlength=nb * B))])
    F = O.ilu0(O.Csr(nb * B, nb * B, sp, c[o], v[o]))
    z = rng.standard_normal(nb * B)
    got = yb.DeviceVector(z)
    yb.ILUPreconditioner(K).solve(got)
    want = O.ilu_solve(F, z)
    assert np.abs(got.numpy() - want).max() <= 1e-11 * np.abs(want).max()
