"""BiCGSTAB's vector kernels (pairs of entries, a grid that follows the rows) against
numpy, at row counts around a block's chunk and the grid's limits, odd and even; and
the change-over from launched to replayed iterations, which must not be visible."""
import numpy as np
import pytest

import yafel_b200 as yb

pytestmark = pytest.mark.gpu


def banded(n, seed):
    """Nonsymmetric, diagonally dominant: a diagonal and up to four bands."""
    rng = np.random.default_rng(seed)
    offs = [o for o in (-7, -1, 0, 1, 5) if abs(o) < n]
    rows = np.concatenate([np.arange(max(0, -o), min(n, n - o)) for o in offs])
    cols = np.concatenate([np.arange(max(0, -o), min(n, n - o)) + o for o in offs])
    vals = np.where(rows == cols, rng.uniform(5, 6, rows.size), rng.uniform(-1, 1, rows.size))
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return ptr, cols, vals, rows


def numpy_bicgstab(A, b, dinv, its):
    ptr, cols, vals, rows = A

    def mul(x):
        return np.bincount(rows, vals * x[cols], minlength=b.size)

    x = np.zeros_like(b)
    r = b.copy()
    rhat, p, v = r.copy(), np.zeros_like(b), np.zeros_like(b)
    rho = alpha = omega = 1.0
    for _ in range(its):
        rho_new = rhat @ r
        beta = rho_new / rho * (alpha / omega)
        rho = rho_new
        p = r + beta * (p - omega * v)
        ph = dinv * p
        v = mul(ph)
        alpha = rho / (rhat @ v)
        s = r - alpha * v
        sh = dinv * s
        t = mul(sh)
        omega = (t @ s) / (t @ t)
        x += alpha * ph + omega * sh
        r = s - omega * t
    return x


# three iterations of systems with condition numbers below 10: rounding alone (1e-11)
@pytest.mark.parametrize("n", [17, 255, 512, 513, 148 * 512 - 1, 148 * 512 + 1, 592 * 512, 592 * 512 + 3, 700001])
@pytest.mark.parametrize("jacobi", [True, False])
def test_three_iterations(n, jacobi):
    A = banded(n, n)
    K = yb.sparse_csr.from_csr(*A[:3])
    b = np.random.default_rng(1).standard_normal(n)
    dinv = 1 / A[2][A[3] == A[1]] if jacobi else np.ones(n)
    M = yb.JacobiPreconditioner(K) if jacobi else None
    x, st = yb.solve(K, b, M=M, method="bicgstab", tol=1e-300, maxiter=3)
    want = numpy_bicgstab(A, b, dinv, 3)
    assert st.iterations == 3
    assert np.abs(x.numpy() - want).max() <= 1e-11 * np.abs(want).max()


@pytest.mark.parametrize("n", [1001, 90000])
def test_iterate_independent_of_change_over(n):
    A = banded(n, 3)
    ptr, cols, vals, rows = A
    K = yb.sparse_csr.from_csr(ptr, cols, np.where(rows == cols, 3.0, vals))  # slower to converge
    K.set_spmv_for(0, 0, 4)
    b = np.random.default_rng(2).standard_normal(n)
    for its in (1, 4, 5, 11):
        got = []
        for every in (2, 8, 64):  # launched until iteration 4, 16, 128
            x, st = yb.solve(K, b, method="bicgstab", tol=1e-300, maxiter=its, check_every=every)
            assert st.iterations == its
            got.append(x.numpy())
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
