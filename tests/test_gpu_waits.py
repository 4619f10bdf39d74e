"""Bounded device waits that expire (a limit of a few polls on a long chain of rows):
the call whose wait it was, or the next that waits for the context, reports it, and the
context stays usable."""
import numpy as np
import pytest

import yafel_b200 as yb
from yafel_b200 import _lib

pytestmark = pytest.mark.gpu


def upper_chain(n, ctx):
    """2 on the diagonal and -1 above: no row of the factorization waits, the backward
    substitution is one chain of n rows."""
    ptr = np.minimum(2 * np.arange(n + 1), 2 * n - 1).astype(np.int32)
    i = np.arange(n)
    col = np.stack([i, i + 1], 1).ravel()[:-1].astype(np.int32)
    return yb.sparse_csr.from_csr(ptr, col, np.tile([2.0, -1.0], n)[:-1], ctx=ctx)


@pytest.fixture
def short_waits(monkeypatch):
    """A context whose ILU(0) waits give up after 32 polls."""
    monkeypatch.setenv("YAFEL_B200_WAIT_POLLS", "32")
    return yb.Context(0)


@pytest.mark.parametrize("criterion", [yb.CRIT_RELRES, yb.CRIT_REFERENCE])
def test_solve_reports_its_own_expired_wait(short_waits, criterion):
    c, n = short_waits, 20000
    A = upper_chain(n, c)
    M = yb.ILUPreconditioner(A)
    b = yb.DeviceVector(np.ones(n), c)
    with pytest.raises(yb.YafelError) as e:
        yb.solve(A, b, M=M, tol=1e-10, criterion=criterion)
    assert e.value.status == _lib.YG_TIMEOUT
    y = A.spmv(b).numpy()  # reported once
    assert np.array_equal(y[:-1], np.ones(n - 1)) and y[-1] == 2.0


def test_apply_is_reported_by_the_download(short_waits, monkeypatch):
    c, n = short_waits, 20000
    A = upper_chain(n, c)
    M = yb.ILUPreconditioner(A)
    with pytest.raises(yb.YafelError) as e:
        M.solve(np.ones(n))
    assert e.value.status == _lib.YG_TIMEOUT
    c.synchronize()
    # rows that wait for nothing: the expired wait before does not end this apply
    D = yb.sparse_csr.from_csr(np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.full(n, 4.0), ctx=c)
    assert np.array_equal(yb.ILUPreconditioner(D).solve(np.ones(n)), np.full(n, 0.25))
    # and with the usual limit the chain is solved: x_i = (1 + x_{i+1}) / 2
    monkeypatch.delenv("YAFEL_B200_WAIT_POLLS")
    full = yb.Context(0)
    x = yb.ILUPreconditioner(upper_chain(n, full)).solve(np.ones(n))
    assert np.all(x[:-1] == (1.0 + x[1:]) / 2.0) and x[-1] == 0.5
