"""Resident PCG iterations of matrices with a few rows much longer than the mean, which a
warp takes: lengths on both sides of where a row counts as long (4 rounds of 2 lanes and
8, 4 or 2 blocks), many of them in one CTA, every block size.  A fixed number of iterations
differs from the streaming iterations by rounding alone (1e-11, as for the other resident
systems: 12 steps, condition numbers below 100)."""
import numpy as np
import pytest

import yafel_b200 as yb
from test_gpu_pcg_resident import device, host_spmv

pytestmark = pytest.mark.gpu


def spiky(nb, B, lengths, seed, extra=2):
    """Diagonally dominant block matrix whose rows 0, 1, ... reach `lengths` other block rows."""
    rng = np.random.default_rng(seed)
    i, j = np.repeat(np.arange(nb), extra), rng.integers(0, nb, nb * extra)
    for r, n in enumerate(lengths):
        i = np.concatenate([i, np.full(n, r)])
        j = np.concatenate([j, len(lengths) + rng.choice(nb - len(lengths), n, replace=False)])
    d = np.arange(nb)
    key = np.unique(np.concatenate([i * nb + j, j * nb + i, d * nb + d]).astype(np.int64))
    r, c = key // nb, key % nb
    vals = np.zeros((key.size, B, B))
    up = r < c
    vals[up] = rng.uniform(-1, 1, (up.sum(), B, B))
    vals[np.searchsorted(key, c[up] * nb + r[up])] = vals[up].transpose(0, 2, 1)
    rowsum = np.zeros((nb, B))
    np.add.at(rowsum, r, np.abs(vals).sum(2))
    vals[r == c] = 0
    vals[np.nonzero(r == c)[0]] += np.einsum("ri,ij->rij", rowsum * 1.2 + rng.uniform(1, 2, (nb, B)), np.eye(B))
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=nb))]), c, vals


CASES = [(3000, 1, [58, 60, 64, 70, 200, 1000, 2500]), (4000, 1, [90] * 120), (1500, 2, [28, 30, 33, 40, 900]),
         (900, 3, [12, 14, 15, 17, 20, 300, 800])]


@pytest.mark.parametrize("nb,B,lengths", CASES)
def test_against_streaming_iterations(ctx, nb, B, lengths):
    sys_ = spiky(nb, B, lengths, nb)
    K = device(*sys_)
    rng = np.random.default_rng(nb)
    b, x0 = rng.standard_normal(nb * B), rng.standard_normal(nb * B)
    M = yb.JacobiPreconditioner(K)
    xa = yb.solve(K, b, x0, M=M, tol=1e-30, maxiter=12)[0].numpy()
    xb = yb.solve(K, b, x0, M=M, tol=1e-30, maxiter=12, profile=True)[0].numpy()
    assert np.linalg.norm(xa - xb) <= 1e-11 * np.linalg.norm(xb)
    for precision in (yb.PREC_FP64, yb.PREC_MIXED_IR):
        x, st = yb.solve(K, b, x0, M=M, tol=1e-10, precision=precision)
        assert st.status == 0
        assert np.linalg.norm(b - host_spmv(*sys_, x.numpy())) <= 1.01e-10 * np.linalg.norm(b)
        assert np.array_equal(x.numpy(), yb.solve(K, b, x0, M=M, tol=1e-10, precision=precision)[0].numpy())


def test_in_a_batch(ctx):
    systems = [spiky(nb, B, lengths, nb) for nb, B, lengths in CASES]
    batch, slots, bs = yb.Batch(len(systems)), [], []
    for s in systems:
        bs.append(np.random.default_rng(1).standard_normal((s[0].size - 1) * s[2].shape[1]))
        slots.append(batch.add(device(*s), bs[-1]))
    assert batch.run() == 0
    for s, b, slot in zip(systems, bs, slots):
        assert batch.stats(slot).status == 0
        assert np.linalg.norm(b - host_spmv(*s, batch.solution(slot).numpy())) <= 1.01e-10 * np.linalg.norm(b)


def test_a_long_row_does_not_hold_up_the_others(ctx):
    """No slower than the streaming kernels, which give a row up to 32 lanes (with the lanes
    that suit the mean, the resident kernel took five times their time here)."""
    s = spiky(40000, 1, [15000], 3)
    K = device(*s)
    b = yb.DeviceVector(np.random.default_rng(2).standard_normal(40000))
    M = yb.JacobiPreconditioner(K)
    ms = {}
    for profile in (False, True):
        ms[profile] = min(yb.solve(K, b, M=M, tol=1e-30, maxiter=200, profile=profile)[1].device_ms for _ in range(4))
    assert ms[False] <= 1.5 * ms[True], ms
