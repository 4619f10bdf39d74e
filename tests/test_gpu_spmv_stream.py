"""Block-stream SpMV (variant 5) against numpy in extended precision where warps'
shares and rows meet awkwardly: fewer blocks than a step, shares that end at and
inside rows, rows without blocks at the ends and between, a row that crosses many
warps, one that spans whole shares, and its fused dot products inside the streaming
solver.  Tolerance per row: (row length) * 2^-52 * sum |a x| for the summation, plus
FP32 rounding of the values (2^-24) where those are used."""
import numpy as np
import pytest

import yafel_b200 as yb
from test_gpu_pcg_resident import device, spd

pytestmark = pytest.mark.gpu


def lengths(kind, rng):
    return {"one": [1], "step": [31], "exact": [32, 32, 64], "over": [33], "short": rng.integers(1, 9, 700),
            "mixed": rng.integers(0, 130, 900), "empty": [0, 0, 5, 0, 0, 0, 40, 0, 27, 0, 0],
            "hub": [20] * 500 + [4000] + [20] * 500, "giant": [3] * 50 + [60000] + [3] * 50,
            "many": rng.integers(20, 60, 20000)}[kind]


@pytest.mark.parametrize("B", [2, 3])
@pytest.mark.parametrize("kind", ["one", "step", "exact", "over", "short", "mixed", "empty", "hub", "giant", "many"])
def test_against_extended_precision(ctx, B, kind):
    rng = np.random.default_rng(B)
    n = np.asarray(lengths(kind, rng))
    nbcols = max(int(n.max()) + 3, 200)
    ptr = np.concatenate([[0], np.cumsum(n)])
    col = np.concatenate([np.sort(rng.permutation(nbcols)[:k]) for k in n]) if ptr[-1] else np.zeros(0, np.int64)
    vals = rng.standard_normal((ptr[-1], B, B))
    K = yb.sparse_bcsr.from_bcsr(B, ptr, col, vals.ravel(), nbcols=nbcols)
    x = rng.standard_normal(nbcols * B)
    xd = yb.DeviceVector(x)
    prod = (vals.astype(np.longdouble) * x.reshape(-1, 1, B)[col])
    want, size = np.zeros((n.size, B), np.longdouble), np.zeros((n.size, B))
    row = np.repeat(np.arange(n.size), n)
    np.add.at(want, row, prod.sum(2))
    np.add.at(size, row, np.abs(prod).sum(2).astype(float))
    for lanes in (1, 2):
        K.set_spmv(5, lanes)
        for prec, eps in ((yb.PREC_FP64, 0.0), (yb.PREC_MIXED, 2.0 ** -24)):
            y = K.spmv(xd, precision=prec).numpy().reshape(-1, B)
            assert np.all(np.abs(y - want) <= (B * n[:, None] * 2.0 ** -52 + eps) * size)
            assert np.array_equal(y, K.spmv(xd, precision=prec).numpy().reshape(-1, B))


@pytest.mark.parametrize("B", [2, 3])
def test_dot_products_and_correction_in_the_solver(ctx, B):
    K = device(*spd(4000, B, 11, extra=12))
    b = np.random.default_rng(3).standard_normal(4000 * B)
    M = yb.JacobiPreconditioner(K)
    for prec in (yb.PREC_FP64, yb.PREC_MIXED_IR):
        K.set_spmv(0, 16)
        x0, s0 = yb.solve(K, b, M=M, tol=1e-10, precision=prec, profile=True)
        for lanes in (1, 2):
            K.set_spmv(5, lanes)
            x, st = yb.solve(K, b, M=M, tol=1e-10, precision=prec, profile=True)
            assert st.status == 0 and abs(st.iterations - s0.iterations) <= 1
            assert np.linalg.norm(x.numpy() - x0.numpy()) <= 1e-8 * np.linalg.norm(x0.numpy())
