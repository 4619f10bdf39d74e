"""Batched PCG in the shared memory of groups of CTAs: one to many CTAs a system, sizes
on both sides of what a group can hold, all block sizes and precisions, systems that
stop by their cap, more systems than one launch takes, and beside systems that the
batch's own kernels iterate.  A result is the same to the bit whatever else is in the
batch and however many blocks a run is cut into."""
import numpy as np
import pytest

import yafel_b200 as yb
from test_gpu_pcg_resident import device, host_spmv, spd

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (40, 2), (300, 1), (700, 3), (2500, 2), (5001, 1), (9000, 3)]


def problems(sizes, seed=0):
    out = []
    for k, (nb, B) in enumerate(sizes):
        sys_ = spd(nb, B, seed + 31 * k + nb)
        out.append((sys_, device(*sys_), np.random.default_rng(k).standard_normal(nb * B)))
    return out


def relres(sys_, x, b):
    return np.linalg.norm(b - host_spmv(*sys_, x)) / np.linalg.norm(b)


def meshes():
    """Poisson and elasticity systems: 4 to 14,406 unknowns, rows of 4 to 125 blocks."""
    out = []
    for dim, n, p, dpn in [(2, 1, 1, 1), (2, 1, 2, 2), (3, 1, 1, 3), (2, 20, 2, 1), (2, 24, 3, 2), (3, 4, 2, 3),
                           (2, 60, 2, 2), (3, 8, 2, 1)]:
        dm = yb.DoFManager.box(dim, (n,) * dim, polyOrder=p, dof_per_node=dpn)
        fe = yb.FESystem(dm, dim, format=yb.BCSR if dpn > 1 else yb.CSR)
        yb.CGAssembly(yb.LinearElasticity(dim) if dpn > 1 else yb.PoissonEquation(dim), fe)
        K = fe.getGlobalTangent()
        F = yb.DeviceVector(np.random.default_rng(n).standard_normal(K.rows()))
        for c in range(dpn):
            bc = yb.DirichletBC(dm, 0.0, c)
            bc.selectByFunction(lambda X: np.abs(X[:, 0]) < 1e-6)
            bc.apply(K, F)
        out.append((fe, K, F.numpy()))
    return out


@pytest.mark.parametrize("precision", [yb.PREC_FP64, yb.PREC_MIXED])
def test_alone_in_mix_and_in_blocks(ctx, precision):
    probs = meshes()
    alone = []
    for _, K, b in probs:
        B = yb.Batch(1, ctx)
        s = B.add(K, b, tol=1e-9, precision=precision, maxiter=2000)
        assert B.run() == 0
        st = B.stats(s)
        assert st.status == 0 and st.iterations > 0
        alone.append((B.solution(s).numpy(), st.iterations, st.refinements))
        assert np.linalg.norm(b - K * alone[-1][0]) <= 1.01e-9 * np.linalg.norm(b)
    for blocks in (0, 1, 3):
        B = yb.Batch(len(probs), ctx)
        slots = [B.add(K, b, tol=1e-9, precision=precision, maxiter=2000) for _, K, b in probs]
        for _ in range(300):
            if B.run(max_blocks=blocks) == 0:
                break
        for s, (x, its, refs) in zip(slots, alone):
            st = B.stats(s)
            assert (st.status, st.iterations, st.refinements) == (0, its, refs)
            assert np.array_equal(B.solution(s).numpy(), x)


@pytest.mark.parametrize("maxiter", [1, 15, 16, 17, 40])
def test_iteration_cap(ctx, maxiter):
    probs = problems(SIZES[3:], seed=5)
    for blocks in (0, 1):
        B = yb.Batch(len(probs), ctx)
        slots = [B.add(K, b, tol=1e-300, maxiter=maxiter) for _, K, b in probs]
        for _ in range(100):
            if B.run(max_blocks=blocks) == 0:
                break
        for s, (_, K, b) in zip(slots, probs):
            assert B.stats(s).iterations == maxiter and B.stats(s).status != 0
            # the single solver's iterate: rounding of at most 40 steps of systems
            # with condition numbers below 100
            x, _ = yb.solve(K, b, M=yb.JacobiPreconditioner(K), tol=1e-300, maxiter=maxiter)
            assert np.abs(B.solution(s).numpy() - x.numpy()).max() <= 1e-10 * np.abs(x.numpy()).max()


def test_beside_systems_of_the_batch_kernels(ctx):
    # BiCGSTAB, a matrix too large for the SMs (68,921 rows, 49 MB), and one with its own launches
    probs = problems(SIZES[2:6], seed=9)
    dm = yb.DoFManager.box(3, (20, 20, 20), polyOrder=2, dof_per_node=1)
    fe = yb.FESystem(dm, 3, format=yb.CSR)
    yb.CGAssembly(yb.PoissonEquation(3), fe)
    big = fe.getGlobalTangent()
    F = yb.DeviceVector(np.random.default_rng(3).standard_normal(big.rows()))
    bc = yb.DirichletBC(dm, 0.0, 0)
    bc.selectByFunction(lambda X: np.abs(X[:, 0]) < 1e-6)
    bc.apply(big, F)
    for blocks in (0, 2):
        B = yb.Batch(len(probs) + 3, ctx)
        systems = [(K, b) for _, K, b in probs] + [(big, F.numpy())]
        slots = [B.add(K, b, tol=1e-9, maxiter=2000) for K, b in systems]
        slots.append(B.add(probs[1][1], probs[1][2], tol=1e-9, method="bicgstab"))
        B.set_solo_bytes(1)
        slots.append(B.add(probs[2][1], probs[2][2], tol=1e-9))
        for _ in range(300):
            if B.run(max_blocks=blocks) == 0:
                break
        for slot, (K, b) in zip(slots, systems + [systems[1], systems[2]]):
            assert B.stats(slot).status == 0
            assert np.linalg.norm(b - K * B.solution(slot).numpy()) <= 1.01e-9 * np.linalg.norm(b)


def test_more_systems_than_a_launch_takes(ctx):
    probs = problems([(20 + k % 7, 1 + k % 3) for k in range(12)], seed=2)
    n = 600
    B = yb.Batch(n, ctx)
    slots = [B.add(probs[k % 12][1], probs[k % 12][2], tol=1e-9) for k in range(n)]
    assert B.run() == 0
    for k, s in enumerate(slots):
        x = B.solution(s).numpy()
        if k < 12:
            assert relres(probs[k][0], x, probs[k][2]) <= 1.01e-9
        else:
            assert np.array_equal(x, B.solution(slots[k % 12]).numpy())
