"""Contexts used from several threads at once, one per thread as the header allows:
every call gives what it gives alone."""
import threading

import numpy as np
import pytest

import yafel_b200 as yb
from test_gpu_pcg_resident import spd

pytestmark = pytest.mark.gpu


def together(*jobs):
    """Runs every job in a thread of its own, started together; their results."""
    out, errors, gate = [None] * len(jobs), [], threading.Barrier(len(jobs))

    def run(i):
        try:
            gate.wait()
            out[i] = jobs[i]()
        except Exception as e:  # (reported by the thread that started this one)
            errors.append(e)
    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return out


def matrix(c, nb, B, seed=1):
    ptr, col, vals = spd(nb, B, seed)
    return (yb.sparse_csr.from_csr(ptr, col, vals.ravel(), ctx=c) if B == 1 else
            yb.sparse_bcsr.from_bcsr(B, ptr, col, vals.ravel(), ctx=c))


def test_solves_of_different_sizes_do_not_lower_each_others_shared_memory(ctx):
    """Systems that need 10 to 200 KB of shared memory an SM, solved side by side."""
    jobs, alone = [], []
    for nb in (300, 40000, 3000, 60000):
        c = yb.Context(0)
        K = matrix(c, nb, 1)
        b = yb.DeviceVector(np.random.default_rng(nb).standard_normal(nb), c)
        M = yb.JacobiPreconditioner(K)

        def job(K=K, b=b, M=M):
            return [yb.solve(K, b, M=M, tol=1e-10)[0].numpy() for _ in range(60)]
        alone.append(job()[0])
        jobs.append(job)
    for xs, ref in zip(together(*jobs), alone):
        for x in xs:
            assert np.array_equal(x, ref)


def test_ilu_factorizations_do_not_lower_each_others_shared_memory(ctx):
    """Rows of about 10 and of about 300 blocks, factored side by side."""
    jobs, refs = [], []
    for nb, extra in ((200, 4), (300, 150)):
        c = yb.Context(0)
        ptr, col, vals = spd(nb, 2, 3, extra=extra)
        K = yb.sparse_bcsr.from_bcsr(2, ptr, col, vals.ravel(), ctx=c)
        z = np.random.default_rng(nb).standard_normal(2 * nb)

        def job(K=K, z=z):
            return [yb.ILUPreconditioner(K).solve(z.copy()) for _ in range(40)]
        refs.append(job()[0])
        jobs.append(job)
    for zs, ref in zip(together(*jobs), refs):
        for z in zs:
            assert np.array_equal(z, ref)


def test_replayed_ilu_applies_beside_resident_solves_and_batches(ctx):
    """ILU(0)-PCG long enough to replay its graph, resident PCG of small and of all-SM
    systems and a resident batch, side by side: each gives what it gives alone."""
    jobs, refs = [], []
    c = yb.Context(0)
    K = matrix(c, 6000, 2, 5)
    b = yb.DeviceVector(np.random.default_rng(5).standard_normal(12000), c)
    M = yb.ILUPreconditioner(K)

    def ilu(K=K, b=b, M=M):  # (a fixed number of iterations, past the directly launched ones)
        return [yb.solve(K, b, M=M, tol=1e-300, maxiter=100)[0].numpy() for _ in range(4)]
    jobs.append(ilu)
    for nb in (2000, 90000):
        c = yb.Context(0)
        K = matrix(c, nb, 1, 6)
        b = yb.DeviceVector(np.random.default_rng(nb).standard_normal(nb), c)

        def resident(K=K, b=b, M=yb.JacobiPreconditioner(K)):
            return [yb.solve(K, b, M=M, tol=1e-10)[0].numpy() for _ in range(30)]
        jobs.append(resident)
    c = yb.Context(0)
    B = yb.Batch(6, c)
    slots = []
    for i in range(6):
        K = matrix(c, 1500 + 700 * i, 1 + i % 2, 7 + i)
        slots.append(B.add(K, np.random.default_rng(i).standard_normal(K.rows())))

    def batch():
        out = []
        for _ in range(8):
            for s in slots:
                B._keep[s][2].fill(0.0)
            B.reset()
            assert B.run() == 0
            out.append(np.concatenate([B.solution(s).numpy() for s in slots]))
        return out
    jobs.append(batch)
    refs = [job()[0] for job in jobs]
    for xs, ref in zip(together(*jobs), refs):
        assert np.all(np.isfinite(ref))
        for x in xs:
            assert np.array_equal(x, ref)
