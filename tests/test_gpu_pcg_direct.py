"""PCG's first iterations are launched one by one and the later ones replayed from a
captured graph: both run the same kernels in the same order, so the iterate does not
depend on where the change-over lies."""
import numpy as np
import pytest

import yafel_b200 as yb

pytestmark = pytest.mark.gpu


def system(n, fmt):
    # 13^3 Q2 elasticity: too large for the shared-memory route in FP64, an odd number of rows
    dm = yb.DoFManager.box(3, (n,) * 3, polyOrder=2, dof_per_node=3)
    fe = yb.FESystem(dm, 3, format=fmt)
    yb.CGAssembly(yb.LinearElasticity(3), fe)
    K = fe.getGlobalTangent()
    F = yb.DeviceVector(np.random.default_rng(5).standard_normal(K.rows()))
    for c in range(3):
        bc = yb.DirichletBC(dm, 0.0, c)
        bc.selectByFunction(lambda X: np.abs(X[:, 0]) < 1e-6)
        bc.apply(K, F)
    K.set_spmv_for(0, 2 if fmt == yb.BCSR else 0, 4)  # one kernel for every solve
    return K, F


@pytest.mark.parametrize("fmt", [yb.BCSR, yb.CSR])
@pytest.mark.parametrize("jacobi", [True, False])
def test_iterate_independent_of_change_over(fmt, jacobi):
    K, F = system(13, fmt)
    assert K.rows() % 2 == 1
    M = yb.JacobiPreconditioner(K) if jacobi else None
    got = {}
    for every in (2, 8, 64):  # direct until iteration 4, 16, 128
        for its in (1, 4, 5, 40):
            x, st = yb.solve(K, F, M=M, tol=1e-300, maxiter=its, check_every=every)
            assert st.iterations == its
            got[every, its] = np.asarray(x.numpy())
    for its in (1, 4, 5, 40):
        assert np.array_equal(got[2, its], got[64, its])
        assert np.array_equal(got[8, its], got[64, its])
    assert not np.array_equal(got[2, 4], got[2, 5])
