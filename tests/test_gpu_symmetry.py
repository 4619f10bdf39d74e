"""The tangents of symmetric forms are symmetric to the bit: entry (B, A) of an element is
entry (A, B), transposed, and both are added in one order of cells."""
import numpy as np
import pytest
import scipy.sparse as sp

import yafel_b200 as yb
from yafel_b200 import meshgen

pytestmark = pytest.mark.gpu

MESHES = {"quads": lambda p: (meshgen.structured_quad(9, 7, order=meshgen.corner_order(p)), 2),
          "mixed": lambda p: (meshgen.jittered_mixed(11, 11, seed=5, order=meshgen.corner_order(p)), 2),
          "hexes": lambda p: (meshgen.structured_hex(4, 3, 3, order=meshgen.corner_order(p)), 3)}


@pytest.mark.parametrize("fmt", [yb.CSR, yb.BCSR])
@pytest.mark.parametrize("phys", ["poisson", "elasticity"])
@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("mesh", sorted(MESHES))
def test_symmetric_to_the_bit(ctx, mesh, p, phys, fmt):
    m, dim = MESHES[mesh](p)
    rng = np.random.default_rng(p)
    m = dict(m, nodes=m["nodes"] + 0.01 * rng.standard_normal(m["nodes"].shape) * (np.arange(3) < dim))
    dm = yb.DoFManager(m, p, dim if phys == "elasticity" else 1)
    fe = yb.FESystem(dm, dim, format=fmt)
    yb.CGAssembly(yb.LinearElasticity(dim) if phys == "elasticity" else yb.PoissonEquation(dim), fe,
                  [yb.AssemblyRequirement.Tangent])
    K = fe.getGlobalTangent()
    ptr, col, val = K.arrays()
    n = len(ptr) - 1
    B = int(round((len(val) / len(col)) ** 0.5))
    A = (sp.csr_matrix((val, col, ptr), shape=(n, n)) if B == 1 else
         sp.bsr_matrix((np.asarray(val).reshape(-1, B, B), col, ptr), shape=(n * B, n * B)).tocsr())
    D = (A - A.T).tocoo()
    assert np.abs(D.data).max(initial=0.0) == 0.0
