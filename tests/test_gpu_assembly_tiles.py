"""The tiled element matrices and the scatter map against the oracle where they
can go wrong: node counts at the edges of the 8-node tiles and of the warp / CTA
teams (4, 25, 64, 100 nodes per cell), more cells than teams in a launch, cells
that list a node twice (no map: searched and added atomically), and a context
whose memory budget does not hold the map.  Tolerance: 1e-13 of a row's largest
entry, the suite's bound for a re-ordered FP64 sum.  From order 7 on the
reference is the same sum in 80-bit arithmetic over the library's element tables
(the oracle's own order-7 matrix is 1.1e-13 off it), and so it is for the cells
that repeat a node (the oracle keeps such columns apart)."""
import numpy as np
import pytest

import yafel_b200 as yb
from oracle import oracle as O
from yafel_b200 import meshgen
from test_gpu_assembly import PHYS, compare, oracle_dofmap

pytestmark = pytest.mark.gpu


def extended(dm, p, okind, dpn, prm):
    """CGAssembly on 2D tensor cells in np.longdouble: (Csr-like K, residual)."""
    ld = np.longdouble
    _, _, W, N, dN = [np.asarray(a, ld) for a in yb.element_table(0, 2, p)]
    n = dm.nNodes() * dpn
    K, R = np.zeros((n, n), ld), np.zeros(n, ld)
    hit = np.zeros((n, n), bool)
    for c in range(dm.nCells()):
        el = dm.getGlobalNodes(c)
        x = np.asarray(dm.dof_nodes[el, :2], ld)
        J = np.einsum("ai,qaj->qij", x, dN)
        w = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
        inv = np.stack([J[:, 1, 1], -J[:, 0, 1], -J[:, 1, 0], J[:, 0, 0]], 1).reshape(-1, 2, 2) / w[:, None, None]
        G = np.einsum("qji,qaj->qai", inv, dN)
        w = w * W
        ix = (el[:, None] * dpn + np.arange(dpn)).ravel()
        M = np.einsum("q,qai,qbk->aibk", w, G, G)
        if okind == O.POISSON:
            Ke, Re = prm[0] * np.einsum("aibi->ab", M), prm[1] * (w @ N)
        elif okind == O.ELASTICITY:
            Ke = prm[1] * M + prm[2] * M.transpose(0, 3, 2, 1)
            for i in range(2):
                Ke[:, i, :, i] += prm[2] * np.einsum("adbd->ab", M)
            Ke, Re = Ke.reshape(ix.size, -1), np.outer(w @ N, np.asarray(prm[3:5], ld)).ravel()
        else:  # SUPG: the advection term once per dimension
            k, h, U, Q = [ld(v) for v in prm]
            a = np.cosh(U * h / (2 * k)) / np.sinh(U * h / (2 * k)) - 2 * k / (U * h)
            Ke = (k + a * h * U / 2) * M[:, 0, :, 0] + k * M[:, 1, :, 1] + 2 * U * np.einsum("q,qa,qb->ab", w, N, G[:, :, 0])
            Re = -(2 * Q * (w @ N) + a * h / 2 * (w @ G[:, :, 0]))
        np.add.at(K, np.ix_(ix, ix), Ke)  # a node listed twice counts twice
        hit[np.ix_(ix, ix)] = True
        np.add.at(R, ix, Re)
    r, c = np.nonzero(hit)
    ptr = np.concatenate([[0], np.cumsum(hit.sum(1))])
    return O.Csr(n, n, ptr, c, K[r, c].astype(np.float64)), R.astype(np.float64)


def check(dm, odm, nsd, phys, fmt):
    okind, mk, oparams = PHYS[phys]
    physics = mk(nsd)
    dpn = nsd if okind == O.ELASTICITY else 1
    if oparams is None:
        oparams = [1.0, physics.lam, physics.mu] + list(physics.body)
    fe = yb.FESystem(dm, nsd, format=fmt)
    yb.CGAssembly(physics, fe)
    if odm is None:
        Ko, Ro = extended(dm, dm.polyOrder, okind, dpn, oparams)
    else:
        Ko, Ro = O.assemble(odm, dpn, nsd, okind, oparams)
    compare(fe.getGlobalTangent(), Ko)
    R = fe.getGlobalResidual().numpy()
    assert np.abs(R - Ro).max() <= 1e-13 * max(np.abs(Ro).max(), 1e-300)
    return fe


@pytest.mark.parametrize("n,p,phys,fmt", [
    (201, 1, "poisson", yb.CSR), (200, 1, "elasticity", yb.BCSR), (97, 1, "supg", yb.CSR),
    (5, 4, "poisson", yb.CSR), (4, 4, "elasticity", yb.BCSR), (4, 4, "elasticity", yb.CSR), (4, 4, "supg", yb.CSR),
    (3, 7, "poisson", yb.CSR), (3, 7, "elasticity", yb.BCSR), (2, 9, "elasticity", yb.BCSR), (2, 9, "supg", yb.CSR)])
def test_tile_edges(ctx, n, p, phys, fmt):
    mesh = meshgen.structured_quad(n, max(2, n - 1), order=meshgen.corner_order(p))
    dm = yb.DoFManager(mesh, p, 2 if phys == "elasticity" else 1)
    check(dm, oracle_dofmap(mesh, p, dm) if p < 7 else None, 2, phys, fmt)


@pytest.mark.parametrize("phys,fmt", [("poisson", yb.CSR), ("elasticity", yb.BCSR), ("elasticity", yb.CSR)])
def test_cells_that_repeat_a_node(ctx, phys, fmt):
    # two quadrilaterals collapsed to triangles beside whole ones
    nodes = np.array([[0, 0, 0], [1, 0, 0], [2, 0, 0], [0, 1, 0], [1, 1, 0], [2, 1, 0], [1, 2, 0.]])
    cells = [[0, 1, 3, 4], [1, 2, 4, 5], [3, 4, 6, 6], [4, 5, 6, 6]]
    mesh = {"nodes": nodes, "cell_nodes": np.array(cells, np.int32).ravel(), "offsets": np.arange(0, 17, 4, dtype=np.int32),
            "cell_types": np.full(4, meshgen.QUAD4, np.int32)}
    dm = yb.DoFManager(mesh, 1, 2 if phys == "elasticity" else 1)
    check(dm, None, 2, phys, fmt)


def test_budget_without_room_for_the_map():
    def build(c):
        dm = yb.DoFManager(meshgen.structured_hex(7, 6, 5), 2, 3, ctx=c)
        fe = yb.FESystem(dm, 3)
        yb.CGAssembly(yb.LinearElasticity(3), fe)
        return fe

    free = yb.Context(0)
    fe = build(free)
    want = fe.getGlobalTangent().arrays()
    held = free.memory()[0]
    tight = yb.Context(0, hbm_budget=held - 1)  # one byte short of the matrix beside the map
    got = build(tight).getGlobalTangent().arrays()
    assert tight.memory()[0] < held - 100_000   # the map went, the matrix came
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert np.abs(got[2] - want[2]).max() <= 1e-13 * np.abs(want[2]).max()
