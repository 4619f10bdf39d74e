"""Scatter maps of the assembly under a memory budget: they go only for an allocation that
needs their place and fits in it, come back at a later assembly when there is room, and
no value depends on them."""
import numpy as np
import pytest

import yafel_b200 as yb
from yafel_b200 import _lib, meshgen

pytestmark = pytest.mark.gpu


def problem(c, mixed):
    mesh = meshgen.jittered_mixed(30, 30, seed=3) if mixed else meshgen.structured_hex(7, 6, 5)
    dim = 2 if mixed else 3
    fe = yb.FESystem(yb.DoFManager(mesh, 2, dim, ctx=c), dim)
    phys = yb.LinearElasticity(dim)
    yb.CGAssembly(phys, fe)
    return fe, phys


@pytest.mark.parametrize("mixed", [False, True])
def test_maps_go_when_they_make_room_and_come_back(mixed):
    free = problem(yb.Context(0), mixed)
    held = free[0].ctx.memory()[0]
    budget = held + (1 << 20)
    c = yb.Context(0, hbm_budget=budget)
    fe, phys = problem(c, mixed)
    assert c.memory()[0] == held
    want = fe.getGlobalTangent().arrays()[2].copy()

    def again():
        yb.CGAssembly(phys, fe)
        assert np.array_equal(fe.getGlobalTangent().arrays()[2], want)

    with pytest.raises(yb.YafelError) as e:  # more than all of the budget: nothing goes for it
        yb.DeviceVector(budget // 8, c)
    assert e.value.status == _lib.YG_OVER_BUDGET and c.memory()[0] == held
    v = yb.DeviceVector((1 << 17) + 100, c)  # a little more than what is left
    assert c.memory()[0] < held + 8 * ((1 << 17) + 100)
    for _ in range(5):  # (there is no room to lay them out again)
        again()
    del v
    small = c.memory()[0]
    assert small < held
    for _ in range(8):
        again()
    assert c.memory()[0] == held
    v = yb.DeviceVector((1 << 17) + 100, c)
    del v
    assert c.memory()[0] == small
    again()
    assert c.memory()[0] == small  # (not at once)
    for _ in range(20):
        again()
    assert c.memory()[0] == held


@pytest.mark.parametrize("phys,fmt", [("poisson", yb.CSR), ("elasticity", yb.BCSR)])
def test_no_maps_for_cells_that_repeat_a_node(phys, fmt):
    """Cells that repeat a node have entries that one cell adds to twice, so they never get a
    map: not even where the pattern was built without room for one and there is room later.
    Tolerance: four contributions of a cell to an entry, summed in any order (1e-13)."""
    mesh = meshgen.structured_quad(40, 40, order=meshgen.corner_order(1))
    mesh["cell_nodes"].reshape(-1, 4)[::7, 2] = mesh["cell_nodes"].reshape(-1, 4)[::7, 3]
    dpn = 2 if phys == "elasticity" else 1
    physics = yb.LinearElasticity(2) if dpn == 2 else yb.PoissonEquation(2)

    def system(c):
        return yb.FESystem(yb.DoFManager(mesh, 1, dpn, ctx=c), 2, format=fmt)

    def values(fe):
        yb.CGAssembly(physics, fe)
        return fe.getGlobalTangent().arrays()[2].copy()

    want = values(system(yb.Context(0)))
    assert np.all(np.isfinite(want))
    refused = 0
    for spare in range(8 << 10, 600 << 10, 16 << 10):  # room for less and more than pattern and maps
        c = yb.Context(0, hbm_budget=64 << 20)
        fe = system(c)
        v = yb.DeviceVector(((64 << 20) - c.memory()[0] - spare) // 8, c)
        try:
            values(fe)
        except yb.YafelError as e:
            assert e.status == _lib.YG_OVER_BUDGET
            refused += 1
        del v
        for _ in range(7):
            assert np.abs(values(fe) - want).max() <= 1e-13 * np.abs(want).max()
    assert refused
