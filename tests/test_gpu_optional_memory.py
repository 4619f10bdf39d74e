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
