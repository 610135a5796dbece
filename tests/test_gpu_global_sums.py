"""The global sums lose nothing when they combine their blocks' sums: total
mass, on states whose blocks' sums are exact, is the exactly rounded sum of
gd areaCell, although single additions of two blocks' sums would drop the
smaller one (it is below half a unit in the last place of the larger)."""
import copy
import math

import numpy as np
import pytest

from tmcore_gb300 import mesh

pytestmark = pytest.mark.gpu


def _unit_areas(level):
    m = copy.copy(mesh.icos_mesh(level))
    m.vars = dict(m.vars, areaCell=np.ones(m.nCells))
    return m


def test_ensemble_mass_is_exact():
    """Slots of 128 cells; warp w of the reduction adds slots w, w + 32, ...,
    the (slot / 32 mod 4)-th of its four accumulators each.  The first holds
    3 2^30, whose unit is 2^-21, the second 0.47 of that, the other two
    together as much."""
    from tmcore_gb300.gpu import TMCoreGPU

    m = _unit_areas(6)
    turn = np.arange(m.nCells) // 128 // 32 % 4
    gd = np.array([2.0 ** 23, 5 * 2.0 ** -33, 15 * 2.0 ** -35, 15 * 2.0 ** -35])[turn]
    g = TMCoreGPU(m, dt=60.0, precision=1, members=16, member_layout=1, renumber=0, radius=1.0, pv_scheme=1,
                  apvm_weight=0.0)
    for k in range(16):
        g.select_member(k)
        g.set_state(np.ldexp(gd, k), np.zeros(g.ne))
    mass = g.diag_all()[:, 0]
    assert np.array_equal(mass, np.ldexp(math.fsum(gd), np.arange(16)))
    g.close()


def test_single_model_mass_is_exact():
    """Blocks of 1024 cells; lane l of a warp takes blocks l and l + 32.
    Blocks 0-8 hold 2^30 each (unit 2^-22), blocks 32-39 0.47 of that unit,
    blocks 9-24 2^-25."""
    from tmcore_gb300.gpu import TMCoreGPU

    m = _unit_areas(6)
    block = np.arange(m.nCells) // 1024
    gd = np.full(m.nCells, 2.0 ** -70)
    gd[block < 9] = 2.0 ** 20
    gd[(block >= 9) & (block < 25)] = 2.0 ** -35
    gd[(block >= 32) & (block < 40)] = 15 * 2.0 ** -37
    g = TMCoreGPU(m, dt=60.0, precision=1, renumber=0, radius=1.0, pv_scheme=1, apvm_weight=0.0)
    g.set_state(gd, np.zeros(g.ne))
    assert g.diag_all()[0, 0] == math.fsum(gd)
    g.close()
