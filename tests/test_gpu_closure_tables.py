"""An ensemble holds the learned closure's mesh tables from the first call on
that needs them, once."""
import pytest

from tmcore_gb300 import cases, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["set_closure", "closure_features"])
def test_tables_on_demand(first):
    from tmcore_gb300.gpu import ClosureMLP, TMCoreGPU

    m = mesh.icos_mesh(3)
    g = TMCoreGPU(m, dt=600.0, precision=1, members=16, member_layout=1, pv_scheme=1, apvm_weight=0.0)
    for k in range(16):
        g.select_member(k)
        g.set_initial(*cases.jet_bumps(m, seed=k))
    net = ClosureMLP(seed=3)
    calls = {"set_closure": lambda: g.set_closure(net), "closure_features": g.closure_features}
    without = g.sizes()[3]
    calls.pop(first)()
    with_tables = g.sizes()[3]
    # a record of 28 words per edge, and a word per vertex of a cell
    assert with_tables == without + 112 * m.nEdges + 4 * 3 * m.nVertices
    calls.popitem()[1]()
    assert g.sizes()[3] == with_tables
    g.set_closure(net)
    g.step(1)
    assert not g.closure_status()
    g.close()
