"""Meshes whose tables disagree (a cell or a vertex that lists an edge which is
not its own, an edge missing from its vertex): the FP64 tendencies are the
oracle's bit for bit all the same."""
import copy

import numpy as np
import pytest

from tmcore_gb300 import cases, mesh

pytestmark = pytest.mark.gpu

CENTRED = dict(pv_scheme=1, apvm_weight=0.0)


def _foreign_edge_on_vertex(m):
    m.vars["edgesOnVertex"][200, 1] = 7


def _foreign_edge_on_cell(m):
    m.vars["edgesOnCell"][100, 2] = 7


def _check(m, **kw):
    from oracle.oracle import Oracle
    from tmcore_gb300.gpu import TMCoreGPU

    gd, u, ghs = cases.jet_bumps(m, seed=5)
    g, o = TMCoreGPU(m, dt=600.0, **kw), Oracle(m, dt=600.0, **kw)
    for x in (g, o):
        x.set_initial(gd, u, ghs)
    iap = o.state()[1]
    for a, b in zip(g.spatial_operators(gd, iap), o.spatial_operators(gd, iap)):
        assert np.all(np.isfinite(b)) and np.array_equal(a, b)
    g.close()
    o.close()


@pytest.mark.parametrize("change", [_foreign_edge_on_vertex, _foreign_edge_on_cell])
def test_foreign_edges(change):
    m = copy.deepcopy(mesh.icos_mesh(3))
    change(m)
    _check(m, **CENTRED)


def _edge_missing_from_vertex(m):
    m.vars["edgesOnVertex"][200, 1] = m.vars["edgesOnVertex"][200, 0]


@pytest.mark.parametrize("order", [3, 4])
def test_upwind_pv_of_an_edge_its_vertex_does_not_list(order):
    """The vertex fits, formed by vertex, would leave the edge's side unset."""
    m = copy.deepcopy(mesh.icos_mesh(3))
    _edge_missing_from_vertex(m)
    _check(m, pv_scheme=3, interp_pv_order=order)


@pytest.mark.parametrize("kw", [CENTRED, dict(pv_scheme=3, interp_pv_order=3)])
def test_wide_neighbour_tables(kw):
    """Six entries per neighbour, with alternating signs but for the first: 60
    of the 64 neighbours a mesh may have, and sums that cancel."""
    m = copy.deepcopy(mesh.icos_mesh(3))
    w = m.vars["weightsOnEdge"][:, :, None] * np.array([1.0, 0.7, -0.7, 0.3, -0.3, 0.0])
    m.vars["weightsOnEdge"] = np.ascontiguousarray(w.reshape(m.nEdges, -1))
    m.vars["edgesOnEdge"] = np.ascontiguousarray(np.repeat(m.vars["edgesOnEdge"], 6, axis=1))
    m.vars["nEdgesOnEdge"] = m.vars["nEdgesOnEdge"] * 6
    m.dims = dict(m.dims, maxEdges2=6 * m.dims["maxEdges2"])
    _check(m, **kw)
