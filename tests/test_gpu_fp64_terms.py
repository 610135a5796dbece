"""The FP64 path's per-edge terms, reciprocal quotients and square roots
against the CPU oracle, bit for bit, on states where the fast forms hand over
to the plain operations: zeros, very large and very small magnitudes, and
meshes whose last block is nearly empty."""
import numpy as np
import pytest

from tmcore_gb300 import cases, mesh

pytestmark = pytest.mark.gpu


def _state(m, scale, still):
    gd, u, ghs = cases.jet_bumps(m, seed=5)
    c1, c2 = m.cellsOnEdge[:, 0] - 1, m.cellsOnEdge[:, 1] - 1
    iap = np.sqrt(0.5 * (gd[c1] + gd[c2])) * u
    if still:  # a calm part of the sphere: zero wind, zero products and quotients
        iap[m.zEdge > 0.2] = 0.0
    return gd * scale, iap * scale, ghs * scale


@pytest.mark.parametrize("level", [1, 3, 4])
@pytest.mark.parametrize("kw", [dict(pv_scheme=1, apvm_weight=0.0), dict(pv_scheme=3, interp_pv_order=3),
                                dict(pv_scheme=1, apvm_weight=0.0, adv_order=3, adv_mono=1)])
@pytest.mark.parametrize("scale,still", [(1.0, False), (1.0, True), (1e-40, True), (1e-130, False), (1e90, False)])
def test_tendencies_bit_identical(level, kw, scale, still):
    from oracle.oracle import Oracle
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(level)
    gd, iap, ghs = _state(m, scale, still)
    g, o = TMCoreGPU(m, dt=600.0, **kw), Oracle(m, dt=600.0, **kw)
    g.set_initial(gd, np.zeros(m.nEdges), ghs)
    o.set_initial(gd, np.zeros(m.nEdges), ghs)
    with np.errstate(all="ignore"):
        want = o.spatial_operators(gd, iap)
    got = g.spatial_operators(gd, iap)
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
    g.close()
    o.close()


@pytest.mark.parametrize("tracers,order", [(1, 2), (4, 2), (5, 2), (2, 3)])
def test_tracer_terms_match_oracle(tracers, order):
    """Tracer edge terms in the fused step: the oracle's tracers to 1e-13 after
    three steps, the tolerance of the coupled tracers (beta's sums are ordered
    differently), and a constant mixing ratio stays constant to round-off."""
    from oracle.oracle import Oracle
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(4)
    gd, u, ghs = cases.jet_bumps(m, seed=6)
    kw = dict(dt=600.0, pv_scheme=1, apvm_weight=0.0, n_tracers=tracers, tracer_adv_order=order)
    q = cases.smooth_tracers(m, tracers, seed=2)
    q[0] = 0.75
    g, o = TMCoreGPU(m, **kw), Oracle(m, **kw)
    for x in (g, o):
        x.set_initial(gd, u, ghs)
        x.set_tracers(q * gd)
        x.step(3)
    a, b = g.get_tracers(), o.tracers()
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))
    assert np.max(np.abs(a[0] / g.get_state()[0] - 0.75)) < 1e-14
    g.close()
    o.close()


@pytest.mark.parametrize("level", [1, 4, 6])
@pytest.mark.parametrize("scale", [1.0, 1e-60, 1e-140, 1e80])
def test_invariants_match_exact_sums(level, scale):
    """Mass, energy and absolute vorticity (integer block sums; FP64 sums for
    extreme exponents) against exactly rounded sums of the same terms.  Terms
    carry at most three roundings of 2^-53 and a thread adds four of them, so
    16 2^-53 of the sum of magnitudes bounds the difference."""
    import math

    from tmcore_gb300.gpu import REF_OMEGA, REF_RADIUS, TMCoreGPU

    m = mesh.icos_mesh(level)
    gd, iap, ghs = _state(m, scale, False)
    g = TMCoreGPU(m, dt=600.0, pv_scheme=1, apvm_weight=0.0)
    g.set_initial(gd, np.zeros(m.nEdges), ghs)
    g.set_state(gd, iap)
    mass, energy, _, av = g.diag()[:4]
    r2 = REF_RADIUS ** 2
    A, Ae, At = m.areaCell * r2, (m.dvEdge * m.dcEdge) * r2, m.areaTriangle * r2
    tol = 16 * 2.0 ** -53
    t = gd * A
    assert abs(mass - math.fsum(t)) <= tol * math.fsum(abs(t))
    t = np.concatenate([(gd * gd + 2.0 * gd * ghs) * A, iap * iap * Ae])
    assert abs(energy - math.fsum(t)) <= tol * math.fsum(abs(t))
    _, vor = g.get_vertex()
    t = (vor + 2.0 * REF_OMEGA * np.sin(m.latVertex)) * At
    assert abs(av * math.fsum(At) - math.fsum(t)) <= tol * math.fsum(abs(t)) + 2.0 ** -51 * abs(math.fsum(t))
    g.close()
