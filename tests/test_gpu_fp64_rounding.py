"""The FP64 path's quotients and square roots are IEEE's, rounded to nearest,
for the arguments where a form by reciprocals goes wrong first: divisors whose
reciprocal lies next to a midpoint of two doubles, quotients next to one, and
arguments whose square root does.

u = iap_u / sqrt(gd_edge) and pv = (f + vorticity) / gd_vertex are read back
and compared with numpy's division and square root, bit for bit."""
import copy

import numpy as np
import pytest

from tmcore_gb300 import mesh

pytestmark = pytest.mark.gpu

ALL_ONES = 2.0 - 2.0 ** -52  # its reciprocal lies 2^-106 above a midpoint


def _velocity(g, gd, iap):
    g.set_state(np.full(g.nc, gd), iap)
    return g.get_state()[2]


def _roots_mod(c, s):
    """The odd x below 2^s with x^2 = c mod 2^s (c = 1 mod 8)."""
    r = 1
    for k in range(3, s):
        if (r * r - c) >> k & 1:
            r += 1 << (k - 1)
    return {q % (1 << s) for q in (r, -r, r + (1 << (s - 1)), -r + (1 << (s - 1)))}


def _hard_squares(cmax):
    """Every double a in [1, 4) (as a 53-bit integer and s: a 2^s) whose root
    is m sqrt(1 - c/m^2) / 2^k for a 54-bit odd m, a midpoint, with |c| <= cmax:
    |c| 2^-56 units in the last place or more from m."""
    out = []
    for c in range(1 - 8 * (cmax // 8), cmax + 1, 8):
        for s in (54, 55):
            for q in _roots_mod(c % (1 << s), s):
                for m in range(q, 1 << 54, 1 << s):
                    a = (m * m - c) >> s
                    if m >= 1 << 53 and 1 << 52 <= a < 1 << 53:
                        out.append(float(a) * 2.0 ** (s % 2 - 52))
    return out


@pytest.fixture(scope="module")
def model():
    from tmcore_gb300.gpu import TMCoreGPU

    g = TMCoreGPU(mesh.icos_mesh(1), dt=600.0, pv_scheme=1, apvm_weight=0.0)
    g.set_initial(np.ones(g.nc), np.zeros(g.ne), np.zeros(g.nc))
    yield g
    g.close()


@pytest.mark.parametrize("exp", [-300, -52, 0, 40, 300])
def test_square_roots_next_to_a_midpoint(model, exp):
    iap = np.ldexp(1.0 + np.random.default_rng(1).random(model.ne), exp // 2)
    hard = _hard_squares(512)
    assert len(hard) > 150
    for a in np.ldexp(np.array(hard), exp):
        assert np.array_equal(_velocity(model, a, iap), iap / np.sqrt(a)), float(a).hex()


@pytest.mark.parametrize("exp", [-200, 0, 200])
def test_quotients_next_to_a_midpoint(model, exp):
    """Divisors 2 - k 2^-52 with odd k: their reciprocals lie k^2 2^-106 above
    a midpoint.  Dividends: powers of two (whose quotient is the reciprocal)
    and those whose quotients lie next to a midpoint, a 2^54 = B m + i with B
    the divisor's 53-bit integer."""
    for k in range(1, 60, 2):
        B = (1 << 53) - k
        gd = float(B * B >> 53) * 2.0 ** -51  # rounds to a root of B 2^-52
        near = np.nextafter(gd, np.array([0.0, 8.0]))
        gd = [x for x in (gd, *near) if np.sqrt(x) == B * 2.0 ** -52]
        assert gd, k
        a = [1 << 52]
        for i in range(-25, 26):
            m = -i * pow(B, -1, 1 << 54) % (1 << 54)
            q = (B * m + i) >> 54
            if 1 << 52 <= q < 1 << 53:
                a.append(q)
        iap = np.ldexp(np.resize(np.array(a, dtype=np.float64), model.ne), exp - 52)
        for x in gd:
            assert np.array_equal(_velocity(model, x, iap), iap / np.sqrt(x)), k


@pytest.mark.parametrize("f", [1.0, 2.0 ** 60, 1.5, 1.0 + 2.0 ** -52])
def test_vertex_quotient_by_a_hard_divisor(f):
    """pv = f / gd_vertex with gd_vertex = gd: one cell's kite is the whole
    triangle, areas are powers of two, and the fluid is at rest."""
    from tmcore_gb300.gpu import TMCoreGPU

    m = copy.deepcopy(mesh.icos_mesh(1))
    m.vars["areaTriangle"][:] = 2.0 ** -6
    m.vars["kiteAreasOnVertex"][:] = 0.0
    m.vars["kiteAreasOnVertex"][:, 0] = 2.0 ** -6
    m.vars["latVertex"][:] = np.pi / 2
    g = TMCoreGPU(m, dt=600.0, pv_scheme=1, apvm_weight=0.0, radius=1.0, omega=0.5 * f)
    for k in range(1, 60, 2):
        gd = 2.0 - k * 2.0 ** -52
        g.set_initial(np.full(g.nc, gd), np.zeros(g.ne), np.zeros(g.nc))
        assert np.array_equal(g.get_vertex()[0], np.full(g.nv, f / gd)), k
    g.close()
