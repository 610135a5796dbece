"""One and four elements per thread give the same results, in FP32 bit for bit
with any block size: a pass of one element per thread stores its terms of the
global sums, and they are added in the order of the four-element launch.  The
levels' element counts are no multiples of a block's 1024."""
import numpy as np
import pytest

from tmcore_gb300 import abi, cases, mesh

pytestmark = pytest.mark.gpu

CENTRED = dict(pv_scheme=1, apvm_weight=0.0)
OPTIONS = [dict(pv_scheme=3, interp_pv_order=3), CENTRED, dict(CENTRED, n_tracers=1), dict(CENTRED, n_tracers=3),
           dict(CENTRED, n_tracers=4), dict(CENTRED, adv_order=3, n_tracers=2), dict(pv_scheme=1, apvm_weight=0.5),
           dict(pv_scheme=2)]


def _run(level, bs, ept, **kw):
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(level)
    gd, u, ghs = cases.jet_bumps(m, seed=3)
    nt = kw.get("n_tracers", 0)
    g = TMCoreGPU(m, dt=200.0, block_size=bs, elements_per_thread=ept, **kw)
    g.set_initial(gd, u, ghs)
    if nt:
        g.set_tracers(cases.smooth_tracers(m, nt, seed=4) * gd)
    out = [g.diag()]
    g.step(3)
    out += [*g.get_state(), g.get_tracers() if nt else np.zeros(1), g.diag()]
    g.close()
    return out


@pytest.mark.parametrize("level", [1, 4, 6])
@pytest.mark.parametrize("kw", OPTIONS)
def test_fp32_bit_identical(level, kw):
    want = _run(level, 256, 4, precision=abi.TMC_FP32, **kw)
    for bs in (0, 32, 224, 512):
        for a, b in zip(_run(level, bs, 1, precision=abi.TMC_FP32, **kw), want):
            assert np.array_equal(a, b), bs


@pytest.mark.parametrize("kw", OPTIONS)
def test_fp64_agree(kw):
    """Beta's and the invariants' sums are ordered differently: 1e-13, as for
    the block sizes."""
    want = _run(4, 256, 4, precision=abi.TMC_FP64, **kw)
    for bs in (0, 224):
        for a, b in zip(_run(4, bs, 1, precision=abi.TMC_FP64, **kw), want):
            assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))
