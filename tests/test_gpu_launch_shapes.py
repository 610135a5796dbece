"""The launch shapes of the fused step (elements per thread, block size) do
not change what an element computes: a small mesh, which runs one element per
thread, stepped with explicit block sizes (other grids, other partial sums)
against the default shapes.  Only beta's sums are ordered differently: their
relative difference is below the block partials' 2^-20 in FP32 and 2^-50 in
FP64, and beta enters as beta dt t_new, so h and iap_u agree to that times
the change of the state, and far closer than 1e-6 / 1e-13 of its size."""
import numpy as np
import pytest

from tmcore_gb300 import abi, cases, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [1, 4, 6])
@pytest.mark.parametrize("precision,tol", [(abi.TMC_FP64, 1e-13), (abi.TMC_FP32, 1e-6)])
@pytest.mark.parametrize("tracers,pv", [(0, dict(pv_scheme=3, interp_pv_order=3)), (3, dict(pv_scheme=1, apvm_weight=0.0)),
                                        (4, dict(pv_scheme=1, apvm_weight=0.0))])
def test_block_sizes_agree(level, precision, tol, tracers, pv):
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(level)
    gd, u, ghs = cases.jet_bumps(m, seed=3)
    q = cases.smooth_tracers(m, tracers, seed=4) if tracers else None
    out = []
    for bs in (0, 32, 224, 512):
        g = TMCoreGPU(m, dt=200.0, precision=precision, n_tracers=tracers, block_size=bs, **pv)
        g.set_initial(gd, u, ghs)
        if tracers:
            g.set_tracers(q * gd)
        g.step(2)
        out.append((*g.get_state()[:2], g.get_tracers() if tracers else np.zeros(1), g.diag()[:1]))
        g.close()
    for other in out[1:]:
        for a, b in zip(other, out[0]):
            assert np.max(np.abs(a - b)) <= tol * np.max(np.abs(b))
