"""Small FP32 models run a step as one chain of dependent launches with the
cell and the vertex pass of a stage in one: what the timing calls report is
that program, and no block size takes a model off it."""
import numpy as np
import pytest

from tmcore_gb300 import abi, cases, mesh

pytestmark = pytest.mark.gpu

CENTRED = dict(pv_scheme=1, apvm_weight=0.0)
UPWIND = dict(pv_scheme=3, interp_pv_order=3)


def _model(level=4, precision=abi.TMC_FP32, **kw):
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(level)
    g = TMCoreGPU(m, dt=60.0, precision=precision, **kw)
    g.set_initial(*cases.jet_bumps(m, seed=1))
    return g


def _launches(g):
    return g.time_steps(1, total=True, flux=False)[3]


@pytest.mark.parametrize("kw,chained,separate", [(CENTRED, 15, 19), (UPWIND, 19, 23),
                                                 (dict(pv_scheme=1, apvm_weight=0.5), 19, 23)])
def test_launch_count(kw, chained, separate):
    """Per stage cell + vertex (one launch in a chain), pv on edges (one, or
    two with the vertex fits or with pv on cells) and flux; then the sums and
    the two final updates."""
    for precision, want in ((abi.TMC_FP32, chained), (abi.TMC_FP64, separate)):
        g = _model(precision=precision, **kw)
        assert _launches(g) == want
        g.close()


@pytest.mark.parametrize("block_size", [32, 224, 256, 288, 512])
def test_block_sizes_keep_the_chain(block_size):
    """The FP32 cell pass takes at most 256 threads per block, the others 512."""
    g = _model(block_size=block_size, **CENTRED)
    assert _launches(g) == 15
    g.close()


@pytest.mark.parametrize("kw", [CENTRED, UPWIND])
def test_pass_times_are_the_chain_s(kw):
    """The merged launch is the cell pass's time; the timed steps give the
    chain's states and invariants bit for bit."""
    g, ref = _model(**kw), _model(**kw)
    t = g.pass_times(3)
    assert t["vertex"] == 0.0 and all(t[k] > 0.0 for k in ("cell", "edge_pv", "edge_flux", "final"))
    ms, flux, n, _ = g.time_steps(2, total=False, flux=True)
    assert flux > 0.0 and n == 8
    ref.step(5 * 3 + 2)
    for a, b in zip(g.get_state() + (g.diag(),), ref.get_state() + (ref.diag(),)):
        assert np.array_equal(a, b)
    g.close()
    ref.close()


@pytest.mark.parametrize("level,kw", [(5, CENTRED), (5, UPWIND), (6, CENTRED)])
def test_autotune_keeps_the_chain(level, kw):
    """Tuning times the program that runs: it keeps the chain, the state and
    the results, and does not make the step slower (measured: 30.8 us to 40.6
    when the passes were tuned one by one; 15% allows for the clock)."""
    g, ref = _model(level, diag_every=0, **kw), _model(level, diag_every=0, **kw)

    def us(x):
        x.step(20)
        return min(x.time_steps(100, total=True, flux=False)[0] for _ in range(5)) * 10.0

    launches, before, state = _launches(g), us(g), g.get_state()
    sizes = g.autotune(3)
    assert sizes["cell"] == sizes["vertex"] <= 256
    assert all(np.array_equal(a, b) for a, b in zip(g.get_state(), state))
    assert _launches(g) == launches and us(g) <= 1.15 * before
    ref.step(1 + 520 + 1 + 520)
    for a, b in zip(g.get_state() + (g.diag(),), ref.get_state() + (ref.diag(),)):
        assert np.array_equal(a, b)
    g.close()
    ref.close()
