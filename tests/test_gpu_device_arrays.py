"""State transfers with device arrays, in place or through the handle's own
arrays (an array not aligned for doubles), against the same calls with host
arrays: bit-identical, for a single model, both precisions, and a member of
either ensemble layout."""
import numpy as np
import pytest

from tmcore_gb300 import abi, cases, mesh

pytestmark = pytest.mark.gpu


def _device(torch, a, offset):
    """The array's bytes on the device, `offset` bytes into an allocation."""
    raw = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda")
    raw[offset:offset + a.nbytes] = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
    return raw


def _host(raw, like, offset):
    return raw[offset:offset + like.nbytes].cpu().numpy().view(np.float64).reshape(like.shape)


@pytest.mark.parametrize("offset", [0, 4, 8])
@pytest.mark.parametrize("kw", [dict(precision=abi.TMC_FP64, n_tracers=2), dict(precision=abi.TMC_FP32, n_tracers=3),
                                dict(precision=abi.TMC_FP32, members=16, member_layout=1),
                                dict(precision=abi.TMC_FP32, members=3)])
def test_device_arrays_match_host_arrays(offset, kw):
    torch = pytest.importorskip("torch")
    from tmcore_gb300.gpu import TMCoreGPU

    m = mesh.icos_mesh(3)
    gd, u, ghs = cases.jet_bumps(m, seed=9)
    g = TMCoreGPU(m, dt=600.0, pv_scheme=1, apvm_weight=0.0, **kw)
    if kw.get("members", 1) > 1:
        for k in range(kw["members"]):
            g.select_member(k)
            g.set_initial(gd, u, ghs)
        g.select_member(kw["members"] - 1)
    g.set_initial(gd, u, ghs)
    nt = kw.get("n_tracers", 0)
    q = cases.smooth_tracers(m, nt, seed=1) * gd if nt else None
    gd1, iap1, _ = g.get_state()
    results = []
    for device in (False, True):
        put = (lambda a: _device(torch, a, offset)) if device else (lambda a: a.copy())
        ptr = (lambda a: a.data_ptr() + offset) if device else (lambda a: a.ctypes.data)
        get = (lambda a, like: _host(a, like, offset)) if device else (lambda a, like: a.copy())
        call = lambda name, *a: g._chk(getattr(g.lib, name)(g.h, *a))  # noqa: E731
        a, b = put(gd1 * 1.001), put(iap1 * 0.999)
        og, oi, ou = put(np.zeros_like(gd1)), put(np.zeros_like(iap1)), put(np.zeros_like(iap1))
        torch.cuda.synchronize()
        call("tmc_set_state", ptr(a), ptr(b))
        res = []
        if nt:
            c, oq = put(q), put(np.zeros_like(q))
            torch.cuda.synchronize()
            call("tmc_set_tracers", ptr(c))
        g.step(2)
        call("tmc_get_state", ptr(og), ptr(oi), ptr(ou))
        res += [get(og, gd1), get(oi, iap1), get(ou, iap1)]
        if nt:
            call("tmc_get_tracers", ptr(oq))
            res.append(get(oq, q))
        if kw.get("members", 1) == 1:
            call("tmc_spatial_operators", ptr(a), ptr(b), ptr(og), ptr(oi))
            res += [get(og, gd1), get(oi, iap1)]
            call("tmc_spatial_operators", ptr(a), ptr(b), ptr(a), ptr(b))  # outputs over the inputs
            res += [get(a, gd1), get(b, iap1)]
        results.append(res)
    for x, y in zip(*results):
        assert np.array_equal(x, y) and np.all(np.isfinite(x))
    g.close()
