"""The workloads whose speed is measured: shallow-water runs, ensembles, the
learned closure and its training, each through the package's public entry
points (the C ABI and its Python mirror).

A model run is what a host program does between two outputs: it hands the
library a state, advances it a number of steps and reads the state back, all
arrays on the device.  An ensemble or a batch of mesh levels is stepped on and
read back, member by member.  ``exact`` integrates the same equations in 64
bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tmcore_gb300 import abi
from tmcore_gb300.gpu import ClosureMLP, TMCoreGPU, TMCoreGroup
from tmcore_gb300.mesh import icos_mesh

RADIUS, GRAV, OMEGA = 6371220.0, 9.80616, 7.292e-5
F64 = torch.float64


def listed():
    return [
        # one tendency evaluation of the drop-in operator interface on a small mesh: latency of a single call
        {"name": "operators_l5_fp64", "kind": "operators", "level": 5, "fp64": True, "upwind": True},
        # the parity configuration (level 5, centred pv, dt 600 s), eight hours between outputs: launches dominate
        {"name": "run_l5_fp64", "kind": "run", "level": 5, "fp64": True, "upwind": False, "tracers": 0, "steps": 48},
        # the shipped namelist (level 6, upwind pv, dt 240 s), two hours between outputs, in both precisions
        {"name": "run_l6_fp64_upwind", "kind": "run", "level": 6, "fp64": True, "upwind": True, "tracers": 0, "steps": 30},
        {"name": "run_l6_fp32_upwind", "kind": "run", "level": 6, "fp64": False, "upwind": True, "tracers": 0, "steps": 30},
        # a high-resolution FP64 run with transported tracers (the closure's truth runs use this level)
        {"name": "run_l8_fp64_tracers", "kind": "run", "level": 8, "fp64": True, "upwind": False, "tracers": 4, "steps": 4},
        # the 2.6-million-cell configuration with four tracers, FP32 state
        {"name": "run_l9_fp32_tracers", "kind": "run", "level": 9, "fp64": False, "upwind": False, "tracers": 4, "steps": 8},
        # the drop-in time_integrate: a host model's page-locked arrays in and out every step
        {"name": "host_l8_fp32_tracers", "kind": "host", "level": 8, "fp64": False, "upwind": False, "tracers": 4},
        # 512 seeded members stepped together for an hour and a half and all read back
        {"name": "ensemble_512_l6", "kind": "ensemble", "level": 6, "members": 512, "upwind": False, "steps": 24},
        # the learned closure in every stage of a 256-member ensemble
        {"name": "closure_256_l6", "kind": "closure", "level": 6, "members": 256, "every_stage": True, "steps": 4},
        # a mixed batch of mesh levels 4-7, each with its own time step, two 1200-s cycles
        {"name": "mixed_l4_l7", "kind": "mixed", "bottom": 4, "top": 7, "members": 16, "cycles": 2},
        # training the closure network: Adam on batches of 65536 edges
        {"name": "train_65536", "kind": "train", "batch": 65536, "steps": 64},
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    kind = rng.choice(["operators", "run", "run", "run", "run", "host", "ensemble", "ensemble", "closure", "mixed", "train"])
    if kind == "operators":
        return {"kind": kind, "level": rng.randint(4, 7), "fp64": rng.random() < 0.7, "upwind": rng.random() < 0.5}
    if kind == "run":
        fp64 = rng.random() < 0.5
        level = rng.randint(4, 8 if fp64 else 9)
        upwind = rng.random() < 0.5 and level < 8
        top = {4: 60, 5: 60, 6: 40, 7: 24, 8: 6, 9: 6}[level]
        return {"kind": kind, "level": level, "fp64": fp64, "upwind": upwind, "tracers": rng.randint(0, 4),
                "steps": rng.randint(max(1, top // 4), top)}
    if kind == "host":
        fp64 = rng.random() < 0.4
        return {"kind": kind, "level": rng.randint(5, 8), "fp64": fp64, "upwind": False, "tracers": rng.randint(0, 4)}
    if kind == "ensemble":
        level = rng.randint(4, 6)
        members = 16 * int(round(2 ** rng.uniform(0.0, 5.0)))
        return {"kind": kind, "level": level, "members": members, "upwind": rng.random() < 0.5, "steps": rng.randint(6, 24)}
    if kind == "closure":
        level = rng.randint(4, 6)
        return {"kind": kind, "level": level, "members": 16 * int(round(2 ** rng.uniform(0.0, 4.0))),
                "every_stage": rng.random() < 0.7, "steps": rng.randint(2, 6)}
    if kind == "mixed":
        return {"kind": kind, "bottom": rng.randint(4, 5), "top": rng.randint(5, 7), "members": 16 * rng.randint(1, 3),
                "cycles": rng.randint(1, 4)}
    return {"kind": kind, "batch": 128 * int(round(2 ** rng.uniform(4.0, 9.5))), "steps": rng.randint(16, 96)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dt(level):
    return {5: 600.0, 6: 240.0, 9: 45.0}.get(level, 1200.0 / 2 ** (level - 4))


def _dev(a, dtype=F64):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


_GEOMETRY: dict = {}


def _geometry(level):
    """Positions and metrics the initial states need, on the device."""
    if level not in _GEOMETRY:
        m = icos_mesh(level)
        _GEOMETRY[level] = {
            "xc": torch.stack([_dev(m.xCell), _dev(m.yCell), _dev(m.zCell)]), "zv": _dev(m.zVertex),
            "v1": _dev(m.verticesOnEdge[:, 0] - 1, torch.int64), "v2": _dev(m.verticesOnEdge[:, 1] - 1, torch.int64),
            "c1": _dev(m.cellsOnEdge[:, 0] - 1, torch.int64), "c2": _dev(m.cellsOnEdge[:, 1] - 1, torch.int64),
            "dv": _dev(m.dvEdge) * RADIUS}
    return _GEOMETRY[level]


def _random(seed, *shape):
    gen = torch.Generator().manual_seed(seed)
    return torch.rand(*shape, generator=gen, dtype=F64)


def _smooth(xc, modes, low, high, seed):
    """A smooth field on the sphere: `modes` plane waves of wavenumbers low..high."""
    r = _random(seed, modes, 6)
    f = torch.zeros_like(xc[0])
    for a, b, c, n, p, w in r.tolist():
        k = torch.tensor([a - 0.5, b - 0.5, c - 0.5], dtype=F64)
        k = (k / k.norm() * (low + n * (high - low))).tolist()
        f += (0.5 + w) * torch.cos(k[0] * xc[0] + k[1] * xc[1] + k[2] * xc[2] + 2.0 * math.pi * p)
    return f


def _initial(level, seed):
    """A seeded zonal jet with a 1% depth perturbation over eight Gaussian mountains: gd, u, iap_u, ghs."""
    G = _geometry(level)
    xc, h0 = G["xc"], 5000.0
    r = _random(seed, 8, 5).tolist()
    u0 = 10.0 + 30.0 * r[0][4]
    ghs = torch.zeros_like(xc[0])
    for a, b, hh, w, _ in r:
        z, lon = 2.0 * a - 1.0, 2.0 * math.pi * b
        s = math.sqrt(1.0 - z * z)
        d = RADIUS * torch.acos((s * math.cos(lon) * xc[0] + s * math.sin(lon) * xc[1] + z * xc[2]).clamp(-1.0, 1.0))
        ghs += GRAV * (500.0 + 1500.0 * hh) * torch.exp(-((d / (500e3 + 1000e3 * w)) ** 2))
    ghs *= torch.clamp(0.6 * GRAV * h0 / ghs.max(), max=1.0)
    pert = _smooth(xc, 12, 4.0, 16.0, seed + 1)
    gd = GRAV * h0 - (RADIUS * OMEGA * u0 + 0.5 * u0 * u0) * xc[2] ** 2 - ghs + GRAV * 0.01 * h0 * pert / pert.abs().max()
    psi = -RADIUS * u0 * G["zv"]
    u = -(psi[G["v2"]] - psi[G["v1"]]) / G["dv"]
    iap = torch.sqrt(0.5 * (gd[G["c1"]] + gd[G["c2"]])) * u
    return gd, u, iap, ghs


def _tracers(level, n, seed):
    """n smooth mixing ratios in [0, 1]."""
    xc = _geometry(level)["xc"]
    q = torch.empty(n, xc.shape[1], dtype=F64, device="cuda")
    for k in range(n):
        f = _smooth(xc, 6, 1.0, 8.0, 1000 * seed + k)
        q[k] = (f - f.min()) / (f.max() - f.min())
    return q


def _model(case, level, dt, **kw):
    pv = dict(pv_scheme=3, interp_pv_order=3) if case.get("upwind") else dict(pv_scheme=1, apvm_weight=0.0)
    return TMCoreGPU(icos_mesh(level), dt=dt, precision=abi.TMC_FP64 if case.get("fp64") else abi.TMC_FP32, **pv, **kw)


def _call(model, name, *args):
    """An entry point of the C ABI with device tensors in place of host arrays."""
    rc = getattr(model.lib, name)(model.h, *[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args])
    if rc != 0:
        raise RuntimeError(f"{name}: {model.lib.tmc_last_error(model.h).decode()}")


def _member_seed(seed, m):
    return 100003 * seed + 17 * m


def _fill_members(model, level, members, seed):
    for m in range(members):
        gd, u, _, ghs = _initial(level, _member_seed(seed, m))
        torch.cuda.current_stream().synchronize()
        model.select_member(m)
        _call(model, "tmc_set_initial", gd, u, ghs)


def _read_members(model, members):
    gd = torch.empty(members, model.nc, dtype=F64, device="cuda")
    iap = torch.empty(members, model.ne, dtype=F64, device="cuda")
    for m in range(members):
        model.select_member(m)
        _call(model, "tmc_get_state", gd[m], iap[m], None)
    return {"gd": gd, "iap": iap}


# the closure network: 24 inputs normalised by typical values of its features, the APVM head
_X_MEAN = [0, 0, 4.6e4, 0, 0, 0, 0, 0, 4.6e4, 4.6e4, 4.9e4, 4.9e4, 2e3, 2e3, 0, 0, 7e4, 1.2e5, 0, 0, 0, 0, 0, 0]
_X_STD = [15, 15, 4e3, 2e-9, 2e-9, 2e-9, 2e-9, 2e-9, 4e3, 4e3, 1e3, 1e3, 4e3, 4e3, 1e-4, 1e-4, 1e4, 1e4, 15, 15, 15, 15, 2e-15, 2e-15]
_LAYERS = [(64, 24), (64, 64), (64, 64), (1, 64)]


def _weights(seed):
    """Network parameters in the library's order, uniform in +-1/sqrt(fan-in)."""
    r = np.random.default_rng(seed)
    parts = []
    for n, k in _LAYERS:
        parts += [r.uniform(-1, 1, n * k) / math.sqrt(k), r.uniform(-1, 1, n) / math.sqrt(k)]
    return np.concatenate(parts).astype(np.float32)


def _train_data(case, seed):
    """A dataset of as many rows as the run of steps reads: features and a smooth target with noise."""
    rows = case["batch"] * min(case["steps"], 16)
    r = np.random.default_rng(seed)
    x = r.standard_normal((rows, 24), dtype=np.float32)
    y = (0.3 * np.tanh(x[:, 0] * x[:, 1]) + 0.1 * x[:, 2] + 0.02 * r.standard_normal(rows, dtype=np.float32)).astype(np.float32)
    return x, y


def _mixed_levels(case):
    return range(case["bottom"], case["top"] + 1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        net = ClosureMLP(seed=1)
        net.set_scaling(np.zeros(24), np.ones(24), 1.0)
        net.set_dataset(*_train_data(case, seed))
        return {"case": case, "net": net, "params": _weights(seed)}
    if kind == "mixed":
        models = []
        for level in _mixed_levels(case):
            m = _model(case, level, 1200.0 / 2 ** (level - 4), members=case["members"], member_layout=1)
            _fill_members(m, level, case["members"], seed)
            models.append(m)
        return {"case": case, "models": models, "group": TMCoreGroup(models, cycle_seconds=1200.0)}
    level = case["level"]
    if kind in ("ensemble", "closure"):
        m = _model(case, level, 1200.0 / 2 ** (level - 4), members=case["members"], member_layout=1)
        _fill_members(m, level, case["members"], seed)
        state = {"case": case, "model": m}
        if kind == "closure":
            net = ClosureMLP(seed=1)
            net.params = _weights(seed)
            net.set_scaling(np.array(_X_MEAN), 1.0 / np.array(_X_STD), 1.0)
            net.set_head(1, 1200.0 / 2 ** (level - 4))
            m.set_closure_stages(case["every_stage"])
            m.set_closure(net)
            state["net"] = net
        return state
    gd, u, iap, ghs = _initial(level, seed)
    nt = case.get("tracers", 0)
    m = _model(case, level, _dt(level), n_tracers=nt)
    torch.cuda.current_stream().synchronize()
    _call(m, "tmc_set_initial", gd, u, ghs)
    state = {"case": case, "model": m, "gd": gd, "iap": iap}
    if nt:
        state["qgd"] = _tracers(level, nt, seed) * gd
    if kind == "host":
        for k in ("gd", "iap", "qgd"):
            if k in state:
                state[k] = state[k].cpu().pin_memory()
                state[k + "_new"] = torch.empty_like(state[k]).pin_memory()
    return state


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        net = s["net"]
        net.params = s["params"]  # also restarts Adam
        losses = net.train(case["steps"], batch=case["batch"], lr=1e-3)
        return {"params": net.params, "losses": losses}
    if kind == "mixed":
        s["group"].run(case["cycles"])
        s["group"].synchronize()
        return [_read_members(m, case["members"]) for m in s["models"]]
    model = s["model"]
    if kind in ("ensemble", "closure"):
        model.step(case["steps"])
        return _read_members(model, case["members"])
    if kind == "host":
        out = [s["gd_new"], s["iap_new"], s.get("qgd_new")]
        _call(model, "tmc_time_integrate", s["gd"], s["iap"], s.get("qgd"), *out)
        return {k: v for k, v in zip(("gd", "iap", "qgd"), out) if v is not None}
    gd, iap = torch.empty_like(s["gd"]), torch.empty_like(s["iap"])
    if kind == "operators":
        _call(model, "tmc_spatial_operators", s["gd"], s["iap"], gd, iap)
        return {"tend_gd": gd, "tend_iap": iap}
    _call(model, "tmc_set_state", s["gd"], s["iap"])
    if "qgd" in s:
        _call(model, "tmc_set_tracers", s["qgd"])
    model.step(case["steps"])
    _call(model, "tmc_get_state", gd, iap, None)
    out = {"gd": gd, "iap": iap}
    if "qgd" in s:
        out["qgd"] = torch.empty_like(s["qgd"])
        _call(model, "tmc_get_tracers", out["qgd"])
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(level, size, tracers, members, upwind):
    """Bytes and operations of one CRK4 step: the state of every member read and written once, the mesh tables
    (connectivity, weights, metrics) read once; four tendency evaluations."""
    nc, ne, nv = 10 * 4 ** level + 2, 30 * 4 ** level, 20 * 4 ** level
    mesh = ne * (56 + 12 * size) + nc * (48 + 2 * size) + nv * (24 + 5 * size)
    if upwind:
        mesh += ne * 24 * (4 + size)
    state = nc * (8 + size * tracers) + ne * size
    ops = 4 * (ne * (75 + (100 if upwind else 0)) + nc * (45 + 40 * tracers) + nv * 15)
    return mesh + 2 * members * state, members * ops


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["batch"] * case["steps"]
        return {"bytes": rows * 100.0 + 12.0 * 9985 * case["steps"], "flops": 6.0 * rows * (24 * 64 + 2 * 64 * 64 + 64)}
    if kind == "mixed":
        b = f = 0.0
        for level in _mixed_levels(case):
            n = case["cycles"] * 2 ** (level - 4)
            x, y = _step_work(level, 4, 0, case["members"], False)
            b += n * x + case["members"] * 8.0 * 40 * 4 ** level
            f += n * y
        return {"bytes": b, "flops": f}
    level, size = case["level"], 8 if case.get("fp64") else 4
    tracers, members = case.get("tracers", 0), case.get("members", 1)
    steps = case.get("steps", 1)
    b, f = _step_work(level, size, tracers, members, case.get("upwind"))
    if kind == "operators":
        return {"bytes": b + 16.0 * 40 * 4 ** level, "flops": f / 4}
    io = 8.0 * members * 4 ** level * (40 + 10 * tracers)
    b, f = steps * b + io * (1 if members > 1 else 2), steps * f
    if kind == "closure":
        nets = 4 if case["every_stage"] else 1
        f += steps * nets * members * 30.0 * 4 ** level * 2 * (24 * 64 + 2 * 64 * 64 + 64)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
class _Exact:
    """CRK4 with the energy-conserving step of the TRiSK shallow-water equations on one mesh; fields are
    [elements, members]."""

    def __init__(self, level, upwind):
        m = icos_mesh(level)
        r, r2 = RADIUS, RADIUS * RADIUS
        idx = lambda a: _dev(np.maximum(a - 1, 0), torch.int64)  # noqa: E731
        self.nc = m.nCells
        self.c1, self.c2 = idx(m.cellsOnEdge[:, 0]), idx(m.cellsOnEdge[:, 1])
        self.v1, self.v2 = idx(m.verticesOnEdge[:, 0]), idx(m.verticesOnEdge[:, 1])
        self.eoc, self.eov, self.cov, self.eoe = (idx(m.edgesOnCell), idx(m.edgesOnVertex), idx(m.cellsOnVertex),
                                                  idx(m.edgesOnEdge))
        col = lambda a: _dev(a)[:, None]  # noqa: E731
        self.dv, self.dc = col(m.dvEdge) * r, col(m.dcEdge) * r
        self.ae, self.ac, self.at = self.dv * self.dc, col(m.areaCell) * r2, col(m.areaTriangle) * r2
        self.kite, self.f = _dev(m.kiteAreasOnVertex) * r2, 2.0 * OMEGA * torch.sin(col(m.latVertex))
        there = _dev(np.arange(m.maxEdges)[None, :] < m.nEdgesOnCell[:, None])
        here = torch.arange(m.nCells, device="cuda")[:, None]
        self.ns = there * torch.where(self.c1[self.eoc] == here, 1.0, -1.0)
        here = torch.arange(m.nVertices, device="cuda")[:, None]
        self.ts = torch.where(self.v1[self.eov] == here, 1.0, -1.0).to(F64)
        self.w = _dev(m.weightsOnEdge) * _dev(np.arange(m.maxEdges2)[None, :] < m.nEdgesOnEdge[:, None])
        self.up = self._fit(m) if upwind else None

    def _fit(self, m):
        """Second derivatives along each edge at its two vertices from quadratic least-squares fits over the
        vertices of the three cells around (and the three neighbours): per side (points [ne, k], weights)."""
        x = torch.stack([_dev(m.xVertex), _dev(m.yVertex), _dev(m.zVertex)], 1)
        x = x / x.norm(dim=1, keepdim=True)
        voc = _dev(m.verticesOnCell, torch.int64) - 1
        voc = torch.where(torch.arange(m.maxEdges, device="cuda")[None, :] < _dev(m.nEdgesOnCell, torch.int64)[:, None], voc, voc[:, :1])
        near = torch.cat([torch.where(self.v1[self.eov] == torch.arange(m.nVertices, device="cuda")[:, None],
                                      self.v2[self.eov], self.v1[self.eov]), voc[self.cov].flatten(1)], 1).sort(1).values
        own = torch.arange(m.nVertices, device="cuda")[:, None]
        drop = (near == own) | torch.cat([torch.zeros_like(own, dtype=torch.bool), near[:, 1:] == near[:, :-1]], 1)
        near = torch.where(drop, -1, near).sort(1, descending=True).values
        near = near[:, : int((near >= 0).sum(1).max())]
        out = []
        for a, b in ((self.v1, self.v2), (self.v2, self.v1)):
            pts = near[a]
            there = pts >= 0
            pts = torch.where(there, pts, a[:, None])
            o, p = x[a], x[pts]
            ex = x[b] - (x[b] * o).sum(1, keepdim=True) * o
            ex = ex / ex.norm(dim=1, keepdim=True)
            ey = torch.linalg.cross(o, ex)
            c = torch.einsum("ek,ejk->ej", o, p)
            px, py = torch.einsum("ek,ejk->ej", ex, p), torch.einsum("ek,ejk->ej", ey, p)
            s = torch.sqrt(px * px + py * py)
            d = torch.where(there, torch.atan2(s, c) / s.clamp(min=1e-300), torch.zeros_like(s))
            scale = self.dv[:, 0] / RADIUS
            px, py = px * d / scale[:, None], py * d / scale[:, None]
            P = torch.stack([px, py, px * px, px * py, py * py], 2)
            B = torch.linalg.solve(P.transpose(1, 2) @ P, P.transpose(1, 2))
            out.append((pts, 2.0 * B[:, 2, :] / (scale[:, None] * RADIUS) ** 2 * there))
        return out

    def tend(self, gd, iap, ghs, q=None, closure=None):
        """Tendencies of gd, iap_u and the tracer masses; closure(self, fields) corrects pv on edges."""
        ge = 0.5 * (gd[self.c1] + gd[self.c2])
        sq = torch.sqrt(ge)
        u = iap / sq
        F = u * ge
        E, tg = gd + ghs, torch.zeros_like(gd)
        tq = None if q is None else [torch.zeros_like(gd) for _ in q]
        qe = None if q is None else [0.5 * (x[self.c1] / gd[self.c1] + x[self.c2] / gd[self.c2]) for x in q]
        for i in range(self.eoc.shape[1]):
            e, n = self.eoc[:, i], self.ns[:, i:i + 1]
            tg -= n * F[e] * self.dv[e] / self.ac
            E = E + n.abs() * 0.25 * u[e] ** 2 * self.ae[e] / self.ac
            for k in range(len(tq or ())):
                tq[k] -= n * (F * qe[k])[e] * self.dv[e] / self.ac
        gv, vo = 0.0, 0.0
        for i in range(3):
            e = self.eov[:, i]
            gv = gv + gd[self.cov[:, i]] * self.kite[:, i:i + 1] / self.at
            vo = vo - self.ts[:, i:i + 1] * u[e] * self.dc[e] / self.at
        pv = (self.f + vo) / gv
        p1, p2 = pv[self.v1], pv[self.v2]
        pe = 0.5 * (p1 + p2)
        if self.up is not None or closure is not None:
            ve = torch.zeros_like(u)
            for i in range(self.eoe.shape[1]):
                ve += self.w[:, i:i + 1] * u[self.eoe[:, i]]
        if self.up is not None:
            d = []
            for (pts, w), ctr in zip(self.up, (p1, p2)):
                acc = torch.zeros_like(pe)
                for j in range(pts.shape[1]):
                    acc += w[:, j:j + 1] * (pv[pts[:, j]] - ctr)
                d.append(acc)
            pe = pe - self.dv ** 2 * ((d[0] + d[1]) - torch.copysign(torch.ones_like(ve), ve) * (d[1] - d[0])) / 12.0
        if closure is not None:
            pe = pe + closure(self, gd, ghs, u, ve, ge, pe, pv, E)
        s = torch.zeros_like(u)
        for i in range(self.eoe.shape[1]):
            e = self.eoe[:, i]
            s += self.w[:, i:i + 1] * F[e] * 0.5 * (pe + pe[e])
        tu = sq * (s - (E[self.c2] - E[self.c1]) / self.dc) + 0.5 * u / sq * 0.5 * (tg[self.c1] + tg[self.c2])
        return tg, tu, tq

    def step(self, gd, iap, ghs, dt, q=None, closure=None):
        t, fac, g, i, x = [], (0.5, 0.5, 1.0), gd, iap, q
        for k in range(4):
            t.append(self.tend(g, i, ghs, x, closure[k] if closure else None))
            if k < 3:
                a = fac[k] * dt
                g, i = gd + a * t[k][0], iap + a * t[k][1]
                x = None if q is None else [y + a * z for y, z in zip(q, t[k][2])]
        mix = lambda a: (a[0] + 2.0 * a[1] + 2.0 * a[2] + a[3]) / 6.0  # noqa: E731
        ng, ni = mix([y[0] for y in t]), mix([y[1] for y in t])
        dot = lambda a, b: (a[0] * b[0] * self.ac).sum(0) + (a[1] * b[1] * self.ae).sum(0)  # noqa: E731
        r = dot(t[0], t[1]) + dot(t[1], t[2]) + dot(t[2], t[3])
        beta = r / (3.0 * dot((ng, ni), (ng, ni)))
        if q is not None:
            q = [y + beta * dt * mix([z[2][k] for z in t]) for k, y in enumerate(q)]
        return gd + beta * dt * ng, iap + beta * dt * ni, q


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _network(p, x):
    o = 0
    for k, (n, m) in enumerate(_LAYERS):
        w, b = p[o:o + n * m].reshape(n, m), p[o + n * m:o + n * m + n]
        o += n * m + n
        x = x @ w.T + b
        if k < 3:
            x = _gelu(x)
    return x[..., 0]


def _closure_fn(p, dt, hold):
    """The APVM-head correction of pv on edges; with `hold` it is computed once and kept."""
    mean, std = torch.tensor(_X_MEAN, dtype=F64, device="cuda"), torch.tensor(_X_STD, dtype=F64, device="cuda")
    kept = []

    def correct(X, gd, ghs, u, ve, ge, pe, pv, E):
        if kept:
            return kept[0]
        pc = torch.zeros_like(gd)
        for i in range(3):
            pc.index_add_(0, X.cov[:, i], pv * X.kite[:, i:i + 1])
        pc = pc / X.ac
        out = torch.empty_like(u)
        p1, p2, q1, q2 = pv[X.v1], pv[X.v2], pc[X.c1], pc[X.c2]
        g1, g2 = (p2 - p1) / X.dv, (q2 - q1) / X.dc
        wide = lambda a: a.expand(-1, 1)  # noqa: E731
        for m in range(u.shape[1]):
            c = slice(m, m + 1)
            cols = [u[:, c], ve[:, c], ge[:, c], pe[:, c], p1[:, c], p2[:, c], q1[:, c], q2[:, c], gd[X.c1, c], gd[X.c2, c],
                    E[X.c1, c], E[X.c2, c], ghs[X.c1, c], ghs[X.c2, c], wide(X.f[X.v1]), wide(X.f[X.v2]), X.dv, X.dc]
            cols += [u[X.eoe[:, i], c] for i in range(4)] + [g1[:, c], g2[:, c]]
            y = _network(p, (torch.cat(cols, 1) - mean) / std)
            out[:, m] = -torch.nn.functional.softplus(y) * dt * (ve[:, m] * g1[:, m] + u[:, m] * g2[:, m])
        if hold:
            kept.append(out)
        return out

    return correct


def _exact_members(level, members, seed, steps, dt, upwind=False, params=None, every_stage=True):
    X = _Exact(level, upwind)
    parts = []
    for m0 in range(0, members, 64):
        ic = [_initial(level, _member_seed(seed, m)) for m in range(m0, min(members, m0 + 64))]
        gd, iap, ghs = (torch.stack([s[k] for s in ic], 1) for k in (0, 2, 3))
        for _ in range(steps):
            closure = None
            if params is not None:
                fn = _closure_fn(params, dt, not every_stage)
                closure = [fn] * 4
            gd, iap, _ = X.step(gd, iap, ghs, dt, closure=closure)
        parts.append((gd.T.contiguous(), iap.T.contiguous()))
    return {"gd": torch.cat([p[0] for p in parts]), "iap": torch.cat([p[1] for p in parts])}


def _exact_train(case, seed):
    x, y = _train_data(case, seed)
    x, y = _dev(x), _dev(y)
    p = _dev(_weights(seed)).requires_grad_(True)
    m, v, losses, at = torch.zeros_like(p), torch.zeros_like(p), [], 0
    for t in range(1, case["steps"] + 1):
        rows = slice(at, at + case["batch"])
        loss = ((_network(p, x[rows]) - y[rows]) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        step = 1e-3 * (m / (1.0 - 0.9 ** t)) / (torch.sqrt(v / (1.0 - 0.999 ** t)) + 1e-8)
        p = (p.detach() - step).requires_grad_(True)
        at = (at + case["batch"]) % len(y)
    return {"params": p.detach(), "losses": np.array(losses)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "mixed":
        return [_exact_members(level, case["members"], seed, case["cycles"] * 2 ** (level - 4), 1200.0 / 2 ** (level - 4))
                for level in _mixed_levels(case)]
    level = case["level"]
    if kind in ("ensemble", "closure"):
        params = _dev(_weights(seed)) if kind == "closure" else None
        return _exact_members(level, case["members"], seed, case["steps"], 1200.0 / 2 ** (level - 4), case.get("upwind"),
                              params, case.get("every_stage", True))
    X = _Exact(level, case["upwind"])
    gd, _, iap, ghs = (a[:, None] for a in _initial(level, seed))
    if kind == "operators":
        tg, tu, _ = X.tend(gd, iap, ghs)
        return {"tend_gd": tg[:, 0], "tend_iap": tu[:, 0]}
    nt = case.get("tracers", 0)
    q = [x[:, None] * gd for x in _tracers(level, nt, seed)] if nt else None
    for _ in range(case.get("steps", 1)):
        gd, iap, q = X.step(gd, iap, ghs, _dt(level), q)
    out = {"gd": gd[:, 0], "iap": iap[:, 0]}
    if nt:
        out["qgd"] = torch.stack([x[:, 0] for x in q])
    return out
