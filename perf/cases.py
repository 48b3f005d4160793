"""The framework's work, as measured cases: what a user's program asks of it,
through the public entry points (``anuga_cuda.GPU_domain``, ``Ensemble``,
``Surrogate`` and the C ABI that they bind).

A case is a dict of plain values.  ``kind`` says which call a pass makes:

* ``step``      one ``GPU_domain.step()``: the smallest call of the evolve loop
* ``evolve``    ``GPU_domain.evolve_steps`` of ``steps`` steps, or the
                ``evolve`` generator over ``yields`` yield intervals
* ``methods``   one Euler step through the per-method entry points
* ``ensemble``  ``Ensemble.evolve`` of several harbours of different sizes,
                with tracking of maximum depth and arrival time
* ``predict``   ``swgpu_mlp_predict`` into a device buffer
* ``gradients`` ``Surrogate.gradients``: forward and backward on given rows
* ``train``     ``swgpu_mlp_train``: Adam steps on random batches

Meshes come from the package's own generators and are built once per process
(a program keeps its mesh); the state on them is made from the seed.
"""
import ctypes as C
import dataclasses
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "anuga-cuda_gb300"))

from anuga_cuda import DEFAULT, GPU_domain, _lib, scenarios  # noqa: E402
from anuga_cuda import surrogate as SG  # noqa: E402
from anuga_cuda.ensemble import Ensemble  # noqa: E402


def listed():
    return [
        # the smallest call: one step of a small basin, as a co-testing or
        # coupled program makes it
        {"name": "step_768_mixed", "kind": "step", "scene": "basin", "m": 16, "n": 12,
         "precision": "mixed", "method": "euler", "flow": 0},
        # the reference's own way of stepping, method by method (FP64)
        {"name": "methods_11k_fp64", "kind": "methods", "scene": "harbour", "m": 11000, "n": 0},
        # a small channel with an inflow hydrograph in the 'tsunami' flow
        # algorithm, two-stage Runge-Kutta
        {"name": "channel_2k_fp64_tsunami", "kind": "evolve", "scene": "channel", "m": 41, "n": 13,
         "precision": "fp64", "method": "rk2", "flow": 1, "steps": 60, "yields": 0},
        # the dam break on 100 x 100 cells in the default precision
        {"name": "dam_40k_fp64", "kind": "evolve", "scene": "dam", "m": 100, "n": 100,
         "precision": "fp64", "method": "euler", "flow": 0, "steps": 54, "yields": 0},
        # the tidal harbour: an irregular mesh of odd size, a run of 400 steps
        {"name": "harbour_45k_mixed", "kind": "evolve", "scene": "harbour", "m": 45000, "n": 0,
         "precision": "mixed", "method": "euler", "flow": 0, "steps": 400, "yields": 0},
        # a wet/dry beach read at yields, three-stage Runge-Kutta
        {"name": "beach_251k_mixed_rk3_yields", "kind": "evolve", "scene": "beach", "m": 251,
         "n": 249, "precision": "mixed", "method": "rk3", "flow": 0, "steps": 0, "yields": 4},
        # the wet/dry beach of a million triangles in the default precision
        {"name": "beach_1M_fp64", "kind": "evolve", "scene": "beach", "m": 500, "n": 500,
         "precision": "fp64", "method": "euler", "flow": 0, "steps": 24, "yields": 0},
        # the largest: the four-million-triangle beach, 200 steps
        {"name": "beach_4M_mixed", "kind": "evolve", "scene": "beach", "m": 1000, "n": 1000,
         "precision": "mixed", "method": "euler", "flow": 0, "steps": 200, "yields": 0},
        # harbours of 2k to 40k triangles side by side (the ensemble)
        {"name": "ensemble_8_mixed", "kind": "ensemble", "count": 8, "nmin": 2000, "nmax": 40000,
         "precision": "mixed", "steps": 200},
        # the surrogate: 16 scenarios of the family mesh into a device buffer
        {"name": "predict_16x200k", "kind": "predict", "cells": 224, "scen": 16, "row0": 0,
         "rows": 16 * 200704},
        # loss and gradients of a ragged set of rows
        {"name": "gradients_4099", "kind": "gradients", "cells": 64, "scen": 8, "rows": 4099},
        # Adam steps of the default batch
        {"name": "train_32k", "kind": "train", "cells": 64, "scen": 16, "batch": 32768,
         "steps": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "methods", "evolve", "evolve", "evolve", "evolve", "ensemble",
                       "predict", "gradients", "train"])
    if kind in ("step", "evolve", "methods"):
        precision = "fp64" if kind == "methods" else rng.choice(["fp64", "mixed"])
        top = 1000000 if precision == "mixed" else 300000
        if kind != "evolve":
            top = 100000
        scene = rng.choice(["basin", "dam", "harbour", "beach", "channel"])
        n_tri = _log_int(rng, 300, min(top, 60000) if scene == "harbour" else top)
        if scene == "harbour":
            m, n = max(n_tri, 1000), 0
        else:
            # rectangular_cross cells, four triangles each, of an odd aspect
            m = max(3, int(math.sqrt(n_tri / 4.0) * rng.uniform(0.7, 1.4)))
            n = max(3, int(round(n_tri / 4.0 / m)))
        case = {"kind": kind, "scene": scene, "m": m, "n": n}
        if kind == "methods":
            return case
        case["precision"] = precision
        case["method"] = rng.choice(["euler", "euler", "rk2", "rk3"])
        case["flow"] = rng.choice([0, 0, 0, 1]) if precision == "fp64" else 0
        if kind == "evolve":
            # about the same work whatever the size
            cost = 3.0e6 if precision == "fp64" else 3.0e7
            stages = {"euler": 1, "rk2": 2, "rk3": 3}[case["method"]]
            steps = int(min(400, max(4, cost / max(n_tri, 3000) / stages)))
            yields = rng.choice([0, 0, 0, 2])
            case["steps"], case["yields"] = (0 if yields else steps), yields
        return case
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(2, 8), "nmin": _log_int(rng, 600, 3000),
                "nmax": _log_int(rng, 3000, 30000), "precision": "mixed",
                "steps": rng.randint(20, 200)}
    cells = rng.randint(12, 120)
    scen = rng.randint(2, 8)
    total = 4 * cells * cells * scen
    if kind == "predict":
        rows = min(total, _log_int(rng, 1, total))
        return {"kind": kind, "cells": cells, "scen": scen, "row0": rng.randint(0, total - rows),
                "rows": rows}
    if kind == "gradients":
        return {"kind": kind, "cells": cells, "scen": scen,
                "rows": min(total, _log_int(rng, 1, 60000))}
    return {"kind": kind, "cells": cells, "scen": scen, "batch": _log_int(rng, 100, 65536),
            "steps": rng.randint(1, 8)}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _scene(scene, m, n):
    if scene == "basin":
        return scenarios.small_basin(m, n, seed=3)
    if scene == "dam":
        return scenarios.dam_break(m, n)
    if scene == "harbour":
        return scenarios.tidal_harbour(m, seed=2)
    if scene == "beach":
        return scenarios.wet_dry(m, n)
    if scene == "channel":
        return scenarios.channel_inflow(m, n, seed=2)
    raise ValueError(scene)


def _scenario(scene, m, n, seed):
    """The scene with a state of the seed: humps on the water surface, a flow
    where it is wet, friction per triangle in ANUGA's usual range."""
    base = _scene(scene, m, n)
    rng = np.random.default_rng(seed)
    c = np.asarray(base.mesh.centroid_coordinates).reshape(-1, 2)
    lo, hi = c.min(axis=0), c.max(axis=0)
    size = float((hi - lo).max())
    zc = base.elevation_vertex.mean(axis=1)
    depth = base.stage_centroid - zc
    top = max(float(depth.max()), 1.0e-3)
    hump = np.zeros(len(zc))
    for _ in range(3):
        x = lo + rng.random(2) * (hi - lo)
        r2 = ((c - x) ** 2).sum(axis=1)
        hump += 0.05 * top * rng.uniform(0.3, 1.0) * np.exp(-r2 / (2 * (0.08 * size) ** 2))
    w = np.maximum(zc, base.stage_centroid + np.where(depth > 0, hump, 0.0))
    h = w - zc
    ang = rng.uniform(0.0, 2.0 * np.pi)
    phase = 2.0 * np.pi * (c - lo) / size
    speed = 0.05 * np.sqrt(9.8 * h) * np.sin(phase[:, 0] + ang) * np.cos(phase[:, 1])
    return dataclasses.replace(base, stage_centroid=w, xmom_centroid=speed * h * np.cos(ang),
                               ymom_centroid=speed * h * np.sin(ang),
                               friction=rng.uniform(0.02, 0.04, len(zc)))


def _params(case):
    return DEFAULT.replace(flow_algorithm=case.get("flow", 0))


@functools.lru_cache(maxsize=None)
def _dt(scene, m, n):
    """A timestep of the scene's size (at rest): yield intervals are cut in it."""
    sc = _scene(scene, m, n)
    h = sc.stage_centroid - sc.elevation_vertex.mean(axis=1)
    return float(np.min(np.asarray(sc.mesh.radii) / np.sqrt(9.8 * np.maximum(h, 0.05))))


@functools.lru_cache(maxsize=None)
def _harbours(count, nmin, nmax):
    return scenarios.ensemble_harbours(count, seed=4, nmin=nmin, nmax=nmax)


def _ensemble(case, seed):
    out = []
    for i, sc in enumerate(_harbours(case["count"], case["nmin"], case["nmax"])):
        rng = np.random.default_rng([seed, i])
        zc = sc.elevation_vertex.mean(axis=1)
        wet = sc.stage_centroid > zc
        w = np.where(wet, np.maximum(zc, sc.stage_centroid + rng.uniform(-0.2, 0.2)
                                     + 0.02 * rng.standard_normal(len(zc))), zc)
        out.append(dataclasses.replace(
            sc, stage_centroid=w, friction=np.full(len(zc), rng.uniform(0.01, 0.05)),
            xmom_centroid=0.05 * rng.standard_normal(len(zc)) * (w - zc)))
    return out


@functools.lru_cache(maxsize=None)
def _family(cells):
    return SG.FamilyMesh(cells=cells)


def _surrogate_inputs(case, seed):
    fm = _family(case["cells"])
    th = SG.sample_params(case["scen"], seed)
    rng = np.random.default_rng(seed + 1)
    # targets of the form that the network learns: a depth excess that decays
    # from the inflow, an arrival time that grows with the distance to it
    d = fm.tri[None, :, 3] / 10000.0
    noise = rng.standard_normal((case["scen"], fm.N, 2)) * 0.05
    t = np.stack([th[:, :1] / 500.0 * np.exp(-3 * d), np.clip(d + 0.1 * th[:, 4:5], 0, 1.25)],
                 axis=2) + noise
    total = case["scen"] * fm.N
    rows = None
    if case["kind"] == "gradients":
        rows = rng.choice(total, case["rows"], replace=False).astype(np.int64)
    return fm, th, t.astype(np.float32), rows


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "evolve", "methods"):
        sc = _scenario(case["scene"], case["m"], case["n"], seed)
        d = GPU_domain(mesh=sc.mesh, parameters=_params(case),
                       precision=case.get("precision", "fp64"))
        sc.apply_to(d)
        d.set_timestepping_method(case.get("method", "euler"))
        if kind != "evolve":
            d.evolve_steps(0)  # the set-up half of evolve
        return case, d
    if kind == "ensemble":
        ens = Ensemble(_ensemble(case, seed), DEFAULT, case["precision"])
        ens.set_tracking(0.02)
        return case, ens
    fm, th, t, rows = _surrogate_inputs(case, seed)
    sg = SG.Surrogate(fm, seed=seed)
    if kind == "predict":
        sg.set_data(th)
        out = torch.empty((case["rows"], 3), dtype=torch.float32, device="cuda")
        return case, sg, out
    sg.set_data(th, t)
    return case, sg, rows, seed


def _conserved(d):
    w, uh, vh = d.get_conserved()
    return {"stage": w, "xmomentum": uh, "ymomentum": vh, "time": d.get_time()}


def run(state):
    case = state[0]
    kind = case["kind"]
    if kind == "step":
        d = state[1]
        d.step()
        return _conserved(d)
    if kind == "evolve":
        d = state[1]
        if case["yields"]:
            dy = 8 * _dt(case["scene"], case["m"], case["n"])
            seen = []
            for t in d.evolve(yieldstep=dy, finaltime=case["yields"] * dy):
                seen.append((t, d.get_water_volume()))
            return dict(_conserved(d), volumes=np.array([v for _, v in seen]))
        d.evolve_steps(case["steps"])
        return _conserved(d)
    if kind == "methods":
        d = state[1]
        d.evolve_one_euler_step(1.0e300, None)
        d.set_time(d.get_time() + d.timestep)
        d.distribute_to_vertices_and_edges()
        d.update_boundary()
        return dict(_conserved(d), stage_update=d.quantities["stage"].explicit_update,
                    stage_edges=d.quantities["stage"].edge_values, max_speed=d.max_speed)
    if kind == "ensemble":
        ens = state[1]
        ens.evolve(1.0e6, max_steps=case["steps"])
        tr = ens.get_tracking()
        return {"stage": ens.centroid_values("stage"), "xmomentum": ens.centroid_values("xmomentum"),
                "ymomentum": ens.centroid_values("ymomentum"), "max_depth": [a for a, _ in tr],
                "masses": ens.masses()}
    sg = state[1]
    if kind == "predict":
        out = state[2]
        sg._check(_lib.lib().swgpu_mlp_predict(sg._h, case["row0"], case["rows"],
                                               C.c_void_p(out.data_ptr()), None), sg._h)
        return out
    if kind == "gradients":
        y, loss, g = sg.gradients(state[2], 1.0, 0.25, 0.02)
        return {"outputs": y, "loss": np.array([loss], np.float32), "gradient": g}
    loss = np.empty(1, np.float32)
    sg._check(_lib.lib().swgpu_mlp_train(sg._h, case["steps"], case["batch"], state[3], 1.0e-3,
                                         1.0, 0.25, 0.02, loss.ctypes.data_as(C.POINTER(C.c_float)),
                                         None), sg._h)
    return {"params": sg.params(), "loss": loss}


# -------------------------------------------------------------------- work

# bytes a triangle's step reads and writes once: geometry, bed, friction and
# neighbours in, the conserved state in and out (FP64 path: all in FP64)
_STEP_BYTES = {"mixed": 200, "fp64": 320}
_STEP_FLOPS = 700  # flux, limiter, balance, friction and update of one triangle


def work(case):
    kind = case["kind"]
    if kind in ("step", "evolve", "methods"):
        sc = _scene(case["scene"], case["m"], case["n"])
        steps = 1
        if kind == "evolve":
            steps = case["steps"] if not case["yields"] else 8 * case["yields"]
        steps *= {"euler": 1, "rk2": 2, "rk3": 3}[case.get("method", "euler")]
        return {"bytes": sc.N * (steps * _STEP_BYTES[case.get("precision", "fp64")] + 24),
                "flops": sc.N * steps * _STEP_FLOPS}
    if kind == "ensemble":
        n = sum(sc.N for sc in _harbours(case["count"], case["nmin"], case["nmax"]))
        return {"bytes": n * (case["steps"] * _STEP_BYTES[case["precision"]] + 28),
                "flops": n * case["steps"] * _STEP_FLOPS}
    products = 2 * (16 * 256 + 2 * 256 * 256 + 256 * 3)
    params = 16 * 256 + 256 + 2 * (256 * 256 + 256) + 256 * 3 + 3
    if kind == "predict":
        return {"bytes": case["rows"] * (12 + 16) + 2 * params, "flops": case["rows"] * products}
    rows = case["rows"] if kind == "gradients" else case["batch"] * case["steps"]
    steps = 1 if kind == "gradients" else case["steps"]
    return {"bytes": rows * (12 + 16 + 8) + steps * 8 * params, "flops": 3 * rows * products}


# ------------------------------------------------------------------- exact

class _Flow:
    """ANUGA's explicit shallow-water step in 64 bits with plain torch, one
    call per stage of the method, for the parameters of DEFAULT."""

    g, eps, H0, mah, CFL, beta = 9.8, 1.0e-12, 1.0e-3, 1.0e-3, 1.0, 0.9

    def __init__(self, sc, flow=0, start=0.0):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        i = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int64), device=dev)  # noqa: E731
        m = sc.mesh
        self.flow, self.time = flow, start
        self.N = N = m.number_of_elements
        nbr = i(m.neighbours).reshape(N, 3)
        self.inner = nbr >= 0
        self.slot = (-nbr - 1).clamp(min=0)
        self.far = nbr.clamp(min=0) * 3 + i(m.neighbour_edges).reshape(N, 3).clamp(min=0)
        self.nbr = nbr.clamp(min=0)
        self.index = torch.arange(N, device=dev)
        self.owner = ~self.inner | (nbr > self.index[:, None])
        self.surr = i(m.surrogate_neighbours).reshape(N, 3)
        self.nb = i(m.number_of_boundaries)
        n = f(m.normals).reshape(N, 3, 2)
        self.n1, self.n2 = n[..., 0], n[..., 1]
        self.len, self.rad, self.area = f(m.edgelengths).reshape(N, 3), f(m.radii), f(m.areas)
        v = f(m.vertex_coordinates).reshape(N, 3, 2)
        c = f(m.centroid_coordinates).reshape(N, 2)
        if flow:
            v_at = 0.5 * (v[:, [1, 2, 0]] + v[:, [2, 0, 1]])
        else:
            v_at = v
        self.vx, self.vy, self.cx, self.cy = v[..., 0], v[..., 1], c[:, 0], c[:, 1]
        self.dxv, self.dyv = v_at[..., 0] - c[:, :1], v_at[..., 1] - c[:, 1:]
        # the mean bed on the host: dry triangles are told by stage == bed, and
        # a division by a constant is rounded once more on the device
        z = np.asarray(sc.elevation_vertex, dtype=np.float64).reshape(N, 3)
        self.zv, self.zc = f(z), f((z[:, 0] + z[:, 1] + z[:, 2]) / 3.0)
        self.ze = self._edges(self.zv)
        self.bcell, self.bedge = i(m.boundary_cells), i(m.boundary_edges)
        self.btag = i(m.boundary_tag)
        self.tags = [(sc.boundaries.get(t), t, m) for t in m.tag_names]
        self.eta = f(sc.friction)
        self.w, self.uh, self.vh = f(sc.stage_centroid), f(sc.xmom_centroid), f(sc.ymom_centroid)
        self.wv, self.uv, self.vv = (q[:, None].repeat(1, 3) for q in (self.w, self.uh, self.vh))
        self.we, self.ue, self.ve = self.wv.clone(), self.uv.clone(), self.vv.clone()
        self.hmax = torch.zeros_like(self.w)
        self.protect()
        self.distribute()
        self.protect()
        self.distribute()
        self.boundary()

    @staticmethod
    def _edges(v):
        return 0.5 * (v[:, [1, 2, 0]] + v[:, [2, 0, 1]])

    def protect(self):
        h = self.w - self.zc
        if self.flow:
            zv = self.zv
            bmax = 0.5 * torch.maximum(zv[:, 0] + zv[:, 1],
                                       torch.maximum(zv[:, 1] + zv[:, 2], zv[:, 2] + zv[:, 0]))
            low = h < torch.clamp(0.1 * (bmax - self.zc), min=self.mah)
            floor = zv.min(dim=1).values - self.mah
            self.w = torch.where(low & (h <= 0) & (self.w < floor), floor, self.w)
        else:
            low = h < self.mah
            self.w = torch.where(low & (h <= 0), self.zc, self.w)
        self.uh = torch.where(low, 0.0, self.uh)
        self.vh = torch.where(low, 0.0, self.vh)

    def _limit(self, d, qmin, qmax):
        tiny, r = 1.0e-100, torch.full_like(qmin, 1000.0)
        r0 = torch.ones_like(qmin)
        for k in range(3):
            x = d[:, k]
            r0 = torch.where(x < -tiny, qmin / x, torch.where(x > tiny, qmax / x, r0))
            r = torch.minimum(r0, r)
        return d * torch.clamp(r * self.beta, max=1.0)[:, None]

    def _aux(self, q, s, geo):
        dx1, dy1, dx2, dy2, inv = geo
        q0, q1, q2 = q[s[:, 0]], q[s[:, 1]], q[s[:, 2]]
        dq0, dq1, dq2 = q0 - q, q1 - q0, q2 - q0
        a, b = (dy2 * dq1 - dy1 * dq2) * inv, (dx1 * dq2 - dx2 * dq1) * inv
        d = a[:, None] * self.dxv + b[:, None] * self.dyv
        e = torch.stack([torch.zeros_like(dq0), dq0, dq0 + dq1, dq0 + dq2])
        return q[:, None] + self._limit(d, e.min(dim=0).values, e.max(dim=0).values)

    def _one(self, q, s):
        dq = q[s] - q
        dx, dy = self.cx[s] - self.cx, self.cy[s] - self.cy
        area2 = dx * dx + dy * dy
        area2 = torch.where(area2 > 0, area2, 1.0)
        d = (dq * dx / area2)[:, None] * self.dxv + (dq * dy / area2)[:, None] * self.dyv
        return q[:, None] + self._limit(d, dq.clamp(max=0.0), dq.clamp(min=0.0))

    def distribute(self):
        w, zc = self.w, self.zc
        dk = torch.clamp(w - zc, min=self.mah)
        u, v = self.uh / dk, self.vh / dk
        s = self.surr
        if self.flow:
            dry = w <= zc
            s = torch.where(dry[s], self.index[:, None], s)
        x, y = self.cx, self.cy
        dx1, dx2 = x[s[:, 1]] - x[s[:, 0]], x[s[:, 2]] - x[s[:, 0]]
        dy1, dy2 = y[s[:, 1]] - y[s[:, 0]], y[s[:, 2]] - y[s[:, 0]]
        area2 = dy2 * dx1 - dy1 * dx2
        aux = (self.nb <= 1) & (area2 > 0)
        geo = (dx1, dy1, dx2, dy2, 1.0 / torch.where(aux, area2, 1.0))
        h = (w - zc)[s]
        keep = aux & (h.max(dim=1).values < self.eps)
        other = torch.where(self.surr[:, 0] != self.index, self.surr[:, 0],
                            torch.where(self.surr[:, 1] != self.index, self.surr[:, 1],
                                        self.surr[:, 2]))
        one = (self.nb == 2) & (other != self.index)
        new = []
        old = (self.we, self.ue, self.ve) if self.flow else (self.wv, self.uv, self.vv)
        for q, o in zip((w, u, v), old):
            r = torch.where(one[:, None], self._one(q, other), q[:, None].expand(-1, 3))
            r = torch.where(aux[:, None], self._aux(q, s, geo), r)
            new.append(torch.where(keep[:, None], o, r))
        if self.flow:
            we, ue, ve = new
            vert = lambda e: e[:, [1, 2, 0]] + e[:, [2, 0, 1]] - e  # noqa: E731
            wv, uv, vv = vert(we), vert(ue), vert(ve)
            de, dv = (we - self.ze).clamp(min=0.0), (wv - self.zv).clamp(min=0.0)
            self.we, self.ue, self.ve = we, ue * de, ve * de
            self.wv, self.uv, self.vv = wv, uv * dv, vv * dv
            return
        wv, uv, vv = new
        dv = (wv - self.zv).clamp(min=0.0)
        uv, vv = uv * dv, vv * dv
        # balance_deep_and_shallow
        hc, hv = w - zc, wv - self.zv
        hd = hc[:, None] - hv
        shallow = hv.min(dim=1).values < self.H0
        a = torch.where(hd <= 0, 1.0, (hc[:, None] - self.H0) / torch.where(hd <= 0, 1.0, hd))
        alpha = torch.where(shallow, a.min(dim=1).values.clamp(0.0, 1.0), 1.0)[:, None]
        some = alpha < 1
        wet = hc > 1.0e-6
        hs = torch.where(wet, hc, 1.0)
        uc, vc = torch.where(wet, self.uh / hs, 0.0), torch.where(wet, self.vh / hs, 0.0)
        wb = self.zv + (1 - alpha) * hc[:, None] + alpha * hv
        self.wv = torch.where(some, wb, wv)
        self.uv = torch.where(some, uc[:, None] * (wb - self.zv), uv)
        self.vv = torch.where(some, vc[:, None] * (wb - self.zv), vv)
        self.we, self.ue, self.ve = (self._edges(q) for q in (self.wv, self.uv, self.vv))

    def boundary(self):
        at = self.bcell * 3 + self.bedge
        w, u, v = (q.reshape(-1)[at] for q in (self.we, self.ue, self.ve))
        n1, n2, z = (q.reshape(-1)[at] for q in (self.n1, self.n2, self.ze))
        bw, bu, bv = w.clone(), torch.zeros_like(u), torch.zeros_like(v)
        for k, (b, name, mesh) in enumerate(self.tags):
            on = self.btag == k
            what = type(b).__name__
            if what == "Dirichlet_boundary":
                q = b.dirichlet_values
                bw[on], bu[on], bv[on] = q[0], q[1], q[2]
            elif what == "Time_stage_sine_boundary":
                bw[on] = b.evaluate(self.time)[0]
            elif what == "Inflow_hydrograph_boundary":
                q = b.discharge(self.time) / mesh.tag_length(name)
                bw[on] = torch.maximum(w, z + (q * q / self.g) ** (1.0 / 3.0))[on]
                bu[on], bv[on] = (-q * n1)[on], (-q * n2)[on]
            elif what == "Transmissive_boundary":
                bu[on], bv[on] = u[on], v[on]
            elif what == "Transmissive_stage_zero_momentum_boundary":
                pass
            else:  # a reflective wall
                r1, r2 = -u * n1 - v * n2, -u * n2 + v * n1
                bu[on], bv[on] = (n1 * r1 - n2 * r2)[on], (n2 * r1 + n1 * r2)[on]
        self.bw, self.bu, self.bv = bw, bu, bv

    def _speed(self, uh, h):
        lim = h < 10 * self.H0
        dry = lim & (h < self.eps)
        h = torch.where(dry, 0.0, h)
        hs = torch.where(dry, 1.0, h)
        u = torch.where(dry, 0.0, torch.where(lim, uh / (hs + self.H0 ** 2 / hs), uh / hs))
        return u, torch.where(lim, u * h, uh), h

    def fluxes(self):
        far = lambda e, b: torch.where(self.inner, e.reshape(-1)[self.far],  # noqa: E731
                                       b[self.slot] if len(b) else 0.0)
        wl, ul0, vl0, zl = self.we, self.ue, self.ve, self.ze
        wr, ur0, vr0 = far(wl, self.bw), far(ul0, self.bu), far(vl0, self.bv)
        zr = torch.where(self.inner, zl.reshape(-1)[self.far], zl)
        n1, n2, g = self.n1, self.n2, self.g
        skip = ((wl - zl).abs() < self.eps) & ((wr - zr).abs() < self.eps)
        al, bl = n1 * ul0 + n2 * vl0, -n2 * ul0 + n1 * vl0
        ar, br = n1 * ur0 + n2 * vr0, -n2 * ur0 + n1 * vr0
        z = 0.5 * (zl + zr)
        ul, uhl, hl = self._speed(al, wl - z)
        ur, uhr, hr = self._speed(ar, wr - z)
        vhl, vhr = self._speed(bl, hl)[1], self._speed(br, hr)[1]
        cl, cr = torch.sqrt(g * hl), torch.sqrt(g * hr)
        smax = torch.maximum(ul + cl, ur + cr).clamp(min=0.0)
        smin = torch.minimum(ul - cl, ur - cr).clamp(max=0.0)
        den = smax - smin
        live = ~skip & ~(den < self.eps)
        inv = 1.0 / torch.where(live, den, 1.0)
        ss = smax * smin
        e0 = (smax * (ul * hl) - smin * (ur * hr) + ss * (wr - wl)) * inv
        e1 = (smax * (ul * uhl + 0.5 * g * hl * hl) - smin * (ur * uhr + 0.5 * g * hr * hr)
              + ss * (ar - al)) * inv
        e2 = (smax * (ul * vhl) - smin * (ur * vhr) + ss * (br - bl)) * inv
        f = lambda q: -(torch.where(live, q, 0.0) * self.len).sum(dim=1) / self.area  # noqa: E731
        self.ew, self.eu, self.ev = f(e0), f(n1 * e1 - n2 * e2), f(n2 * e1 + n1 * e2)
        ms = torch.where(live, torch.maximum(smax.abs(), smin.abs()), 0.0)
        fast = ms > self.eps
        r = torch.minimum(self.rad[:, None].expand(-1, 3),
                          torch.where(self.inner, self.rad[self.nbr], math.inf))
        dt = torch.where(fast, r / torch.where(fast, ms, 1.0), math.inf).min()
        self.max_speed = torch.where(self.owner, ms, 0.0).max(dim=1).values
        # gravity on the free surface, and the edges' pressure
        x, y, q = self.vx, self.vy, self.wv
        y20, y10, x10, x20 = (y[:, 2] - y[:, 0], y[:, 1] - y[:, 0], x[:, 1] - x[:, 0],
                              x[:, 2] - x[:, 0])
        det = y20 * x10 - y10 * x20
        d1, d2 = q[:, 1] - q[:, 0], q[:, 2] - q[:, 0]
        wx, wy = (y20 * d1 - y10 * d2) / det, (x10 * d2 - x20 * d1) / det
        h = self.w - self.zc
        p = -0.5 * g * (wl - zl) ** 2 * self.len
        self.eu = self.eu - g * wx * h - (p * n1).sum(dim=1) / self.area
        self.ev = self.ev - g * wy * h - (p * n2).sum(dim=1) / self.area
        return float(dt)

    def update(self, dt):
        h = self.w - self.zc
        on = (self.eta > self.mah) & (h >= self.mah)
        hs = torch.where(on, h, 1.0)
        S = torch.where(on, -self.g * self.eta ** 2 * torch.sqrt(self.uh ** 2 + self.vh ** 2)
                        / hs ** (7.0 / 3.0), 0.0)
        self.w = self.w + dt * self.ew
        den_u = 1.0 - dt * torch.where(self.uh == 0, 0.0, S)
        den_v = 1.0 - dt * torch.where(self.vh == 0, 0.0, S)
        self.uh = (self.uh + dt * self.eu) / den_u
        self.vh = (self.vh + dt * self.ev) / den_v

    def step(self, method="euler", until=math.inf):
        stages = {"euler": [(0.0, 1.0)], "rk2": [(0.0, 1.0), (0.5, 1.0)],
                  "rk3": [(0.0, 1.0), (0.75, 0.5), (1.0 / 3.0, 1.0)]}[method]
        t0, back, dt = self.time, (self.w, self.uh, self.vh), None
        for k, (b, at) in enumerate(stages):
            ft = self.fluxes()
            if k == 0:
                dt = min(self.CFL * ft, 1.0e100, until - t0)
            self.update(dt)
            if k:
                self.w, self.uh, self.vh = ((1.0 - b) * q + b * o for q, o in
                                            zip((self.w, self.uh, self.vh), back))
            self.protect()
            self.time = t0 + at * dt
            if k == len(stages) - 1:
                self.hmax = torch.maximum(self.hmax, self.w - self.zc)
            self.distribute()
            self.boundary()

    def conserved(self):
        return {"stage": self.w.cpu().numpy(), "xmomentum": self.uh.cpu().numpy(),
                "ymomentum": self.vh.cpu().numpy(), "time": float(self.time)}

    def volume(self):
        return float((self.area * (self.w - self.zc)).sum())


def _network(p):
    shapes = [(16, 256), (256,), (256, 256), (256,), (256, 256), (256,), (256, 3), (3,)]
    out, o = [], 0
    for s in shapes:
        n = int(np.prod(s))
        out.append(p[o:o + n].reshape(s))
        o += n
    return out


def _exact_surrogate(case, seed):
    fm, th, t, rows = _surrogate_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    mu, isd = SG.feature_normalisation(fm)
    scen, tri = f(th.astype(np.float32)), f(fm.tri)
    params = f(SG.init_params(seed))
    N, total = fm.N, case["scen"] * fm.N
    target = f(t).reshape(total, 2)

    def features(r):
        s, k = torch.div(r, N, rounding_mode="floor"), r % N
        raw = torch.zeros((len(r), 16), dtype=torch.float64, device=dev)
        raw[:, :9], raw[:, 9:13] = scen[s], tri[k][:, [2, 0, 1, 3]]
        return (raw - f(mu)) * f(isd)

    def forward(p, r):
        W1, b1, W2, b2, W3, b3, W4, b4 = _network(p)
        x = torch.relu(features(r) @ W1 + b1)
        x = torch.relu(x @ W2 + b2)
        return torch.relu(x @ W3 + b3) @ W4 + b4

    if case["kind"] == "predict":
        r = torch.arange(case["row0"], case["row0"] + case["rows"], device=dev)
        return torch.cat([forward(params, part).float() for part in r.split(1 << 19)])

    def loss_and_gradient(p, r):
        q = p.clone().requires_grad_(True)
        y = forward(q, r)
        e0, e1 = y[:, 0] - target[r, 0], y[:, 1] - target[r, 1]
        u = e0.detach().abs() - y[:, 2]
        pin = torch.where(u >= 0, 0.9 * u, -0.1 * u)
        loss = (e0 * e0 + 0.25 * e1 * e1 + 0.02 * pin).mean()
        loss.backward()
        return y.detach(), float(loss), q.grad

    if case["kind"] == "gradients":
        y, loss, g = loss_and_gradient(params, torch.as_tensor(rows, device=dev))
        return {"outputs": y.cpu().numpy(), "loss": np.array([loss]),
                "gradient": g.cpu().numpy()}
    m, v, loss = torch.zeros_like(params), torch.zeros_like(params), 0.0
    mask = (1 << 64) - 1
    for s in range(case["steps"]):
        key = (seed * 0x9E3779B97F4A7C15 + s) & mask
        z = np.uint64(key) ^ (np.arange(case["batch"], dtype=np.uint64)
                              * np.uint64(0xD1B54A32D192ED03))
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        r = ((z ^ (z >> np.uint64(31))) % np.uint64(total)).astype(np.int64)
        _, loss, g = loss_and_gradient(params, torch.as_tensor(r, device=dev))
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        params = params - 1.0e-3 * (m / (1 - 0.9 ** (s + 1))) / (
            torch.sqrt(v / (1 - 0.999 ** (s + 1))) + 1.0e-8)
    return {"params": params.cpu().numpy(), "loss": np.array([loss])}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("predict", "gradients", "train"):
        return _exact_surrogate(case, seed)
    if kind == "ensemble":
        flows = [_Flow(sc) for sc in _ensemble(case, seed)]
        for f in flows:
            for _ in range(case["steps"]):
                f.step()
        got = [f.conserved() for f in flows]
        return {"stage": [q["stage"] for q in got], "xmomentum": [q["xmomentum"] for q in got],
                "ymomentum": [q["ymomentum"] for q in got],
                "max_depth": [f.hmax.cpu().numpy() for f in flows],
                "masses": np.array([f.volume() for f in flows])}
    sc = _scenario(case["scene"], case["m"], case["n"], seed)
    f = _Flow(sc, case.get("flow", 0))
    method = case.get("method", "euler")
    if kind == "step":
        f.step(method)
        return f.conserved()
    if kind == "methods":
        f.step()
        return dict(f.conserved(), stage_update=f.ew.cpu().numpy(),
                    stage_edges=f.we.cpu().numpy(), max_speed=f.max_speed.cpu().numpy())
    if not case["yields"]:
        for _ in range(case["steps"]):
            f.step(method)
        return f.conserved()
    dy = 8 * _dt(case["scene"], case["m"], case["n"])
    volumes, end = [f.volume()], case["yields"] * dy
    for k in range(1, case["yields"] + 1):
        until = min(k * dy, end)
        while f.time < until - 1.0e-12:
            f.step(method, until)
        volumes.append(f.volume())
    f.time = end
    return dict(f.conserved(), volumes=np.array(volumes))
