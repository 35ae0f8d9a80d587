"""What a user of dgrain has it do, as measurable cases.

Every pass goes through the package's public calls, from host arrays to host arrays: state up,
device work, results down.  A case is a dict of plain values:

  kind       "run"        Solver.time_evolution, the device-resident time loop
             "host_loop"  the reference's own loop: set_boundary and oneTimeStep2D per step,
                          the next dt from the returned wave speed
             "operators"  compute2DL, SlopeLimiter, PDop2D, wetDryStatus2D on host arrays
             "ensemble"   Ensemble.run over meshes of uneven size, tide and rain per mesh
             "gradient"   GaugeMisfit.forward and .backward (recorded run, discrete adjoint)
  nx, ny     cells of the rectangle (two triangles each); an ensemble has `meshes` of them,
             with triangle counts log-uniform in [least, most]
  land       True: the coastal rectangle with dry land and a moving shoreline, wet/dry on;
             False: a submerged basin
  order, stages, flux, friction ("node": n per node, "element": n per element), steps,
  checkpoint (gradient: steps between checkpoints), gauges
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dg-rain_b200"))

import dgrain  # noqa: E402
from dgrain import p2  # noqa: E402

FLUX = {"roe": 0, "llf": 1, "hllc": 2}
TIDE_PERIOD = 44712.0
FILM = 0.9e-3       # water on dry land, just below the wet/dry threshold

BASE = dict(kind="run", nx=0, ny=0, land=False, order=1, stages=2, flux="roe", friction="node", steps=1, gauges=0,
            checkpoint=0, meshes=1, least=0, most=0)


def _case(**kw):
    return {**BASE, **kw}


def listed():
    return [
        # the 250 m test mesh and a calibration-sized estuary: many short launches per step
        _case(name="coast_1600", nx=40, ny=20, land=True, steps=60),
        _case(name="coast_24k", nx=157, ny=77, land=True, friction="element", steps=50, gauges=8),
        # the mesh of the adjoint studies, and the largest mesh of the benchmark
        _case(name="coast_200k", nx=448, ny=223, land=True, steps=100),
        _case(name="coast_4m", nx=2000, ny=1000, land=True, steps=100),
        # the extensions for flows that stay wet: SSP(3,3) with another numerical flux
        _case(name="basin_91k_rk3_hllc", nx=300, ny=151, stages=3, flux="hllc", steps=60),
        # code written against the reference's call surface: its own time loop, its operators
        _case(name="host_loop_10k", kind="host_loop", nx=101, ny=49, steps=50),
        _case(name="operators_44k", kind="operators", nx=211, ny=103, land=True),
        # scenario studies: many small meshes at once
        _case(name="ensemble_32", kind="ensemble", meshes=32, least=5000, most=80000, steps=40),
        # the p = 2 step alone and under the zonal calibration (one objective and gradient)
        _case(name="p2_163k", nx=401, ny=203, order=2, stages=3, steps=30, gauges=32),
        _case(name="p2_calibration_8", kind="gradient", meshes=8, least=5000, most=30000, order=2, stages=3,
              friction="element", steps=20, checkpoint=10, gauges=16),
        # gradients of the wet/dry step on a small and on an ordinary mesh
        _case(name="gradient_5k", kind="gradient", nx=71, ny=35, land=True, friction="element", steps=30,
              checkpoint=10, gauges=8),
        _case(name="gradient_200k", kind="gradient", nx=448, ny=223, land=True, friction="element", steps=20,
              checkpoint=10, gauges=32),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "host_loop", "operators", "ensemble", "gradient"])
    order = 2 if kind in ("run", "gradient") and rng.random() < 0.35 else 1
    largest = {"run": 1.2e6 if order == 1 else 2.5e5, "host_loop": 2e5, "operators": 5e5, "ensemble": 0,
               "gradient": 2e5 if order == 1 else 6e4}[kind]
    if kind == "ensemble":
        least = int(math.exp(rng.uniform(math.log(1000), math.log(10000))))
        return _case(kind=kind, meshes=rng.randint(3, 32), least=least, most=least * rng.randint(2, 8),
                     stages=rng.choice([2, 3]), steps=rng.randint(10, 40))
    cells = math.exp(rng.uniform(math.log(400), math.log(largest / 2)))
    nx = max(16, int(math.sqrt(2 * cells) * rng.uniform(0.95, 1.05)))
    land = order == 1 and kind != "host_loop" and rng.random() < 0.6
    steps = {"run": rng.randint(20, 80), "host_loop": rng.randint(10, 50), "operators": 1,
             "gradient": rng.randint(8, 30)}[kind]
    return _case(kind=kind, nx=nx, ny=max(8, int(cells / nx)), land=land, order=order,
                 stages=3 if order == 2 else rng.choice([2, 2, 3]),
                 flux="roe" if land else rng.choice(["roe", "roe", "llf", "hllc"]),
                 friction="element" if kind == "gradient" else rng.choice(["node", "element"]), steps=steps,
                 checkpoint=rng.randint(4, 12) if kind == "gradient" else 0,
                 gauges=rng.randint(4, 32) if kind == "gradient" else rng.choice([0, 0, 8]))


# ------------------------------------------------------------------------------ inputs ----


def _mesh(nx, ny, land, seed):
    m = dgrain.rectangle(nx, ny, jitter=0.1, seed=seed, datum=0.0 if land else 7.0, connect=False)
    return dgrain.build_connectivity(m, device=True)


def _fields(m, rng):
    """smooth zeta, Qx, Qy as functions of (x, y, depth): a hump off the coast and a slow basin
    circulation that dies out towards the shore (the scheme itself stops at some shorelines
    once a wave runs up them, so the waves start well away from the shore)"""
    lx, ly = float(m.x.max()), float(m.y.max())
    amp, cx, cy = rng.uniform(0.05, 0.2), rng.uniform(0.08, 0.2) * lx, rng.uniform(0.3, 0.7) * ly
    wid, tilt, turn, ph = 0.06 * lx, rng.uniform(0.005, 0.02), rng.uniform(0.05, 0.2), rng.uniform(0.0, 6.0, 2)
    deep = lambda z: np.clip((z - 1.5) / 2, 0.0, 1.0) ** 2  # noqa: E731
    wave = lambda x, y, k: np.sin(4 * x / lx + ph[k]) * np.cos(5 * y / ly + ph[1 - k])  # noqa: E731

    def zeta(x, y, z):
        hump = amp * np.maximum(np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * wid * wid)) - 0.05, 0.0)
        return hump + tilt * deep(z) * wave(x, y, 0)

    return (zeta, lambda x, y, z: turn * deep(z) * wave(x, y, 1),
            lambda x, y, z: turn * deep(z) * wave(y * lx / ly, x * ly / lx, 0))


def _one(case, nx, ny, seed):
    """mesh, initial state, per-element n, tide amplitude and rain of one mesh"""
    m = _mesh(nx, ny, case["land"], seed)
    rng = np.random.default_rng(seed)
    fz, fx, fy = _fields(m, rng)
    if case["order"] == 2:
        far = lambda f: p2.project(m, lambda x, y: f(x, y, 9.0))  # noqa: E731
        state = (far(fz), far(fx), far(fy), np.zeros(m.num_el, dtype=np.int32))
    else:
        zn = fz(m.x, m.y, m.z)
        zeta, _, _, wd = dgrain.initial_state(m, np.maximum(zn, FILM - m.z) if case["land"] else zn)
        mid = [(a[m.el2v] + a[m.el2v[:, [1, 2, 0]]]).ravel() / 2 for a in (m.x, m.y, m.z)]
        state = (zeta, fx(*mid), fy(*mid), wd)
    n_el = rng.uniform(0.02, 0.05, m.num_el) if case["friction"] == "element" else None
    rain = 0.0 if case["land"] else float(rng.uniform(0.0, 2e-5))
    return dict(mesh=m, state=state, n_el=n_el, amp=float(rng.uniform(0.3, 0.6)), rain=rain,
                points=np.column_stack([rng.uniform(0.1, 0.5 if case["land"] else 0.9, case["gauges"]) * m.x.max(),
                                        rng.uniform(0.1, 0.9, case["gauges"]) * m.y.max()]))


def _inputs(case, seed):
    if not case["least"]:
        return [_one(case, case["nx"], case["ny"], seed)]
    sizes = np.exp(np.random.default_rng(case["meshes"]).uniform(np.log(case["least"]), np.log(case["most"]),
                                                                 case["meshes"]))
    return [_one(case, max(2, round(math.sqrt(s))), max(1, round(math.sqrt(s)) // 2), 1000 * seed + k)
            for k, s in enumerate(sizes)]


def _common(case):
    return dict(order=case["order"], rk_stages=case["stages"], flux=FLUX[case["flux"]],
                wet_dry=int(case["land"]), cfl=0.1 if case["order"] == 2 else 0.3)


def _gauges(case, ins):
    """flattened gauge elements and weights"""
    place = p2.gauge_weights if case["order"] == 2 else dgrain.place_gauges
    els, ws, off = [], [], 0
    for i in ins:
        el, w = place(i["mesh"], [tuple(p) for p in i["points"]])
        els.append(el + off)
        ws.append(w)
        off += i["mesh"].num_el
    return np.concatenate(els), np.concatenate(ws)


def _target(case, ngauges, seed):
    return 0.05 * np.random.default_rng(seed + 1).standard_normal((case["steps"], ngauges))


def prepare(case, seed):
    ins = _inputs(case, seed)
    s = dict(case=case, ins=ins)
    if case["least"]:
        scen = [dict(tide_on=1, tide_amp=i["amp"], tide_period=TIDE_PERIOD, rain=i["rain"], n_el=i["n_el"])
                for i in ins]
        s["solver"] = dgrain.Ensemble([i["mesh"] for i in ins], scen, **_common(case))
    else:
        i = ins[0]
        s["solver"] = dgrain.Solver(i["mesh"], tide_on=1, tide_amp=i["amp"], tide_period=TIDE_PERIOD,
                                    rain=i["rain"], **_common(case))
        if i["n_el"] is not None:
            s["solver"].set_element_manning(i["n_el"])
    if case["kind"] == "gradient":
        el, w = _gauges(case, ins)
        s["misfit"] = dgrain.GaugeMisfit(s["solver"], case["steps"], case["checkpoint"], el, w,
                                         _target(case, len(el), seed))
        s["state"] = s["solver"].flatten_states([i["state"] for i in ins]) if case["least"] else ins[0]["state"]
    elif case["gauges"]:
        s["solver"].set_gauges(*_gauges(case, ins), case["steps"])
    if case["kind"] == "host_loop":
        m = ins[0]["mesh"]
        s["bzeta"], s["bqn"] = np.zeros(m.num_edges), np.full(m.num_edges, 1e6)
        s["sea"] = np.flatnonzero(m.bdry == 2)
    return s


# -------------------------------------------------------------------------------- pass ----


def run(s):
    case, solver, ins = s["case"], s["solver"], s["ins"]
    if case["kind"] == "gradient":
        J, values = s["misfit"].forward(s["state"])
        return {"J": J, "gauges": values, **s["misfit"].backward()}
    if case["kind"] == "ensemble":
        for k, i in enumerate(ins):
            solver.upload_state(k, *i["state"])
        t, dt, n = solver.run(case["steps"])
        down = [solver.download_state(k) for k in range(len(ins))]
        out = {name: np.concatenate([d[v] for d in down]) for v, name in enumerate(("zeta", "qx", "qy", "wd"))}
        return {**out, "time": t, "dt": dt, "steps": n}
    solver.upload_state(*ins[0]["state"])
    if case["kind"] == "operators":
        solver.boundary_conditions(0.0)
        solver.wetDryStatus2D()
        rz, rx, ry, lam = solver.compute2DL()
        solver.SlopeLimiter()
        solver.PDop2D()
        solver.wetDryStatus2D()
        z, x, y, wd = solver.download_state()
        return {"rz": rz, "rx": rx, "ry": ry, "speed": lam, "zeta": z, "qx": x, "qy": y, "wd": wd}
    if case["kind"] == "host_loop":
        t, dt = 0.0, solver.params.dt0
        for _ in range(case["steps"]):
            s["bzeta"][s["sea"]] = ins[0]["amp"] * math.sin(2 * math.pi * t / TIDE_PERIOD)
            solver.set_boundary(s["bzeta"], s["bqn"])
            lam = solver.oneTimeStep2D(t, dt)
            t, dt = t + dt, solver.params.cfl * ins[0]["mesh"].min_edge / lam
        n = case["steps"]
    else:
        t, dt, n = solver.time_evolution(1e9, case["steps"])
    z, x, y, wd = solver.download_state()
    out = {"zeta": z, "qx": x, "qy": y, "wd": wd, "time": t, "dt": dt, "steps": n}
    if case["gauges"]:
        out["gauges"] = solver.gauge_series()
    return out


def work(case):
    """Bytes: per stage and element the stage input and the step input read, the output
    written (3 x 72 B, or 3 x 144 B at p = 2), the states up and down once; a gradient reads
    and writes them again for the reversed run.  Operations: of the scheme's fluxes, fits,
    quadrature and limiter, per element and stage."""
    if case["least"]:
        ne = sum(2 * max(2, round(math.sqrt(v))) * max(1, round(math.sqrt(v)) // 2) for v in np.exp(
            np.random.default_rng(case["meshes"]).uniform(np.log(case["least"]), np.log(case["most"]),
                                                          case["meshes"])))
    else:
        ne = 2 * case["nx"] * case["ny"]
    state, ops = (144, 3600) if case["order"] == 2 else (72, 1500)
    if case["kind"] == "operators":
        return {"bytes": 5 * 72 * ne, "flops": ops * ne}
    sweeps = 3 if case["kind"] == "gradient" else 1
    stages = case["steps"] * case["stages"]
    return {"bytes": ne * (2 * state + sweeps * stages * 3 * state), "flops": sweeps * stages * ops * ne}


# --------------------------------------------------------------------- 64-bit reference ----
#
# The scheme in plain torch, whole arrays at a time: state S [3, k, ne] (zeta, Qx, Qy; k = 3
# edge midpoints or 6 modes).  Maxima and minima are written as where() on strict comparisons,
# so that derivatives of ties follow the first operand.

G, H0, VELZERO = 9.81, 1e-3, 1e-2


def _pick(cond, a, b):
    return torch.where(cond, a, b)


def _max(a, b):
    return _pick(b > a, b, a)


def _min(a, b):
    return _pick(b < a, b, a)


def _length(u, v):
    q = u * u + v * v
    return _pick(q > 0, torch.sqrt(_pick(q > 0, q, 1.0)), 0.0)


class _Scheme:
    def __init__(self, case, i, dev):
        m = i["mesh"]
        t = lambda a: torch.as_tensor(np.asarray(a), device=dev)  # noqa: E731
        self.case, self.i, self.dev, self.ne, self.nn = case, i, dev, m.num_el, m.num_nodes
        self.x, self.y, self.z = t(m.x), t(m.y), t(m.z)
        self.v = t(m.el2v).long().T.contiguous()
        self.ein, self.eex = t(m.ed2el).long().T
        ends, self.bdry = t(m.ed2v).long().sort(1)[0], t(m.bdry)
        self.min_edge = float(m.min_edge)
        sides = torch.stack([self.v, self.v.roll(-1, 0)], -1).sort(-1)[0]      # [3, ne, 2]
        same = lambda el: (sides[:, el] == ends).all(-1).int().argmax(0)       # noqa: E731
        self.kin, self.kex = same(self.ein), same(self.eex)
        self.wall = (self.bdry == 0) & (self.ein == self.eex)
        self.va = self.v[self.kin, self.ein]
        self.vb = self.v[(self.kin + 1) % 3, self.ein]
        xa, xb, ya, yb = self.x[self.va], self.x[self.vb], self.y[self.va], self.y[self.vb]
        xv, yv = self.x[self.v], self.y[self.v]
        self.jac = xv[0] * (yv[1] - yv[2]) + xv[1] * (yv[2] - yv[0]) + xv[2] * (yv[0] - yv[1])
        sg = torch.sign(self.jac)[self.ein]
        length = torch.sqrt((xb - xa) ** 2 + (yb - ya) ** 2)
        self.nx, self.ny = sg * (yb - ya) / length, sg * (xa - xb) / length
        self.edge_of = torch.zeros(3, self.ne, dtype=torch.long, device=dev)
        self.side_of = torch.zeros(3, self.ne, dtype=torch.bool, device=dev)
        ids, two = torch.arange(len(self.ein), device=dev), self.ein != self.eex
        self.edge_of[self.kin, self.ein] = ids
        self.edge_of[self.kex[two], self.eex[two]] = ids[two]
        self.side_of[self.kex[two], self.eex[two]] = True
        self.turned = self.v[self.kex, self.eex] != self.va                    # neighbours run it the other way
        order = torch.sort(self.v.T.reshape(-1), stable=True)
        start = torch.searchsorted(order[0], torch.arange(self.nn + 1, device=dev))
        most = int((start[1:] - start[:-1]).max())
        at = start[:-1, None] + torch.arange(most, device=dev)[None]
        self.around = torch.where(at < start[1:, None], order[1][at.clamp(max=3 * self.ne - 1)] // 3, -1).T
        self.n_el = t(i["n_el"]) if i["n_el"] is not None else None
        self.n_node = t(m.nfric)
        self._geometry()
        if case["order"] == 2:
            self._tables()

    def _geometry(self):
        xv, yv = self.x[self.v], self.y[self.v]
        nxt = lambda a: a.roll(-1, 0)  # noqa: E731
        self.len = torch.sqrt((nxt(xv) - xv) ** 2 + (nxt(yv) - yv) ** 2)
        self.xm, self.ym = (xv + nxt(xv)) / 2, (yv + nxt(yv)) / 2
        sj = torch.sign(self.jac)
        self.enx, self.eny = sj * (nxt(yv) - yv) / self.len, sj * (xv - nxt(xv)) / self.len
        x, y = self.xm, self.ym
        self.mjac = 4 * (x[1] - x[2]) * (y[1] - y[0]) - 4 * (x[1] - x[0]) * (y[1] - y[2])
        a, b, c = [0, 1, 2], [1, 2, 0], [2, 0, 1]
        self.gx, self.gy = 4 / self.mjac * (y[b] - y[c]), 4 / self.mjac * (x[c] - x[b])
        self.gp = self.gx * x.sum(0) + self.gy * y.sum(0)
        s3 = math.sqrt(3.0)
        # Gauss points of edge e lie at its midpoint -+ half the edge / sqrt(3)
        self.qx = torch.stack([x + sgn * (x[b] - x[c]) / s3 for sgn in (-1, 1)])  # [2, 3, ne]
        self.qy = torch.stack([y + sgn * (y[b] - y[c]) / s3 for sgn in (-1, 1)])
        den = x[0] * y[1] - x[0] * y[2] + x[1] * y[2] - x[1] * y[0] + x[2] * y[0] - x[2] * y[1]
        psi = [-(self.qy * x[j] - self.qy * x[k] - self.qx * y[j] + x[k] * y[j] + self.qx * y[k] - x[j] * y[k]) / den
               for j, k in ((1, 2), (2, 0), (0, 1))]
        self.psi = torch.stack(psi)                                              # [3, 2, 3, ne]
        self.m2 = x * self.enx + y * self.eny
        A, B, C = self.enx, self.m2, self.eny
        self.dm = (C[0] * B[1] * A[2] - B[0] * C[1] * A[2] - C[0] * A[1] * B[2] + A[0] * C[1] * B[2]
                   + B[0] * A[1] * C[2] - A[0] * B[1] * C[2])

    # ---- numerical fluxes: in and ex traces [3, nf] -> (Fhat.n [3, nf], largest speed [nf])

    def flux(self, wi, we, zed, g_press, kind):
        nx, ny = self.nx, self.ny
        hi, he = wi[0] + zed, we[0] + zed
        ui, vi, ue, ve = wi[1] / hi, wi[2] / hi, we[1] / he, we[2] / he

        def normal(h, u, v):
            p = 0.5 * g_press * (h * h - zed * zed)
            huv = h * u * v
            return torch.stack([h * u * nx + h * v * ny, (h * u * u + p) * nx + huv * ny,
                                huv * nx + (h * v * v + p) * ny])

        uni, une = ui * nx + vi * ny, ue * nx + ve * ny
        ci, ce = torch.sqrt(G * hi), torch.sqrt(G * he)
        speed = torch.zeros_like(hi)
        for s in (uni - ci, une - ce, uni, une, uni + ci, une + ce):
            speed = _max(speed, s.abs())
        if kind == "llf":
            return 0.5 * (normal(hi, ui, vi) + normal(he, ue, ve)) - 0.5 * speed * (we - wi), speed
        if kind == "hllc":
            uti, ute = -ui * ny + vi * nx, -ue * ny + ve * nx
            hs = 1.0 / G * (0.5 * (ci + ce) + 0.25 * (uni - une)) ** 2
            li = _pick(hs > hi, torch.sqrt((hs * hs + hs * hi) / (2 * hi * hi)), 1.0)
            le = _pick(hs > he, torch.sqrt((hs * hs + hs * he) / (2 * he * he)), 1.0)
            si, se = uni - ci * li, une + ce * le
            A, B = une - se, uni - si
            st = (si * he * A - se * hi * B) / (he * A - hi * B)
            inside = (si >= 0) | (st >= 0)
            star = (si < 0) & ((st >= 0) | (se >= 0))
            w, h, u, v = _pick(inside, wi, we), _pick(inside, hi, he), _pick(inside, ui, ue), _pick(inside, vi, ve)
            S, un, ut = _pick(inside, si, se), _pick(inside, uni, une), _pick(inside, uti, ute)
            q1 = h * ((S - un) / (S - st))
            d = torch.stack([q1 - h, q1 * st - (w[1] * nx + w[2] * ny), q1 * ut - (-w[1] * ny + w[2] * nx)])
            add = S * torch.stack([d[0], d[1] * nx - d[2] * ny, d[1] * ny + d[2] * nx])
            return normal(h, u, v) + _pick(star, add, 0.0), speed
        ri, re = torch.sqrt(hi), torch.sqrt(he)
        u, v = (ui * ri + ue * re) / (ri + re), (vi * ri + ve * re) / (ri + re)
        c = torch.sqrt(G * (0.5 * (hi + he)))
        un = u * nx + v * ny
        lam = []
        for lh, a, b in ((un - c, uni - ci, une - ce), (un, uni, une), (un + c, uni + ci, une + ce)):
            e = _max(_max(torch.zeros_like(c), lh - a), b - lh)
            lam.append(_max(e, _pick(lh < 0, -lh, lh)))
        j, den = wi - we, -2 * c
        k0 = lam[0] * ((-c - un) / den * j[0] + nx / den * j[1] + ny / den * j[2])
        k1 = lam[1] * ((-2 * c * ny * u + 2 * c * nx * v) / den * j[0] + 2 * c * ny / den * j[1]
                       + -2 * c * nx / den * j[2])
        k2 = lam[2] * ((-c + un) / den * j[0] - nx / den * j[1] - ny / den * j[2])
        diss = torch.stack([k0 + k2, (u - c * nx) * k0 - ny * k1 + (u + c * nx) * k2,
                            (v - c * ny) * k0 + nx * k1 + (v + c * ny) * k2])
        return 0.5 * (normal(hi, ui, vi) + normal(he, ue, ve)) + 0.5 * diss, speed

    def mirror(self, w):
        """the trace behind a wall: normal discharge reflected"""
        qn, qt = w[1] * self.nx + w[2] * self.ny, -w[1] * self.ny + w[2] * self.nx
        return torch.stack([w[0], -qn * self.nx - qt * self.ny, -qn * self.ny + qt * self.nx])

    def outside(self, wi, we, bz):
        """exterior traces: the neighbour's, a wall's, or the sea's level bz (its own if negative)"""
        sea = torch.stack([wi[0] if bz < 0 else torch.full_like(wi[0], bz), wi[1], wi[2]])
        return _pick(self.wall, self.mirror(wi), _pick(self.bdry > 0, sea, we))

    # ---- p = 1

    def rhs1(self, S, wd, bz, z, n_el):
        wi, we = S[:, self.kin, self.ein], S[:, self.kex, self.eex]
        we = self.outside(wi, we, bz)
        zed = (z[self.va] + z[self.vb]) / 2
        kind = self.case["flux"]
        fin, lam = self.flux(wi, we, zed, G, kind)
        fex = fin
        if wd is not None:
            di, de = wd[self.ein] != 1, wd[self.eex] != 1
            f0, l0 = self.flux(wi, we, zed, 0.0, kind)
            both = (wd[self.ein] == 0) & (wd[self.eex] == 0)
            fi2, li2 = self.flux(wi, self.mirror(wi), zed, 0.0, kind)
            fe2, le2 = self.flux(self.mirror(we), we, zed, 0.0, kind)
            fin, fex = _pick(both, fi2, _pick(di, f0, fin)), _pick(both, fe2, _pick(de, f0, fin))
            lam = _pick(both, _max(li2, le2), _pick(di | de, _max(lam, l0), lam))
        F = _pick(self.side_of, -fex[:, self.edge_of], fin[:, self.edge_of])     # [3, 3, ne]
        enx, eny, A, B, C = self.enx, self.eny, self.enx, self.m2, self.eny

        def fit(R):
            a = (R[2] * C[0] * B[1] - R[2] * B[0] * C[1] - R[1] * C[0] * B[2] + R[0] * C[1] * B[2]
                 + R[1] * B[0] * C[2] - R[0] * B[1] * C[2]) / self.dm
            b = -(R[2] * C[0] * A[1] - R[2] * A[0] * C[1] - R[1] * C[0] * A[2] + R[0] * C[1] * A[2]
                  + R[1] * A[0] * C[2] - R[0] * A[1] * C[2]) / self.dm
            c = (R[2] * B[0] * A[1] - R[2] * A[0] * B[1] - R[1] * B[0] * A[2] + R[0] * B[1] * A[2]
                 + R[1] * A[0] * B[2] - R[0] * A[1] * B[2]) / self.dm
            return a, b, c

        midz = 0.5 * (z[self.v] + z[self.v].roll(-1, 0))
        n = n_el.expand(3, -1) if n_el is not None else \
            0.5 * (self.n_node[self.v] + self.n_node[self.v].roll(-1, 0))
        H = S[0] + midz
        u, v = S[1] / H, S[2] / H
        tau = G * n * n * _length(u, v) / H ** (4.0 / 3)
        gl = G if wd is None else _pick(wd == 0, 0.0, torch.full_like(H[0], G))
        pr = 0.5 * gl * (H * H - midz * midz)
        qxy = S[1] * S[2] / H
        R = (S[1] * enx + S[2] * eny, (S[1] * S[1] / H + pr) * enx + qxy * eny,
             qxy * enx + (S[2] * S[2] / H + pr) * eny)
        aj = self.mjac.abs()
        X = []
        for k in range(3):
            a, b, c = fit(F[k])
            fd = (a + b * self.qx) * enx + (c + b * self.qy) * eny               # [2, 3, ne]
            si = (self.len / 2 * (fd * self.psi).sum(1)).sum(1)
            a, b, c = fit(R[k])
            dv = aj * (0.5 * a * self.gx + 0.5 * c * self.gy + b / 6 * self.gp)
            x = dv - si
            if k:
                grad = (midz * (self.gx if k == 1 else self.gy)).sum(0)
                x = x + gl * aj * grad / 6 * S[0] - aj / 6 * tau * S[k]
            X.append(x)
        rhs = 6 / self.jac.abs() * torch.stack(X)
        rhs = torch.cat([rhs[:1] + self.i["rain"], rhs[1:]])
        return rhs, lam.detach()

    def limit(self, S, z):
        avg = S.sum(1) / 3
        hi = torch.full((3, self.nn), -99999.0, device=self.dev, dtype=S.dtype)
        lo = -hi
        for el in self.around:
            a = avg[:, el.clamp(min=0)]
            hi, lo = _pick((el >= 0) & (a > hi), a, hi), _pick((el >= 0) & (a < lo), a, lo)
        hi, lo, zn = hi[:, self.v], lo[:, self.v], z[self.v]
        vx = torch.stack([S[:, 0] - S[:, 1] + S[:, 2], S[:, 0] + S[:, 1] - S[:, 2], -S[:, 0] + S[:, 1] + S[:, 2]], 1)
        use = ((vx[0] + zn > H0) & (lo[0] + zn > H0)).all(0)
        vx = list((_max(_min(hi, vx), lo)).unbind(1))
        for _ in range(3):
            diff = ((vx[0] + vx[1] + vx[2]) / 3 - avg) * 3
            sd = torch.sign(diff.detach())
            up = [((v - avg) * sd) > 0 for v in vx]
            left = sum(p.to(S.dtype) for p in up)
            for k in range(3):
                red = _pick(up[k], diff * sd / left.clamp(min=1.0), 0.0)
                left = left - up[k].to(S.dtype)
                room = _pick(sd > 0, vx[k] - lo[:, k], hi[:, k] - vx[k])
                red = _min(room, red)
                diff, vx[k] = diff - red * sd, vx[k] - red * sd
        use = use & (torch.stack([v[0] for v in vx]) + zn >= H0).all(0)
        return _pick(use, torch.stack([(vx[0] + vx[1]) / 2, (vx[1] + vx[2]) / 2, (vx[2] + vx[0]) / 2], 1), S)

    def positive(self, S, z):
        zn = z[self.v]
        midz = 0.5 * (zn + zn.roll(-1, 0))
        mh = S[0] + midz
        ht = torch.stack([mh[0] - mh[1] + mh[2], mh[0] + mh[1] - mh[2], -mh[0] + mh[1] + mh[2]])
        avg = ht.sum(0) / 3
        low = (ht <= H0).any(0)
        hmin, imin = ht[0], torch.zeros_like(self.v[0])
        for k in (1, 2):
            less = ht[k] < hmin
            hmin, imin = _pick(less, ht[k], hmin), _pick(less, k, imin)
        hnext, inext = ht[1], torch.ones_like(imin)
        for k in range(3):
            less = (ht[k] < hnext) & (imin != k)
            hnext, inext = _pick(less, ht[k], hnext), _pick(less, k, inext)
        rest = _pick((imin != 0) & (inext != 0), 0, _pick((imin != 1) & (inext != 1), 1, torch.full_like(imin, 2)))
        ids = torch.arange(3, device=self.dev)[:, None]
        hh = _pick(ids == imin, torch.full_like(ht, H0), ht)
        low_next = 0.5 * (hh.gather(0, imin[None])[0] - hmin)
        hh = _pick(ids == inext, _max(torch.full_like(hnext, H0), hnext - low_next), hh)
        gone = (hh.gather(0, imin[None])[0] - hmin), (hh.gather(0, inext[None])[0] - hnext)
        hh = _pick(ids == rest, hh - gone[0] - gone[1], hh)
        ht = _pick(low, _pick(avg <= H0, avg.expand(3, -1), hh), ht)
        zeta = _pick(low, 0.5 * (ht + ht.roll(-1, 0)) - midz, S[0])
        wet = ht > H0
        count = wet.sum(0).to(S.dtype)
        out = [zeta]
        for k in (1, 2):
            q = S[k]
            qe = torch.stack([q[0] - q[1] + q[2], q[0] + q[1] - q[2], -q[0] + q[1] + q[2]])
            u = qe / _pick(ht != 0, ht, 1.0)
            spare = _pick(~wet & (qe.abs() > VELZERO), u, 0.0).sum(0) / count.clamp(min=1.0)
            qe = ht * _pick(wet, u + spare, 0.0)
            part = 0.5 * (qe + qe.roll(-1, 0))
            out.append(_pick(count == 0, 0.0, _pick(count == 3, q, part)))
        return torch.stack(out)

    def status(self, S, z, wd):
        zn = z[self.v]
        s = S[0]
        zv = torch.stack([s[0] - s[1] + s[2], s[0] + s[1] - s[2], -s[0] + s[1] + s[2]])
        h = zv + zn
        deep, top = h.sum(0) / 3 > H0, zv.gather(0, h.argmax(0)[None])[0] > H0 - zn.amin(0)
        return _pick(wd == -1, deep & top, _pick(wd == 1, deep, deep & top)).to(wd.dtype)

    # ---- p = 2

    def _tables(self):
        def basis(r, s):
            A, B = r + (1 + s) / 2, (1 - s) / 2
            o = np.ones_like(r)
            phi = [o, (3 * s + 1) / 2, A, (5 * s * s + 2 * s - 1) / 2, A * (5 * s + 3) / 2, (3 * A * A - B * B) / 2]
            dr = [0 * o, 0 * o, o, 0 * o, (5 * s + 3) / 2, 3 * A]
            ds = [0 * o, 1.5 * o, 0.5 * o, 5 * s + 1, (5 * s + 3) / 4 + 2.5 * A, 1.5 * A + 0.5 * B]
            return [torch.as_tensor(np.stack(p, -1), device=self.dev) for p in (phi, dr, ds)]

        q = math.sqrt(15.0)
        bary = [(1 / 3, 1 / 3, 1 / 3)]
        for a in ((6 - q) / 21, (6 + q) / 21):
            bary += [(1 - 2 * a, a, a), (a, 1 - 2 * a, a), (a, a, 1 - 2 * a)]
        self.bary = torch.as_tensor(np.array(bary), device=self.dev)
        self.wq = [9 / 40] + [(155 - q) / 1200] * 3 + [(155 + q) / 1200] * 3
        lam = np.array(bary)
        self.phi, self.dr, self.ds = basis(-lam[:, 0] + lam[:, 1] - lam[:, 2], -lam[:, 0] - lam[:, 1] + lam[:, 2])
        self.te, self.wg = [-math.sqrt(0.6), 0.0, math.sqrt(0.6)], [5 / 9, 8 / 9, 5 / 9]
        t, corner = np.array(self.te), np.array([(-1, -1), (1, -1), (-1, 1)], dtype=float)
        self.phie = torch.stack([basis(*(corner[k][:, None] * (1 - t) / 2 + corner[(k + 1) % 3][:, None] * (1 + t) / 2))
                                 [0] for k in range(3)])                          # [3, 3, 6]
        self.mass = torch.as_tensor([2, 1, 1 / 3, 2 / 3, 2 / 9, 2 / 15], dtype=torch.float64, device=self.dev)
        xv, yv = self.x[self.v], self.y[self.v]
        xr, xs, yr, ys = (xv[1] - xv[0]) / 2, (xv[2] - xv[0]) / 2, (yv[1] - yv[0]) / 2, (yv[2] - yv[0]) / 2
        det = xr * ys - xs * yr
        self.det, self.rx, self.ry, self.sx, self.sy = det.abs(), ys / det, -xs / det, -yr / det, xr / det

    def rhs2(self, S, wd, bz, z, n_el):
        F, lam = [], None
        for gp in range(3):
            t = self.te[gp]
            zed = z[self.va] * ((1 - t) / 2) + z[self.vb] * ((1 + t) / 2)
            wi = (S[:, :, self.ein] * self.phie[self.kin, gp].T).sum(1)
            ge = torch.where(self.turned, 2 - gp, gp)
            we = (S[:, :, self.eex] * self.phie[self.kex, ge].T).sum(1)
            f, l = self.flux(wi, self.outside(wi, we, bz), zed, G, self.case["flux"])
            F.append(f)
            lam = l if lam is None else _max(lam, l)
        F = torch.stack(F)                                                        # [3 points, 3, nf]
        zv = z[self.v]
        zr, zs = (zv[1] - zv[0]) / 2, (zv[2] - zv[0]) / 2
        dzx, dzy = zr * self.rx + zs * self.sx, zr * self.ry + zs * self.sy
        n = n_el if n_el is not None else self.n_node[self.v].sum(0) / 3
        acc = torch.zeros_like(S)
        for q in range(7):
            uq = (S * self.phi[q][:, None]).sum(1)
            zq = (self.bary[q][:, None] * zv).sum(0)
            H = uq[0] + zq
            u, v = uq[1] / H, uq[2] / H
            p = 0.5 * G * (H * H - zq * zq)
            tau = G * n * n * _length(u, v) / H ** (4.0 / 3)
            fx = torch.stack([uq[1], uq[1] * u + p, uq[1] * v])
            fy = torch.stack([uq[2], uq[1] * v, uq[2] * v + p])
            src = torch.stack([torch.full_like(H, self.i["rain"]), G * uq[0] * dzx - tau * uq[1],
                               G * uq[0] * dzy - tau * uq[2]])
            gx = self.dr[q][:, None] * self.rx + self.ds[q][:, None] * self.sx
            gy = self.dr[q][:, None] * self.ry + self.ds[q][:, None] * self.sy
            acc = acc + 2 * self.wq[q] * self.det * (fx[:, None] * gx + fy[:, None] * gy
                                                     + src[:, None] * self.phi[q][:, None])
        turned = self.turned[self.edge_of] & self.side_of
        for k in range(3):
            for gp in range(3):
                f = _pick(turned[k], F[2 - gp][:, self.edge_of[k]], F[gp][:, self.edge_of[k]])
                f = _pick(self.side_of[k], -f, f)
                acc = acc - self.wg[gp] * self.len[k] / 2 * f[:, None] * self.phie[k, gp][:, None]
        return acc / (self.det * self.mass[:, None]), lam.detach()

    # ---- time loop

    def step(self, S, wd, dt, bz, z, n_el):
        U, ns = S, self.case["stages"]
        for st in range(ns):
            R, lam = (self.rhs2 if self.case["order"] == 2 else self.rhs1)(S, wd, bz, z, n_el)
            E = S + dt * R
            S = E if st == 0 else 0.5 * (U + E) if ns == 2 else 0.75 * U + 0.25 * E if st == 1 else \
                1.0 / 3 * U + 2.0 / 3 * E
            if self.case["order"] == 1:
                S = self.limit(S, z)
            last = wd
            if wd is not None:
                S = self.positive(S, z)
                wd = self.status(S, z, wd)
        return S, wd, last, float(lam.max())

    def state(self):
        k = 6 if self.case["order"] == 2 else 3
        S = torch.stack([torch.as_tensor(a, device=self.dev).reshape(-1, k).T for a in self.i["state"][:3]])
        wd = torch.as_tensor(self.i["state"][3], device=self.dev) if self.case["land"] else None
        return S, self.status(S, self.z, wd) if wd is not None else None

    def evolve(self, z, n_el, S, wd, each=None):
        """`steps` steps; each(S) sees the state after every step"""
        from torch.utils.checkpoint import checkpoint

        t, dt, cfl, last = 0.0, 1e-7, _common(self.case)["cfl"], wd
        grad = torch.is_grad_enabled() and any(a is not None and a.requires_grad for a in (z, n_el, S))
        for _ in range(self.case["steps"]):
            bz = self.i["amp"] * math.sin(2 * math.pi * t / TIDE_PERIOD)
            args = (S, wd, dt, bz, z, n_el)
            S, wd, last, lam = checkpoint(self.step, *args, use_reentrant=False) if grad else self.step(*args)
            t, dt = t + dt, cfl * self.min_edge / lam
            if each:
                each(S)
        return S, last, t, dt


def _rows(a):
    return a.transpose(-1, -2).reshape(-1)


def exact(case, seed):
    """What run() returns, from the whole-array form above: values, and by automatic
    differentiation the gradients (time steps and decisions held, as the adjoint holds them)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ins = _inputs(case, seed)
    ne = sum(i["mesh"].num_el for i in ins)
    stages = case["steps"] * case["stages"]
    if ne * stages > 1e9 or len(ins) * stages > (500 if case["kind"] == "gradient" else 3000):
        return None  # more than about 20 seconds
    parts = [_Scheme(case, i, dev) for i in ins]
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed, ins, parts)
    with torch.no_grad():
        if case["kind"] == "operators":
            p = parts[0]
            S, _ = p.state()
            wd = p.status(S, p.z, torch.as_tensor(p.i["state"][3], device=dev))
            R, lam = p.rhs1(S, wd if case["land"] else None, 0.0, p.z, p.n_el)
            S = p.positive(p.limit(S, p.z), p.z)
            out = p.status(S, p.z, wd)
            return {"rz": _rows(R[0]), "rx": _rows(R[1]), "ry": _rows(R[2]), "speed": float(lam.max()),
                    "zeta": _rows(S[0]), "qx": _rows(S[1]), "qy": _rows(S[2]), "wd": out}
        done, series = [], []
        if case["gauges"]:
            el, w = (torch.as_tensor(a, device=dev) for a in _gauges(case, ins))
            el = el.long()
        for p in parts:
            see = (lambda S: series.append((S[0][:, el] * w.T).sum(0))) if case["gauges"] else None
            S, wd = p.state()
            done.append(p.evolve(p.z, p.n_el, S, wd, see))
    out = {name: torch.cat([_rows(d[0][v]) for d in done]) for v, name in enumerate(("zeta", "qx", "qy"))}
    out["wd"] = torch.cat([torch.as_tensor(p.i["state"][3], device=dev) if d[1] is None else d[1]
                           for p, d in zip(parts, done)])
    single = not case["least"]
    out["time"] = done[0][2] if single else np.array([d[2] for d in done])
    out["dt"] = done[0][3] if single else np.array([d[3] for d in done])
    out["steps"] = case["steps"] if single else np.full(len(done), case["steps"], dtype=np.int32)
    if series:
        out["gauges"] = torch.stack(series)
    return out


def _exact_gradient(case, seed, ins, parts):
    dev = parts[0].dev
    el, w = _gauges(case, ins)
    target = torch.as_tensor(_target(case, len(el), seed), device=dev)
    off, total = 0, 0.0
    values, grads = [], {k: [] for k in ("n_el", "z", "zeta0", "qx0", "qy0")}
    for p, i in zip(parts, ins):
        mine = (el >= off) & (el < off + p.ne)
        ge, gw = torch.as_tensor(el[mine] - off, device=dev).long(), torch.as_tensor(w[mine], device=dev)
        z, n_el = p.z.clone().requires_grad_(), p.n_el.clone().requires_grad_()
        S, wd = p.state()
        S = S.clone().requires_grad_()
        seen = []
        p.evolve(z, n_el, S, wd, lambda S: seen.append((S[0][:, ge] * gw.T).sum(0)))
        got = torch.stack(seen)
        J = ((got - target[:, torch.as_tensor(mine, device=dev)]) ** 2).sum()
        gn, gz, gs = torch.autograd.grad(J, (n_el, z, S))
        total, off = total + float(J), off + p.ne
        values.append(got.detach())
        for k, g in zip(grads, (gn, gz, _rows(gs[0]), _rows(gs[1]), _rows(gs[2]))):
            grads[k].append(g)
    return {"J": total, "gauges": torch.cat(values, 1), **{k: torch.cat(v) for k, v in grads.items()}}
