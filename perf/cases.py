"""Timed workloads of the shallow-water timestep, one entry per way of calling it.

Each case is one use of the library through its public Python entry points:
a rollout replayed from a captured CUDA graph, single steps, the drop-in
CalculateFlux / UpdateCell pair on reference-layout arrays, the end-to-end
call with host buffers, a batch of scenarios, and the gradient of a gauge
loss.  Meshes are generated here in memory, as a program that has its own
mesh would hand them over (``hb_mesh_desc``): jittered lattices of triangles
(quads among them where the count is odd or the mesh is mixed), with the
boundary codes, depths and bed shapes of the repository's channel and
dam-break configurations.

``exact`` restates the step in 64-bit torch, without the library.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hydro-bench_b200"))

import hydrob200 as hb  # noqa: E402
from hydrob200 import _lib  # noqa: E402
from hydrob200.adjoint import Adjoint, gauge_loss_function  # noqa: E402

HX = 56.0           # lattice spacing (m); two triangles of about 1,544 m^2 per lattice square, as the 207,234-cell channel
HM1, HM2 = 0.001, 0.01


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a coupled program that advances one step at a time on a small mixed mesh with open boundaries: launches count
        {"name": "step_1k5_mixed", "path": "step", "mesh": "mixed", "cells": 1500, "steps": 20,
         "variant": "H", "precision": "fp64", "layout": "edge"},
        # the F1 configuration: 6,675 cells, 100 steps replayed from one graph
        {"name": "graph_f1", "path": "graph", "mesh": "channel", "cells": 6675, "steps": 100,
         "variant": "H", "precision": "fp64", "layout": "edge"},
        # the second reference deck's size with the CFL-limited update variant
        {"name": "graph_24k_variant_f", "path": "graph", "mesh": "channel", "cells": 24021, "steps": 60,
         "variant": "F", "precision": "fp64", "layout": "edge"},
        # the headline configuration: the plain fp64 step at 207,234 cells
        {"name": "graph_207k", "path": "graph", "mesh": "channel", "cells": 207234, "steps": 40,
         "variant": "H", "precision": "fp64", "layout": "edge"},
        # the same mesh in split precision, and an odd mixed mesh in fp32 (tile layout, their recommended form)
        {"name": "graph_207k_split", "path": "graph", "mesh": "channel", "cells": 207234, "steps": 40,
         "variant": "H", "precision": "split", "layout": "tile"},
        {"name": "graph_61k_fp32", "path": "graph", "mesh": "mixed", "cells": 61003, "steps": 40,
         "variant": "H", "precision": "fp32", "layout": "tile"},
        # wetting and drying at the largest size: the fp64 dam break, whose state and terms exceed the L2
        {"name": "graph_dam_2m", "path": "graph", "mesh": "dam", "cells": 2000000, "steps": 20,
         "variant": "H", "precision": "fp64", "layout": "edge"},
        # ... and half a million cells of it in split precision
        {"name": "graph_dam_500k_split", "path": "graph", "mesh": "dam", "cells": 500001, "steps": 20,
         "variant": "H", "precision": "split", "layout": "tile"},
        # an ensemble of uneven scenarios stepped by one launch, split precision
        {"name": "batch_16_split", "path": "batch", "mesh": "channel", "cells": 5000, "most": 50000, "scenarios": 16,
         "steps": 40, "variant": "H", "precision": "split", "layout": "tile"},
        # calibration: loss and gradient (forward and backward) on the 24,020-cell mesh, checkpoints every 10 steps
        {"name": "adjoint_24k", "path": "adjoint", "mesh": "channel", "cells": 24020, "steps": 200, "every": 10,
         "gauges": 50, "variant": "H", "precision": "fp64", "layout": "edge"},
        # the drop-in call pair over the caller's own reference-layout arrays, at the headline size
        {"name": "dropin_207k", "path": "dropin", "mesh": "channel", "cells": 207234, "steps": 5,
         "variant": "H", "precision": "fp64", "layout": "edge"},
        # state kept on the host: one step per call, page-locked buffers in and out
        {"name": "host_207k", "path": "host", "mesh": "channel", "cells": 207234, "steps": 1,
         "variant": "H", "precision": "fp64", "layout": "edge"},
    ]


def draw(rng):
    path = rng.choice(["graph", "graph", "graph", "step", "dropin", "batch", "adjoint", "host"])
    mesh = rng.choice(["channel", "channel", "mixed", "dam"])
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    case = {"path": path, "mesh": mesh, "variant": rng.choice("HHHF"), "precision": "fp64", "layout": "edge"}
    if path == "graph":
        case["precision"] = rng.choice(["fp64", "fp64", "fp32", "split"])
        case["layout"] = "edge" if case["precision"] == "fp64" else rng.choice(["tile", "tile", "edge"])
        case.update(cells=size(1500, 700000), steps=rng.choice([10, 20, 40]))
    elif path == "step":
        case.update(cells=size(1000, 100000), steps=rng.choice([5, 10, 20]))
    elif path == "dropin":
        case["precision"] = rng.choice(["fp64", "fp64", "fp32"])
        case.update(cells=size(2000, 300000), steps=rng.choice([2, 5, 10]))
    elif path == "batch":
        lo = size(1000, 8000)
        case["precision"] = rng.choice(["split", "split", "fp32", "fp64"])
        case["layout"] = "edge" if case["precision"] == "fp64" else "tile"
        case.update(cells=lo, most=lo * rng.choice([4, 10]), scenarios=rng.randint(3, 20), steps=rng.choice([10, 20]))
    elif path == "adjoint":
        case["mesh"] = "channel"
        case["variant"] = "H"
        case.update(cells=size(2000, 40000), steps=rng.choice([50, 100, 150]), every=rng.choice([10, 25, 50]),
                    gauges=rng.randint(5, 60))
    else:
        case.update(cells=size(5000, 300000), steps=rng.choice([1, 1, 4]))
    return case


# ---------------------------------------------------------------------------
# meshes
# ---------------------------------------------------------------------------
def _lattice(kind, cells):
    """(mx, my, quads): 2 mx my - quads cells."""
    aspect = 1.0 if kind == "dam" else 5.0
    squares = cells / 1.5 if kind == "mixed" else cells / 2.0
    my = max(2, int(round(math.sqrt(squares / aspect))))
    mx = max(2, int(math.ceil(squares / my)))
    while 2 * mx * my < cells:
        mx += 1
    return mx, my, 2 * mx * my - cells


class Mesh:
    """A mesh, its tables and its initial state, in reference order: what the
    solver classes take in place of a deck read from files."""

    def __init__(self, kind, cells, seed):
        rng = np.random.default_rng([seed, cells, len(kind)])
        mx, my, quads = _lattice(kind, cells)
        self.cells = cells
        # nodes
        x = np.repeat(np.arange(mx + 1) * HX, my + 1).reshape(mx + 1, my + 1)
        y = np.tile(np.arange(my + 1) * HX, mx + 1).reshape(mx + 1, my + 1)
        x[1:-1, 1:-1] += rng.uniform(-0.15, 0.15, (mx - 1, my - 1)) * HX
        y[1:-1, 1:-1] += rng.uniform(-0.15, 0.15, (mx - 1, my - 1)) * HX
        x[1:-1, [0, -1]] += rng.uniform(-0.15, 0.15, (mx - 1, 2)) * HX
        y[[0, -1], 1:-1] += rng.uniform(-0.15, 0.15, (2, my - 1)) * HX
        x, y = x.ravel(), y.ravel()
        # squares split along one diagonal or the other, `quads` of them kept whole
        n = mx * my
        kind_of = rng.integers(0, 2, n)
        kind_of[rng.permutation(n)[:quads]] = 2
        first = np.concatenate([[0], np.cumsum(np.where(kind_of == 2, 1, 2))])[:-1]
        a = (np.arange(mx)[:, None] * (my + 1) + np.arange(my)[None, :]).ravel()
        b, c, d = a + my + 1, a + my + 2, a + 1
        nodes = np.full((cells, 4), -1, dtype=np.int64)
        # owner cell and slot of each square's south, east, north and west side
        own = np.empty((4, n), dtype=np.int64)
        slot = np.empty((4, n), dtype=np.int64)
        nac = np.zeros((cells, 4), dtype=np.int64)
        for k, (tris, sides, diag) in enumerate([
                ((("a", "b", "c"), ("a", "c", "d")), ((0, 0), (0, 1), (1, 1), (1, 2)), ((0, 2), (1, 0))),
                ((("a", "b", "d"), ("b", "c", "d")), ((0, 0), (1, 0), (1, 1), (0, 2)), ((0, 1), (1, 2))),
                ((("a", "b", "c", "d"),), ((0, 0), (0, 1), (0, 2), (0, 3)), None)]):
            q = np.nonzero(kind_of == k)[0]
            for t, tri in enumerate(tris):
                for s, name in enumerate(tri):
                    nodes[first[q] + t, s] = {"a": a, "b": b, "c": c, "d": d}[name][q]
            for side, (t, s) in enumerate(sides):
                own[side, q] = first[q] + t
                slot[side, q] = s
            if diag:
                (t0, s0), (t1, s1) = diag
                nac[first[q] + t0, s0] = first[q] + t1 + 1
                nac[first[q] + t1, s1] = first[q] + t0 + 1
        g = lambda side: (own[side].reshape(mx, my), slot[side].reshape(mx, my))
        (so, ss), (eo, es), (no, ns), (wo, ws) = g(0), g(1), g(2), g(3)
        for (o0, s0), (o1, s1) in (((eo[:-1], es[:-1]), (wo[1:], ws[1:])), ((no[:, :-1], ns[:, :-1]), (so[:, 1:], ss[:, 1:]))):
            nac[o0, s0] = o1 + 1
            nac[o1, s1] = o0 + 1
        klas = np.zeros((cells, 4))
        west, east = (wo[0], ws[0]), (eo[-1], es[-1])
        south, north = (so[:, 0], ss[:, 0]), (no[:, -1], ns[:, -1])
        for o, s in (west, east, south, north):
            klas[o, s] = 4.0
        if kind != "dam":
            klas[west] = 10.0
            klas[east] = 1.0
            free = rng.permutation(mx - 2)[:min(8, mx - 2)] + 1     # zero-discharge edges on the long side
            klas[south[0][free], south[1][free]] = 10.0
        if kind == "mixed":
            half = np.arange(mx // 3, mx // 2 + 1)                  # an open stretch of the other long side
            klas[north[0][half], north[1][half]] = 5.0
        if kind == "mixed":                                        # numbered without any order
            to = rng.permutation(cells)
            back = np.empty_like(to)
            back[to] = np.arange(cells)
            nodes, klas = nodes[back], klas[back]
            nac = nac[back]
            nac = np.where(nac > 0, to[np.maximum(nac, 1) - 1] + 1, 0)
        # geometry (outward normal (dy, -dx) / L of the edge from node j to node j + 1)
        nv = np.where(nodes[:, 3] < 0, 3, 4)
        nxt = np.concatenate([nodes[:, 1:], nodes[:, :1]], axis=1)
        nxt[nv == 3, 2] = nodes[nv == 3, 0]
        has = np.arange(4)[None, :] < nv[:, None]
        p, q = np.where(has, nodes, 0), np.where(has, nxt, 0)
        dx, dy = np.where(has, x[q] - x[p], 0.0), np.where(has, y[q] - y[p], 0.0)
        side = np.sqrt(dx * dx + dy * dy)
        cosf = np.where(has, dy / np.where(has, side, 1.0), 0.0)
        sinf = np.where(has, -dx / np.where(has, side, 1.0), 0.0)
        area = 0.5 * np.where(has, x[p] * y[q] - x[q] * y[p], 0.0).sum(axis=1)
        cx, cy = np.where(has, x[p], 0.0).sum(axis=1) / nv, np.where(has, y[p], 0.0).sum(axis=1) / nv
        lx, ly = mx * HX, my * HX
        # bed and level
        z = np.zeros(cells)
        if kind == "dam":
            for k in range(1, 9):                                  # rough bed, spectral slope about -2, 5 m relief
                for _ in range(3):
                    kx, ky, ph = rng.normal(0, 1), rng.normal(0, 1), rng.uniform(0, 2 * np.pi)
                    z += np.sin(2 * np.pi * 2 ** (0.5 * k) * (kx * cx / lx + ky * cy / ly) + ph) / 2 ** (0.5 * k)
            zbc = 0.05 + 5.0 * (z - z.min()) / max(z.max() - z.min(), 1e-9)
            level = np.where(cx < 0.5 * lx, 5.0, zbc - 1.0)
            self.dt = 0.5
        else:
            plane = 0.05 + 1e-4 * (lx - cx)
            for _ in range(3):
                bx, by = rng.uniform(0.2, 0.8) * lx, rng.uniform(0.25, 0.75) * ly
                z += np.exp(-((cx - bx) ** 2 + (cy - by) ** 2) / (2.0 * max(300.0, 0.015 * lx) ** 2))
            zbc = plane + 1.0 * z
            level = plane + 2.0 + 0.02 * rng.standard_normal(cells)
            if kind == "mixed":                                    # a high bank that stays dry, a shallow shelf
                zbc = np.where((np.abs(cx - 0.5 * lx) < 0.05 * lx) & (cy > 0.6 * ly), plane + 4.0, zbc)
                shelf = (cx > 0.7 * lx) & (cx < 0.8 * lx) & (cy < 0.3 * ly)
                zbc = np.where(shelf, level - rng.uniform(0.1, 0.3, cells), zbc)
            self.dt = 1.0
        wet = level > zbc
        h = np.where(wet, level - zbc, HM1)
        zz = np.where(wet, level, zbc + HM1)
        u = np.where(wet & (h > HM2), (0.0 if kind == "dam" else 0.5) + 0.05 * rng.standard_normal(cells), 0.0)
        v = np.where(wet & (h > HM2), 0.05 * rng.standard_normal(cells), 0.0)
        manning = rng.uniform(0.02, 0.035, cells)
        self.start = {"H": h, "U": u, "V": v, "Z": zz, "W": np.sqrt(u * u + v * v)}
        # tables: hourly intervals
        ndays = 2 if cells > 400000 else 6
        self.ndays, self.steps_per_day = ndays, int(3600 / self.dt)
        qt, dqt = np.zeros((ndays, cells)), np.zeros((ndays, cells))
        zt, dzt = np.zeros((ndays, cells)), np.zeros((ndays, cells))
        if kind != "dam":
            ins = np.nonzero(((klas == 10.0) & (cx < HX)[:, None]).any(axis=1))[0]
            outs = np.nonzero((klas == 1.0).any(axis=1))[0]
            per = rng.uniform(0.9, 1.3, ndays)
            for t in range(ndays):
                qt[t, ins] = per[t] * HX
                dqt[t, ins] = 1e-5 * HX
                zt[t, outs] = 2.05 + 0.02 * t
                dzt[t, outs] = 1e-6
        flat = lambda w: np.ascontiguousarray(w, dtype=np.float64).reshape(-1)
        self.arrays = dict(nac=flat(nac), klas=flat(klas), side=flat(side), cosf=flat(cosf), sinf=flat(sinf),
                           slcos=flat(side * cosf), slsin=flat(side * sinf), zbc=flat(zbc), zb1=flat(zbc + HM1), area=flat(area),
                           fnc=flat(9.81 * manning * manning), bfeat=np.zeros(cells), zw=np.zeros(0), qw=np.zeros(0),
                           qt=qt.reshape(-1), dqt=dqt.reshape(-1), zt=zt.reshape(-1), dzt=dzt.reshape(-1))
        self.arrays["nhq1"] = np.zeros(cells, dtype=np.int32)
        m = _lib.MeshDesc()
        m.cells, m.ndays, m.nhq, m.steps_per_day = cells, ndays, 0, self.steps_per_day
        m.dt, m.hm1, m.hm2, m.jl = self.dt, HM1, HM2, 0.0
        for k, w in self.arrays.items():
            setattr(m, k, w.ctypes.data_as(ctypes.POINTER(ctypes.c_int32 if k == "nhq1" else ctypes.c_double)))
        self.mesh = m

    def array(self, name):
        return self.arrays[name]

    def state(self):
        return self.start

    @property
    def limit(self):
        """Steps that the boundary tables cover."""
        return self.ndays * (self.steps_per_day - 1)


def _meshes(case, seed):
    if case["path"] != "batch":
        return [Mesh(case["mesh"], case["cells"], seed)]
    rng = np.random.default_rng([seed, 77])
    # the scenario sizes belong to the case, the meshes themselves to the seed
    sizes = np.exp(np.random.default_rng(case["cells"] * 31 + case["scenarios"]).uniform(
        math.log(case["cells"]), math.log(case["most"]), case["scenarios"])).round().astype(int)
    return [Mesh(case["mesh"], int(n), int(rng.integers(1 << 30))) for n in sizes]


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _problem(case, mesh, seed):
    """Gauges, observations and parameters of a calibration."""
    rng = np.random.default_rng([seed, 5])
    gauges = np.sort(rng.choice(mesh.cells, case["gauges"], replace=False)).astype(np.int32)
    obs = mesh.start["H"][gauges][None, :] + 0.05 * rng.standard_normal((case["steps"] // 10, case["gauges"]))
    manning = rng.uniform(0.02, 0.035, mesh.cells)
    return gauges, obs, manning, mesh.array("zbc") + 0.01 * rng.standard_normal(mesh.cells)


def prepare(case, seed):
    meshes = _meshes(case, seed)
    opts = dict(variant=case["variant"], precision=case["precision"])
    state = {"case": case, "steps": case["steps"], "limit": min(m.limit for m in meshes)}
    path = case["path"]
    if path == "dropin":
        state["mesh"] = hb.RefLayoutMesh(meshes[0], **opts)
        return state
    if path == "adjoint":
        gauges, obs, manning, zbc = _problem(case, meshes[0], seed)
        adj = Adjoint(meshes[0], gauges, 10, case["steps"], case["every"])
        adj.set_observations(obs)
        state.update(adjoint=adj, loss=gauge_loss_function().apply,
                     n=torch.tensor(manning, requires_grad=True), zbc=torch.tensor(zbc, requires_grad=True))
        return state
    if path == "batch":
        s = hb.Batch(meshes, layout=case["layout"], **opts)
        perm, at = [], 0
        for i, m in enumerate(meshes):
            perm.append(s.permutation(i).astype(np.int64) + at)
            at += m.cells
        perm = np.concatenate(perm)
    else:
        s = hb.Solver(meshes[0], layout=case["layout"], **opts)
        perm = s.permutation().astype(np.int64)
    state["solver"] = s
    if path == "host":
        block = torch.empty(4, meshes[0].cells, dtype=torch.float64, pin_memory=True)
        for k, name in enumerate("HUVZ"):
            block[k] = torch.from_numpy(meshes[0].start[name])
        state["block"] = block
        return state
    where = np.empty_like(perm)
    where[perm] = np.arange(perm.size)
    state["where"] = 4 * torch.as_tensor(where, device="cuda")[:, None] + torch.arange(4, device="cuda")   # device place of each value
    if path in ("graph", "batch"):
        s.capture_graph(case["steps"])
    return state


class _Records:
    """The state records that begin at the view of H, as an array [C][4]."""

    def __init__(self, h):
        self.__cuda_array_interface__ = {"shape": (h.shape[0], 4), "typestr": "<f%d" % h.element_size(),
                                         "data": (h.data_ptr(), False), "version": 3}


def _read(state):
    """The state [C][4] in reference order: {H, U, V, Z} ({H, U, V, H_lo} in split precision), a copy on the device."""
    h = state["solver"].device_state()["H"]
    return torch.as_tensor(_Records(h), device="cuda").view(-1)[state["where"]]


def run(state):
    path, n = state["case"]["path"], state["steps"]
    if path == "dropin":
        m = state["mesh"]
        if m.steps_done + n > state["limit"]:
            m.steps_done = 0                       # the tables start over
        m.run(n)
        return {k: m.T[k] for k in ("H", "U", "V", "W", "Z", "FLUX0", "FLUX1", "FLUX2", "FLUX3")}
    if path == "adjoint":
        loss = state["loss"](state["n"], state["zbc"], state["adjoint"])
        gn, gz = torch.autograd.grad(loss, (state["n"], state["zbc"]))
        return {"loss": loss.detach(), "grad_n": gn, "grad_zbc": gz}
    s = state["solver"]
    if s.position[0] + n > state["limit"]:
        s.set_position(0)
    if path == "host":
        b = state["block"]
        s.step_host(b[0], b[1], b[2], b[3], None, n)
        s.sync()
        return b
    if path == "step":
        for _ in range(n):
            s.step(1)
    else:
        s.graph_launch()
    return _read(state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _sizes(case):
    """(cells, unique edges) of the case's meshes."""
    if case["path"] == "batch":
        sizes = np.exp(np.random.default_rng(case["cells"] * 31 + case["scenarios"]).uniform(
            math.log(case["cells"]), math.log(case["most"]), case["scenarios"])).round().astype(int)
    else:
        sizes = [case["cells"]]
    cells = edges = 0
    for n in sizes:
        mx, my, quads = _lattice(case["mesh"], int(n))
        cells += int(n)
        edges += mx * (my + 1) + my * (mx + 1) + mx * my - quads
    return cells, edges


def work(case):
    """Per step: the state in and out, AREA, ZBC and FNC per cell; two cell
    ids, a code byte, SIDE, COSF and SINF per unique edge.  About 90
    operations per edge and 45 per cell (a square root, power or division
    counted as one).  A gradient needs a forward and, by the operations of a
    reverse sweep, about twice as much again."""
    w = 8 if case["precision"] == "fp64" else 4
    cells, edges = _sizes(case)
    n = case["steps"]
    if case["path"] == "dropin":          # the pair also leaves the fluxes and W, and codes and ids are reals
        slots = 4 * cells
        step = cells * (13 * w) + slots * (2 * w + 3 * w + 4 * w)
        return {"bytes": n * step, "flops": n * (90 * edges + 45 * cells)}
    if case["path"] == "host":
        return {"bytes": n * (12 * w * cells + edges * (9 + 3 * w)) + 2 * 32 * cells, "flops": n * (90 * edges + 45 * cells)}
    step = 12 * w * cells + edges * (9 + 3 * w)
    if case["path"] == "adjoint":
        return {"bytes": 3 * n * step, "flops": 3 * n * (90 * edges + 45 * cells)}
    return {"bytes": n * step, "flops": n * (90 * edges + 45 * cells)}


# ---------------------------------------------------------------------------
# the step in 64-bit torch
# ---------------------------------------------------------------------------
class Step64:
    """CalculateFlux and UpdateCell restated in float64 torch, differentiable
    with the branches frozen where the state put them."""

    def __init__(self, mesh, variant, device, zbc=None, fnc=None):
        t = lambda k: torch.as_tensor(mesh.array(k), device=device)
        four = lambda k: t(k).view(-1, 4)
        self.variant, self.dt = variant, mesh.dt
        self.cells, self.per_day, self.ndays = mesh.cells, mesh.steps_per_day - 1, mesh.ndays
        self.zbc = t("zbc") if zbc is None else zbc
        self.fnc = t("fnc") if fnc is None else fnc
        self.area = t("area")
        self.klas, self.side = four("klas"), four("side")
        self.cos, self.sin = four("cosf"), four("sinf")
        nac = four("nac").long() - 1
        self.has = nac >= 0
        self.nb = nac.clamp(min=0)
        self.first = torch.arange(self.cells, device=device)[:, None] < nac
        self.tables = {k: t(k).view(mesh.ndays, -1) for k in ("qt", "dqt", "zt", "dzt")}
        edges = self.klas != 0
        self.rows, self.cols = torch.nonzero(edges, as_tuple=True)

    def osher(self, hl, hr, ql1, ql2, qr1, qr2, cl):
        fil = ql1 + 2 * cl
        cr = (9.81 * hr).sqrt()
        fir = qr1 - 2 * cr
        ua, ca = (fil + fir) / 2, ((fil - fir) / 4).abs()
        k2 = torch.where(ca < ua, 1, torch.where(ua >= 0, 2, torch.where(ua >= -ca, 3, 4)))
        k1 = torch.where(qr1 >= -cr, torch.where(ql1 < cl, 1, 2), torch.where(ql1 < cl, 3, 4))
        out = [0, 0, 0, 0]

        def add(on, sign, h, u, v):
            f = torch.where(on, 1.0, 0.0).to(h.dtype) * sign
            out[0] = out[0] + f * h * u
            out[1] = out[1] + f * h * u * u
            out[2] = out[2] + f * h * u * v
            out[3] = out[3] + f * 4.905 * h * h

        odd, even = (k1 == 1) | (k1 == 3), (k1 == 2) | (k1 == 4)
        add(even, 1.0, hl, ql1, ql2)
        us = fil / 3
        add(torch.where(k2 == 1, odd, even), torch.where(k2 == 1, 1.0, -1.0), us * us / 9.81, us, ql2)
        add(k2 == 2, 1.0, (fil - ua) ** 2 / 39.24, ua, ql2)
        fir5 = fir - ua
        add(k2 == 3, 1.0, fir5 ** 2 / 39.24, ua, qr2)
        us = torch.where(k2 == 3, fir5, fir) / 3
        add(torch.where(k2 == 4, k1 <= 2, k1 >= 3), torch.where(k2 == 4, 1.0, -1.0), us * us / 9.81, us, qr2)
        add(k1 >= 3, 1.0, hr, qr1, qr2)
        return out

    def boundary(self, kt, jt, h, u, v):
        """The four fluxes of the slots with a code, [n] each."""
        r, c = self.rows, self.cols
        k, side, cs, sn = self.klas[r, c], self.side[r, c], self.cos[r, c], self.sin[r, c]
        h, u, v, zbc = h[r], u[r], v[r], self.zbc[r]
        ql1, ql2 = u * cs + v * sn, v * cs - u * sn
        cl = (9.81 * h).sqrt()
        press = 4.905 * h * h
        # given discharge
        q = -(self.tables["qt"][jt][r] + self.tables["dqt"][jt][r] * kt) / side
        fil, hb, hb0, live = ql1 + 2 * cl, h, h, k == 10
        for _ in range(20):
            w = fil - q / hb0
            new = w * w / 39.24
            hb = torch.where(live, new, hb)
            live = live & ((hb0 - new).abs() > 0.005)
            hb0 = torch.where(live, (hb0 + new) / 2, hb0)
        f10 = [q, torch.where(hb <= 1, torch.zeros_like(q), q * q / hb), torch.zeros_like(q), 4.905 * hb * hb]
        # given level
        mult = kt if self.variant == "F" else jt
        hb1 = (self.tables["zt"][jt][r] + self.tables["dzt"][jt][r] * mult - zbc)
        hb1 = torch.where((k == 1) & (hb1 > HM2), hb1, torch.full_like(hb1, HM2))
        fial, ur0, urb, live = ql1 + 6.264 * h.sqrt(), ql1, ql1, k == 1
        for _ in range(30):
            fiar = urb - 6.264 * hb1.sqrt()
            new = (fial + fiar) * (fial - fiar) ** 2 / hb1 / 313.92
            urb = torch.where(live, new, urb)
            live = live & ((new - ur0).abs() > 0.0001)
            ur0 = torch.where(live, new, ur0)
        along = torch.where(ql1 > 0, h * ql1 * ql2, torch.zeros_like(h))
        f1 = [hb1 * urb, hb1 * urb * urb, along, 4.905 * hb1 * hb1]
        # wall; open
        zero = torch.zeros_like(h)
        f4 = [zero, zero, zero, press]
        out = torch.where(ql1 > 0, ql1, zero)
        f5 = [h * out, h * out * out, along, press]
        fast = (ql1 > cl) if self.variant == "F" else (ql1 > cl) & (h < HM2)
        ff = [h * ql1, h * ql1 * ql1, h * ql1 * ql2, press]
        pick = lambda i: torch.where(fast, ff[i], torch.where(k == 10, f10[i], torch.where(k == 1, f1[i], torch.where(k == 4, f4[i], f5[i]))))
        return [pick(i) for i in range(4)]

    def flux(self, step, h, u, v, z):
        kt, jt = 1 + step % self.per_day, step // self.per_day
        zbc, cs, sn, has, nb = self.zbc, self.cos, self.sin, self.has, self.nb
        C1 = 1.7
        one = lambda w: w[:, None].expand(-1, 4)
        h1, u1, v1, z1, b1 = one(h), one(u), one(v), one(z), one(zbc)
        ql1, ql2 = u1 * cs + v1 * sn, v1 * cs - u1 * sn
        zi = torch.where(z1 > b1 + HM1, z1, b1 + HM1)
        zero = torch.zeros_like(h1)
        there = lambda w: torch.where(has, w[nb], zero)
        hn, uc, vc, bc, zn = there(h), there(u), there(v), there(zbc), there(z)
        hc = torch.where(has, torch.where(hn > HM1, hn, torch.full_like(hn, HM1)), zero)
        zc = torch.where(bc > zn, bc, zn)
        # Osher across the edge, from the lower-numbered cell
        lo = self.first | ~has
        pick = lambda p, q: torch.where(lo, p, q)
        one_ = torch.ones_like(h1)
        hR, uR, vR = pick(torch.where(has, hn, one_), h1), pick(uc, u1), pick(vc, v1)
        hL, uL, vL, bL = pick(h1, torch.where(has, hn, one_)), pick(u1, uc), pick(v1, vc), pick(b1, bc)
        zR, bR = pick(torch.where(has, zn, z1), z1), pick(bc, b1)
        sg = torch.where(lo, 1.0, -1.0).to(h1.dtype)
        c, s = cs * sg, sn * sg
        hcR = torch.where(hR > HM1, hR, torch.full_like(hR, HM1))
        top = torch.where(bR > zR, bR, zR) - bL
        qr0 = torch.where(top > HM1, top, torch.full_like(top, HM1))
        ur = uR * c + vR * s
        ratio = hcR / qr0
        ratio = torch.where(ratio < 1.5, ratio, torch.full_like(ratio, 1.5))
        thin = (hcR <= HM2) | (qr0 <= HM2)
        qr1 = torch.where(thin, torch.copysign(torch.full_like(ur, 0.001), ur.detach()), ur * ratio)
        o = self.osher(hL, qr0, uL * c + vL * s, vL * c - uL * s, qr1, vR * c - uR * s, (9.81 * hL).sqrt())
        o1 = o[1] + (1 - ratio) * hcR * ur * ur / 2
        ok = o[3] > 0
        za = torch.where(ok, torch.where(ok, o[3], one_) / 4.905, one_).sqrt() * ok + bL
        h3 = torch.where(za > b1, za - b1, zero)
        f = [o[0] * sg, o1, o[2], torch.where(lo, o[3], 4.905 * h3 * h3)]
        # the chain before it
        p = 4.905 * h1 * h1
        pos = lambda w: torch.where(w > HM1, w, torch.full_like(w, HM1))
        p15 = lambda w: pos(w) ** 1.5

        def put(on, g):
            for i in range(4):
                f[i] = torch.where(on, g[i], f[i])

        dh = pos(zi - bc)
        un, hc1 = C1 * dh.sqrt(), zc - b1
        thinR = hc <= HM2
        put(thinR, [-C1 * p15(hc), h1 * ql1 * ql1, zero, p])
        put(thinR & (zi > zc), [dh * un, dh * un * un, dh * un * ql2, 4.905 * hc1 * hc1])
        dh = pos(zc - b1)
        un = -C1 * dh.sqrt()
        thinL = h1 <= HM2
        put(thinL, [C1 * p15(h1), zero, zero, p])
        put(thinL & (zc > zi), [dh * un, dh * un * un, dh * un * (vc * cs - uc * sn), p])
        put(zc <= b1, [C1 * p15(h1), h1 * ql1.abs() * ql1, h1 * ql1.abs() * ql2, zero])
        put(zi <= bc, [-C1 * p15(hc), h1 * ql1 * ql1.abs(), zero, p])
        put((h1 <= HM1) & (hc <= HM1), [zero] * 4)
        b = self.boundary(kt, jt, h, u, v)
        return [f[i].index_put((self.rows, self.cols), b[i]) for i in range(4)]

    def step(self, step, h, u, v, z):
        f = self.flux(step, h, u, v, z)
        fr = f[1] + f[3]
        sc, ss = self.side * self.cos, self.side * self.sin
        wh = (self.side * f[0]).sum(1)
        wu = (sc * fr - ss * f[2]).sum(1)
        wv = (ss * fr + sc * f[2]).sum(1)
        if self.variant == "F":
            s = self.side
            tri = s[:, 3] == 0
            mid = torch.minimum((s[:, 0] + s[:, 2]) / 2, (s[:, 1] + s[:, 3]) / 2)
            ph = (s[:, 0] + s[:, 1] + s[:, 2]) / 2
            inr = ((ph - s[:, 0]) * (ph - s[:, 1]) * (ph - s[:, 2]) / ph).clamp(min=0).sqrt()
            dt2 = torch.where(tri, inr, mid) / (u + (9.81 * h.clamp(min=HM1)).sqrt())
            dta = dt2.clamp(max=self.dt).clamp(min=self.dt / 10) / self.area
            cap = 5.0
        else:
            dta, cap = self.dt / self.area, 15.0
        new = h - dta * wh
        h2 = torch.where(new > HM1, new, torch.full_like(new, HM1))
        s2 = u * u + v * v
        sq = torch.where(s2 > 0, torch.where(s2 > 0, s2, torch.ones_like(s2)).sqrt(), torch.zeros_like(s2))
        dtw = self.dt * self.fnc * sq / h ** 0.33333
        lim = lambda w: torch.where(w.abs() < cap, w, torch.copysign(torch.full_like(w, cap), w.detach()))
        u2 = lim((h * u - dta * wu - dtw * u) / h2)
        v2 = lim((h * v - dta * wv - dtw * v) / h2)
        small = lambda w: torch.where(w.abs() < 0.001, w, torch.copysign(torch.full_like(w, 0.001), w.detach()))
        zero = torch.zeros_like(u)
        u2 = torch.where(h2 <= HM1, zero, torch.where(h2 <= HM2, small(u), u2))
        v2 = torch.where(h2 <= HM1, zero, torch.where(h2 <= HM2, small(v), v2))
        return (h2, u2, v2, h2 + self.zbc), f


def _gradient64(case, mesh, seed, device):
    gauges, obs, manning, zbc = _problem(case, mesh, seed)
    t = lambda w: torch.as_tensor(w, device=device)
    gauges, obs = t(gauges.astype(np.int64)), t(obs)
    n, b = t(manning).requires_grad_(), t(zbc).requires_grad_()

    def begin():
        z0 = t(mesh.start["Z"])
        wet = z0 > b.detach()
        return (torch.where(wet, z0 - b, torch.full_like(b, HM1)), t(mesh.start["U"]), t(mesh.start["V"]), torch.where(wet, z0, b + HM1))

    def advance(s, t0, t1):
        m = Step64(mesh, case["variant"], device, b, 9.81 * n * n)
        loss = torch.zeros((), dtype=torch.float64, device=device)
        for k in range(t0, t1):
            s, _ = m.step(k, *s)
            if (k + 1) % 10 == 0:
                loss = loss + ((s[0][gauges] - obs[(k + 1) // 10 - 1]) ** 2).sum()
        return s, loss

    cuts = list(range(0, case["steps"], 10)) + [case["steps"]]
    saved, total = [], 0.0
    with torch.no_grad():
        s = begin()
        for t0, t1 in zip(cuts, cuts[1:]):
            saved.append(s)
            s, loss = advance(s, t0, t1)
            total += float(loss)
    gn, gz = torch.zeros_like(n), torch.zeros_like(b)
    bar = [torch.zeros_like(w) for w in s]
    for (t0, t1), s in zip(reversed(list(zip(cuts, cuts[1:]))), reversed(saved)):
        s = begin() if t0 == 0 else tuple(w.detach().requires_grad_() for w in s)
        end, loss = advance(s, t0, t1)
        whole = loss + sum((w * g).sum() for w, g in zip(end, bar))
        ins = [n, b] + ([] if t0 == 0 else list(s))
        got = torch.autograd.grad(whole, ins, allow_unused=True)
        got = [torch.zeros_like(i) if g is None else g for i, g in zip(ins, got)]
        gn, gz, bar = gn + got[0], gz + got[1], got[2:]
    return {"loss": torch.tensor(total, dtype=torch.float64), "grad_n": gn.cpu(), "grad_zbc": gz.cpu()}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    meshes = _meshes(case, seed)
    if case["path"] == "adjoint":
        return _gradient64(case, meshes[0], seed, device)
    outs = []
    with torch.no_grad():
        for mesh in meshes:
            m = Step64(mesh, case["variant"], device)
            s = tuple(torch.as_tensor(mesh.start[k], device=device) for k in "HUVZ")
            for k in range(case["steps"]):
                s, f = m.step(k, *s)
            if case["path"] == "dropin":
                got = dict(zip("HUVZ", s))
                got["W"] = (s[1] ** 2 + s[2] ** 2).sqrt()
                got.update({"FLUX%d" % i: f[i].reshape(-1) for i in range(4)})
                return {k: w.cpu() for k, w in got.items()}
            if case["path"] == "host":
                return torch.stack(s).cpu()
            if case["precision"] == "split":        # the depth as the sum of two fp32 numbers
                outs.append(torch.stack([s[0].float().double(), s[1], s[2], s[0] - s[0].float().double()], dim=1))
            else:
                outs.append(torch.stack(s, dim=1))
    return torch.cat(outs).cpu()
