"""The work a user has this library do, as measured cases.

Each propagate case is one job through the C ABI as bench.py and the
integration notes use it: the initial fields of every case of a handle go in
from page-locked host arrays, the solver takes its steps, the final fields
come back into page-locked arrays.  The other cases are the reference's
functions one at a time (a program that keeps the reference's own loop) and
the update on device arrays that the caller owns.

A handle (mesh layout, device memory) is what a program sets up once and
keeps; the fields are the inputs, made from the seed.  FP64 results come back
as the library gives them.  The mixed path keeps its primitives in FP32 and
widens them on download, so its fields are stored in single precision here,
which loses nothing.

`exact` is the same job in plain torch, in 64 bits: reconstruction, limiters,
fluxes, boundary states, viscous source, update and node averages written
from the formulas, over the same meshes.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()


# ------------------------------------------------------------------ cases


def _case(name, call, flow, nodes, steps, *, precision="f64", count=1, loop="tile", flux="ausm", limiter="minmod",
          viscous=False, quads=False, dt_mode=2):
    return {"name": name, "call": call, "flow": flow, "nodes": nodes, "steps": steps, "precision": precision,
            "count": count, "loop": loop, "flux": flux, "limiter": limiter, "viscous": viscous, "quads": quads,
            "dt_mode": dt_mode}


def listed():
    return [
        # a small mesh stepped one call at a time, the statistics looked at
        # after each (a convergence loop): launches and call overhead
        _case("square33 f64 step by step", "steps", "square", 33, 16),
        # the plain inviscid square of the benchmark's first configuration
        _case("square101 f64", "propagate", "square", 101, 96),
        # the same loop with the Roe flux and another limiter, an odd size
        _case("square267 f64 roe", "propagate", "square", 267, 48, flux="roe", limiter="vanalbada"),
        # the reference's own Taylor-Green box: quads, its viscous term, its
        # analytic ghost states, its fixed time step
        _case("tgvbox161 f64 quads", "propagate", "tgv_box", 161, 64, viscous=True, quads=True, dt_mode=0),
        # an ordinary viscous cylinder
        _case("cylinder273 f64", "propagate", "cylinder", 273, 48, limiter="venkat", viscous=True),
        # what a C or Julia caller without a launch record gets: the
        # cell-centred loop
        _case("cylinder257 f64 cell loop", "propagate", "cylinder", 257, 32, limiter="venkat", viscous=True,
              loop="cell"),
        # the headline: the 2.09M-cell viscous cylinder, both precisions
        _case("cylinder1025 f64", "propagate", "cylinder", 1025, 64, limiter="venkat", viscous=True),
        _case("cylinder1025 mixed", "propagate", "cylinder", 1025, 128, precision="mixed", limiter="venkat",
              viscous=True),
        # a parameter sweep in one handle: Taylor-Green vortices of several sizes
        _case("tgv batch10 mixed", "propagate", "tgv", 257, 64, precision="mixed", count=10, viscous=True),
        # a small mesh in mixed precision
        _case("square135 mixed", "propagate", "square", 135, 96, precision="mixed"),
        # the reference's functions one at a time, its loop kept by the caller
        _case("stages cylinder129 f64", "stages", "cylinder", 129, 4, limiter="venkat", viscous=True),
        # updateVariablesSA with residuals on the caller's own device arrays
        _case("update 4194301 cells", "update", "none", 4194301, 2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(["f64", "f64", "mixed"])
    loop = rng.choice(["tile", "tile", "tile", "cell"])
    flow = rng.choice(["square", "square", "cylinder", "cylinder", "tgv", "tgv_box", "stages", "update"])
    steps = _log_int(rng, 4, 100)
    if flow == "update":
        c = _case("", "update", "none", _log_int(rng, 1000, 12_000_000), 2)
    elif flow == "stages":
        c = _case("", "stages", "cylinder", _log_int(rng, 97, 300), rng.randint(1, 6), limiter="venkat", viscous=True)
    elif flow == "square":
        c = _case("", rng.choice(["propagate", "propagate", "steps"]), "square", _log_int(rng, 17, 500), steps,
                  precision=precision, loop=loop, flux=rng.choice(["ausm", "ausm", "roe", "ausm_m2020"]),
                  limiter=rng.choice(["minmod", "minmod", "vanleer", "vanalbada", "none", "venkat"]),
                  dt_mode=rng.choice([1, 2]))
    elif flow == "cylinder":
        c = _case("", "propagate", "cylinder", _log_int(rng, 97, 600), steps, precision=precision, loop=loop,
                  count=rng.choice([1, 1, 3]), limiter=rng.choice(["venkat", "venkat", "minmod"]),
                  viscous=rng.random() < 0.75)
    elif flow == "tgv":
        c = _case("", "propagate", "tgv", _log_int(rng, 33, 400), steps, precision=precision, loop=loop,
                  count=rng.choice([1, 2, 5]), viscous=True)
    else:
        c = _case("", "propagate", "tgv_box", _log_int(rng, 33, 300), steps, precision=precision, loop=loop,
                  viscous=True, quads=rng.random() < 0.5, dt_mode=0)
    del c["name"]
    return c


# ----------------------------------------------------------------- inputs


@functools.lru_cache(maxsize=64)
def _flow(flow, nodes, index, flux, limiter, viscous, quads, dt_mode):
    """Mesh, configuration and smooth initial fields of one case (no seed)."""
    if flow == "cylinder":
        r = np.random.default_rng(1000 + index)
        mach, re, rad = (3.5, 1.0e4, 0.5) if index == 0 else (r.uniform(2.0, 4.0), r.uniform(2e3, 2e4),
                                                              r.uniform(0.35, 0.7))
        mesh, cfg, prims = pkg.cases.cylinder_case(nodes, mach=float(mach), re_d=float(re), radius=float(rad),
                                                   flux=flux, limiter=limiter, viscous=viscous)
        # gas at rest at the wall, the stream a diameter away: the impulsive
        # start empties the wake of some staircase walls below zero pressure
        d = np.maximum(np.hypot(mesh.cell_mid_points[:, 0], mesh.cell_mid_points[:, 1]) - rad, 0.0)
        prims = (prims[0], prims[1] * -np.expm1(-d * d), prims[2], prims[3])
    elif flow == "tgv":
        r = np.random.default_rng(2000 + index)
        mesh, cfg, prims = pkg.cases.tgv_case(nodes, float(r.uniform(0.1, 0.5)), float(r.uniform(100.0, 1600.0)),
                                              flux=flux, limiter=limiter)
    else:
        mesh, cfg, prims = pkg.cases.reference_tgv_case(nodes, quads=quads)
        # a fixed step of CFL about 0.3 on this mesh, so that the fields move
        cfg = dict(cfg, dt=0.1 * 2.0 * math.pi / (nodes - 1) / 420.0)
    return mesh, dict(cfg, dt_mode=dt_mode), prims


def _sizes(case):
    """Nodes per side of each case of the handle: from the largest down."""
    n, k = case["nodes"], case["count"]
    least = 97 if case["flow"] == "cylinder" else 17
    return [max(least, int(round(n * (1.0 - 0.7 * i / k)))) for i in range(k)]


def _inputs(case, seed):
    """[(mesh, cfg, (rho, u, v, p))] of the handle's cases."""
    out = []
    for i, n in enumerate(_sizes(case)):
        if case["flow"] == "square":
            mesh, cfg, prims = pkg.cases.square_inviscid(n, seed=seed + i, flux=case["flux"], limiter=case["limiter"])
            # the reference's tau goes by the longest edge of the mesh: a
            # smaller CFL number gives a step of the same length
            cfl = 0.08 if case["dt_mode"] == 1 else cfg["CFL"]
            out.append((mesh, dict(cfg, dt_mode=case["dt_mode"], CFL=cfl), prims))
            continue
        mesh, cfg, (rho, u, v, p) = _flow(case["flow"], n, i, case["flux"], case["limiter"], case["viscous"],
                                          case["quads"], case["dt_mode"])
        # a smooth disturbance of half a percent
        rng = np.random.default_rng([seed, i])
        x, y = mesh.cell_mid_points[:, 0], mesh.cell_mid_points[:, 1]
        e = [0.005 * np.sin(kx * x + ky * y + ph) for kx, ky, ph in
             zip(rng.uniform(0.5, 2.0, 2), rng.uniform(0.5, 2.0, 2), rng.uniform(0.0, 2.0 * math.pi, 2))]
        out.append((mesh, cfg, (rho * (1.0 + e[0]), u, v, p * (1.0 + e[1]))))
    return out


def _update_inputs(case, seed):
    """Two conservative states (4 x n each, the columns of an n x 4 matrix)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    n = case["nodes"]
    x = torch.rand((2, 4, n), generator=g, device=dev, dtype=torch.float64)
    U = torch.empty_like(x)
    U[:, 0] = 0.8 + 0.4 * x[:, 0]
    U[:, 1] = U[:, 0] * (2.0 + 0.2 * x[:, 1])
    U[:, 2] = U[:, 0] * (0.2 * x[:, 2] - 0.1)
    U[:, 3] = (0.6 + 0.3 * x[:, 3]) / 0.4 + 0.5 * (U[:, 1] ** 2 + U[:, 2] ** 2) / U[:, 0]
    return U[0].contiguous(), U[1].contiguous()


def _pinned(shape, dtype=torch.float64):
    return torch.zeros(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    if case["call"] == "update":
        a, b = _update_inputs(case, seed)
        return {"case": case, "new": (a, b), "old": torch.zeros_like(a), "prims": torch.zeros_like(a),
                "stats": torch.zeros(6, dtype=torch.float64, device=a.device)}
    inputs = _inputs(case, seed)
    solver = pkg.setupSolver([m for m, _, _ in inputs], [c for _, c, _ in inputs], precision=case["precision"],
                             loop=case["loop"])
    st = {"case": case, "solver": solver, "fields": [], "cells": [], "nodes": [], "out": []}
    for mesh, cfg, prims in inputs:
        f = _pinned((4, mesh.nCells))
        for k in range(4):
            f[k] = torch.from_numpy(prims[k])
        st["fields"].append(f)
        st["cells"].append(_pinned((4, mesh.nCells)))
        st["nodes"].append(_pinned((4, mesh.nNodes)))
        if case["precision"] == "mixed":
            st["out"].append((torch.zeros((4, mesh.nCells)), torch.zeros((4, mesh.nNodes))))
    st["dt"] = [float(c.get("dt", 0.0)) for _, c, _ in inputs]
    return st


def _stats_row(s, dtype):
    return np.array([s["dt"], s["tau"], s["velmax"], *s["residual"], s["rhoMin"], s["rhoMax"], *s["totals"], s["Ek"]],
                    dtype=dtype)


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


STAGE_DT = 1.0e-6  # the time step of the loop that the caller keeps (cylinder)


def run(state):
    case = state["case"]
    if case["call"] == "update":
        lib = pkg._native.load()
        stream = torch.cuda.current_stream().cuda_stream if torch.cuda.is_available() else None
        for u in state["new"]:  # two steps of the caller's loop
            pkg._native.check(lib.gd2d_update_variables_noalloc(u.data_ptr(), state["old"].data_ptr(),
                                                                state["prims"].data_ptr(), case["nodes"], 1.4,
                                                                state["stats"].data_ptr(), stream))
        return {"uold": state["old"], "prims": state["prims"], "stats": state["stats"]}
    s = state["solver"]
    for i, f in enumerate(state["fields"]):
        s.createFields2d(i, *[f[k].numpy() for k in range(4)])
    if case["call"] == "stages":
        t = 0.0
        for _ in range(case["steps"]):
            diff = s.calcDiffTerm(0)
            flux, unew = s.calcOneStageMUSCLcpuFast(0, 1.0, STAGE_DT, t)
            delta = s.updateVariablesSA(0)
            s.cells2nodesSolutionReconstructionWithStencils()
            t += STAGE_DT
        return {"diff": diff, "flux": flux, "unew": unew, "delta": delta, "nodes": _read(s, 0, state)[1]}
    mixed = case["precision"] == "mixed"
    if case["call"] == "steps":
        for _ in range(case["steps"]):
            stats = s.propagate2d(1)
    else:
        stats = s.propagate2d(case["steps"])
    kind = np.float32 if mixed else np.float64
    out = {"stats": [_stats_row(x, kind) for x in stats], "cells": [], "nodes": []}
    for i in range(len(state["fields"])):
        cells, nodes = _read(s, i, state)
        if mixed:
            c, n = state["out"][i]
            cells, nodes = c.copy_(cells), n.copy_(nodes)
        out["cells"].append(cells)
        out["nodes"].append(nodes)
    return out


def _read(s, i, state):
    """The case's fields into its page-locked arrays: FP64 conservatives
    (mixed: primitives) of the cells, primitives of the nodes."""
    mixed = state["case"]["precision"] == "mixed"
    cells, nodes = state["cells"][i], state["nodes"][i]
    pkg._native.check(s.L.gd2d_get_state(s.h, i, None if mixed else _dp(cells), _dp(cells) if mixed else None,
                                         _dp(nodes)), s.h)
    return cells, nodes


# ------------------------------------------------------------------- work

# Bytes a cell and step cannot do without (state read and written, face
# geometry, connectivity, cluster data; intermediates none), and operations:
# 1.5 faces a cell of reconstruction, eight limiters and a flux, the update,
# the node averages, and with viscosity two Green-Gauss gradients.
BYTES = {("f64", False): 216, ("f64", True): 248, ("mixed", False): 164, ("mixed", True): 192}
FLOPS = {False: 450, True: 650}


def _cells(case):
    total = 0
    for n in _sizes(case):
        total += (n - 1) ** 2 * (1 if case["quads"] else 2)
    return total


def work(case):
    if case["call"] == "update":
        return {"bytes": 2.0 * 16 * 8 * case["nodes"], "flops": 2.0 * 40 * case["nodes"]}
    n = _cells(case)
    b = n * case["steps"] * BYTES[case["precision"], case["viscous"]] + n * (32 + 32 + 16)
    if case["call"] == "stages":
        b += n * case["steps"] * 4 * 32  # the four matrices each step hands back
    return {"bytes": float(b), "flops": float(n * case["steps"] * FLOPS[case["viscous"]])}


# ------------------------------------------------------------------ exact


class _Exact:
    """The explicit step in 64 bits, plain torch over a mesh's arrays."""

    def __init__(self, mesh, cfg, prims):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev = dev

        def t(a, kind):
            return torch.from_numpy(np.ascontiguousarray(a)).to(dev, kind)

        f, i = torch.float64, torch.int64
        self.cfg, self.g = cfg, cfg["thermo"]["Gamma"]
        self.R = cfg["thermo"]["RGAS"]
        nf = t(mesh.mesh_connectivity[:, 2], i)
        self.quad = (nf == 4)[:, None]
        K = 4 if bool(self.quad.any()) else 3
        self.K = K
        live = torch.arange(K, device=dev)[None, :] < nf[:, None]
        self.live = live
        stiff = t(mesh.cell_stiffness[:, :K], i)
        self.inner = (stiff >= 1) & live
        self.nb = torch.where(self.inner, stiff - 1, torch.arange(mesh.nCells, device=dev)[:, None])
        self.tags = [(b, (stiff == b["tag"]) & live) for b in cfg["bc"]]
        self.nx, self.ny = t(mesh.cell_edges_Nx[:, :K], f), t(mesh.cell_edges_Ny[:, :K], f)
        self.len = torch.where(live, t(mesh.cell_edges_length[:, :K], f), 0.0)
        self.area, self.hx = t(mesh.cell_areas, f), t(mesh.HX, f)
        self.charlen = 2.0 * self.area / self.len.sum(1)

        def nodes(a, first):
            return torch.clamp(t(a[:, first:2 * K:2], i) - 1, min=0)

        self.up, self.up2 = nodes(mesh.node2cellL2up, 0), nodes(mesh.node2cellL2up, 1)
        self.dn, self.dn2 = nodes(mesh.node2cellL2down, 0), nodes(mesh.node2cellL2down, 1)
        self.ea, self.eb = nodes(mesh.cells2nodes, 0), nodes(mesh.cells2nodes, 1)
        cl = t(mesh.cell_clusters, i)
        self.cl = torch.where(cl > 0, cl - 1, mesh.nCells)  # row nCells: zeros
        self.w = torch.where(cl > 0, t(mesh.node_stencils, f), 0.0)
        self.one = (cl > 0).to(f)
        self.mid = t(mesh.cell_mid_points, f)
        self.xy = torch.stack([t(mesh.xNodes, f), t(mesh.yNodes, f)], 1)
        self.P = torch.stack([t(x, f) for x in prims], 1)
        r, u, v, p = self.P.unbind(1)
        self.U = torch.stack([r, r * u, r * v, p / (self.g - 1.0) + 0.5 * r * (u * u + v * v)], 1)
        self.N = torch.zeros((mesh.nNodes, 4), dtype=f, device=dev)
        self.t = 0.0

    def _means(self, q, w):
        q = torch.cat([q, torch.zeros((1, q.shape[1]), dtype=q.dtype, device=q.device)])
        s = torch.zeros((self.cl.shape[0], q.shape[1]), dtype=q.dtype, device=q.device)
        for j in range(self.cl.shape[1]):
            s += q[self.cl[:, j]] * w[:, j:j + 1]
        d = w.sum(1, keepdim=True)
        return torch.where(d != 0.0, s / torch.where(d != 0.0, d, 1.0), 0.0)

    def _edge_sums(self, at_nodes, nx, ny):
        """Green-Gauss sums over a cell's edges of node values, per component."""
        m = 0.5 * (at_nodes[self.ea] + at_nodes[self.eb])
        gx = (m * (-nx * self.len)[..., None]).sum(1) / self.area[:, None]
        gy = (m * (-ny * self.len)[..., None]).sum(1) / self.area[:, None]
        return gx, gy

    def diff_term(self):
        c, g = self.cfg, self.g
        r, u, v, p = self.P.unbind(1)
        T = p / r / self.R
        prim = c["viscosity"] != "reference"
        q = (torch.stack([u, v, 0.5 * (u * u + v * v) + g / c["Pr"] * (p / ((g - 1.0) * r))], 1) if prim
             else self.U[:, 1:])
        gx, gy = self._edge_sums(self._means(q, self.one), self.ny, self.nx)
        gxx, _ = self._edge_sums(self._means(gx, self.one), self.ny, self.nx)
        _, gyy = self._edge_sums(self._means(gy, self.one), self.ny, self.nx)
        lap = gxx + gyy
        D = torch.zeros_like(self.U)
        if not prim:
            iT = 1.0 / T
            low = (2898903.0 * iT**2 - 56496.26 * iT + 1437.799 - 1.653609 * T + 0.003062254 * T**2
                   - 2.279138e-6 * T**3 + 6.272365e-10 * T**4)
            assert bool(((T > 200.0) & (T < 1000.0)).all())
            k = (15.0 / 4.0 * 8.314462 / 28.9647 * 1.716e-5 * (T / 273.11) ** (2.0 / 3.0)
                 * (4.0 / 15.0 * low * 28.9647 / 8.314462 + 1.0 / 3.0))
            D[:, 1:] = c["mu_ref"] * lap
            D[:, 3] *= k
            return D
        mu = torch.full_like(T, c["mu_ref"])
        if c["viscosity"] == "sutherland":
            mu = mu * (torch.sqrt(T / c["T_ref"]) * (1.0 + 116.0 / c["T_ref"]) / (1.0 + 116.0 / T))
        if c["art_viscosity"]:
            gx, gy = self._edge_sums(self.N[:, 1:3], self.nx, self.ny)
            div = gx[:, 0] + gy[:, 1]
            a = 0.05 * torch.sqrt(g * p / r) / self.hx / math.sqrt(2.0)
            on = (-div > a) & (div * div - a * a > 0.0)
            mu = mu + torch.where(on, 0.25 * r * self.hx**2 * torch.sqrt(torch.clamp(div * div - a * a, min=0.0))
                                  * 1.0e-5, 0.0)
        D[:, 1:] = mu[:, None] * lap
        return D

    def _ghost(self, b, L, nx, ny, cells, k):
        G = L.clone()
        if b["kind"] == "inflow":
            for j, n in enumerate(("rho", "u", "v", "p")):
                G[:, j] = b[n]
        elif b["kind"] == "slip":
            G[:, 1] = L[:, 1] * (ny * ny - nx * nx) - 2.0 * nx * ny * L[:, 2]
            G[:, 2] = L[:, 2] * (nx * nx - ny * ny) - 2.0 * nx * ny * L[:, 1]
        elif b["kind"] == "noslip_isothermal":
            G[:, 0] = L[:, 3] / (self.R * b["Tw"])
            G[:, 1:3] = -L[:, 1:3]
        elif b["kind"] == "tgv":
            a, e = self.xy[self.ea[cells, k]], self.xy[self.eb[cells, k]]
            d, w = e - a, self.mid[cells] - a
            q = (d * d).sum(1)
            ca, cb = (d[:, 0] ** 2 - d[:, 1] ** 2) / q, 2.0 * d[:, 0] * d[:, 1] / q
            x, y = ca * w[:, 0] + cb * w[:, 1] + a[:, 0], cb * w[:, 0] - ca * w[:, 1] + a[:, 1]
            z = self.cfg["tgv"]
            U, L0, f = z["U0"], z["L"], math.exp(-2.0 * z["mu"] * self.t / z["L"] ** 2)
            G[:, 0] = 1.0
            G[:, 1] = U * torch.sin(x / L0) * torch.cos(y / L0) * f
            G[:, 2] = -U * torch.cos(x / L0) * torch.sin(y / L0) * f
            G[:, 3] = z["P0"] + 0.25 * U * U * (torch.cos(2 * x / L0) + torch.cos(2 * y / L0)) * f * f
        return G

    def _limit(self, a, b, e2):
        kind, c = self.cfg["limiter"], self.cfg["ksi"]
        if kind == "venkat":
            b = torch.where(a * b < 0.0, 0.0, b)
            d = b * b + 2.0 * a * a + a * b + e2
            return torch.where(d == 0.0, 0.0, ((b * b + e2) * a + 2.0 * a * a * b) / torch.where(d == 0.0, 1.0, d))
        if kind == "minmod":
            return (torch.sign(a) + torch.sign(b)) * (a * b).abs() / (a.abs() + b.abs() + c)
        if kind == "vanleer":
            return (a * b + (a * b).abs()) / (a + b + c)
        if kind == "vanalbada":
            return (a * (b * b + c) + b * (a * a + c)) / (a * a + b * b + 2.0 * c)
        return torch.zeros_like(a)

    def _flux(self, L, R, nx, ny, side):
        g, kind = self.g, self.cfg["flux"]
        rL, uL, vL, pL = L.unbind(-1)
        rR, uR, vR, pR = R.unbind(-1)
        nL, nR = uL * nx + vL * ny, uR * nx + vR * ny
        hL = 0.5 * (uL * uL + vL * vL) + g / (g - 1.0) * pL / rL
        hR = 0.5 * (uR * uR + vR * vR) + g / (g - 1.0) * pR / rR
        if kind == "roe":
            aL, aR = torch.sqrt(g * pL / rL), torch.sqrt(g * pR / rR)
            mx, my = -ny, nx
            w = torch.sqrt(rR / rL)
            u, v, H = (uL + w * uR) / (1 + w), (vL + w * vR) / (1 + w), (hL + w * hR) / (1 + w)
            r = w * rL
            a = torch.sqrt((g - 1.0) * (H - 0.5 * (u * u + v * v)))
            un, um = u * nx + v * ny, u * mx + v * my
            dn, dm, dp = nR - nL, (uR - uL) * mx + (vR - vL) * my, pR - pL

            def fix(x):
                return torch.where(x < 0.2, 0.5 * (x * x / 0.2 + 0.2), x)

            w1 = fix((un - a).abs()) * (dp - r * a * dn) / (2 * a * a)
            w2 = un.abs() * r * dm
            w3 = un.abs() * (rR - rL - dp / (a * a))
            w4 = fix((un + a).abs()) * (dp + r * a * dn) / (2 * a * a)
            diss = [w1 + w3 + w4, w1 * (u - a * nx) + w2 * mx + w3 * u + w4 * (u + a * nx),
                    w1 * (v - a * ny) + w2 * my + w3 * v + w4 * (v + a * ny),
                    w1 * (H - un * a) + w2 * um + w3 * 0.5 * (u * u + v * v) + w4 * (H + un * a)]
            both = [rL * nL + rR * nR, rL * nL * uL + pL * nx + rR * nR * uR + pR * nx,
                    rL * nL * vL + pL * ny + rR * nR * vR + pR * ny, rL * nL * hL + rR * nR * hR]
            return torch.stack([-0.5 * (f - d) * side for f, d in zip(both, diss)], -1)
        g2 = 2.0 * (g - 1.0) / (g + 1.0)

        def split(M, sign, beta):
            q = M * M - 1.0
            out = torch.where(M.abs() >= 1.0, 0.5 * (M + sign * M.abs()),
                              sign * (0.25 * (M + sign) ** 2 + beta * q * q))
            return out

        def press(M, sign, alpha):
            q = M * M - 1.0
            return torch.where(M.abs() >= 1.0, 0.5 * (1.0 + sign * torch.sign(M)),
                               0.25 * (M + sign) ** 2 * (2.0 - sign * M) + sign * alpha * M * q * q)

        if kind == "ausm":
            sL, sR = torch.sqrt(g2 * hL), torch.sqrt(g2 * hR)
            a = torch.minimum(torch.minimum(sL, sL * sL / nL.abs()), torch.minimum(sR, sR * sR / nR.abs()))
            m = split(nL / a, 1.0, 0.125) + split(nR / a, -1.0, 0.125)
            ps = press(nL / a, 1.0, 0.1875) * pL + press(nR / a, -1.0, 0.1875) * pR
            mL, mR = a * torch.clamp(m, min=0.0) * rL, a * torch.clamp(m, max=0.0) * rR
            f = [mL + mR, mL * uL + mR * uR + ps * nx, mL * vL + mR * vR + ps * ny, mL * hL + mR * hR]
            return torch.stack([-x * side for x in f], -1)
        tL, tR = uL * ny - vL * nx, uR * ny - vR * nx
        s = torch.sqrt(g2 * 0.5 * (hL + hR - 0.5 * (tL * tL + tR * tR)))
        a = s * s / torch.maximum(torch.where(0.5 * (nL + nR) >= 0.0, nL.abs(), nR.abs()), s)
        ML, MR = nL / a, nR / a
        f = 0.5 * (1.0 - torch.cos(math.pi * torch.clamp(torch.maximum(ML.abs(), MR.abs()), max=1.0)))
        h = 0.5 * (1.0 + torch.cos(math.pi * torch.minimum(pL / pR, pR / pL)))
        p12 = -h * g * (pL + pR) * 0.5 / a * press(ML, 1.0, 0.1875) * press(MR, -1.0, 0.1875)
        ps = 0.5 * (pL + pR) - 0.25 * (rL + rR) * a * (uR - uL)
        m = (split(ML, 1.0, 0.125) + split(MR, -1.0, 0.125)
             - 0.5 * (1.0 - f) * (pR - pL) * 2.0 / (rL + rR) / a / a * (1.0 - h))
        m = torch.where(m >= 0.0, m * a * rL, m * a * rR)
        mL, mR = torch.clamp(m, min=0.0), torch.clamp(m, max=0.0)
        out = [mL + mR, mL * uL + mR * uR + ps * nx + p12 * (uR - uL), mL * vL + mR * vR + ps * ny + p12 * (vR - vL),
               mL * hL + mR * hR]
        return torch.stack([-x * side for x in out], -1)

    def fluxes(self):
        total = torch.zeros_like(self.P)
        for k in range(self.K):
            nx, ny, inner = self.nx[:, k], self.ny[:, k], self.inner[:, k:k + 1]
            L, R = self.P, self.P[self.nb[:, k]].clone()
            dn, up = self.N[self.dn[:, k]], self.N[self.up[:, k]]
            if self.K == 4:
                dn = torch.where(self.quad, 0.5 * (dn + self.N[self.dn2[:, k]]), dn)
                up = torch.where(self.quad, 0.5 * (up + self.N[self.up2[:, k]]), up)
            for b, mask in self.tags:
                cells = mask[:, k].nonzero()[:, 0]
                if cells.numel():
                    R[cells] = self._ghost(b, L[cells], nx[cells], ny[cells], cells, k)
            dn, up = torch.where(inner, dn, L), torch.where(inner, up, R)
            sc = 0.5 * (L * L + R * R)
            if self.cfg["limiter"] == "venkat":
                K3 = self.cfg.get("venkat_K", 5.0) ** 3
                eL = K3 * self.hx[:, None] ** 3 * sc
                eR = K3 * self.hx[self.nb[:, k]][:, None] ** 3 * sc
                a = L + 0.5 * self._limit(L - dn, R - L, eL)
                c = R + 0.5 * self._limit(R - up, L - R, eR)
            else:
                a = L + 0.5 * self._limit(L - dn, R - L, None)
                c = R - 0.5 * self._limit(R - L, up - R, None)
            f = self._flux(c, a, nx, ny, self.len[:, k])
            total += torch.where(self.live[:, k:k + 1], f, 0.0)
        return total

    def update(self, Un):
        if self.cfg.get("densityConstrained", 0):
            Un[:, 0].clamp_(self.cfg["minDensityConstrained"], self.cfg["maxDensityConstrained"])
        delta = Un - self.U
        self.U = Un
        r, mu, mv, E = Un.unbind(1)
        self.P = torch.stack([r, mu / r, mv / r, (self.g - 1.0) * (E - 0.5 * (mu * mu + mv * mv) / r)], 1)
        return delta

    def nodes(self):
        self.N = self._means(self.P, self.w)

    def step(self):
        c = self.cfg
        r, u, v, p = self.P.unbind(1)
        vmax = torch.sqrt(u * u + v * v) + torch.sqrt(self.g * p / r)
        tau = c["CFL"] * float(self.hx.max()) / max(float(vmax.max()), 1.0e-6)
        dt = {0: c.get("dt", 0.0), 1: tau, 2: c["CFL"] * float((self.charlen / vmax).min())}[c["dt_mode"]]
        D = self.diff_term() if c["viscosity"] != "none" else 0.0
        F = self.fluxes()
        lo, hi = float(r.min()), float(r.max())
        d = self.update(self.U - F * dt / self.area[:, None] + dt * D)
        self.nodes()
        self.t += dt
        q = self.P
        ek = (0.5 * q[:, 0] * (q[:, 1] ** 2 + q[:, 2] ** 2) * self.area).sum()
        return [dt, tau, float(vmax.max()), *(d * d).sum(0).tolist(), lo, hi,
                *(self.U * self.area[:, None]).sum(0).tolist(), float(ek)]


def exact(case, seed):
    if case["call"] == "update":
        a, b = _update_inputs(case, seed)
        r, mu, mv, E = b
        u, v, p = mu / r, mv / r, 0.4 * (E - 0.5 * (mu * mu + mv * mv) / r)
        vm = torch.sqrt(u * u + v * v) + torch.sqrt(1.4 * p / r)
        st = torch.cat([((b - a) ** 2).sum(1), vm.max().reshape(1), torch.zeros_like(vm[:1])])
        return {"uold": b, "prims": torch.stack([r, u, v, p]), "stats": st}
    out = {"stats": [], "cells": [], "nodes": []}
    for mesh, cfg, prims in _inputs(case, seed):
        x = _Exact(mesh, cfg, prims)
        if case["call"] == "stages":
            for _ in range(case["steps"]):
                D = x.diff_term()
                F = x.fluxes()
                Un = x.U - F * STAGE_DT / x.area[:, None] + STAGE_DT * D
                d = x.update(Un.clone())
                x.nodes()
            return {"diff": D, "flux": F, "unew": Un, "delta": d, "nodes": x.N.T.contiguous()}
        for _ in range(case["steps"]):
            st = x.step()
        out["stats"].append(np.array(st, dtype=np.float64))
        cells = x.P if case["precision"] == "mixed" else x.U
        out["cells"].append(cells.T.contiguous())
        out["nodes"].append(x.N.T.contiguous())
        del x
    return out
