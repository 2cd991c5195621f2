"""The work a user of this framework has it do, as timed cases.

A case is a plain dict.  Three kinds:

* "march":    a batch of coarse time steps of one simulation on the drop-in
              path (solver.execute_timestep_batch), as the main loop runs it;
* "pool":     a chunk of coarse steps of several cases in one block pool
              (native.Context), then what the serving loop reads at a chunk's
              end: every case's force coefficients, and the fields of a case
              that retires;
* "diagnose": the main loop's diagnostics (flow statistics of level 1, forces
              with surface maps and net forces on the finest level).

prepare() makes the flow state from the seed; the case's domain (blocks,
masks, Bouzidi lists) is static and built once per process.  exact() repeats a
pass in 64 bits with plain torch (tensors over all cells of a level).
"""
from __future__ import annotations

import dataclasses as dc
import functools
import math

import numpy as np
import torch

from openludwig_b200 import domain, native, scaling, solver, workloads

DEV = "cuda:0"


# ------------------------------------------------------------------- cases

def _march(name, body, size, levels, steps, **kw):
    c = dict(kind="march", body=body, size=size, levels=levels, steps=steps,
             operator="cumulant", c_wale=0.5, wall_model=False, limiter="factored",
             compressible=False, ddf=False, sponge_blend=False, turbulence=0.0, u=0.05)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _pool(name, storage, size, count, steps, mix):
    c = dict(kind="pool", storage=storage, size=size, count=count, steps=steps, mix=mix)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a 64x32x32 single-level run, bound by launches
        _march("sphere_64", "sphere", 8, 1, 8, c_wale=0.0),
        # the single-level sphere of 128x64x64 (the reference's CPU-runnable case)
        _march("sphere_128", "sphere", 16, 1, 8, c_wale=0.0),
        # a small refined case of the batch mix's sizes (24 finest cells)
        _march("cube_24", "mix_cube", 24, 2, 8),
        # the three-level cube of the headline configuration
        _march("cube_3lvl", "cube", 64, 3, 2, wall_model=True),
        # the same at one and a half times the resolution: the largest run
        _march("cube_96", "cube", 96, 3, 2, wall_model=True),
        # Mach 0.6 thermal sphere: O(u^4) equilibria and the thermal populations
        _march("sphere_ddf", "sphere_ddf", 48, 2, 2, compressible=True, ddf=True, u=0.346),
        # the other collision operator, with inlet turbulence and WALE
        _march("sphere_bgk", "sphere", 32, 2, 4, operator="regularized_bgk", turbulence=0.02),
        # an odd size with the options that are off by default
        _march("sphere_odd", "sphere", 37, 3, 4, limiter="positivity", sponge_blend=True,
               wall_model=True, u=0.08),
        # batched cases in one pool, both storages
        _pool("pool_f32", "f32", 32, 6, 8, 1234),
        _pool("pool_f16", "f16", 32, 6, 8, 1234),
        # what the main loop prints and writes at a diagnostics step
        dict(name="diagnose_ddf", kind="diagnose", body="sphere_ddf", size=48, levels=2,
             ddf=True, u=0.346, c_wale=0.5, search_radius=5),
    ]


def draw(rng):
    """One more case: sizes log-uniform over 8..64 cells of body length."""
    size = int(round(8.0 * 8.0 ** rng.random()))
    kind = rng.choice(["march"] * 6 + ["pool"] * 2 + ["diagnose"])
    if kind == "pool":
        return _pool(None, rng.choice(["f32", "f16"]), rng.randint(16, 32), rng.randint(2, 6),
                     rng.choice([2, 4, 8]), rng.randint(1, 10 ** 6))
    body = rng.choice(["sphere", "cube", "mix_cube", "mix_sphere", "sphere_ddf"])
    ddf = body == "sphere_ddf"
    levels = rng.randint(1, 3)
    if levels == 1 or ddf:
        size = min(size, 28 + 12 * levels)
    u = 0.346 if ddf else round(rng.uniform(0.04, 0.1), 3)
    if kind == "diagnose":
        return dict(kind="diagnose", body=body, size=size, levels=levels, ddf=ddf, u=u,
                    c_wale=0.5, search_radius=5)
    op = rng.choice(["cumulant"] * 4 + ["regularized_bgk"])
    return _march(None, body, size, levels, rng.choice([1, 2, 4]), operator=op,
                  c_wale=rng.choice([0.0, 0.2, 0.5]), wall_model=rng.random() < 0.4,
                  limiter=rng.choice(["factored", "factored", "positivity", "none"]),
                  compressible=ddf or rng.random() < 0.2, ddf=ddf,
                  sponge_blend=rng.random() < 0.3,
                  turbulence=rng.choice([0.0, 0.0, 0.02]), u=u)


# ----------------------------------------------------------------- domains

@functools.lru_cache(maxsize=None)
def _domain(body, size, levels, alpha=None, beta=None):
    """(config, mesh, domain parameters, host levels) with wall distances."""
    if body == "sphere":
        cfg, mesh = workloads.sphere_1lvl(size)
    elif body == "sphere_ddf":
        cfg, mesh = workloads.sphere_ddf()
    elif body == "cube":
        cfg, mesh = workloads.cube_3lvl()
    else:  # a case of the batch mix
        m = workloads.MixCase(body[4:], size, levels, 1e5, 3.0 if alpha is None else alpha,
                              -2.0 if beta is None else beta)
        cfg, mesh = workloads.mix_case_config(m)
    cfg.surface_resolution = size
    cfg.num_levels_config = levels
    cfg.wall_model_enabled = True  # wall distances, used when the case turns the model on
    p = scaling.compute_domain_from_mesh(cfg, mesh.min_bounds, mesh.max_bounds)
    return cfg, mesh, p, domain.setup_multilevel_domain(cfg, mesh, p, device=0)


def _with_options(case, base, **over):
    """The case's own config and scaling over a cached domain (same blocks)."""
    cfg, mesh, p, hosts = base
    cfg = dc.replace(cfg, wall_model_enabled=bool(case.get("wall_model", False)),
                     c_wale=float(np.float32(case["c_wale"])),
                     u_target=float(np.float32(case["u"])), ddf_enabled=bool(case.get("ddf")),
                     collision_operator=case.get("operator", "cumulant"),
                     cumulant_limiter=case.get("limiter", "factored"),
                     compressibility_correction=bool(case.get("compressible", False)),
                     sponge_blend_distributions=bool(case.get("sponge_blend", False)),
                     inlet_turbulence_intensity=float(np.float32(case.get("turbulence", 0.0))),
                     **over)
    p = scaling.compute_domain_from_mesh(cfg, mesh.min_bounds, mesh.max_bounds)
    hosts = [dc.replace(h, tau=p.tau_levels[i], tau_g=p.tau_g_levels[i] if p.tau_g_levels else 0.0)
             for i, h in enumerate(hosts)]
    return cfg, mesh, p, hosts


def _pool_cases(case, seed):
    """The pool's prepared cases: bodies, depths and angles from the mix
    number, Reynolds number and inlet speed from the seed."""
    pick = np.random.default_rng(case["mix"])
    flow = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        body = ["mix_cube", "mix_sphere"][int(pick.integers(2))]
        size = int(case["size"] * [0.5, 0.75, 1.0][int(pick.integers(3))])
        levels = 1 + i % 3
        alpha, beta = float(pick.uniform(-4, 12)), float(pick.uniform(-5, 5))
        re, u = float(10 ** flow.uniform(3, 6)), float(flow.uniform(0.04, 0.06))
        cfg, mesh, p, hosts = _with_options(
            dict(c_wale=0.5, u=u), _domain(body, size, levels, alpha, beta),
            fluid_kinematic_viscosity=1.0 / re)
        out.append(native.PreparedCase(cfg, mesh, p, hosts,
                                       solver.StepSettings.from_config(cfg, False)))
    return out


# Steps a pool's cases have taken before the first pass: the start's pressure
# wave (0.58 cells a step) has passed every body, at most 48 cells downstream.
# Odd, so that after a pass the pool's velocity readout is the newest step's.
POOL_WARM = 161


# ------------------------------------------------------------------- state

_CX = [k % 3 - 1 for k in range(27)]
_CY = [k // 3 % 3 - 1 for k in range(27)]
_CZ = [k // 9 - 1 for k in range(27)]
_W = [[8 / 27, 2 / 27, 1 / 54, 1 / 216][abs(x) + abs(y) + abs(z)] for x, y, z in zip(_CX, _CY, _CZ)]


def _cells(h):
    """1-based global coordinates of a level's cells, [512 n] each."""
    c = torch.from_numpy(np.ascontiguousarray(h.coords)).to(DEV).long()
    t = torch.arange(512, device=DEV)
    return [((c[:, a, None] - 1) * 8 + loc[None] + 1).reshape(-1)
            for a, loc in enumerate((t & 7, t >> 3 & 7, t >> 6))]


def _flow_state(h, dims, u0, seed, ddf):
    """A developed-looking flow on a level: the mean flow with a few seeded
    waves in velocity, density and temperature (the same field on every level)
    and per-population non-equilibrium noise."""
    rng = np.random.default_rng(seed)
    scale = 2.0 ** (h.level_id - 1)
    pos = [(g.float() - 0.5) / (scale * d) for g, d in zip(_cells(h), dims)]

    def waves():
        v = torch.zeros_like(pos[0])
        for _ in range(4):
            k = rng.integers(1, 7, 3) * 2.0 * math.pi
            v += torch.sin(k[0] * pos[0] + k[1] * pos[1] + k[2] * pos[2] + rng.uniform(0, 6.28))
        return v / 4

    solid = torch.from_numpy(h.obstacle).to(DEV) != 0
    u = [u0 * (1.0 + 0.2 * waves()), 0.1 * u0 * waves(), 0.1 * u0 * waves()]
    u = [torch.where(solid, 0.0, v) for v in u]
    rho = torch.where(solid, 1.0, 1.0 + 0.5 * u0 * u0 * waves())
    T = 1.0 + 0.02 * waves()
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 8 + h.level_id)
    usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    f = torch.empty((27, rho.numel()), device=DEV)
    g = torch.empty_like(f) if ddf else None
    for k in range(27):
        cu = _CX[k] * u[0] + _CY[k] * u[1] + _CZ[k] * u[2]
        noise = 1.0 + 1e-3 * u0 * torch.randn(rho.numel(), generator=gen, device=DEV)
        f[k] = rho * _W[k] * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * usq) * noise
        if ddf:
            g[k] = _W[k] * T * (1 + 3 * cu)
    return dict(f=f.reshape(-1), rho=rho, vel=torch.cat(u), g=None if g is None else g.reshape(-1),
                T=g.sum(0) if ddf else None)


def prepare(case, seed):
    if case["kind"] == "pool":
        cases = _pool_cases(case, seed)
        blocks = sum(h.n_blocks for c in cases for h in c.levels)
        per = 512 * ((2 if case["storage"] == "f16" else 4) * 54 + 41)
        ctx = native.Context(budget_bytes=int(1.3 * blocks * per) + (64 << 20),
                             storage=case["storage"])
        ids = [ctx.add_case(c) for c in cases]
        ctx.step(POOL_WARM)
        ctx.sync()
        return dict(case=case, ctx=ctx, ids=ids, cases=cases)
    cfg, mesh, p, hosts = _with_options(case, _domain(case["body"], case["size"], case["levels"]))
    sim = solver.Simulation(cfg, mesh, p, hosts)
    for lv in sim.levels:
        s = _flow_state(lv.host, sim.dims, cfg.u_target, seed, cfg.ddf_enabled)
        lv.f.copy_(s["f"]), lv.f_temp.copy_(s["f"])
        lv.vel.copy_(s["vel"]), lv.vel_temp.copy_(s["vel"])
        lv.rho.copy_(s["rho"])
        if cfg.ddf_enabled:
            lv.g.copy_(s["g"]), lv.g_temp.copy_(s["g"])
            lv.temperature.copy_(s["T"])
    return dict(case=case, sim=sim, t=0)


# -------------------------------------------------------------------- pass

def run(state):
    case = state["case"]
    if case["kind"] == "pool":
        ctx, ids = state["ctx"], state["ids"]
        ctx.step(case["steps"])
        coef = [np.array(list(ctx.coefficient_record(i).values())) for i in ids]
        # the case that retires: its fields go back to the host
        fields = [ctx.download(ids[-1], lv + 1)[:2] for lv in range(len(state["cases"][-1].levels))]
        return {"coefficients": coef, "fields": fields}
    sim = state["sim"]
    if case["kind"] == "diagnose":
        lv = sim.levels[-1]
        raw, maps = solver.compute_aerodynamics(lv, sim.dmesh, sim.p, sim.cfg, maps=True,
                                                search_radius=case["search_radius"])
        net = solver.compute_net_aerodynamics(lv, sim.dmesh, sim.p, sim.cfg,
                                              search_radius=case["search_radius"])
        return {"stats": solver.flow_stats(sim.levels[0]), "raw": raw, "maps": maps, "net": net}
    n = case["steps"]
    solver.execute_timestep_batch(sim.levels, sim.settings, state["t"] + 1, n, sim.cfg.u_target,
                                  sim.dims)
    state["t"] += n
    out = []
    for i, lv in enumerate(sim.levels):
        temp = i == 0 and state["t"] % 2 == 0  # an even step writes the second buffer
        o = {"f": lv.f_temp if temp else lv.f, "rho": lv.rho,
             "vel": lv.vel_temp if temp else lv.vel}
        if case["ddf"]:
            o["g"], o["T"] = lv.g_temp if temp else lv.g, lv.temperature
        out.append(o)
    return out


# -------------------------------------------------------------------- work

def _level_hosts(case):
    if case["kind"] == "pool":
        return [c.levels for c in _pool_cases(case, 1)]
    return [_domain(case["body"], case["size"], case["levels"])[3]]


def work(case):
    """Bytes and operations of one pass: per cell update every population
    read and written once, the macroscopic fields written (and the velocity
    read for WALE), the masks read; about 700 FP32 operations (250 for the
    thermal update)."""
    hosts = _level_hosts(case)
    if case["kind"] == "diagnose":
        tri = _domain(case["body"], case["size"], case["levels"])[1].n
        coarse = hosts[0][0].n_blocks * 512
        return {"bytes": coarse * 17.0 + tri * (8 * 17 + 7 * 4 + 16 + 12) * 2, "flops": tri * 400.0}
    updates = sum(h.n_blocks * 512 * 2 ** i for hs in hosts for i, h in enumerate(hs)) * case["steps"]
    pop = 2 if case.get("storage") == "f16" else 4
    wale = case["kind"] == "pool" or case["c_wale"] != 0.0
    per = 54 * pop + 16 + 5 + (12 if wale else 0) + (4 if case.get("wall_model") else 0)
    flops = 700
    if case.get("ddf"):
        per, flops = per + 54 * pop + 4, flops + 250
    return {"bytes": float(updates * per), "flops": float(updates * flops)}


def tolerance(case):
    """About four times what the FP32 path is off the 64-bit one (march: 1.3e-6
    on the velocities; forces: cancellation on faces across an axis, 3.7e-4 on
    cubes) or two kernels with other roundings differ by after 16 steps (pool)."""
    if case["kind"] == "diagnose":
        return {"rel": 1.5e-3 if "cube" in case["body"] else 2e-4, "max": 1e-2}
    if case["kind"] == "pool":
        return {"rel": 2.2e-3, "max": 1e-2} if case["storage"] == "f16" else {"rel": 3e-5, "max": 1e-3}
    return {"rel": 5e-6, "max": 2e-4}


# ------------------------------------------------- one pass in 64 bits
#
# The method as plain tensor operations: lattice k = (cx+1) + 3 (cy+1) +
# 9 (cz+1), arrays [27, 512 n] per level, everything float64.

class _Level:
    def __init__(self, h, tau, tau_g):
        d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        self.n = h.n_blocks
        self.tau, self.tau_g = float(np.float32(tau)), float(np.float32(tau_g))
        self.nbr = d(h.neighbor_table).long().reshape(27, self.n) - 1
        self.ptr, self.dim = d(h.block_ptr).long(), h.grid_dim
        self.pos = _cells(h)
        self.solid = d(h.obstacle) != 0
        self.sponge = d(h.sponge).double()
        self.wall = d(h.wall_dist).double()
        self.links = None
        if h.bouzidi and h.n_boundary > 0:
            cell = ((d(h.cell_block).long() - 1) * 512 + d(h.cell_x).long() - 1 +
                    8 * (d(h.cell_y).long() - 1) + 64 * (d(h.cell_z).long() - 1))
            q = d(h.q_map.view(np.float16)).reshape(27, -1)[:, cell].double()
            self.links = (cell, q)
        self.t = torch.arange(512 * self.n, device=DEV)

    def neighbor(self, dx, dy, dz, cells=None):
        """Index of the cell at an offset, -1 where its block is absent."""
        t = self.t if cells is None else cells
        b, c = t >> 9, t & 511
        x, y, z = (c & 7) + dx, (c >> 3 & 7) + dy, (c >> 6) + dz
        d = (1 + (x > 7).long() - (x < 0).long()) + 3 * (1 + (y > 7).long() - (y < 0).long()) + \
            9 * (1 + (z > 7).long() - (z < 0).long())
        nb = torch.where(d == 13, b, self.nbr[d, b])
        return torch.where(nb < 0, -1, nb * 512 + (x & 7) + 8 * (y & 7) + 64 * (z & 7))


def _feq(rho, u, k, order4):
    cu = _CX[k] * u[0] + _CY[k] * u[1] + _CZ[k] * u[2]
    sq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    v = 1 + 3 * cu + 4.5 * cu * cu - 1.5 * sq
    if order4:
        v = v + 4.5 * cu ** 3 - 4.5 * cu * sq + 3.375 * cu ** 4 - 6.75 * cu * cu * sq + 1.125 * sq * sq
    return rho * _W[k] * v


def _geq(T, u, k):
    return _W[k] * T * (1 + 3 * (_CX[k] * u[0] + _CY[k] * u[1] + _CZ[k] * u[2]))


def _noise(gx, gy, gz):
    """The inlet's integer hash noise in [-1, 1), 32-bit wrap-around products."""
    m = 0xFFFFFFFF
    h = (gx * 374761393 + gy * 668265263 + gz * 1274126177 + 1234) & m
    h = ((h ^ (h >> 16)) * 0x85ebca6b) & m
    h = ((h ^ (h >> 13)) * 0xc2b2ae35) & m
    return ((h ^ (h >> 16)) & 0xFFFF).double() / 32768.0 - 1.0


def _from_parent(P, pos, w, values):
    """Trilinear values at fine positions from the parent's cells.  values:
    list of (parent field, value where the parent cell is absent)."""
    lo, frac = [], []
    for g in pos:
        c = (g.double() - 0.5) * 0.5
        f = torch.floor(c)
        lo.append(f.long()), frac.append(c - f)
    v = [[None] * 8 for _ in values]
    for s in range(8):
        g = [lo[a] + 1 if s >> a & 1 else lo[a].clamp(min=1) for a in range(3)]
        bl = [(x - 1) // 8 for x in g]
        ok = torch.ones_like(g[0], dtype=torch.bool)
        for a in range(3):
            ok &= (bl[a] >= 0) & (bl[a] < P.dim[a])
        i = bl[0] + P.dim[0] * (bl[1] + P.dim[1] * bl[2])
        pb = torch.where(ok, P.ptr[torch.where(ok, i, 0)], 0) - 1
        cell = pb.clamp(min=0) * 512 + (g[0] - 1) % 8 + 8 * ((g[1] - 1) % 8) + 64 * ((g[2] - 1) % 8)
        for j, (field, none) in enumerate(values):
            x = torch.where(pb >= 0, field[cell], none)
            v[j][s] = x if s == 0 else torch.where(pb >= 0, x, v[j][0])
    out = []
    for c in v:
        for a in range(3):
            c = [c[2 * i] * (1 - frac[a]) + c[2 * i + 1] * frac[a] for i in range(len(c) // 2)]
        out.append(c[0])
    return out


def _pull(L, P, f, st, dims, u_in, step, tw, thermal):
    out = torch.empty_like(f)
    for k in range(27):
        c = (_CX[k], _CY[k], _CZ[k])
        i = L.neighbor(-c[0], -c[1], -c[2])
        out[k] = f[k][i.clamp(min=0)]
        m = torch.nonzero(i < 0).reshape(-1)
        if m.numel() == 0:
            continue
        src = [L.pos[a][m] - c[a] for a in range(3)]
        one = torch.ones(m.numel(), dtype=torch.float64, device=DEV)
        zero = 0 * one
        if P is None:
            v = _W[k] * one * (st.t_inlet if thermal else 1.0)
        else:
            old, new = P.old, P.new

            def mix(name, row=None):
                o, x = (old[name], new[name]) if row is None else (old[name][row], new[name][row])
                return o * (1 - tw) + x * tw

            names = ("g", "T") if thermal else ("f", "rho")
            a, r, ux, uy, uz = _from_parent(P, src, _W[k], [
                (mix(names[0], k), _W[k]), (mix(names[1]), 1.0), (mix("vel", 0), 0.0),
                (mix("vel", 1), 0.0), (mix("vel", 2), 0.0)])
            e = _geq(r, (ux, uy, uz), k) if thermal else _feq(r, (ux, uy, uz), k, st.compressible)
            tc, tf = (P.tau_g - 0.5, L.tau_g - 0.5) if thermal else (P.tau - 0.5, L.tau - 0.5)
            v = e + (a - e) * (min(max(tf / tc, 0.01), 100.0) if tc > 1e-6 else 1.0)
        my, mz = k - 6 * c[1], k - 18 * c[2]
        v = torch.where((src[2] < 1) | (src[2] > dims[2]), f[mz][m], v)
        v = torch.where((src[1] < 1) | (src[1] > dims[1]), f[my][m], v)
        if thermal:
            edge = _geq(st.t_inlet * one, (u_in * one, zero, zero), k)
            v = torch.where((src[0] < 1) | (src[0] > dims[0]), edge, v)
        else:
            v = torch.where(src[0] > dims[0], _feq(one, (u_in * one, zero, zero), k, st.compressible), v)
            ui = u_in * one
            if st.inlet_turbulence > 0:
                # the noise is indexed by the pulling cell's y, z and the sub-step
                ui = ui + _noise(L.pos[1][m], L.pos[2][m], step % 1000000) * st.inlet_turbulence * u_in
            v = torch.where(src[0] < 1, _feq(one, (ui, zero, zero), k, st.compressible), v)
        out[k][m] = v
    return out


def _wale(L, vel, c_wale):
    G = [[None] * 3 for _ in range(3)]
    for j in range(3):
        e = [0, 0, 0]
        e[j] = 1
        hi, lo = L.neighbor(*e), L.neighbor(*[-x for x in e])
        hi, lo = torch.where(hi < 0, L.t, hi), torch.where(lo < 0, L.t, lo)
        for i in range(3):
            G[i][j] = 0.5 * (vel[i][hi] - vel[i][lo])
    q = [[sum(G[i][a] * G[a][j] for a in range(3)) for j in range(3)] for i in range(3)]
    tr = (q[0][0] + q[1][1] + q[2][2]) / 3
    a = b = 0
    for i in range(3):
        for j in range(3):
            sd = 0.5 * (q[i][j] + q[j][i]) - (tr if i == j else 0)
            s = 0.5 * (G[i][j] + G[j][i])
            a, b = a + sd * sd, b + s * s
    den = b * b * torch.sqrt(b.clamp(min=1e-12)) + a * a.clamp(min=1e-12) ** 0.25
    return torch.where((a > 1e-12) & (den > 1e-12), c_wale ** 2 * a ** 1.5 / den.clamp(min=1e-300), 0.0)


def _wall_force(L, rho, u):
    d, nu = L.wall, (L.tau - 0.5) / 3
    um = torch.sqrt(u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    on = (d > 0) & (d < 10) & (um > 1e-6) & (nu > 1e-10)
    um = um.clamp(min=1e-30)
    ut = (um * (nu / (d * um + 1e-10)) ** (1 / 7) * 16.6 ** (-1 / 7)).clamp(min=1e-6)
    yp = ut * d / nu
    up = torch.log(yp.clamp(min=1e-30)) / 0.41 + 5.2
    ut = torch.where((yp > 11.81) & (up > 0.1), (um / up.clamp(min=0.1)).clamp(min=1e-6), ut)
    tw, tr = rho * ut * ut, rho * nu * um / d
    fm = torch.where(on & (tw > tr), (tw - tr) / d, 0.0)
    return [-fm * v / um for v in u]


def _shift(a, u, back):
    """Raw to central moments along one axis (triples in a), or back."""
    x, y, z = a
    if not back:
        m0, m1, m2 = x + y + z, z - x, x + z
        return m0, m1 - u * m0, m2 - 2 * u * m1 + u * u * m0
    m0, m1, m2 = x, y + u * x, z + 2 * u * y + u * u * x
    return 0.5 * (m2 - m1), m0 - m2, 0.5 * (m2 + m1)


def _cumulant(A, u, omega, st):
    A = list(A)

    def axis(a, back):
        for i in range(27):
            if i // 3 ** a % 3 == 0:
                j = (i, i + 3 ** a, i + 2 * 3 ** a)
                A[j[0]], A[j[1]], A[j[2]] = _shift([A[x] for x in j], u[a], back)

    for a in range(3):
        axis(a, False)
    r = A[0]
    inv = 1 / r.clamp(min=0.01)
    m = {(i % 3, i // 3 % 3, i // 9): A[i] * inv for i in range(27)}
    o4d = st.omega_4
    if st.adaptive_omega4:
        o4d = (-(omega - 2) ** 2 / (st.lambda_param * omega + 1e-10)).clamp(0.01, 2.0)
    s2 = [m[2, 0, 0], m[0, 2, 0], m[0, 0, 2]]
    off = {0: m[0, 1, 1], 1: m[1, 0, 1], 2: m[1, 1, 0]}  # by the axis left out
    pairs = [(0, 1, 2), (0, 2, 1), (1, 2, 0)]            # (i, j, axis left out)

    def e(*ax):
        v = [0, 0, 0]
        for x in ax:
            v[x] += 1
        return tuple(v)

    Cd = {c: m[e(i, i, j, j)] - s2[i] * s2[j] - 2 * off[c] ** 2 for i, j, c in pairs}
    # C211 and its permutations: axis a twice, the other two once
    Co = {}
    for a in range(3):
        b, c = [x for x in range(3) if x != a]
        Co[a] = m[e(a, a, b, c)] - s2[a] * off[a] - 2 * off[c] * off[b]
    tr = s2[0] + s2[1] + s2[2]
    trs = (1 - st.omega_bulk) * tr + st.omega_bulk
    d1, d2 = (1 - omega) * (s2[0] - s2[1]), (1 - omega) * (s2[0] - s2[2])
    n2 = [(trs + d1 + d2) / 3, (trs - 2 * d1 + d2) / 3, (trs + d1 - 2 * d2) / 3]
    no = {a: (1 - omega) * off[a] for a in range(3)}
    if st.limiter == 1:
        for i, j, c in pairs:
            bnd = torch.sqrt((n2[i] * n2[j]).clamp(min=0))
            no[c] = torch.maximum(torch.minimum(no[c], bnd), -bnd)
    o3 = 1 - st.omega_3
    n = {k: o3 * v for k, v in m.items() if sum(k) == 3}
    n111 = n[1, 1, 1]
    nCd = {c: (1 - o4d) * v for c, v in Cd.items()}
    nCo = {a: (1 - st.omega_4) * v for a, v in Co.items()}
    n[0, 0, 0] = torch.ones_like(r)
    n[1, 0, 0] = n[0, 1, 0] = n[0, 0, 1] = torch.zeros_like(r)
    n[2, 0, 0], n[0, 2, 0], n[0, 0, 2] = n2
    n[0, 1, 1], n[1, 0, 1], n[1, 1, 0] = no[0], no[1], no[2]
    for i, j, c in pairs:
        n[e(i, i, j, j)] = nCd[c] + n2[i] * n2[j] + 2 * no[c] ** 2
    for a in range(3):
        b, c = [x for x in range(3) if x != a]
        n[e(a, a, b, c)] = nCo[a] + n2[a] * no[a] + 2 * no[c] * no[b]
    for i, j, c in pairs:  # 221: axes i, j twice, c once
        n[e(i, i, j, j, c)] = (n2[i] * n[e(j, j, c)] + n2[j] * n[e(i, i, c)] + 4 * no[c] * n111 +
                               2 * no[j] * n[e(i, j, j)] + 2 * no[i] * n[e(i, i, j)])
    v = sum(n2[c] * nCd[c] for c in range(3)) + 4 * sum(no[a] * nCo[a] for a in range(3))
    v = v + 2 * (n[2, 1, 0] * n[0, 1, 2] + n[2, 0, 1] * n[0, 2, 1] + n[1, 2, 0] * n[1, 0, 2]) + 4 * n111 ** 2
    v = v + n2[0] * n2[1] * n2[2] + 2 * sum(n2[a] * no[a] ** 2 for a in range(3)) + 8 * no[0] * no[1] * no[2]
    n[2, 2, 2] = v
    A = [r * n[i % 3, i // 3 % 3, i // 9] for i in range(27)]
    for a in (2, 1, 0):
        axis(a, True)
    return A


def _bgk(A, rho, u, omega, st):
    fe = [_feq(rho, u, k, st.compressible) for k in range(27)]
    c = list(zip(_CX, _CY, _CZ))
    P = [[sum((A[k] - fe[k]) * (c[k][i] * c[k][j]) for k in range(27) if c[k][i] * c[k][j])
          for j in range(3)] for i in range(3)]
    out = []
    for k in range(27):
        s = sum(P[i][j] * (c[k][i] * c[k][j] - (1 / 3 if i == j else 0)) for i in range(3) for j in range(3))
        out.append(fe[k] + (1 - omega) * _W[k] * 4.5 * s)
    return out


def _positivity(A, rho, u, st):
    fe = [_feq(rho, u, k, st.compressible) for k in range(27)]
    low = torch.stack(A).min(0).values < 0
    alpha = torch.ones_like(rho)
    for k in range(27):
        fn = A[k] - fe[k]
        lim = fe[k] / (fe[k] - fn + 1e-15)
        alpha = torch.where((fn < 0) & (fe[k] > 1e-15), torch.minimum(alpha, lim), alpha)
    alpha = alpha.clamp(min=0)
    return [torch.where(low, fe[k] + alpha * (A[k] - fe[k]), A[k]) for k in range(27)]


def _bouzidi(L, f, q_min):
    post = f.clone()
    cells, q = L.links
    for k in range(27):
        on = torch.nonzero((q[k] > q_min) & (q[k] <= 1)).reshape(-1)
        if on.numel() == 0:
            continue
        x, qk = cells[on], q[k][on]
        far = L.neighbor(-_CX[k], -_CY[k], -_CZ[k], x)
        fk = post[k][x]
        ff = torch.where(far >= 0, post[k][far.clamp(min=0)], fk)
        f[26 - k][x] = torch.where(qk < 0.5, 2 * qk * fk + (1 - 2 * qk) * ff,
                                   fk / (2 * qk) + (2 * qk - 1) / (2 * qk) * post[26 - k][x])


def _exact_step(L, P, s, st, dims, u_in, step, tw):
    """One sub-step of a level: state s = {f, rho, vel, g, T} -> the new one."""
    A = _pull(L, P, s["f"], st, dims, u_in, step, tw, False)
    bounced = A.flip(0)
    rho = A.sum(0)
    u = [sum(c[k] * A[k] for k in range(27) if c[k]) for c in (_CX, _CY, _CZ)]
    rho = rho.clamp(min=0.01)
    inv = 1 / rho
    g = L.sponge
    u = [v * inv for v in u]
    rho = rho * (1 - g) + g
    u = [u[0] * (1 - g) + u_in * g, u[1] * (1 - g), u[2] * (1 - g)]
    if st.sponge_blend:
        one = torch.ones_like(rho)
        for k in range(27):
            A[k] = A[k] * (1 - g) + _feq(one, (u_in * one, 0 * one, 0 * one), k, st.compressible) * g
    F = _wall_force(L, rho, u) if st.wall_model else [0 * rho] * 3
    ue = [v + 0.5 * x * inv for v, x in zip(u, F)]
    nu_t = _wale(L, s["vel"], st.c_wale) if st.c_wale else 0 * rho
    nu_t = nu_t.clamp(min=st.nu_sgs_bg)
    omega = 1 / (L.tau + 3 * nu_t).clamp(min=0.500001)
    if st.op == 0:
        B = _cumulant(A, ue, omega, st)
        if st.limiter == 2:
            B = _positivity(B, rho, ue, st)
    else:
        B = _bgk(A, rho, ue, omega, st)
    del A
    for k in range(27):
        c = (_CX[k], _CY[k], _CZ[k])
        if st.wall_model:
            cu = sum(a * b for a, b in zip(c, ue))
            ft = 3 * _W[k] * sum((c[i] - u[i] + 3 * cu * c[i]) * F[i] for i in range(3))
            B[k] = B[k] + (1 - 0.5 * omega) * ft
        B[k] = torch.where(L.solid, bounced[k], B[k])
    f = torch.stack(B)
    del B, bounced
    out = {"f": f, "rho": torch.where(L.solid, 1.0, rho),
           "vel": torch.stack([torch.where(L.solid, 0.0, v) for v in u])}
    if L.links is not None:
        _bouzidi(L, f, st.q_min)
    if st.ddf:
        G = _pull(L, P, s["g"], st, dims, u_in, step, tw, True)
        Ts = G.sum(0)
        v = out["vel"]
        T = Ts.clamp(min=0.01) * (1 - g) + st.t_inlet * g
        v = [v[0] * (1 - g) + u_in * g, v[1] * (1 - g), v[2] * (1 - g)]
        og = 1 / max(L.tau_g, 0.500001)
        one = torch.ones_like(T)
        for k in range(27):
            gs = G[k]
            if st.sponge_blend:
                gs = gs * (1 - g) + _geq(st.t_inlet * one, (u_in * one, 0 * one, 0 * one), k) * g
            back = s["g"][26 - k]
            if not st.wall_bc_adiabatic:
                back = 2 * _W[k] * st.t_wall - back
            G[k] = torch.where(L.solid, back, gs - og * (gs - _geq(T, v, k)))
        out["g"] = G
        out["T"] = torch.where(L.solid, Ts if st.wall_bc_adiabatic else st.t_wall * one, T)
        if L.links is not None:
            _bouzidi(L, G, st.q_min)
    return out


def _exact_march(levels, states, st, dims, u_in, first, steps):
    def go(i, step, tw):
        L = levels[i]
        d = [x * 2 ** i for x in dims]
        old = states[i]
        states[i] = _exact_step(L, levels[i - 1] if i else None, old, st, d, u_in, step, tw)
        if i + 1 < len(levels):
            L.old, L.new = old, states[i]
            go(i + 1, 2 * step, 0.0)
            go(i + 1, 2 * step + 1, 0.5)
    for s in range(steps):
        go(0, first + s, 0.0)


def _exact_forces(sim, lv, vel, rho, radius):
    """Surface maps, their sums and (closed body) net forces of a level."""
    p, cfg, h, mesh = sim.p, sim.cfg, lv.host, sim.mesh
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a.astype(np.float32))).to(DEV).double()  # noqa: E731
    c, nrm, area = d(mesh.centers), d(mesh.normals), d(mesh.areas)
    fp = solver.force_params_for(lv, p, cfg, radius)
    dx = fp.dx
    c = c + torch.tensor([fp.offset_x, fp.offset_y, fp.offset_z], dtype=torch.float64, device=DEV)
    L = _Level(h, h.tau, h.tau_g)
    best = torch.zeros((len(c), 5), dtype=torch.float64, device=DEV)
    best[:, 0], wbest = 1.0, torch.zeros(len(c), dtype=torch.float64, device=DEV)
    done = torch.zeros(len(c), dtype=torch.bool, device=DEV)
    for r in range(1, radius + 1):
        x = (c + nrm * ((r + 0.5) * dx)) / dx - 0.5
        lo = torch.floor(x)
        fr, lo = (x - lo).clamp(0, 1), lo.long() + 1
        acc = torch.zeros((len(c), 5), dtype=torch.float64, device=DEV)
        for s in range(8):
            g = [lo[:, a] + (s >> a & 1) for a in range(3)]
            w = 1.0
            ok = torch.ones(len(c), dtype=torch.bool, device=DEV)
            for a in range(3):
                w = w * (fr[:, a] if s >> a & 1 else 1 - fr[:, a])
                ok &= (g[a] >= 1) & ((g[a] - 1) // 8 < L.dim[a])
            i = (g[0] - 1) // 8 + L.dim[0] * ((g[1] - 1) // 8 + L.dim[1] * ((g[2] - 1) // 8))
            b = torch.where(ok, L.ptr[torch.where(ok, i, 0)], 0) - 1
            cell = b.clamp(min=0) * 512 + (g[0] - 1) % 8 + 8 * ((g[1] - 1) % 8) + 64 * ((g[2] - 1) % 8)
            w = torch.where((b >= 0) & ~L.solid[cell], w, 0.0)
            acc += w[:, None] * torch.stack([rho[cell], vel[0][cell], vel[1][cell], vel[2][cell],
                                             torch.ones_like(w)], 1)
        w = acc[:, 4]
        use = ~done & (w > 0.01) & ((w >= 0.5) | (w > wbest))
        new = torch.cat([acc[:, :4] / w.clamp(min=1e-30)[:, None], torch.full_like(w, r + 0.5)[:, None]], 1)
        best = torch.where(use[:, None], new, best)
        wbest = torch.where(use, w, wbest)
        done |= (w > 0.01) & (w >= 0.5)
    if bool((wbest <= 0).any()):
        return None  # a triangle that needs the nearest-cell search
    rr, u, dist = best[:, 0], best[:, 1:4], best[:, 4]
    pr = (rr - 1) / 3 * fp.pressure_scale
    ut = u - (u * nrm).sum(1, keepdim=True) * nrm
    um = ut.norm(dim=1)
    nu = (fp.tau_molecular - 0.5) / 3
    nus = torch.where(um > 1e-10, fp.c_wale ** 2 * um / dist, 0.0).clamp(min=fp.nu_sgs_bg)
    tau = torch.where(um > 1e-10, rr * (nu + nus) / dist * fp.stress_scale, 0.0)[:, None] * ut
    Fp, Fv = -pr[:, None] * nrm * area[:, None], tau * area[:, None]
    arm = c - torch.tensor([fp.ref_x, fp.ref_y, fp.ref_z], dtype=torch.float64, device=DEV)
    raw = torch.cat([Fp.sum(0), Fv.sum(0), torch.linalg.cross(arm, Fp + Fv).sum(0)])
    maps = torch.stack([pr, tau[:, 0], tau[:, 1], tau[:, 2]])
    return raw, maps, tuple((Fp + Fv).T)


def _exact_stats(L, rho, vel):
    fl = ~L.solid
    r, v2 = rho[fl], (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)[fl]
    return {"n_fluid": int(fl.sum()), "rho_mean": float(r.mean()), "rho_min": float(r.min()),
            "rho_max": float(r.max()), "v_max": float(v2.max().sqrt()),
            "kinetic_energy": float((0.5 * r * v2).sum()), "mass": float(rho.sum())}


def exact(case, seed):
    if case["kind"] == "pool":
        # the retiring case alone: the others would take minutes
        pc = _pool_cases(case, seed)[-1]
        levels = [_Level(h, h.tau, h.tau_g) for h in pc.levels]
        w = torch.tensor(_W, dtype=torch.float64, device=DEV)
        states = [{"f": w[:, None].repeat(1, 512 * L.n),
                   "rho": torch.ones(512 * L.n, dtype=torch.float64, device=DEV),
                   "vel": torch.zeros((3, 512 * L.n), dtype=torch.float64, device=DEV)}
                  for L in levels]
        p = pc.params
        _exact_march(levels, states, pc.settings, (p.nx_coarse, p.ny_coarse, p.nz_coarse),
                     float(np.float32(pc.cfg.u_target)), 1, POOL_WARM + case["steps"])
        view = type("V", (), dict(p=p, cfg=pc.cfg, mesh=pc.mesh))()
        lv = type("V", (), dict(host=pc.levels[-1]))()
        got = _exact_forces(view, lv, states[-1]["vel"], states[-1]["rho"], 5)
        coef = None
        if got is not None:
            F, M = got[0][:3] + got[0][3:6], got[0][6:]
            ref = 0.5 * p.rho_physical * p.u_physical ** 2 * p.reference_area
            coef = torch.cat([F[[0, 2, 1]] / ref, M / (ref * p.reference_chord), F, M])
        return {"coefficients": [None] * (case["count"] - 1) + [coef],
                "fields": [(s["rho"], s["vel"].reshape(-1)) for s in states]}
    cfg, mesh, p, hosts = _with_options(case, _domain(case["body"], case["size"], case["levels"]))
    dims = (p.nx_coarse, p.ny_coarse, p.nz_coarse)
    st = solver.StepSettings.from_config(cfg, cfg.wall_model_enabled)
    levels = [_Level(h, h.tau, h.tau_g) for h in hosts]
    states = []
    for h in hosts:
        s = _flow_state(h, dims, cfg.u_target, seed, cfg.ddf_enabled)
        x = {"f": s["f"].double().reshape(27, -1), "rho": s["rho"].double(),
             "vel": s["vel"].double().reshape(3, -1)}
        if cfg.ddf_enabled:
            x["g"], x["T"] = s["g"].double().reshape(27, -1), s["T"].double()
        states.append(x)
    if case["kind"] == "diagnose":
        view = type("V", (), dict(p=p, cfg=cfg, mesh=mesh))()
        lv = type("V", (), dict(host=hosts[-1]))()
        got = _exact_forces(view, lv, states[-1]["vel"], states[-1]["rho"], case["search_radius"])
        raw, maps, net = got if got else (None, None, None)
        return {"stats": _exact_stats(levels[0], states[0]["rho"], states[0]["vel"]), "raw": raw,
                "maps": maps, "net": net}
    _exact_march(levels, states, st, dims, cfg.u_target, 1, case["steps"])
    return [{k: v.reshape(-1) for k, v in s.items()} for s in states]
