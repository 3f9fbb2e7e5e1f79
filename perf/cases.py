"""What the framework's time is measured on: calls through its public entry
points, over the sizes, patch widths, boundary rules, friction options and
forms (host arrays, device-resident levels, forests, served scenarios,
topography) that a flood program uses.

Inputs are synthetic and made from a seed: fractal beds, ponds and rivers
with fractal shore lines, smooth currents and waves on them, so that every
kind of face occurs: still and moving water, shocks and rarefactions, wet/dry
fronts and dry land.

A device-resident step starts from the saved state of the step (one copy on
the device): the driver saves the state of a step before it takes it, to
retake it when the CFL number comes out too large.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import geoflood_gb300 as gf
from geoflood_gb300 import _lib, synth
from geoflood_gb300.forest import batch_run
from geoflood_gb300.topo import Topo

MBC = 2
G = 9.81
DRY = 1.0e-3


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the per-patch solver hook on one patch of the default dam-break
        # configuration: the smallest call, host arrays in and out
        dict(name="patch_one", kind="batch", m=32, n=1, wet=0.8, maux=1, friction="manning"),
        # the buffered hook's flush of a small AMR level: an odd number of 16^2 patches
        dict(name="patch_batch", kind="batch", m=16, n=129, wet=0.6, maux=1, friction="manning"),
        # a coarse level of a small run, 8^2 patches: launch and latency bound
        dict(name="level_small", kind="level", m=8, npx=6, npy=4, wet=0.7, maux=1,
             friction="manning", order=2, transverse=2, limiter=4, bc=3),
        # an ordinary level: more patches than SMs, fewer than two for each
        dict(name="level_mid", kind="level", m=32, npx=19, npy=13, wet=0.7, maux=1,
             friction="manning", order=2, transverse=2, limiter=4, bc=1),
        # a large wet level of 16^2 patches with a land-cover friction field
        dict(name="level_wide", kind="level", m=16, npx=83, npy=67, wet=0.9, maux=2,
             friction="variable", order=2, transverse=2, limiter=4, bc=3),
        # the uniform dam-break level of the benchmark: 4096 patches of 32^2, a third wet
        dict(name="level_flood", kind="level", m=32, npx=64, npy=64, wet=0.35, maux=1,
             friction="manning", order=2, transverse=2, limiter=4, bc=1),
        # the same step when the state lives on the host (pinned arrays), as a
        # driver that keeps its own patches calls it
        dict(name="level_host", kind="host", m=32, npx=37, npy=29, wet=0.5, maux=1,
             friction="manning", order=2, transverse=2, limiter=4, bc=1),
        # one AMR exchange between two levels (fine to coarse, coarse to fine),
        # the fill of new children and the refinement tags of a regrid
        dict(name="exchange", kind="exchange", m=16, n=311, wet=0.6),
        # an adaptive dam-break run from its initial refinement, regrid every second step
        dict(name="forest_run", kind="forest", m=16, nbx=2, nby=1, lmin=1, lmax=3, steps=12),
        # a batch of adaptive river floods of all patch widths in shared launches
        dict(name="forest_batch", kind="forests", n=6, patches=120.0, lmin=1, lmax=4, t=2.0),
        # single-level river floods of mixed patch widths through the scenario server
        dict(name="served", kind="served", n=9, cells=20000.0, t=8.0),
        # cell-averaged bathymetry of a level from a DEM with a finer inset
        dict(name="dem", kind="dem", n0=1025, n1=513, nx=1531, ny=1531),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _brick(rng, lo, hi):
    """npx, npy of a brick of about lo..hi patches."""
    n = _log(rng, lo, hi)
    npx = max(1, min(int(hi), int(round(math.sqrt(n) * rng.uniform(0.7, 1.4)))))
    return npx, max(1, min(int(n // npx), int(hi) // npx))


def draw(rng):
    kind = rng.choice(["batch", "batch", "level", "level", "level", "level", "level", "host", "host",
                       "exchange", "forest", "forests", "served", "dem"])
    m = rng.choice([8, 16, 32])
    cap = {8: 16000, 16: 8000, 32: 4000}[m]
    c = dict(kind=kind)
    if kind == "batch":
        c.update(m=m, n=int(_log(rng, 1, 600)), wet=round(rng.uniform(0.2, 1.0), 3),
                 maux=rng.choice([1, 2, 3]), friction=rng.choice(["manning", "table", "none"]))
    elif kind in ("level", "host"):
        npx, npy = _brick(rng, 1, cap if kind == "level" else cap // 3)
        friction = rng.choice(["manning", "manning", "table", "variable", "none"])
        c.update(m=m, npx=npx, npy=npy, wet=round(rng.uniform(0.1, 1.0), 3),
                 maux=2 if friction == "variable" else rng.choice([1, 1, 3]), friction=friction,
                 order=rng.choice([2, 2, 2, 2, 1]), transverse=rng.choice([2, 2, 2, 1, 0]),
                 limiter=rng.choice([4, 4, 4, 1, 2, 3]), bc=rng.choice([1, 3]))
    elif kind == "exchange":
        c.update(m=m, n=int(_log(rng, 3, 1500)), wet=round(rng.uniform(0.2, 1.0), 3))
    elif kind == "forest":
        c.update(m=rng.choice([8, 16]), nbx=rng.choice([1, 2]), nby=rng.choice([1, 2]), lmin=1, lmax=3,
                 steps=rng.randint(4, 12))
    elif kind == "forests":
        c.update(n=rng.randint(2, 6), patches=round(_log(rng, 30, 120), 1), lmin=1, lmax=4,
                 t=round(rng.uniform(0.8, 2.0), 3))
    elif kind == "served":
        c.update(n=rng.randint(2, 9), cells=round(_log(rng, 4000, 20000), 0), t=round(rng.uniform(3.0, 8.0), 3))
    else:
        c.update(n0=rng.randint(200, 1025), n1=rng.randint(100, 513), nx=rng.randint(100, 1531),
                 ny=rng.randint(100, 1531))
    return c


def work(case):
    """Algorithmic bytes: each state, bathymetry or node value read once and
    each result written once. Operations: about 420 for a wet cell's update (two
    face solves with their limiter, transverse split and friction), 25 for a
    cell of a transfer or a node cell of an integral."""
    k = case["kind"]
    if k in ("batch", "level", "host"):
        n = case["n"] if k == "batch" else case["npx"] * case["npy"]
        cells = n * case["m"] ** 2
        ghost = 0 if k == "batch" else n * ((case["m"] + 4) ** 2 - case["m"] ** 2) * 24
        extra = 8 if case["friction"] == "variable" else 0
        return {"bytes": cells * (56 + extra) + ghost, "flops": 420.0 * cells * case["wet"]}
    if k == "exchange":
        m, n = case["m"], case["n"]
        cells = n * (2 * m + 2 * (2 * m) * 2 + 4 * (m + 2) ** 2)
        return {"bytes": 56.0 * cells + 2 * n * m * m * 32, "flops": 25.0 * cells}
    if k == "forest":
        cells = case["nbx"] * case["nby"] * case["m"] ** 2 * 4 ** case["lmax"] // 3
        return {"bytes": 56.0 * cells * case["steps"], "flops": 420.0 * cells * case["steps"]}
    if k == "forests":
        cells = case["n"] * case["patches"] * 448
        steps = case["t"] / 0.15
        return {"bytes": 56.0 * cells * steps, "flops": 200.0 * cells * steps}
    if k == "served":
        cells = case["n"] * case["cells"]
        steps = case["t"] / 0.6
        return {"bytes": 56.0 * cells * steps, "flops": 60.0 * cells * steps}
    nodes = case["n0"] ** 2 + case["n1"] ** 2
    cells = case["nx"] * case["ny"]
    return {"bytes": 8.0 * (nodes + cells), "flops": 25.0 * (nodes + cells)}


# ----------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _surface(ny, nx, gen, power):
    """(ny, nx) random surface with spectrum k^-power, values in [0, 1]."""
    w = torch.randn((ny, nx), dtype=torch.float64, device="cuda", generator=gen)
    kx = torch.fft.rfftfreq(nx, dtype=torch.float64, device="cuda") * nx / max(nx, ny)
    ky = torch.fft.fftfreq(ny, dtype=torch.float64, device="cuda") * ny / max(nx, ny)
    k = torch.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2)
    k[0, 0] = 1.0
    a = torch.fft.irfft2(torch.fft.rfft2(w) * k ** (-power), s=(ny, nx))
    return (a - a.min()) / (a.max() - a.min())


def _state(ny, nx, dx, wet, seed):
    """Global (ny, nx) bed and flow: b, h, hu, hv."""
    gen = _gen(seed)
    relief = 30.0 * min(1.0, max(nx, ny) * dx / 512.0)
    b = relief * _surface(ny, nx, gen, 1.8)
    level = torch.quantile(b.flatten()[:: max(1, b.numel() // 100000)], wet)
    eta = level + 1.0 * (_surface(ny, nx, gen, 3.0) - 0.5)
    h = torch.clamp(eta - b, min=0.0)
    h = torch.where(h < 0.5 * DRY, torch.zeros_like(h), h)
    u = 3.0 * (_surface(ny, nx, gen, 3.0) - 0.5)
    v = 3.0 * (_surface(ny, nx, gen, 3.0) - 0.5)
    return b, h, h * u, h * v


def _pad(a, bc, neg_x=False, neg_y=False):
    """Two ghost cells by extrapolation (bc 1) or a wall (bc 3), x sides then y sides."""
    if bc == 1:
        ix = torch.arange(-MBC, a.shape[1] + MBC, device=a.device).clamp(0, a.shape[1] - 1)
        iy = torch.arange(-MBC, a.shape[0] + MBC, device=a.device).clamp(0, a.shape[0] - 1)
        return a[:, ix][iy]
    sx, sy = (-1.0 if neg_x else 1.0), (-1.0 if neg_y else 1.0)
    a = torch.cat([sx * a[:, :MBC].flip(1), a, sx * a[:, -MBC:].flip(1)], dim=1)
    return torch.cat([sy * a[:MBC].flip(0), a, sy * a[-MBC:].flip(0)], dim=0)


def _tiles(a, m):
    """(patches, m + 4, m + 4) windows of a padded global array."""
    w = a.unfold(0, m + 2 * MBC, m).unfold(1, m + 2 * MBC, m)
    return w.reshape(-1, m + 2 * MBC, m + 2 * MBC).contiguous()


def _pad_state(h, hu, hv, bc):
    return _pad(h, bc), _pad(hu, bc, neg_x=True), _pad(hv, bc, neg_y=True)


def _dt(h, hu, hv, dx, cfl):
    w = h > DRY
    hs = torch.where(w, h, torch.ones_like(h))
    sp = torch.where(w, torch.maximum(hu.abs(), hv.abs()) / hs + torch.sqrt(G * hs), torch.zeros_like(h))
    return cfl * dx / max(float(sp.max()), 1.0)


def _phys(case):
    f = case["friction"]
    lim = case.get("limiter", 4)
    kw = dict(order=case.get("order", 2), transverse=case.get("transverse", 2), mthlim=(lim, lim, lim))
    if f == "none":
        return gf.Phys(friction_forcing=False, **kw)
    if f == "table":  # river bed and flood plain by bed elevation
        return gf.Phys(manning_coefficient=(0.03, 0.06), manning_break=(8.0, 1.0e10), **kw)
    if f == "variable":
        return gf.Phys(variable_friction=True, friction_index=2, **kw)
    return gf.Phys(**kw)


def _patches(case, seed):
    """Inputs of a brick: q (P, 3, n4, n4), aux (P, maux, n4, n4), dx, dt."""
    m, dx, bc = case["m"], 2.0, case.get("bc", 1)
    npx, npy = (case["npx"], case["npy"]) if "npx" in case else (case["n"], 1)
    b, h, hu, hv = _state(npy * m, npx * m, dx, case["wet"], seed)
    q = torch.stack([_tiles(a, m) for a in _pad_state(h, hu, hv, bc)], dim=1)
    aux = [_tiles(_pad(b, bc), m)]
    gen = _gen(seed + 77)
    for _ in range(1, case["maux"]):  # land cover: Manning coefficients
        aux.append(_tiles(_pad(0.02 + 0.06 * _surface(npy * m, npx * m, gen, 2.0), bc), m))
    cfl = 0.45 if case["kind"] == "host" else 0.8
    return q, torch.stack(aux, dim=1), dx, _dt(h, hu, hv, dx, cfl)


def _host(a):
    """Planes (P, nf, n4, n4) as the hooks' Fortran layout (P, n4, n4, nf) on the host."""
    return a.permute(0, 2, 3, 1).contiguous().cpu().numpy()


class _Planes:
    """Device memory of a level as an array interface; a tensor made from it keeps the level alive."""

    def __init__(self, lev, ptr, shape):
        self.level = lev
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _planes(lev):
    q = _lib._dp()
    assert lev._lib.gf_level_device_planes(lev.h, C.byref(q), None) == 0
    n4 = lev.m + 2 * MBC
    return torch.as_tensor(_Planes(lev, C.cast(q, C.c_void_p).value, (lev.npatch, 3, n4, n4)), device="cuda")


def _level(ctx, case, q, aux, dx):
    m, npx, npy = case["m"], case["npx"], case["npy"]
    lev = gf.Level(ctx, q.shape[0], m, aux.shape[1])
    lev.set_geometry(dx, dx)
    nbr, xl, yl = synth.brick_layout(npy, npx, m, dx)
    lev.set_layout(nbr, xl, yl)
    lev.set_bc([case["bc"]] * 4)
    lev.upload(_host(q), _host(aux))
    return lev


def prepare(case, seed):
    return {"batch": _prepare_batch, "level": _prepare_level, "host": _prepare_level,
            "exchange": _prepare_exchange, "forest": _prepare_forest, "forests": _prepare_forests,
            "served": _prepare_served, "dem": _prepare_dem}[case["kind"]](case, int(seed))


def _prepare_batch(case, seed):
    q, aux, dx, dt = _patches(case, seed)
    q0, a0 = _host(q), _host(aux)
    cur = q0.copy()
    return dict(case=case, ctx=gf.Context(0, _phys(case)), q0=q0, cur=cur, qs=list(cur), auxs=list(a0),
                dx=dx, dt=dt)


def _prepare_level(case, seed):
    q, aux, dx, dt = _patches(case, seed)
    ctx = gf.Context(0, _phys(case))
    lev = _level(ctx, case, q, aux, dx)
    s = dict(case=case, ctx=ctx, lev=lev, dt=dt)
    if case["kind"] == "host":
        n4 = case["m"] + 2 * MBC
        pin = torch.empty((q.shape[0], n4, n4, 3), dtype=torch.float64, pin_memory=True)
        pin.copy_(q.permute(0, 2, 3, 1))
        s.update(pin=pin, qh=pin.numpy())
    else:
        s.update(q0=q, planes=_planes(lev), stream=torch.cuda.ExternalStream(ctx.stream))
    torch.cuda.synchronize()
    return s


def _amr(case, seed):
    """A column of n coarse patches, the 2 n fine patches to the right of it
    and the 4 n children of the coarse patches: planes of each, by seed."""
    m, n, dx = case["m"], case["n"], 4.0
    b, h, hu, hv = _state(2 * n * m, 2 * m, dx / 2, case["wet"], seed)
    fine = torch.stack([_tiles(a, m) for a in _pad_state(h, hu, hv, 1)], dim=1)
    fineb = _tiles(_pad(b, 1), m)
    fine, fineb = fine[0::2].contiguous(), fineb[0::2].contiguous()  # the left column of fine patches
    cb, ch, chu, chv = _state(n * m, m, dx, case["wet"], seed + 1)
    coarse = torch.stack([_tiles(a, m) for a in _pad_state(ch, chu, chv, 1)], dim=1)
    coarseb = _tiles(_pad(cb, 1), m)
    kb = _tiles(_pad(cb.repeat_interleave(2, 0).repeat_interleave(2, 1), 1), m)
    return coarse, coarseb, fine, fineb, kb


def _prepare_exchange(case, seed):
    m, n = case["m"], case["n"]
    coarse, coarseb, fine, fineb, kb = _amr(case, seed)
    ctx = gf.Context(0, gf.Phys())
    lv = []
    for q, b, dx in ((coarse, coarseb, 4.0), (fine, fineb, 2.0), (torch.zeros_like(kb)[:, None].repeat(1, 3, 1, 1), kb, 2.0)):
        lev = gf.Level(ctx, q.shape[0], m, 1)
        lev.set_geometry(dx, dx)
        lev.upload(_host(q), _host(b[:, None]))
        lv.append(lev)
    avg, itp, new = [], [], []
    for k in range(n):
        for half in range(2):
            avg.append((0, k, 2 * k + half, 1, -2 * m, -half * m))
            itp.append((2, k, 2 * k + half, 1, -2 * m, -half * m))
        for igrid in range(4):  # children in the brick's row-major order
            new.append((4, k, (2 * k + igrid // 2) * 2 + igrid % 2, igrid, 0, 0))
    lists = [(len(t), (_lib.gf_transfer * len(t))(*[_lib.gf_transfer(*x) for x in t])) for t in (avg, itp, new)]
    rf = gf.Refine(wave_tolerance=1e9, flowgrades=((1.5, 2, 1, 4),))
    torch.cuda.synchronize()
    return dict(case=case, ctx=ctx, lv=lv, lists=lists, rf=rf, planes=[_planes(x) for x in lv])


def _frames(F, nbx, nby):
    """Buffers that hold any set of leaves: cells and (level, I, J)."""
    cap = nbx * nby * 4 ** F.maxlevel
    return np.zeros((cap, F.mx, F.mx, 3)), np.full((cap, 3), -1, np.int64)


def _frame(F, out):
    """The current leaves into `out`; ghost cells are scratch between steps."""
    q, leaves = out
    n = F.npatch
    q[:n] = F.download()[:, MBC:-MBC, MBC:-MBC]
    q[n:] = 0.0
    leaves[:n] = F.patches()
    leaves[n:] = -1
    return {"q": q, "leaves": leaves}


def _prepare_forest(case, seed):
    m, nbx, nby, lmin, lmax = case["m"], case["nbx"], case["nby"], case["lmin"], case["lmax"]
    dx0 = 1000.0 / m
    nx, ny = nbx * m << lmax, nby * m << lmax
    dxf = dx0 / (1 << lmax)
    b = synth.bump_ramp_dem(nx, ny, dxf, dxf, seed=seed)
    q = synth.dam_break_state(b, dxf, x_dam=0.6 * 500.0 * nbx)
    ctx = gf.Context(0, gf.Phys())
    rf = gf.Refine(wave_tolerance=1e9, flowgrades=((1.0, 2, 1, lmax),))
    F = gf.Forest(ctx, m, nbx, nby, lmin, lmax, dx0, dx0, b, q, mthbc=(3, 3, 3, 3), regrid_interval=2, refine=rf)
    return dict(case=case, ctx=ctx, forest=F, out=_frames(F, nbx, nby))


def _prepare_forests(case, seed):
    ctx = gf.Context(0, gf.Phys())
    fs, outs = [], []
    for k in range(case["n"]):
        sp = synth.flood_forest(seed * 31 + k, case["patches"], mx=(8, 16, 32)[k % 3], minlevel=case["lmin"],
                                maxlevel=case["lmax"])
        ctx.set_phys(1 + k, sp["phys"])
        F = gf.Forest(ctx, sp["mx"], sp["nbx"], sp["nby"], sp["minlevel"], sp["maxlevel"], sp["dx0"], sp["dy0"],
                      sp["aux"], sp["q"], mthbc=sp["mthbc"], regrid_interval=sp["regrid_interval"],
                      refine=sp["refine"], phys_slot=1 + k)
        F.set_hydrograph(*sp["hydro"])
        fs.append(F)
        outs.append(_frames(F, sp["nbx"], sp["nby"]))
    return dict(case=case, ctx=ctx, forests=fs, outs=outs)


def _prepare_served(case, seed):
    scs = []
    for k in range(case["n"]):
        cells = case["cells"] * (0.4, 1.0, 1.6)[(k // 3) % 3]
        sc = synth.flood_scenario(seed * 17 + k, cells, mx=(8, 16, 32)[k % 3], time_scale=1.0 / 300.0)
        sc.t_final = case["t"]
        scs.append(sc)
    return dict(case=case, server=gf.Server(0), scs=scs, outs=[np.zeros_like(s.q) for s in scs])


def _dem(case, seed):
    """Two DEM grids (node values, south first), (z, x0, y0, spacing): a fine
    inset inside a coarse one over [0, L]^2."""
    gen = _gen(seed)
    n0, n1 = case["n0"], case["n1"]
    d0 = 2.0
    L = (n0 - 1) * d0
    d1 = 0.45 * L / (n1 - 1)
    za = 40.0 * _surface(n0, n0, gen, 1.8)
    zb = 40.0 * _surface(n1, n1, gen, 1.8)
    return [(za, 0.0, 0.0, d0), (zb, 0.21 * L, 0.33 * L, d1)], L


def _prepare_dem(case, seed):
    grids, L = _dem(case, seed)
    topo = Topo()
    for z, x0, y0, d in grids:
        topo.add_grid(z.flip(0).contiguous().cpu().numpy(), x0, y0, d, d)
    return dict(case=case, ctx=gf.Context(0, gf.Phys()), topo=topo, L=L)


# -------------------------------------------------------------------- run

def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "batch":
        np.copyto(s["cur"], s["q0"])
        if case["n"] == 1:
            cfl = s["ctx"].patch_update(s["qs"][0], s["auxs"][0], s["dx"], s["dx"], 0.0, s["dt"])
            return {"q": s["cur"], "cfl": cfl}
        cfls, cfl = s["ctx"].patch_update_batch(s["qs"], s["auxs"], s["dx"], s["dx"], 0.0, s["dt"])
        return {"q": s["cur"], "cfl": cfl, "cfls": cfls}
    if k == "level":
        with torch.cuda.stream(s["stream"]):
            s["planes"].copy_(s["q0"])
        cfl = s["lev"].step(0.0, s["dt"])
        s["lev"].ghost_fill_async(s["dt"])
        return {"q": s["planes"], "cfl": cfl}
    if k == "host":
        cfl = s["lev"].step_host(s["qh"], 0.0, s["dt"])
        return {"q": s["qh"], "cfl": cfl}
    if k == "exchange":
        coarse, fine, kids = s["lv"]
        lib = coarse._lib
        for (n, tasks), to in zip(s["lists"], (fine, fine, kids)):
            if lib.gf_level_transfer(coarse.h, to.h, n, tasks) != 0:
                raise RuntimeError("gf_level_transfer")
        tags = fine.tag4refinement(s["rf"], 2, 3, 0, 0.0)
        return {"coarse": s["planes"][0], "fine": s["planes"][1], "new": s["planes"][2], "tags": tags}
    if k == "forest":
        F = s["forest"]
        F.init()
        st = F.run(1e9, 1, 5.0, 0.9, 1.0, max_steps=case["steps"])
        return {"t": st["t"], "steps": st["steps"], **_frame(F, s["out"])}
    if k == "forests":
        for F in s["forests"]:
            F.init()
        batch_run(s["forests"], case["t"], 1, 0.8, 0.9, 1.0)
        return [{"steps": F.stats()["steps"], **_frame(F, o)} for F, o in zip(s["forests"], s["outs"])]
    if k == "served":
        srv = s["server"]
        ids = [srv.submit(sc, o) for sc, o in zip(s["scs"], s["outs"])]
        srv.run_until_idle()
        steps = [srv.poll(i)["steps"] for i in ids]
        for i in ids:
            srv.release(i)
        return {"q": [o[:, MBC:-MBC, MBC:-MBC] for o in s["outs"]], "steps": steps}
    dx, dy = s["L"] / case["nx"], s["L"] / case["ny"]
    return s["topo"].raster(s["ctx"], case["nx"], case["ny"], 2, 0.0, 0.0, dx, dy, s["L"], s["L"])


# -------------------------------------- the same in 64 bits, plain tensors

def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        return _exact_batch(case, int(seed))
    if k in ("level", "host"):
        return _exact_level(case, int(seed))
    if k == "exchange":
        return _exact_exchange(case, int(seed))
    if k == "dem":
        return _exact_dem(case, int(seed))
    return None  # whole runs: many steps with their own time-step control


def _maxmod(x, y, z):
    return torch.maximum(torch.minimum(x, y), z)


def _where0(c, x):
    return torch.where(c, x, torch.zeros_like(x))


def _middle(hL, hR, uL, uR):
    """Speeds at the middle state of a Riemann problem over a flat bed, one
    Newton or secant step from the bound; depths are positive."""
    lo, hi = torch.minimum(hL, hR), torch.maximum(hL, hR)
    du = uR - uL
    cL, cR = torch.sqrt(G * hL), torch.sqrt(G * hR)
    clo, chi = torch.sqrt(G * lo), torch.sqrt(G * hi)
    Fmin = du + 2.0 * (clo - chi)
    Fmax = du + (hi - lo) * torch.sqrt(0.5 * G * (hi + lo) / (hi * lo))
    t = torch.clamp(-du + 2.0 * (cL + cR), min=0.0)
    c2 = torch.sqrt(G * (t * t / (16.0 * G)))
    r1, r2 = uL + 2.0 * cL - 3.0 * c2, uR - 2.0 * cR + 3.0 * c2
    gL = torch.sqrt(0.5 * G * (1.0 / hi + 1.0 / hL))
    gR = torch.sqrt(0.5 * G * (1.0 / hi + 1.0 / hR))
    F0 = du + (hi - hL) * gL + (hi - hR) * gR
    dF = gL - G * (hi - hL) / (4.0 * hi * hi * gL) + gR - G * (hi - hR) / (4.0 * hi * hi * gR)
    hm = (torch.sqrt(hi) - F0 / (2.0 * torch.sqrt(hi) * dF)) ** 2
    hm = torch.where(hm > 0, hm, torch.ones_like(hm))
    s1 = uL - (hm - hL) * torch.sqrt(0.5 * G * (1.0 / hm + 1.0 / hL)) - torch.sqrt(G * hm)
    s2 = uR + (hm - hR) * torch.sqrt(0.5 * G * (1.0 / hm + 1.0 / hR)) + torch.sqrt(G * hm)
    gap = torch.where(hi > lo, hi - lo, torch.ones_like(hi))
    slope = (Fmax - Fmin) / gap
    hx = lo - Fmin / torch.where(slope != 0, slope, torch.ones_like(slope))
    cx = torch.sqrt(G * torch.clamp(hx, min=0.0))
    x1 = torch.where(hL > hR, uL + 2.0 * cL - 3.0 * cx, uR - 2.0 * cR + cx)
    x2 = torch.where(hL > hR, uL + 2.0 * cL - cx, uR - 2.0 * cR + 3.0 * cx)
    rare, shock = Fmin > 0, Fmax <= 0
    h_out = torch.where(rare, t * t / (16.0 * G), torch.where(shock, hm, hx))
    return (h_out, torch.where(rare, r1, torch.where(shock, s1, x1)), torch.where(rare, r2, torch.where(shock, s2, x2)))


def _faces(h, hu, hv, b):
    """Speeds (3 of (..., n-1)) and f-waves [wave][component] at the faces
    along the last axis: the augmented solver with its wall and steady-state rules."""
    hL, hR, huL, huR = h[..., :-1], h[..., 1:], hu[..., :-1], hu[..., 1:]
    hvL, hvR, bL, bR = hv[..., :-1], hv[..., 1:], b[..., :-1], b[..., 1:]
    wL, wR = hL > DRY, hR > DRY
    some = wL | wR
    one = torch.ones_like(hL)

    def cell(w, hh, m1, m2):
        hs = torch.where(w, hh, one)
        return _where0(w, hh), _where0(w, m1), _where0(w, m1 / hs), _where0(w, m2 / hs), _where0(w, 0.5 * G * hh * hh + m1 * m1 / hs)

    hL, huL, uL, vL, pL = cell(wL, hL, huL, hvL)
    hR, huR, uR, vR, pR = cell(wR, hR, huR, hvR)
    keep = [one, one, one]
    # a dry right side, then a dry left side: a wall where the water does not reach over the step
    hs, _, _ = _middle(torch.where(wL, hL, one), torch.where(wL, hL, one), uL, -uL)
    top = torch.maximum(hL, hs) + bL
    dryR = wL & ~wR
    wall = dryR & (top < bR)
    step = dryR & ~wall & (hL + bL < bR)
    bR = torch.where(wall, bL, torch.where(step, hL + bL, bR))
    hR, huR, pR = torch.where(wall, hL, hR), torch.where(wall, -huL, huR), torch.where(wall, pL, pR)
    uR, vR = torch.where(wall, -uL, uR), torch.where(wall, vL, vR)
    keep[1], keep[2] = torch.where(wall, 0 * one, keep[1]), torch.where(wall, 0 * one, keep[2])
    hs, _, _ = _middle(torch.where(wR, hR, one), torch.where(wR, hR, one), -uR, uR)
    top = torch.maximum(hR, hs) + bR
    dryL = wR & ~wL
    wall = dryL & (top < bL)
    step = dryL & ~wall & (hR + bR < bL)
    bL = torch.where(wall, bR, torch.where(step, hR + bR, bL))
    hL, huL, pL = torch.where(wall, hR, hL), torch.where(wall, -huR, huL), torch.where(wall, pR, pL)
    uL, vL = torch.where(wall, -uR, uL), torch.where(wall, vR, vL)
    keep[0], keep[1] = torch.where(wall, 0 * one, keep[0]), torch.where(wall, 0 * one, keep[1])

    cL, cR = torch.sqrt(G * hL), torch.sqrt(G * hR)
    csum = torch.where(some, cL + cR, one)
    uhat = (cL * uL + cR * uR) / csum
    chat = torch.sqrt(G * 0.5 * (hR + hL))
    both = (hL > DRY) & (hR > DRY)
    _, m1, m2 = _middle(torch.where(both, hL, one), torch.where(both, hR, one), uL, uR)
    flat = uR + uL - 2.0 * cR + 2.0 * cL
    m1, m2 = torch.where(both, m1, flat), torch.where(both, m2, flat)
    l1 = torch.minimum(torch.minimum(uL - cL, uhat - chat), m2)
    l3 = torch.maximum(torch.maximum(uR + cR, uhat + chat), m1)
    gap = torch.where(some, l3 - l1, one)
    hll = torch.clamp((huL - huR + l3 * hR - l1 * hL) / gap, min=0.0)
    dh, dhu, dphi, db = hR - hL, huR - huL, pR - pL, bR - bL
    crit = max(DRY * G, 1e-6)
    crit2 = math.sqrt(crit)
    hbar = torch.clamp(0.5 * (hL + hR), min=0.0)
    sb = 0.25 * (uL + uR) ** 2 - G * hbar
    st = torch.clamp(uL * uR, min=0.0) - G * hbar
    sonic = ((sb.abs() <= crit) | (sb * st <= crit ** 2) | (sb * l1 * l3 <= crit ** 2)
             | (torch.minimum(l1.abs(), l3.abs()) < crit2) | ((l1 < crit2) & (m1 > -crit2))
             | ((l3 > -crit2) & (m2 < crit2)) | ((uL + cL) * (uR + cR) < 0) | ((uL - cL) * (uR - cR) < 0))
    sbs = torch.where(sonic, one, sb)
    ddh = torch.where(sonic, -db, db * G * hbar / sbs)
    l1s, l3s = torch.where(l1 != 0, l1, one), torch.where(l3 != 0, l3, one)
    sub, right, left = (l1 < -crit) & (l3 > crit), l1 >= crit, l3 <= -crit
    a = hll * (l3 - l1)
    ddh = torch.where(sub, _maxmod(ddh, a / l3s, a / l1s),
                      torch.where(right, _maxmod(ddh, a / l1s, -hL),
                                  torch.where(left, _maxmod(ddh, hR, a / l3s), ddh)))
    ddp = torch.where(sonic, -G * hbar * db, -db * G * hbar * st / sbs)
    ddp = _maxmod(ddp, G * torch.maximum(-hL * db, -hR * db), G * torch.minimum(-hL * db, -hR * db))
    d1, d2, d3 = dh - ddh, dhu, dphi - ddp
    b1, b3 = (d1 * l3 - d2) / gap, (d2 - d1 * l1) / gap
    b2 = d3 - l1 * l1 * b1 - l3 * l3 * b3
    f1, f2, f3 = [b1 * l1, b1 * l1 * l1, b1 * l1 * vL], [0 * one, b2, 0 * one], [b3 * l3, b3 * l3 * l3, b3 * l3 * vR]
    fix = hR * uR * vR - hL * uL * vL - f1[2] - f3[2]
    toward = huL + f1[0] <= 0
    f1[2] = f1[2] + torch.where(toward, fix, 0 * one)
    f3[2] = f3[2] + torch.where(toward, 0 * one, fix)
    s = [_where0(some, x * w) for x, w in zip((l1, 0.5 * (l1 + l3), l3), keep)]
    fw = [[_where0(some, x * w) for x in f] for f, w in zip((f1, f2, f3), keep)]
    return s, fw


def _limit(r, how):
    if how == 2:
        return torch.maximum(torch.clamp(2.0 * r, 0.0, 1.0), torch.clamp(r, max=2.0))
    if how == 3:
        return (r + r.abs()) / (1.0 + r.abs())
    if how == 4:
        return torch.clamp(torch.minimum(torch.clamp(0.5 * (1.0 + r), max=2.0), 2.0 * r), min=0.0)
    return torch.clamp(r, 0.0, 1.0)


def _sweep(h, hu, hv, b, r, order, transverse, how):
    """One direction, cells along the last axis, slices along the one before it;
    r = dt / dx. Returns the cells' flux difference, their down- and up-going
    transverse parts (3 components each, cells 1..n-2 of each slice; the
    interior lies inside) and the largest speed over the slices 1..n-2."""
    s, fw = _faces(h, hu, hv, b)
    am = [sum(torch.where(s[w] < 0, fw[w][c], torch.where(s[w] > 0, 0 * s[w], 0.5 * fw[w][c])) for w in range(3)) for c in range(3)]
    ap = [sum(torch.where(s[w] > 0, fw[w][c], torch.where(s[w] < 0, 0 * s[w], 0.5 * fw[w][c])) for w in range(3)) for c in range(3)]
    cq = [torch.zeros_like(s[0]) for _ in range(3)]
    if order == 2:
        for w in range(3):
            norm = sum(f * f for f in fw[w])
            dot = sum(f[..., :-1] * f[..., 1:] for f in fw[w])
            z = torch.zeros_like(norm[..., :1])
            up = torch.where(s[w] > 0, torch.cat([z, dot], -1), torch.cat([dot, z], -1))
            nz = norm != 0
            lim = torch.where(nz, _limit(up / torch.where(nz, norm, torch.ones_like(norm)), how), torch.ones_like(norm))
            sg = torch.where(torch.signbit(s[w]), -torch.ones_like(norm), torch.ones_like(norm))
            fac = sg * (1.0 - s[w].abs() * r) * lim
            cq = [cq[c] + fac * fw[w][c] for c in range(3)]
    lo, hi = slice(None, -1), slice(1, None)  # left and right face of a cell
    P = [am[c][..., hi] + ap[c][..., lo] for c in range(3)]
    Q = [cq[c][..., hi] - cq[c][..., lo] for c in range(3)]
    N = [P[c] + 0.5 * Q[c] for c in range(3)]
    smax = torch.stack([x[..., 1:-1, :].abs().amax(dim=(-1, -2)) for x in s]).amax(dim=0)
    zero = torch.zeros_like(P[0])
    if transverse == 0:
        return N, [zero] * 3, [zero] * 3, smax
    x = [P[c] + Q[c] if transverse == 2 else P[c] for c in range(3)]
    hc, huc, hvc, bc = (a[..., 1:-1] for a in (h, hu, hv, b))
    wet = hc > DRY
    hs = torch.where(wet, hc, torch.ones_like(hc))
    u, v, c0 = huc / hs, hvc / hs, torch.sqrt(G * hs)
    below = torch.cat([bc[..., :1, :], bc[..., :-1, :]], -2)
    above = torch.cat([bc[..., 1:, :], bc[..., -1:, :]], -2)
    eta = hc + bc
    on = wet & (eta >= torch.minimum(below, above))
    sp = [v - c0, v, v + c0]
    be = [(sp[2] * x[0] - x[2]) / (2.0 * c0), x[1] - u * x[0], (x[2] - sp[0] * x[0]) / (2.0 * c0)]
    vec = [[torch.ones_like(u), u, sp[0]], [zero, torch.ones_like(u), zero], [torch.ones_like(u), u, sp[2]]]
    dn = [sum(_where0(on & (sp[w] < 0) & (eta >= below), sp[w] * be[w] * vec[w][c]) for w in range(3)) for c in range(3)]
    up = [sum(_where0(on & (sp[w] > 0) & (eta >= above), sp[w] * be[w] * vec[w][c]) for w in range(3)) for c in range(3)]
    return N, dn, up, smax


def _update(case, q, aux, dx, dt):
    """One step of every patch: interior (P, 3, m, m) and CFL of each patch."""
    order, transverse, how = case.get("order", 2), case.get("transverse", 2), case.get("limiter", 4)
    dry = q[:, 0] < DRY
    h = torch.where(dry, torch.clamp(q[:, 0], min=0.0), q[:, 0])
    hu, hv = (torch.where(dry, torch.zeros_like(h), q[:, c]) for c in (1, 2))
    b, r = aux[:, 0], dt / dx
    t = lambda a: a.transpose(-1, -2)  # noqa: E731
    Nx, dx_, ux, sx = _sweep(h, hu, hv, b, r, order, transverse, how)
    Ny, dy_, uy, sy = _sweep(t(h), t(hv), t(hu), t(b), r, order, transverse, how)
    new = []
    for c, (h0, cy) in enumerate(((h, 0), (hu, 2), (hv, 1))):  # component c is number cy of the y sweep
        inner = slice(1, -1)
        d = Nx[c][:, 2:-2, inner] + t(Ny[cy][:, 2:-2, inner])
        for up, dn, turn in ((ux[c], dx_[c], False), (uy[cy], dy_[cy], True)):
            part = 0.5 * r * (up[:, 1:-3] + dn[:, 2:-2] - up[:, 2:-2] - dn[:, 3:-1])[:, :, inner]
            d = d + (t(part) if turn else part)
        new.append(h0[:, 2:-2, 2:-2] - r * d)
    h1, hu1, hv1 = new
    if case["friction"] != "none":
        bi = b[:, 2:-2, 2:-2]
        if case["friction"] == "variable":
            n = aux[:, 1, 2:-2, 2:-2]
        elif case["friction"] == "table":
            n = torch.where(bi < 8.0, 0.03, 0.06).double()
        else:
            n = torch.full_like(bi, 0.035)
        none = h1 < 1e-30
        hs = torch.where(none, torch.ones_like(h1), h1)
        gam = 1.0 + dt * torch.sqrt(hu1 ** 2 + hv1 ** 2) * G * n * n / hs ** (7.0 / 3.0)
        hu1, hv1 = torch.where(none, torch.zeros_like(hu1), hu1 / gam), torch.where(none, torch.zeros_like(hv1), hv1 / gam)
    cfl = r * torch.maximum(sx, sy)
    return torch.stack([h1, hu1, hv1], dim=1), torch.where(cfl > 100.0, torch.zeros_like(cfl), cfl)


def _exact_update(case, seed):
    q, aux, dx, dt = _patches(case, seed)
    parts = [_update(case, q[k:k + 512], aux[k:k + 512], dx, dt) for k in range(0, q.shape[0], 512)]
    return q, torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])


def _exact_batch(case, seed):
    q, new, cfl = _exact_update(case, seed)
    q = q.clone()
    q[:, :, 2:-2, 2:-2] = new
    out = {"q": q.permute(0, 2, 3, 1).contiguous(), "cfl": float(cfl.max())}
    if case["n"] > 1:
        out["cfls"] = cfl
    return out


def _exact_level(case, seed):
    _, new, cfl = _exact_update(case, seed)
    m, npx, npy = case["m"], case["npx"], case["npy"]
    glob = new.reshape(npy, npx, 3, m, m).permute(2, 0, 3, 1, 4).reshape(3, npy * m, npx * m)
    q = torch.stack([_tiles(a, m) for a in _pad_state(*glob, case["bc"])], dim=1)
    if case["kind"] == "host":
        q = q.permute(0, 2, 3, 1).contiguous()
    return {"q": q, "cfl": float(cfl.max())}


def _average4(q, b, target_b):
    """Fine cells (..., 4) under a coarse cell to its h, hu, hv."""
    h, hu, hv = q
    wet = h > DRY
    n = wet.sum(-1)
    ns = torch.clamp(n, min=1).double()
    hsum = h.sum(-1)
    hc = torch.minimum(hsum / ns, torch.clamp(_where0(wet, h + b).sum(-1) / ns - target_b, min=0.0))
    f = hc / torch.where(n > 0, hsum, torch.ones_like(hsum))
    return [_where0(n > 0, x) for x in (hc, f * _where0(wet, hu).sum(-1), f * _where0(wet, hv).sum(-1))]


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _exact_exchange(case, seed):
    m, n = case["m"], case["n"]
    coarse, cb, fine, fb, kb = _amr(case, seed)
    coarse, fine = coarse.clone(), fine.clone()
    n4 = m + 4
    # fine interiors next to the coarse patches' right side -> two ghost columns
    cols = fine[:, :, 2:-2, 2:6].reshape(n, 2, 3, m, 4).permute(0, 2, 1, 3, 4).reshape(n, 3, m, 2, 2, 2)
    cols = cols.permute(0, 1, 2, 4, 3, 5).reshape(n, 3, m, 2, 4)
    bcols = fb[:, 2:-2, 2:6].reshape(n, 2 * m, 4).reshape(n, m, 2, 2, 2).permute(0, 1, 3, 2, 4).reshape(n, m, 2, 4)
    got = _average4([cols[:, c] for c in range(3)], bcols, cb[:, 2:-2, m + 2:])
    coarse[:, :, 2:-2, m + 2:] = torch.stack(got, dim=1)

    def children(j0, j1, i0, i1):
        """Values of the 2 x 2 fine cells in the coarse cells j0..j1-1, i0..i1-1 (array indices)."""
        h, hu, hv = coarse[:, 0], coarse[:, 1], coarse[:, 2]
        eta = torch.where(h < DRY, torch.zeros_like(h), h + cb)
        out = []
        for a in (eta, hu, hv):
            z = a[:, j0:j1, i0:i1]
            gx = _minmod(z - a[:, j0:j1, i0 - 1:i1 - 1], a[:, j0:j1, i0 + 1:i1 + 1] - z)
            gy = _minmod(z - a[:, j0 - 1:j1 - 1, i0:i1], a[:, j0 + 1:j1 + 1, i0:i1] - z)
            v = torch.empty((n, j1 - j0, 2, i1 - i0, 2), dtype=torch.float64, device=a.device)
            for y in range(2):
                for x in range(2):
                    v[:, :, y, :, x] = z + gx * (x - 0.5) / 2.0 + gy * (y - 0.5) / 2.0
            out.append(v.reshape(n, 2 * (j1 - j0), 2 * (i1 - i0)))
        return out

    eta, mu, mv = children(2, m + 2, m + 1, m + 2)
    # both fine patches also take the two ghost rows that lie over this coarse patch
    for half, rows, to in ((0, slice(0, m + 2), slice(2, m + 4)), (1, slice(m - 2, 2 * m), slice(0, m + 2))):
        p = 2 * torch.arange(n, device=fine.device) + half
        v = torch.stack([torch.clamp(eta[:, rows] - fb[p][:, to, 0:2], min=0.0), mu[:, rows], mv[:, rows]], dim=1)
        got = fine[p]
        got[:, :, to, 0:2] = v
        fine[p] = got
    new = torch.zeros((4 * n, 3, n4, n4), dtype=torch.float64, device=fine.device)
    kids = children(1, m + 3, 1, m + 3)  # with one ghost layer of coarse cells
    for g in range(4):
        # child g: its interior and the outer ghost layers the rule reaches
        ig, jg = g % 2, g // 2
        w, at = m + 2, torch.arange(n, device=fine.device)
        # coarse cells i1..i1+m/2 (1-based, i1 = 1 - ig) plus the half's offset, fine index 2 (i - 1) + 1
        i1, j1 = 1 - ig, 1 - jg
        fi0, fj0 = (i1 - 1) * 2 + 1, (j1 - 1) * 2 + 1
        ci, cj = i1 + ig * m // 2, j1 + jg * m // 2
        p = (2 * at + jg) * 2 + ig
        sy, sx = slice(fj0 + 1, fj0 + 1 + w), slice(fi0 + 1, fi0 + 1 + w)
        ky, kx = slice(2 * cj, 2 * cj + w), slice(2 * ci, 2 * ci + w)
        for c in range(3):
            v = kids[c][:, ky, kx]
            if c == 0:
                v = v - kb[p][:, sy, sx]
            buf = new[p, c]
            buf[:, sy, sx] = v
            new[p, c] = buf
    h, hu, hv, b = fine[:, 0, 2:-2, 2:-2], fine[:, 1, 2:-2, 2:-2], fine[:, 2, 2:-2, 2:-2], fb[:, 2:-2, 2:-2]
    return {"coarse": coarse, "fine": fine, "new": new, "tags": None}


def _hats(x1, x2, x0, d, n):
    """Integrals of the n hat functions of nodes x0 + k d over the intervals [x1, x2]."""
    k = torch.arange(n, dtype=torch.float64, device=x1.device)[None, :]

    def primitive(x):
        s = (x[:, None] - x0) / d - k
        return torch.where(s < -1, 0 * s, torch.where(s < 0, 0.5 * (s + 1) ** 2, torch.where(s < 1, 0.5 + s - 0.5 * s * s, 1.0 + 0 * s)))

    return d * (primitive(x2) - primitive(x1))


def _exact_dem(case, seed):
    (A, B), L = _dem(case, seed)
    edge = [torch.arange(n + 1, dtype=torch.float64, device="cuda") * (L / n) for n in (case["nx"], case["ny"])]

    def integral(grid, clip):
        z, x0, y0, d = grid
        w = []
        for e, o, n in ((edge[1], y0, z.shape[0]), (edge[0], x0, z.shape[1])):
            a, c = e[:-1], e[1:]
            if clip is not None:
                lo = clip[0] if e is edge[0] else clip[1]
                hi = lo + clip[2]
                a, c = a.clamp(lo, hi), c.clamp(lo, hi)
            w.append(_hats(a, c, o, d, n))
        return w[0] @ z @ w[1].T

    inset = (B[1], B[2], (B[0].shape[0] - 1) * B[3])
    v = integral(A, None) - integral(A, inset) + integral(B, inset)
    v = v / ((L / case["nx"]) * (L / case["ny"]))
    return _pad(v, 1)
