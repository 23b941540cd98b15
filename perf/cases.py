"""Performance cases of the diffusion library: what its users run, through
its public entry points, over the range of grids, kernel widths and substep
counts that the configurations, the tests and the benchmark name.

Kinds
  tick      one resident world, vfd.World.tick (the ABM's per-tick call)
  ensemble  many uneven worlds ticked together, vfd.Batch.tick
  served    requests with host fields through vfd.Server (continuous batching)
  fft3d     the general 3D transform with a dense window and the chemical
            update on the device, vfd.World.tick_update
  host      host buffers in and out, vfd.World.diffuse_update_host (what the
            Diffuser drop-in calls each tick), then the totals
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vf-version_7_3_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import vfd  # noqa: E402
from vfd import configs  # noqa: E402

SIGMA, DECAY = configs.SIGMA0, configs.DECAY0
# retention factors of the chemical update (p = d + factor * t)
RETAIN = [1.0 - d for d in DECAY]
LAMBDA = 0.1333  # the human-VF stencil's arm weight


def listed():
    return [
        # the smallest plain world: one substep a tick; launches and latency
        dict(name="tick_small", kind="tick", grid="64x64x32", fields=8, scale=1.0, substeps=1, sources=500, vf=False),
        # a single chemical on an odd grid (rows not 16-byte aligned) under the vocal-fold boundary rule
        dict(name="tick_odd", kind="tick", grid="97x61x45", fields=3, scale=1.3, substeps=10, sources=300, vf=True),
        # the human-scale world, ten substeps a tick (the benchmark's flagship step)
        dict(name="tick_human", kind="tick", grid="512x256x384", fields=8, scale=1.5, substeps=10, sources=200000,
             vf=False),
        # the human-scale world with one substep a tick under the vocal-fold boundary rule
        dict(name="tick_human_single", kind="tick", grid="512x256x384", fields=8, scale=1.5, substeps=1,
             sources=200000, vf=True),
        # the large world: the largest fields and source lists, wider kernels
        dict(name="tick_large", kind="tick", grid="768x384x576", fields=8, scale=2.0, substeps=10, sources=1000000,
             vf=False),
        # fast-diffusing chemicals: kernel radii 10 to 16
        dict(name="tick_wide", kind="tick", grid="256x128x192", fields=8, scale=4.0, substeps=2, sources=20000,
             vf=False),
        # the sensitivity ensemble: 32 uneven worlds, ten substeps a tick
        dict(name="ensemble", kind="ensemble", worlds=32, substeps=10, sources=500),
        # few worlds ticked one substep at a time (a lightly loaded ensemble)
        dict(name="ensemble_single", kind="ensemble", worlds=6, substeps=1, sources=500),
        # a burst of requests of mixed sizes, fields from and to the host
        dict(name="served_burst", kind="served", grids="64x64x32,64x64x32,64x64x32,64x64x32,128x96x96,128x96x96,"
             "128x96x96,256x128x192", fields=8, ticks=20, sources=1000),
        # the reference's own transform at human scale, resident, with the chemical update
        dict(name="fft3d_human", kind="fft3d", grid="512x256x384", fields=8, half=6, substeps=1, vf=True),
        # the same on a small odd grid
        dict(name="fft3d_odd", kind="fft3d", grid="75x50x33", fields=8, half=8, substeps=1, vf=True),
        # the drop-in's call: host fields in and out through the general transform
        dict(name="host_dropin", kind="host", grid="256x128x192", fields=8, half=6, substeps=1, vf=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tick", "tick", "tick", "tick", "ensemble", "served", "fft3d", "host"])
    if kind == "ensemble":
        return dict(kind=kind, worlds=_log_int(rng, 2, 32), substeps=rng.choice([1, 2, 5, 10]),
                    sources=_log_int(rng, 100, 2000))
    if kind == "served":
        n = rng.randint(3, 8)
        grids = ",".join("%dx%dx%d" % tuple(rng.choice(configs.CFG3["grids"][:2])) for _ in range(n))
        return dict(kind=kind, grids=grids, fields=8, ticks=rng.randint(5, 30), sources=_log_int(rng, 1000, 5000))
    top = {"tick": 640, "fft3d": 400, "host": 200}[kind]
    while True:
        g = [_log_int(rng, 24, top) for _ in range(3)]
        if rng.random() < 0.5:  # half of the grids are multiples of 16, the others as they come
            g = [16 * max(2, round(v / 16)) for v in g]
        if g[0] * g[1] * g[2] <= 768 * 384 * 576 // 2:
            break
    fields, grid = rng.randint(1, 8), "%dx%dx%d" % tuple(g)
    vf = rng.random() < 0.4
    if kind == "tick":
        V = g[0] * g[1] * g[2]
        scale = math.exp(rng.uniform(math.log(0.6), math.log(5.0)))
        return dict(kind=kind, grid=grid, fields=fields, scale=round(scale, 3),
                    substeps=rng.choice([1, 1, 2, 4, 7, 10]),
                    sources=min(_log_int(rng, 100, 1000000), V), vf=vf)
    return dict(kind=kind, grid=grid, fields=fields, half=rng.randint(2, 12), substeps=rng.choice([1, 1, 2]), vf=vf)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _grid(text):
    return tuple(int(v) for v in text.split("x"))


def _gen(seed, *salt):
    g = torch.Generator(device="cuda")
    k = int(seed) & 0xFFFFFFFF
    for s in salt:
        k = (k * 1000003 + int(s) + 1) & 0x7FFFFFFFFFFF
    g.manual_seed(k)
    return g


def _field(seed, world, f, grid):
    nx, ny, nz = grid
    return torch.rand((nz, ny, nx), generator=_gen(seed, world, f, 0), device="cuda", dtype=torch.float32) * 1e-3


def _sources(seed, world, f, grid, n):
    g = _gen(seed, world, f, 1)
    V = grid[0] * grid[1] * grid[2]
    idx = torch.randint(0, V, (n,), generator=g, device="cuda", dtype=torch.int64)
    amt = torch.exp(torch.randn((n,), generator=g, device="cuda", dtype=torch.float32) - 6.0)
    return idx, amt


def _update_d(seed, f, grid):
    """The secreted amounts (dChem): a tenth of the voxels hold some."""
    nx, ny, nz = grid
    g = _gen(seed, 0, f, 2)
    u = torch.rand((nz, ny, nx), generator=g, device="cuda", dtype=torch.float32)
    return torch.where(u < 0.1, u * 1e-3, torch.zeros((), device="cuda"))


def _params(case):
    """(sigma, decay, baseline) per field of a tick case."""
    return [(SIGMA[f] * case["scale"], DECAY[f], 1e-4 * (f + 1) if case["vf"] else 0.0) for f in range(case["fields"])]


def _ensemble(case):
    return [(w["grid"], list(zip(w["sigma"], w["decay"]))) for w in configs.cfg2_worlds(case["worlds"])]


def _windows(case):
    """One stencil-power window a field: field f is the stencil applied
    2 + f % (half - 1) times, cropped to the case's half-width."""
    h = case["half"]
    n = 2 * h + 1
    w = np.zeros((n + 2,) * 3)
    w[h + 1, h + 1, h + 1] = 1.0
    by_steps = {}
    for s in range(1, h + 1):
        a = (1.0 - 6.0 * LAMBDA) * w
        for ax in range(3):
            for d in (-1, 1):
                a += LAMBDA * np.roll(w, d, axis=ax)
        w = a
        by_steps[s] = w[1:-1, 1:-1, 1:-1].astype(np.float32)
    return [by_steps[min(h, 2 + f % max(1, h - 1))] for f in range(case["fields"])]


def _epi(case, grid):
    return grid[0] - 1 if case["vf"] else 0


def _pad(case):
    return vfd.PAD_CONSTANT_VF if case["vf"] else vfd.PAD_ZERO


class _View:
    """A world's resident fields (fields, nz, ny, nx) as torch sees them; the
    tensor keeps this object, and so the world and its device memory."""

    def __init__(self, world):
        self.world = world
        self.__cuda_array_interface__ = {"shape": (world.nf,) + world.shape, "typestr": "<f4", "version": 3,
                                         "strides": None, "data": (world.device_ptr(0), False)}


def _view(world):
    return torch.as_tensor(_View(world), device="cuda")


def _resident(grid, params, case, seed, world_id, method, sources, fft=(0, 0, 0)):
    w = vfd.World(*grid, params, pad_mode=_pad(case), epi_boundary=_epi(case, grid), method=method, fft=fft)
    view = _view(w)
    for f, v in enumerate(view):
        v.copy_(_field(seed, world_id, f, grid))
        if sources:
            idx, amt = _sources(seed, world_id, f, grid, sources)
            w.set_sources(f, idx.to(torch.int32).cpu().numpy(), amt.cpu().numpy())
    return w, view


def _general_world(case, seed):
    grid = _grid(case["grid"])
    h = case["half"]
    params = [vfd.field_params(1.0, 0.0, radius=h, baseline=1e-4 * (f + 1) if case["vf"] else 0.0)
              for f in range(case["fields"])]
    w, view = _resident(grid, params, case, seed, 0, vfd.METHOD_FFT3D, 0)
    for f, win in enumerate(_windows(case)):
        w.set_window(f, win)
    return w, view


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tick":
        params = [vfd.field_params(s, d, baseline=b) for s, d, b in _params(case)]
        w, view = _resident(_grid(case["grid"]), params, case, seed, 0, vfd.METHOD_SEPARABLE, case["sources"])
        return dict(kind=kind, world=w, view=view, substeps=case["substeps"])
    if kind == "ensemble":
        worlds, views = [], []
        for i, (grid, fp) in enumerate(_ensemble(case)):
            w, v = _resident(grid, [vfd.field_params(s, d) for s, d in fp], dict(vf=False), seed, i,
                             vfd.METHOD_SEPARABLE, case["sources"])
            worlds.append(w)
            views.append(v)
        b = vfd.Batch(worlds)
        return dict(kind=kind, batch=b, views=views, substeps=case["substeps"])
    if kind == "served":
        s = vfd.Server(64 << 30, max_active=16)
        reqs = []
        for i, g in enumerate(case["grids"].split(",")):
            grid = _grid(g)
            nf = case["fields"]
            init = [_field(seed, i, f, grid).cpu().numpy() for f in range(nf)]
            src = []
            for f in range(nf):
                idx, amt = _sources(seed, i, f, grid, case["sources"])
                src.append((idx.to(torch.int32).cpu().numpy(), amt.cpu().numpy()))
            out = np.empty((nf,) + init[0].shape, np.float32)
            reqs.append((grid, [vfd.field_params(SIGMA[f], DECAY[f]) for f in range(nf)], init, src, out))
        return dict(kind=kind, server=s, reqs=reqs, ticks=case["ticks"])
    if kind == "fft3d":
        w, view = _general_world(case, seed)
        d = [_update_d(seed, f, _grid(case["grid"])) for f in range(case["fields"])]
        return dict(kind=kind, world=w, view=view, d=d, ptrs=[t.data_ptr() for t in d],
                    retain=np.array(RETAIN[:case["fields"]], np.float32), substeps=case["substeps"])
    w, view = _general_world(case, seed)
    grid = _grid(case["grid"])
    p = [v.cpu().pin_memory().numpy() for v in view]
    d = [_update_d(seed, f, grid).cpu().pin_memory().numpy() for f in range(case["fields"])]
    return dict(kind=kind, world=w, p=p, d=d, retain=np.array(RETAIN[:case["fields"]], np.float32),
                substeps=case["substeps"])


def run(state):
    kind = state["kind"]
    if kind == "tick":
        state["world"].tick(state["substeps"])
        return state["view"]
    if kind == "ensemble":
        state["batch"].tick(state["substeps"])
        return state["views"]
    if kind == "served":
        s = state["server"]
        ids = [s.submit(grid, params, state["ticks"], init=init, sources=src, result=list(out))
               for grid, params, init, src, out in state["reqs"]]
        for i in ids:
            s.wait(i)
        return [out for _, _, _, _, out in state["reqs"]]
    if kind == "fft3d":
        state["world"].tick_update(state["retain"], state["ptrs"], state["substeps"])
        return state["view"]
    w = state["world"]
    w.diffuse_update_host(state["p"], state["d"], state["retain"], state["substeps"])
    return {"p": state["p"], "totals": [m["total"] for m in w.mass()]}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _radius(sigma):
    return math.ceil(3.0 * sigma)


def _separable_work(grid, sigmas, substeps, sources):
    V = grid[0] * grid[1] * grid[2]
    flops = sum(3.0 * 2.0 * (2 * _radius(s) + 1) * V * substeps for s in sigmas)
    return len(sigmas) * (8.0 * V + 8.0 * sources), flops


def _general_work(case, arrays):
    nx, ny, nz = _grid(case["grid"])
    h, nf, V = case["half"], case["fields"], nx * ny * nz
    N = (nx + h) * (ny + h) * (nz + h)
    # the window is read once; two real transforms and a multiply a substep
    return (nf * (arrays * 4.0 * V + 4.0 * (2 * h + 1) ** 3),
            nf * case["substeps"] * (2 * 2.5 * N * math.log2(N) + 3.0 * N))


def work(case):
    kind = case["kind"]
    if kind == "tick":
        b, f = _separable_work(_grid(case["grid"]), [p[0] for p in _params(case)], case["substeps"], case["sources"])
    elif kind == "ensemble":
        parts = [_separable_work(g, [s for s, _ in fp], case["substeps"], case["sources"]) for g, fp in _ensemble(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "served":
        parts = [_separable_work(_grid(g), SIGMA[:case["fields"]], case["ticks"], case["sources"])
                 for g in case["grids"].split(",")]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    else:
        b, f = _general_work(case, 3)
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _taps(sigma):
    r = _radius(sigma)
    j = np.arange(-r, r + 1, dtype=np.float64)
    g = np.exp(-j * j / (2.0 * sigma * sigma))
    return g / g.sum()


def _conv_axis(v, taps, dim):
    """The zero-extended line convolution along `dim`, cropped."""
    r, n = len(taps) // 2, v.shape[dim]
    out = v * taps[r]
    for j in range(1, min(r, n - 1) + 1):
        a, b = out.narrow(dim, j, n - j), out.narrow(dim, 0, n - j)
        a.add_(v.narrow(dim, 0, n - j), alpha=float(taps[r + j]))
        b.add_(v.narrow(dim, j, n - j), alpha=float(taps[r + j]))
    return out


def _mask(shape, epi):
    nz, ny, nx = shape
    m = torch.zeros(shape, dtype=torch.float64, device="cuda")
    m[1:nz - 1, 1:ny - 1, 1:min(epi, nx)] = 1.0
    return m


def _exact_ticks(u, sigma, decay, b, mask, substeps, ticks, src):
    u = u.double()
    taps = _taps(sigma)
    idx, amt = src
    for _ in range(ticks):
        for _ in range(substeps):
            v = u - b if mask is None else (u - b) * mask
            for dim in (2, 1, 0):
                v = _conv_axis(v, taps, dim)
            u = (v + b) * (1.0 - decay)
        u.view(-1).index_add_(0, idx, amt.double())
    return u


def _exact_general(u, win, b, mask, substeps, retain, d):
    nz, ny, nx = u.shape
    h = win.shape[0] // 2
    F = (nz + h, ny + h, nx + h)
    w = torch.zeros(F, dtype=torch.float64, device="cuda")
    w[:2 * h + 1, :2 * h + 1, :2 * h + 1] = torch.from_numpy(win.astype(np.float64)).cuda()
    K = torch.fft.rfftn(torch.roll(w, (-h, -h, -h), (0, 1, 2)))
    k0 = float(win.astype(np.float64).sum())
    u = u.double()
    for _ in range(substeps):
        v = u - b if mask is None else (u - b) * mask
        t = torch.fft.irfftn(torch.fft.rfftn(v, s=F) * K, s=F)
        u = t[:nz, :ny, :nx] + b * k0
    return d.double() + u * float(np.float32(retain))


def exact(case, seed):
    kind = case["kind"]
    if kind == "tick":
        grid = _grid(case["grid"])
        mask = _mask(grid[::-1], _epi(case, grid)) if case["vf"] else None
        return torch.stack([_exact_ticks(_field(seed, 0, f, grid), s, d, float(np.float32(b)), mask, case["substeps"],
                                         1, _sources(seed, 0, f, grid, case["sources"]))
                            for f, (s, d, b) in enumerate(_params(case))])
    if kind in ("ensemble", "served"):
        served = kind == "served"
        worlds = _ensemble(case) if not served else [
            (_grid(g), list(zip(SIGMA, DECAY))[:case["fields"]]) for g in case["grids"].split(",")]
        return [torch.stack([_exact_ticks(_field(seed, i, f, grid), s, d, 0.0, None, 1 if served else case["substeps"],
                                          case["ticks"] if served else 1, _sources(seed, i, f, grid, case["sources"]))
                             for f, (s, d) in enumerate(fp)]) for i, (grid, fp) in enumerate(worlds)]
    grid = _grid(case["grid"])
    mask = _mask(grid[::-1], _epi(case, grid)) if case["vf"] else None
    outs = [_exact_general(_field(seed, 0, f, grid), win, float(np.float32(1e-4 * (f + 1))) if case["vf"] else 0.0,
                           mask, case["substeps"], RETAIN[f], _update_d(seed, f, grid))
            for f, win in enumerate(_windows(case))]
    if kind == "fft3d":
        return torch.stack(outs)
    return {"p": outs, "totals": [float(u.sum()) for u in outs]}
