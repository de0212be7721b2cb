"""Workloads of the FDK engine as its users run them, through the public Python entry points.

A case describes one scan (detector kind, views, detector and grid sizes), how it is reconstructed
(storage, ramp filter, apodisation) and the entry point (`op`):

* ``execute``      FdkPlan.execute on device buffers, the plan kept between scans
* ``reconstruct``  gct_b200.reconstruct, host array in and out, no plan kept
* ``forward``      gct_b200.forward_project of a volume
* ``batch``        FdkBatch.launch over an uneven mix of plans

Lengths are in mm; `du` is in radians for the arc detectors. Inputs are line integrals of seeded
ellipsoids with photon noise, made on the GPU. ``exact`` restates the path in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gct_b200 as g

FILTERS = {"fft": g.FILTER_FFT, "toeplitz_f16x2": g.FILTER_TOEPLITZ_F16X2, "toeplitz_bf16x4": g.FILTER_TOEPLITZ_BF16X4}
APODS = {"none": g.ApodFunc.NONE, "hann": g.ApodFunc.HANN, "hamming": g.ApodFunc.HAMMING}
PARALLEL = ("parallel_1d", "parallel_2d", "cone_parallel")
ARC = ("fan_arc", "cone_cyl")
PLANAR = ("parallel_1d", "fan_arc", "fan_line")

DEFAULTS = dict(op="execute", kind="cone_flat", nv=360, nc=512, nr=1, du=1.0, dv=1.0, sod=0.0, sdd=0.0, nx=256, ny=256,
                nz=1, vox=1.0, voxz=1.0, mx=0.0, my=0.0, mz=0.0, scan="full", turns=1, pitch=0.0, ccw=False,
                storage="f32", filter="fft", apod="none", cutoff=1.0)


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one fan-beam slice, host arrays in and out through the drop-in entry
        # point with its defaults (the repository's fan-beam benchmark geometry)
        _case("fan256_host", op="reconstruct", kind="fan_line", nv=360, nc=512, du=1.2, sod=570.0, sdd=1040.0, nx=256,
              ny=256),
        # one slice of the serving mix's commonest class: 2D fan, FP16 storage, plan kept
        _case("fan512_f16", kind="fan_line", nv=720, nc=768, du=1.0, sod=570.0, sdd=1040.0, nx=512, ny=512, vox=0.8,
              storage="f16"),
        # a parallel-beam slice (synchrotron, rebinned fan), default options
        _case("par1024_f32", kind="parallel_1d", nv=900, nc=1455, du=250.0 / 1024, nx=1024, ny=1024, vox=250.0 / 1024),
        # an off-centre region of a fan-arc scan, nothing a round number: no symmetry, no alignment
        _case("arc_odd_f32", kind="fan_arc", nv=1151, nc=671, du=0.907 / 672, sod=570.0, sdd=1040.0, nx=509, ny=387,
              vox=0.7, mx=11.0, my=-23.0, ccw=True, apod="hann"),
        # the flat-panel full scan at default options (FP32 throughout)
        _case("flat256_f32", nv=360, nc=512, nr=384, du=0.8, dv=0.8, sod=750.0, sdd=1200.0, nz=256),
        # the benchmark's flat-panel full scan, mixed precision: the largest listed case
        _case("flat512_mixed", nv=720, nc=1024, nr=768, du=0.4, dv=0.4, sod=750.0, sdd=1200.0, nx=512, ny=512, nz=512,
              vox=0.5, voxz=0.5, storage="f16", filter="toeplitz_f16x2"),
        # a C-arm short scan (pi plus the fan angle), mixed precision
        _case("short384_mixed", nv=496, nc=1240, nr=960, du=0.3, dv=0.3, sod=785.0, sdd=1200.0, nx=512, ny=512, nz=384,
              vox=0.5, voxz=0.5, scan="short", storage="f16", filter="toeplitz_f16x2"),
        # a short scan of odd sizes into an off-centre grid, apodised, FP32
        _case("short_odd_f32", nv=247, nc=619, nr=477, du=0.6, dv=0.6, sod=785.0, sdd=1200.0, nx=253, ny=241, nz=187,
              mx=5.0, my=-7.0, mz=3.0, scan="short", apod="hamming", cutoff=0.9),
        # a diagnostic multi-slice scanner's axial rotation (cylindrical detector), FP16 storage
        _case("cyl64_f16", kind="cone_cyl", nv=1152, nc=896, nr=64, du=0.0011, dv=1.0, sod=600.0, sdd=1100.0, nx=512,
              ny=512, nz=64, vox=0.9, voxz=0.55, storage="f16"),
        # the same scanner in spiral mode, four rotations, default options
        _case("spiral_cyl_f32", kind="cone_cyl", nv=2304, nc=448, nr=64, du=0.0022, dv=1.0, sod=600.0, sdd=1100.0,
              nz=96, scan="spiral", turns=4, pitch=3.5),
        # the projection direction: forward projection of a volume for iterative or consistency work
        _case("forward192", op="forward", nv=180, nc=384, nr=288, du=1.0667, dv=1.0667, sod=750.0, sdd=1200.0, nx=192,
              ny=192, nz=192, vox=1.3333, voxz=1.3333),
        # a quarter of the repository's uneven batch (parallel slices of four sizes, fan arcs,
        # cylindrical and rebinned cone scans) in one launch, FP16 storage
        _case("batch12_f16", op="batch", storage="f16"),
    ]


def _near(n, multiple=1):
    """A whole number near n: any, or a multiple of what symmetric scans need."""
    return max(multiple, int(round(n / multiple)) * multiple)


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: kinds, entry points, storage and filters as listed, sizes
    over the listed range (2D slices of 128 to 2048 pixels, volumes of 64 to 512 voxels a side and
    at most 2e10 updates), half of them as the scanner gives them and half of any size."""
    op = rng.choices(["execute", "reconstruct", "forward", "spiral"], [0.7, 0.1, 0.1, 0.1])[0]
    even = rng.random() < 0.5
    m = 4 if even else 1
    if op == "spiral":
        kind = rng.choice(["cone_cyl", "cone_flat"])
    elif op == "forward":
        kind = rng.choice(["parallel_2d", "cone_cyl", "cone_flat", "fan_line", "parallel_1d"])
    else:
        kind = rng.choice(["parallel_1d", "fan_arc", "fan_line", "parallel_2d", "cone_parallel", "cone_cyl", "cone_flat",
                           "cone_flat"])
    planar = kind in PLANAR
    n = _near(_log(rng, 128, 2048 if op == "execute" else 512) if planar else
             _log(rng, 64, 128 if op == "reconstruct" else 192 if op == "forward" else 512), m)
    c = dict(op="execute" if op == "spiral" else op, kind=kind, nx=n, ny=n if even else max(8, n - rng.randint(0, n // 8)))
    fov = rng.uniform(200.0, 400.0)
    c["vox"] = c["voxz"] = round(fov / n, 4)
    c["nv"] = _near(n * rng.uniform(0.7, 1.6), m) if n < 1024 else _near(n * rng.uniform(0.5, 0.9), m)
    c["nc"] = _near(n * rng.uniform(1.3, 2.1), m)
    if kind not in PARALLEL or kind == "cone_parallel":
        c["sod"] = round(rng.uniform(550.0, 800.0), 1)
        c["sdd"] = round(c["sod"] * rng.uniform(1.5, 1.9), 1)
    mag = c["sdd"] / c["sod"] if c.get("sdd") else 1.0
    cover = rng.uniform(0.9, 1.25)
    if kind in ARC:
        c["du"] = round(2.0 * math.asin(min(0.9, cover * fov / 2 / c["sod"])) / c["nc"], 7)
    else:
        c["du"] = round(cover * fov * (mag if kind not in PARALLEL else 1.0) / c["nc"], 5)
    if not planar:
        c["nz"] = _near(min(n * rng.uniform(0.2, 0.9), 2e10 / (n * n * c["nv"])), 2 if even else 1)
        c["nr"] = _near(c["nz"] * rng.uniform(0.9, 1.8), m)
        c["dv"] = round(cover * c["nz"] * c["voxz"] * mag / c["nr"], 5)
    if not even:
        c["mx"], c["my"] = round(rng.uniform(-10, 10), 2), round(rng.uniform(-10, 10), 2)
        c["mz"] = 0.0 if planar else round(rng.uniform(-4, 4), 2)
    c["ccw"] = rng.random() < 0.3
    if op == "spiral":
        turns = rng.randint(3, 5)
        npr = _near(n * rng.uniform(0.8, 1.5), m)
        c.update(scan="spiral", turns=turns, nv=npr * turns, mx=0.0, my=0.0, mz=0.0, nr=_near(rng.uniform(24, 96), m))
        c["pitch"] = round(c["nz"] * c["voxz"] / (turns - 1.0) / (2 * math.pi), 4)
        c["dv"] = round(1.3 * c["nz"] * c["voxz"] / (turns - 1.0) * mag / c["nr"], 5)
    elif kind in ("fan_line", "cone_flat") and op == "execute" and rng.random() < 0.4:
        c["scan"] = "short"
    if op == "execute":
        c["storage"] = rng.choice(["f32", "f16"])
        if c["storage"] == "f16":
            c["filter"] = rng.choice(["fft", "toeplitz_f16x2", "toeplitz_bf16x4"])
    if op != "forward":
        c["apod"] = rng.choice(["none", "none", "hann", "hamming"])
        c["cutoff"] = 1.0 if c["apod"] == "none" else round(rng.uniform(0.7, 1.0), 2)
    return _case(**c)


# ---- geometry in the framework's terms ---------------------------------------------------------

def _span(c):
    """(total rotation angle, angle step)."""
    if c["scan"] == "short":
        span = math.pi + 2.0 * math.atan(c["nc"] * c["du"] / 2.0 / c["sdd"])
    else:
        span = 2.0 * math.pi * c["turns"]
    return span, span / c["nv"]


def _geometry(c):
    _, incr = _span(c)
    rot = g.RotationParams(g.RotDir.CCW if c["ccw"] else g.RotDir.CW, 0.0, incr, c["nv"], c["pitch"])
    nc, nr, k = c["nc"], c["nr"], c["kind"]
    c0, r0 = (nc - 1) / 2.0, (nr - 1) / 2.0
    row = {"parallel_1d": g.DetParallel, "parallel_2d": g.DetParallel, "cone_parallel": g.DetParallel,
           "fan_arc": g.DetFanArc, "cone_cyl": g.DetFanArc}.get(k, g.DetFanLine)(nc, c["du"])
    if k in PLANAR:
        det = (row,)
        params = (g.Parallel1DProjGeomParams(c0, rot) if k == "parallel_1d"
                  else g.FanBeamProjGeomParams(c0, rot, c["sdd"], c["sod"]))
    else:
        det = (row, (g.DetParallel if k == "parallel_2d" else g.DetFanLine)(nr, c["dv"]))
        params = (g.Parallel2DProjGeomParams(c0, rot, r0) if k == "parallel_2d"
                  else g.ConeBeamProjGeomParams(c0, rot, c["sdd"], c["sod"], r0))
    if c["scan"] == "spiral":
        cg = g.SpiralCTGeom(det, g.ProjGeomFactory(*(type(d) for d in det)).create_all(params))
    else:
        cg = g.AxialCTGeom.from_params(det, params)
    x, y = g.EqDistSampler(c["nx"], c["vox"]), g.EqDistSampler(c["ny"], c["vox"])
    if k in PLANAR:
        return cg, g.ReconImgGeom(x, y, None, (c["mx"], c["my"]))
    return cg, g.ReconImgGeom(x, y, g.EqDistSampler(c["nz"], c["voxz"]), (c["mx"], c["my"], _mid_z(c)))


def _mid_z(c):
    if c["scan"] != "spiral":
        return c["mz"]
    return -c["pitch"] * _span(c)[1] * (c["nv"] - 1) / 2.0  # the middle of the helix


def _options(c):
    o = g.FdkOptions(filter=FILTERS[c["filter"]], storage=g.STORAGE_F16 if c["storage"] == "f16" else g.STORAGE_F32)
    if c["scan"] == "spiral":
        o.scan = g.SCAN_SPIRAL
    return o


def _filt(c):
    return g.FiltParams(c["cutoff"], APODS[c["apod"]])


def _batch_items():
    """A quarter of the uneven batch mix: six parallel slices, two fan arcs, two cylindrical cones,
    two rebinned cones."""
    items = []
    for n, nv in [(256, 180), (512, 360), (1024, 900), (2048, 1800), (256, 180), (512, 360)]:
        items.append(_case(kind="parallel_1d", nv=nv, nc=int(math.ceil(1.42 * n)), du=250.0 / n, nx=n, ny=n,
                           vox=250.0 / n, storage="f16"))
    items += [_case(kind="fan_arc", nv=1152, nc=672, du=0.907 / 672, sod=570.0, sdd=1040.0, nx=512, ny=512, vox=0.9,
                    storage="f16")] * 2
    items += [_case(kind="cone_cyl", nv=1152, nc=896, nr=64, du=0.0011, sod=600.0, sdd=1100.0, nx=512, ny=512, nz=64,
                    vox=0.9, voxz=0.55, storage="f16")] * 2
    items += [_case(kind="cone_parallel", nv=1152, nc=736, nr=64, du=0.65, sod=600.0, sdd=1100.0, nx=512, ny=512, nz=64,
                    vox=0.9, voxz=0.55, storage="f16")] * 2
    return items


# ---- the same geometry from its definition, in 64 bits -----------------------------------------

class _Scan:
    """Views of a circular or helical scan: source, detector axes and angles as 64-bit tensors."""

    def __init__(self, c, dev):
        f = dict(dtype=torch.float64, device=dev)
        _, self.incr = _span(c)
        th = torch.arange(c["nv"], **f) * self.incr
        phi = -th if c["ccw"] else th
        cs, sn, zero = torch.cos(phi), torch.sin(phi), torch.zeros_like(phi)
        self.theta = th
        self.src = torch.stack([c["sod"] * cs, c["sod"] * sn, -c["pitch"] * th], 1)
        self.eu = torch.stack([-sn, cs, zero], 1)
        self.ew = torch.stack([-cs, -sn, zero], 1)
        self.c0, self.r0 = (c["nc"] - 1) / 2.0, (c["nr"] - 1) / 2.0
        self.u = (torch.arange(c["nc"], **f) - self.c0) * c["du"]
        self.v = (torch.arange(c["nr"], **f) - self.r0) * (c["dv"] if c["kind"] not in PLANAR else 0.0)
        self.mid = (c["mx"], c["my"], 0.0 if c["kind"] in PLANAR else _mid_z(c))

    def rays(self, c, v0, v1):
        """Origins and directions [views][rows][cols] of the rays of views [v0, v1)."""
        u, t = self.u[None, None, :], self.v[None, :, None]
        if c["kind"] in PARALLEL:  # detector coordinate along (-sin, cos), rays along (cos, sin)
            cs, sn = torch.cos(self.theta[v0:v1, None, None]), torch.sin(self.theta[v0:v1, None, None])
            z = -t * (c["sod"] / c["sdd"] if c["kind"] == "cone_parallel" else 1.0)
            o = torch.broadcast_tensors(-sn * u, cs * u, z + 0 * u + 0 * sn)
            d = torch.broadcast_tensors(cs + 0 * o[0], sn + 0 * o[0], 0 * o[0])
            return o, d
        e = [x[v0:v1, None, None, :] for x in (self.src, self.eu, self.ew)]
        if c["kind"] in ARC:
            a, b, z = torch.cos(u), torch.sin(u), -t / c["sdd"]
        else:
            a, b, z = torch.full_like(u, c["sdd"]), u, -t
        d = [a * e[2][..., k] + b * e[1][..., k] + (z if k == 2 else 0.0) + 0 * t for k in range(3)]
        o = [e[0][..., k] + 0 * d[0] for k in range(3)]
        return o, d


def _ellipsoids(c, seed):
    """Seeded body and inserts (centre, semi-axes, angle, attenuation) scaled to the grid."""
    rs = np.random.RandomState(seed % (1 << 32))
    rx = 0.5 * c["vox"] * min(c["nx"], c["ny"])
    rz = 0.5 * c["voxz"] * c["nz"] if c["kind"] not in PLANAR else rx
    z0 = 0.0 if c["kind"] in PLANAR else _mid_z(c)
    ell = [(0.0, 0.0, z0, 0.80 * rx, 0.65 * rx, 0.9 * rz, 0.0, 0.019)]
    for _ in range(5):
        r, t = 0.5 * rx * math.sqrt(rs.uniform()), rs.uniform(0, 2 * math.pi)
        a = rs.uniform(0.05, 0.25, size=3)
        ell.append((r * math.cos(t), r * math.sin(t), z0 + rs.uniform(-0.5, 0.5) * rz, a[0] * rx, a[1] * rx, a[2] * rz,
                    rs.uniform(0, math.pi), rs.uniform(-0.008, 0.02)))
    return ell


def _projections(c, seed, dev="cuda"):
    """Line integrals of the seeded phantom with photon noise (I0 = 1e5), float32 [view][row][col]."""
    s = _Scan(c, dev)
    out = torch.empty((c["nv"], c["nr"], c["nc"]), dtype=torch.float32, device=dev)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    ell = _ellipsoids(c, seed)
    step = max(1, (1 << 23) // (c["nr"] * c["nc"]))
    for v0 in range(0, c["nv"], step):
        v1 = min(c["nv"], v0 + step)
        o, d = s.rays(c, v0, v1)
        dn = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        total = torch.zeros_like(dn)
        for cx, cy, cz, ax, ay, az, ang, mu in ell:
            cp, sp = math.cos(ang), math.sin(ang)
            px, py, pz = o[0] - cx, o[1] - cy, (o[2] - cz) / az
            px, py = (cp * px + sp * py) / ax, (-sp * px + cp * py) / ay
            qx, qy, qz = (cp * d[0] + sp * d[1]) / ax, (-sp * d[0] + cp * d[1]) / ay, d[2] / az
            if c["kind"] in PLANAR:
                pz, qz = 0.0 * pz, 0.0 * qz
            A = qx * qx + qy * qy + qz * qz
            B = px * qx + py * qy + pz * qz
            C = px * px + py * py + pz * pz - 1.0
            total += 2.0 * mu * torch.sqrt((B * B - A * C).clamp_(min=0.0)) / A * dn
        counts = torch.poisson(1e5 * torch.exp(-total), generator=gen).clamp_(min=1.0)
        out[v0:v1] = -torch.log(counts / 1e5)
    return out


def _volume(c, seed, dev="cuda"):
    """The seeded phantom on the grid, with a little texture, float32 [z][y][x] (2D: [y][x])."""
    x, y, z = _axes(c, dev)
    vol = torch.zeros((len(z), len(y), len(x)), dtype=torch.float32, device=dev)
    for cx, cy, cz, ax, ay, az, ang, mu in _ellipsoids(c, seed):
        cp, sp = math.cos(ang), math.sin(ang)
        dx, dy = x[None, None, :] - cx, y[None, :, None] - cy
        r = ((cp * dx + sp * dy) / ax) ** 2 + ((-sp * dx + cp * dy) / ay) ** 2
        if c["kind"] not in PLANAR:
            r = r + ((z[:, None, None] - cz) / az) ** 2
        vol += torch.where(r <= 1.0, mu, 0.0).float()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    vol += 5e-4 * torch.randn(vol.shape, generator=gen, device=dev)
    return vol[0] if c["kind"] in PLANAR else vol


def _axes(c, dev):
    """Voxel centre coordinates along x, y, z."""
    f = dict(dtype=torch.float64, device=dev)
    mid = (c["mx"], c["my"], 0.0 if c["kind"] in PLANAR else _mid_z(c))
    return [m + (torch.arange(n, **f) - (n - 1) / 2.0) * w
            for m, n, w in zip(mid, (c["nx"], c["ny"], c["nz"]), (c["vox"], c["vox"], c["voxz"]))]


# ---- what a user's program has and calls -------------------------------------------------------

def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    if c["op"] == "batch":
        items = []
        for i, it in enumerate(_batch_items()):
            cg, vg = _geometry(it)
            items.append((g.FdkPlan(cg, vg, _filt(it), _options(it)), _projections(it, seed + 1000 * i),
                          torch.empty(vg.shape, dtype=torch.float32, device="cuda")))
        return dict(op="batch", items=items, batch=g.FdkBatch(items))
    cg, vg = _geometry(c)
    if c["op"] == "forward":
        return dict(op="forward", cg=cg, vg=vg, vol=_volume(c, seed),
                    proj=torch.empty((c["nv"], c["nr"], c["nc"]), dtype=torch.float32, device="cuda"))
    proj = _projections(c, seed)
    if c["op"] == "reconstruct":
        return dict(op="reconstruct", cg=cg, vol=g.ReconImg(vg), proj=proj.cpu().numpy(), filt=_filt(c),
                    opts=_options(c))
    return dict(op="execute", plan=g.FdkPlan(cg, vg, _filt(c), _options(c)), proj=proj,
                vol=torch.empty(vg.shape, dtype=torch.float32, device="cuda"))


def run(state):
    op = state["op"]
    if op == "execute":
        state["plan"].execute(state["proj"], state["vol"])
        return state["vol"]
    if op == "reconstruct":
        g.reconstruct(state["cg"], state["proj"], state["vol"], state["filt"], state["opts"])
        return state["vol"].elements
    if op == "forward":
        g.forward_project(state["cg"], state["vg"], state["vol"], state["proj"])
        return state["proj"]
    state["batch"].launch()
    return [vol for _, _, vol in state["items"]]


def work(case):
    """Projections read once, volume written once (forward projection: the reverse); ten operations
    per voxel-view update (bilinear blend, weight, sum) plus the ramp filter as two real transforms of
    twice the row, or seventeen per trilinear sample at half a voxel along the rays."""
    c = dict(DEFAULTS, **case)
    if c["op"] == "batch":
        parts = [work(it) for it in _batch_items()]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    pixels, voxels = c["nv"] * c["nr"] * c["nc"], c["nx"] * c["ny"] * c["nz"]
    moved = 4.0 * (pixels + voxels)
    if c["op"] == "forward":
        along = 0.6 * 2.0 * max(c["nx"], c["ny"])  # samples of a central ray that meets the grid
        return {"bytes": moved, "flops": 17.0 * along * pixels}
    views = c["nv"] / c["turns"]
    return {"bytes": moved, "flops": 10.0 * voxels * views + pixels * 10.0 * math.log2(2 * c["nc"])}


# ---- 64-bit results ----------------------------------------------------------------------------

def _taps(c, dev):
    """Ramp kernel g(m), m = -N/2 .. N-1-N/2, with cut-off and apodisation; the arc detectors' taps
    carry (b / sin b)^2."""
    n = c["nc"]
    m = torch.arange(n, dtype=torch.float64, device=dev) - n // 2

    def big_m(t):
        s = torch.where(t == 0, 1.0, t)
        return torch.where(t == 0, 0.5, torch.sin(s) / s + (torch.cos(s) - 1.0) / (s * s))

    a = {"none": 1.0, "hann": 0.5, "hamming": 0.54}[c["apod"]]
    fc = c["cutoff"]
    k = fc * math.pi * m
    h = fc * fc / (2.0 * c["du"]) * (a * big_m(k) + (1 - a) / 2 * (big_m(k + math.pi) + big_m(k - math.pi)))
    if c["kind"] in ARC:
        b = torch.where(m == 0, 1.0, m * c["du"])
        h = torch.where(m == 0, h, h * (b / torch.sin(b)) ** 2)
    return h


def _redundancy(c, s):
    """Weights [view][col] for rays measured more than once."""
    one = torch.ones((c["nv"], c["nc"]), dtype=torch.float64, device=s.u.device)
    if c["scan"] == "spiral":
        return one
    phi = s.incr * c["nv"]
    if c["kind"] in PARALLEL:
        return one * (1.0 if phi <= s.incr + math.pi else 0.5)
    b = (s.theta.flip(0) if c["ccw"] else s.theta)[:, None]
    gm = (s.u if c["kind"] in ARC else torch.atan2(s.u, torch.full_like(s.u, c["sdd"])))[None, :]
    t2, t3 = 2 * gm + phi - math.pi, 2 * gm + math.pi
    rise = torch.sin(math.pi * b / (2 * (phi - math.pi) + 4 * gm)) ** 2
    fall = torch.sin(math.pi * (phi - b) / (2 * (phi - math.pi) - 4 * gm)) ** 2
    w = torch.where(b <= t2, rise, torch.where(b <= t3, one, torch.where((b >= t3) & (b <= phi), fall, 0 * one)))
    return w


def _filtered(c, s, proj):
    """Weighted and ramp-filtered views, 64-bit [view][row][col]."""
    u, t = s.u[None, :], s.v[:, None]
    k, sdd = c["kind"], c["sdd"]
    if k in ("parallel_1d", "parallel_2d"):
        cosw = torch.ones_like(u + t)
    elif k == "cone_parallel":
        cosw = sdd / torch.sqrt(t * t + sdd * sdd) + 0 * u
    elif k in ARC:
        cosw = torch.cos(u) * sdd / torch.sqrt(t * t + sdd * sdd)
    else:
        cosw = sdd / torch.sqrt(u * u + t * t + sdd * sdd)
    w = _redundancy(c, s)
    n = c["nc"]
    length = 1 << (2 * n).bit_length()
    kern = torch.zeros(length, dtype=torch.float64, device=u.device)
    kern[(torch.arange(n, device=u.device) - n // 2) % length] = _taps(c, u.device)
    spec = torch.fft.rfft(kern)
    out = torch.empty(proj.shape, dtype=torch.float64, device=u.device)
    step = max(1, (1 << 24) // (c["nr"] * length))
    for v in range(0, c["nv"], step):
        x = proj[v:v + step].double() * cosw * w[v:v + step, None, :]
        out[v:v + step] = torch.fft.irfft(torch.fft.rfft(x, length) * spec, length)[..., :n]
    return out


def _spiral_windows(c, s, z):
    """Views [first, last) of every slice: the rotation centred on the view nearest the slice."""
    npr = c["nv"] // c["turns"]
    first = torch.argmin(torch.abs(s.src[None, :, 2] - z[:, None]), 1) - npr // 2
    last = first + npr
    good = (first > 0) & (last < c["nv"])
    return torch.where(good, first, 0), torch.where(good, last, 0)


def _fdk(c, proj):
    dev = proj.device
    s = _Scan(c, dev)
    filt = _filtered(c, s, proj)
    x, y, z = _axes(c, dev)
    nr, nc = c["nr"], c["nc"]
    planar = c["kind"] in PLANAR
    vol = torch.zeros((len(z), len(y), len(x)), dtype=torch.float64, device=dev)
    if c["scan"] == "spiral":
        first, last = _spiral_windows(c, s, z)
    pad = torch.zeros((nr + 4, nc + 4), dtype=torch.float64, device=dev)
    X, Y = x[None, :], y[:, None]
    for v in range(c["nv"]):
        ks = slice(None)
        if c["scan"] == "spiral":
            used = torch.nonzero((first <= v) & (v < last))[:, 0]
            if len(used) == 0:
                continue
            ks = slice(int(used[0]), int(used[-1]) + 1)
        Z = z[ks, None, None]
        pad[2:nr + 2, 2:nc + 2] = filt[v]
        if c["kind"] in PARALLEL:
            th = float(s.theta[v]) + math.pi / 2
            u = (X * math.cos(th) + Y * math.sin(th)) / c["du"] + s.c0
            mag = c["sdd"] / c["sod"] if c["kind"] == "cone_parallel" else 1.0
            row = (-Z * mag / c["dv"] + s.r0).expand(-1, len(y), len(x))
            wt = torch.full_like(u, s.incr)
        else:
            sx, sy, sz = s.src[v].tolist()
            eu, ew = s.eu[v].tolist(), s.ew[v].tolist()
            sid = math.sqrt(sx * sx + sy * sy + sz * sz)
            A = eu[0] * (X - sx) + eu[1] * (Y - sy)
            D = ew[0] * (X - sx) + ew[1] * (Y - sy)
            T = sz - Z
            if c["kind"] in ARC:
                rho2 = A * A + D * D
                u = torch.atan2(A, D) / c["du"] + s.c0
                row = c["sdd"] / c["dv"] * T / torch.sqrt(rho2) + s.r0
                wt = s.incr * sid / (rho2 if planar else rho2 + T * T)
            else:
                u = c["sdd"] * A / D / c["du"] + s.c0
                row = c["sdd"] / c["dv"] * T / D + s.r0
                wt = s.incr * c["sdd"] * sid / (D * D)
        u = u.clamp(-1.5, nc + 0.5)
        iu = torch.floor(u)
        fu = u - iu
        if planar:
            at = iu.long() + 2
            vol[0] += wt * torch.lerp(pad[2][at], pad[2][at + 1], fu)
            continue
        row = row.clamp(-1.5, nr + 0.5)
        iv = torch.floor(row)
        fv = row - iv
        fu = fu.expand_as(fv)
        at = ((iv + 2) * (nc + 4) + (iu + 2)).long()
        flat = pad.view(-1)
        top = torch.lerp(flat[at], flat[at + 1], fu)
        at += nc + 4
        bot = torch.lerp(flat[at], flat[at + 1], fu)
        val = torch.lerp(top, bot, fv).mul_(wt)
        if c["scan"] == "spiral":
            val *= ((first[ks] <= v) & (v < last[ks]))[:, None, None]
        vol[ks] += val
    return vol[0] if planar else vol


def _forward(c, vol):
    """Midpoint sums of trilinear samples every half voxel between a ray's two crossings of the
    grid's outer faces; samples outside the outermost voxel centres blend with zero."""
    dev = vol.device
    s = _Scan(c, dev)
    planar = c["kind"] in PLANAR
    n = [c["nx"], c["ny"], c["nz"]]
    w = [c["vox"], c["vox"], c["voxz"]]
    lo = [float(a[0]) for a in _axes(c, dev)]
    axes = [0, 1] if planar else [0, 1, 2]
    h = 0.5 * min(w[a] for a in axes)
    grid = vol.double()[None, None] if not planar else vol.double()[None, None, None]
    out = torch.zeros((c["nv"], c["nr"], c["nc"]), dtype=torch.float64, device=dev)
    for v in range(c["nv"]):
        o, d = s.rays(c, v, v + 1)
        if planar:
            d = [d[0], d[1], 0 * d[0]]
        dn = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        d = [x / dn for x in d]
        t0, t1 = torch.full_like(dn, -1e300), torch.full_like(dn, 1e300)
        hit = torch.ones_like(dn, dtype=torch.bool)
        for a in axes:
            l, r = lo[a] - 0.5 * w[a], lo[a] + (n[a] - 0.5) * w[a]
            flat = d[a].abs() < 1e-15
            da = torch.where(flat, 1.0, d[a])
            ta, tb = (l - o[a]) / da, (r - o[a]) / da
            t0 = torch.where(flat, t0, torch.maximum(t0, torch.minimum(ta, tb)))
            t1 = torch.where(flat, t1, torch.minimum(t1, torch.maximum(ta, tb)))
            hit &= ~flat | ((o[a] >= l) & (o[a] <= r))
        hit &= t1 > t0
        if not bool(hit.any()):
            continue
        o, d = [x[hit] for x in o], [x[hit] for x in d]
        t0, t1 = t0[hit], t1[hit]
        steps = torch.ceil((t1 - t0) / h)
        total = torch.zeros_like(t0)
        most, part = int(steps.max()), 64
        for k0 in range(0, most, part):
            k = torch.arange(k0, min(most, k0 + part), dtype=torch.float64, device=dev)
            t = t0[:, None] + (k + 0.5) * h
            # grid_sample's coordinates: -1 and 1 at the outermost voxel centres
            p = [2.0 * (o[a][:, None] + t * d[a][:, None] - lo[a]) / (w[a] * (n[a] - 1.0)) - 1.0 if a in axes
                 else 0 * t for a in range(3)]
            got = torch.nn.functional.grid_sample(grid, torch.stack(p, -1)[None, None], mode="bilinear",
                                                  padding_mode="zeros", align_corners=True)[0, 0, 0]
            total += torch.where(k < steps[:, None], got, 0.0).sum(1)
        out[v][hit[0]] = total * h
    return out


def exact(case, seed):
    c = dict(DEFAULTS, **case)
    if c["op"] == "batch":
        return [_fdk(it, _projections(it, seed + 1000 * i)) for i, it in enumerate(_batch_items())]
    if c["op"] == "forward":
        return _forward(c, _volume(c, seed))
    if c["nx"] * c["ny"] * c["nz"] * c["nv"] > 6e10:
        return None  # minutes in 64 bits
    return _fdk(c, _projections(c, seed))
