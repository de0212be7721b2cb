"""gct_forward_project against its definition in FP64 numpy: midpoint sums of trilinear samples
every step_vox smallest voxel lengths between a ray's crossings of the grid's outer faces, with
zero outside the outermost voxel centres.

The cases sit where the kernel's paths meet: grids below and above the size that is read through
copies (pairs of planes, x and y exchanged), rays along x, along y and at 45 degrees, odd sides,
grids one voxel thick, off the axis and missed by rays, steps of a quarter voxel and steps longer
than a voxel along a ray (the range-checked path), anisotropic voxels.

Tolerance: a sample's position is within 8e-6 voxels of its FP64 value and the values lie in
[0, 1), so a blend is off by at most 3 x 8e-6; 8 blends' roundings and the FP32 sum of n samples add
(8 + n / 2) x 6e-8. With n <= 700 that is below 5e-5 of a sample, hence 5e-5 of the ray's length."""
import math

import numpy as np
import pytest

import gct_b200 as g

pytestmark = pytest.mark.gpu


def _rays(kind, nv, nc, nr, du, dv, sid, sdd):
    th = 2 * math.pi * np.arange(nv) / nv
    cs, sn = (f(th)[:, None, None] for f in (np.cos, np.sin))
    u = ((np.arange(nc) - (nc - 1) / 2) * du)[None, None, :]
    t = ((np.arange(nr) - (nr - 1) / 2) * dv)[None, :, None]
    zero = np.zeros((nv, nr, nc))
    if kind == "parallel_2d":
        return [-sn * u + zero, cs * u + zero, -t + zero], [cs + zero, sn + zero, zero]
    if kind in ("cone_cyl", "fan_arc"):
        a, b, w = np.cos(u), np.sin(u), -t / sdd
    else:
        a, b, w = sdd + 0 * u, u, -t
    if kind in ("fan_arc", "fan_line"):
        w = 0 * t
    return [sid * cs + zero, sid * sn + zero, zero], [-a * cs - b * sn + zero, -a * sn + b * cs + zero, w + zero]


def _reference(o, d, vol, lo, w, step, planar):
    axes = [0, 1] if planar else [0, 1, 2]
    n = vol.shape[::-1]
    dn = np.sqrt(sum(x * x for x in d))
    d = [x / dn for x in d]
    h = step * min(w[a] for a in axes)
    out = np.zeros(dn.shape)
    length = np.zeros(dn.shape)
    pad = np.zeros(tuple(k + 4 for k in vol.shape))
    pad[2:-2, 2:-2, 2:-2] = vol
    for at in np.ndindex(dn.shape):
        t0, t1 = -1e300, 1e300
        for a in axes:
            l, r = lo[a] - 0.5 * w[a], lo[a] + (n[a] - 0.5) * w[a]
            if abs(d[a][at]) < 1e-15:
                if not l <= o[a][at] <= r:
                    t1 = -1e300
                continue
            ta, tb = sorted(((l - o[a][at]) / d[a][at], (r - o[a][at]) / d[a][at]))
            t0, t1 = max(t0, ta), min(t1, tb)
        if not t1 > t0:
            continue
        t = t0 + (np.arange(math.ceil((t1 - t0) / h)) + 0.5) * h
        p = [np.clip((o[a][at] + t * d[a][at] - lo[a]) / w[a], -1.5, n[a] + 0.5) if a in axes else 0 * t
             for a in range(3)]
        i = [np.floor(x).astype(int) for x in p]
        f = [x - k for x, k in zip(p, i)]
        s = 0.0
        for k in range(8):
            b = [k & 1, k >> 1 & 1, k >> 2]
            wt = np.prod([f[a] if b[a] else 1 - f[a] for a in range(3)], axis=0)
            s = s + wt * pad[i[2] + 2 + b[2], i[1] + 2 + b[1], i[0] + 2 + b[0]]
        out[at] = s.sum() * h
        length[at] = t1 - t0
    return out, length


@pytest.mark.parametrize("kind,n,vox,mid,step", [
    ("cone_flat", (24, 22, 20), (1.0, 1.0, 1.0), (0, 0, 0), 0.5),       # read as it is
    ("cone_flat", (33, 31, 37), (1.0, 1.0, 0.7), (2.0, -1.0, 1.5), 0.5),  # through copies
    ("cone_flat", (130, 128, 1), (0.4, 0.4, 3.0), (0, 0, 0), 0.5),      # one plane: no interior
    ("cone_flat", (40, 36, 32), (1.0, 1.0, 0.25), (0, 0, 0), 0.25),     # short steps
    ("cone_flat", (40, 36, 32), (1.0, 0.5, 1.0), (0, 0, 0), 2.5),       # steps longer than a voxel
    ("cone_cyl", (65, 17, 19), (0.5, 2.0, 1.0), (-6.0, 3.0, 0), 0.5),
    ("parallel_2d", (32, 32, 33), (1.0, 1.0, 1.0), (0, 0, 0), 0.5),     # rays along the axes
    ("parallel_2d", (128, 2, 70), (0.3, 5.0, 0.5), (0, 9.0, 0), 0.5),   # two voxels across
    ("fan_line", (101, 99, 1), (0.4, 0.4, 1.0), (0, 0, 0), 0.5),
    ("fan_line", (203, 187, 1), (0.2, 0.2, 1.0), (4.0, 0, 0), 0.5),
    ("fan_arc", (257, 129, 1), (0.15, 0.3, 1.0), (0, 5.0, 0), 0.37),
])
def test_forward_project_is_the_sum_of_its_samples(kind, n, vox, mid, step):
    import torch
    planar = kind in ("fan_line", "fan_arc")
    nv, nc, nr = 8, 37, 1 if planar else 11
    du, dv, sid, sdd = (0.0031 if kind in ("fan_arc", "cone_cyl") else 1.9 if kind != "parallel_2d" else 1.1), 2.3, 300.0, 500.0
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
    c0, r0 = (nc - 1) / 2, (nr - 1) / 2
    if planar:
        det = ((g.DetFanArc if kind == "fan_arc" else g.DetFanLine)(nc, du),)
        params = g.FanBeamProjGeomParams(c0, rot, sdd, sid)
    elif kind == "parallel_2d":
        det, params = (g.DetParallel(nc, du), g.DetParallel(nr, dv)), g.Parallel2DProjGeomParams(c0, rot, r0)
    else:
        det = ((g.DetFanArc if kind == "cone_cyl" else g.DetFanLine)(nc, du), g.DetFanLine(nr, dv))
        params = g.ConeBeamProjGeomParams(c0, rot, sdd, sid, r0)
    cg = g.AxialCTGeom.from_params(det, params)
    x, y = g.EqDistSampler(n[0], vox[0]), g.EqDistSampler(n[1], vox[1])
    vg = g.ReconImgGeom(x, y, None, mid[:2]) if planar else g.ReconImgGeom(x, y, g.EqDistSampler(n[2], vox[2]), mid)
    vol = np.random.RandomState(3).rand(n[2], n[1], n[0]).astype(np.float32)
    out = torch.full((nv, nr, nc), float("nan"), dtype=torch.float32, device="cuda")
    g.forward_project(cg, vg, torch.from_numpy(vol.reshape(vg.shape)).cuda(), out, step_vox=step)
    got = out.cpu().numpy().astype(np.float64)
    lo = [m - (k - 1) * w / 2 for m, k, w in zip((mid[0], mid[1], 0.0 if planar else mid[2]), n, vox)]
    o, d = _rays(kind, nv, nc, nr, du, dv, sid, sdd)
    ref, length = _reference(o, d, vol.astype(np.float64), lo, vox, step, planar)
    assert (length > 0).mean() > 0.2
    err = np.abs(got - ref)
    assert (err <= 5e-5 * (length + max(vox))).all(), float((err / (length + max(vox))).max())
