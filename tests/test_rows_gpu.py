"""The planar kinds' backprojector (row pairs, 32 x 32 pixel cells) against its definition: FP64 sums of
linear interpolations in the filtered rows, at coordinates taken in the FP32 steps that all
backprojection kernels share (per-view forms in voxel indices rounded to FP32, fused multiply-adds, then
the quotient or the angle). No cells, no classes, no chunks: every pixel and view in turn.

The cases sit at the edges of the kernel's cells and view chunks: images of one pixel, of one cell and of
one pixel more or less, wide and tall ones, fewer views than one stage (32) and counts that leave empty or
short chunks, images that reach past the detector's field (cells off the row, partly off it) and close to
the source (beyond the angles of the arc kind's polynomial), odd rows, both turns, and the image added to
in chunks.

Tolerance: the approximate reciprocal and the angle are off by a unit or two in the last place, 1e-5 of
a sample at 130 columns, and a random row changes by its own size per sample; the sum over n views adds
sqrt(n) x 6e-8. Together below 2e-5 relative RMS. FP16 storage and the split filters round samples to
2^-11 and drop parts of the rows: 1e-3."""
import math

import numpy as np
import pytest

import gct_b200 as g
pytestmark = pytest.mark.gpu

# kind, views, columns, nx, ny, pixel (mm), centre, turn, storage, filter
CASES = [
    ("parallel_1d", 5, 64, 1, 1, 1.0, (0.0, 0.0), 1, "f32", "fft"),
    ("parallel_1d", 33, 97, 31, 33, 1.0, (2.0, -3.0), 1, "f32", "fft"),
    ("parallel_1d", 130, 101, 32, 64, 1.0, (0.0, 0.0), -1, "f16", "fft"),
    ("parallel_1d", 90, 80, 95, 65, 2.0, (0.0, 0.0), 1, "f32", "fft"),
    ("fan_line", 17, 66, 32, 32, 1.0, (0.0, 0.0), 1, "f32", "fft"),
    ("fan_line", 129, 131, 33, 97, 1.0, (-4.0, 6.0), -1, "f32", "fft"),
    ("fan_line", 120, 60, 128, 96, 6.0, (0.0, 0.0), 1, "f32", "fft"),
    ("fan_line", 64, 96, 64, 64, 1.0, (0.0, 0.0), 1, "f16", "fft"),
    ("fan_line", 36, 40, 2, 2, 1.0, (0.0, 0.0), 1, "f16", "fft"),  # quarter turns: partners interleaved
    ("fan_line", 132, 90, 70, 70, 1.0, (0.0, 0.0), -1, "f16", "fft"),
    ("fan_line", 64, 60, 96, 96, 6.0, (0.0, 0.0), 1, "f16", "fft"),
    ("fan_line", 66, 60, 64, 64, 1.0, (0.0, 0.0), 1, "f16", "fft"),  # no quarter turns
    ("fan_arc", 9, 67, 33, 31, 1.0, (0.0, 0.0), 1, "f32", "fft"),
    ("fan_arc", 131, 128, 65, 40, 1.0, (5.0, 3.0), -1, "f32", "fft"),
    ("fan_arc", 120, 61, 96, 96, 6.0, (0.0, 0.0), 1, "f32", "fft"),
    ("fan_arc", 72, 96, 64, 64, 1.0, (0.0, 0.0), 1, "f32", "toeplitz_bf16x4"),
]


def _scan(kind, nv, nc, nx, ny, vox, mid, turn):
    rot = g.RotationParams(g.RotDir.CW if turn > 0 else g.RotDir.CCW, 0.3, 2 * math.pi / nv, nv)
    c0 = (nc - 1) / 2
    reach = 1.1 * min(max(nx, ny), 64)
    if kind == "parallel_1d":
        det, params = g.DetParallel(nc, reach / nc), g.Parallel1DProjGeomParams(c0, rot)
    elif kind == "fan_line":
        det, params = g.DetFanLine(nc, 1.6 * reach / nc), g.FanBeamProjGeomParams(c0, rot, 960.0, 600.0)
    else:
        det, params = g.DetFanArc(nc, reach / 600 / nc), g.FanBeamProjGeomParams(c0, rot, 960.0, 600.0)
    cg = g.AxialCTGeom.from_params((det,), params)
    return cg, g.ReconImgGeom(g.EqDistSampler(nx, vox), g.EqDistSampler(ny, vox), None, mid)


def _fma(a, b, c):
    a, b, c = (np.asarray(z, np.float64) for z in (a, b, c))
    return (a * b + c).astype(np.float32)


def _reference(kind, cg, rows, nx, ny, vox, mid, nv):
    """Image of the filtered rows [view][col]."""
    f32 = np.float32
    nc, du = rows.shape[1], cg.det_geom()[0].sampling_width
    x0, y0 = (m - (n - 1) * vox / 2 for m, n in zip(mid, (nx, ny)))
    i, j = np.arange(nx, dtype=f32)[None, :], np.arange(ny, dtype=f32)[:, None]
    pad = np.zeros((nv, nc + 4))
    pad[:, 2:-2] = rows
    out = np.zeros((ny, nx))
    for v in range(nv):
        w = cg.views[v]
        c0, sdd = float(w["det_row_center"]), float(w["src_det_dist"])
        if kind == "parallel_1d":
            t = float(w["rot_ang"]) + math.pi / 2
            u0, ui, uj = (f32(z) for z in ((x0 * math.cos(t) + y0 * math.sin(t)) / du + c0, vox * math.cos(t) / du,
                                           vox * math.sin(t) / du))
            k0 = np.floor(j / 16) * 16  # rows in steps of 16 from the coordinate of their first
            u = _fma(uj, j - k0, _fma(uj, k0, _fma(ui, i, u0)) - f32(0.5)).astype(np.float64) + 0.5
            wt = np.ones((ny, nx))
        else:
            s, eu = np.array(w["src_pos"][:2], float), np.array(w["det_row_dir"][:2], float)
            ew = np.array([-eu[1], eu[0]]) if kind == "fan_line" else np.array(w["iso_ray_dir"][:2], float)
            a = np.array([eu @ (np.array([x0, y0]) - s), eu[0] * vox, eu[1] * vox])
            d = np.array([ew @ (np.array([x0, y0]) - s), ew[0] * vox, ew[1] * vox])
            if kind == "fan_line":
                a = sdd / du * a + c0 * d
            a, d = a.astype(f32), d.astype(f32)
            A, D = (_fma(c[2], j, _fma(c[1], i, c[0])) for c in (a, d))
            if kind == "fan_line":
                u = A.astype(np.float64) / D
                wt = sdd * np.hypot(*s) / D.astype(np.float64) ** 2
            else:
                g32 = np.arctan2(A.astype(np.float64), D.astype(np.float64)).astype(f32)
                u = _fma(g32, f32(1 / du), f32(c0)).astype(np.float64)
                wt = np.hypot(*s) / (A.astype(np.float64) ** 2 + D.astype(np.float64) ** 2)
        u = np.clip(u, -1.0, nc) + 2
        k = np.minimum(np.floor(u).astype(int), nc + 2)
        out += wt * (pad[v][k] + (u - k) * (pad[v][k + 1] - pad[v][k]))
    return out * 2 * math.pi / nv


@pytest.mark.parametrize("kind,nv,nc,nx,ny,vox,mid,turn,storage,filt", CASES)
def test_rows_against_definition(kind, nv, nc, nx, ny, vox, mid, turn, storage, filt):
    import torch
    cg, vg = _scan(kind, nv, nc, nx, ny, vox, mid, turn)
    proj = np.random.default_rng(7).uniform(0.0, 1.0, (nv, 1, nc)).astype(np.float32)
    opts = g.FdkOptions(storage=g.STORAGE_F16 if storage == "f16" else g.STORAGE_F32,
                        filter={"fft": g.FILTER_FFT, "toeplitz_f16x2": g.FILTER_TOEPLITZ_F16X2,
                                "toeplitz_bf16x4": g.FILTER_TOEPLITZ_BF16X4}[filt])
    p = torch.from_numpy(proj).cuda()
    got, twice = (torch.full(vg.shape, float("nan"), dtype=torch.float32, device="cuda") for _ in range(2))
    rows = torch.empty_like(p)
    with g.FdkPlan(cg, vg, opts=opts) as plan:
        plan.filter(p, rows)
        plan.execute(p, got)
        plan.prepare(p)
        half = nv // 2
        plan.backproject(twice, view_begin=0, view_count=half)
        plan.backproject(twice, view_begin=half, view_count=nv - half, accumulate=True)
        plan.check()
    ref = _reference(kind, cg, rows.cpu().numpy()[:, 0].astype(np.float64), nx, ny, vox, mid, nv).reshape(vg.shape)
    scale = np.sqrt(np.mean(ref ** 2))
    tol = 2e-5 if storage == "f32" else 1e-3
    assert np.sqrt(np.mean((got.cpu().numpy() - ref) ** 2)) <= tol * scale
    # the two halves are the same terms summed in another order
    assert np.sqrt(np.mean((twice - got).cpu().numpy() ** 2)) <= 1e-6 * scale
