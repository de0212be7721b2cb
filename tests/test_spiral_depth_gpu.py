"""The number of slices a thread takes of a spiral scan is chosen from the slices' view windows and the size
of the image: at default options a backprojection takes no longer than with one slice per thread (a tenth
for the timing), from dense slices of large images to slices whose windows hardly meet and small volumes,
and with dense slices no longer than with the best fixed number. Results agree between the depths within FP32 rounding (1e-5, FP16 blends 1e-3)."""
import math

import pytest

import gct_b200 as g
from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _plan(kind, npr, shift, n, nz, storage, zpt):
    """Slices one mm apart, between which the source moves on by `shift` views."""
    turns = math.ceil(nz * shift / npr) + 3
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / npr, npr * turns, npr / shift / (2 * math.pi))
    nc, nr = int(1.5 * n), 32
    row = g.DetFanArc(nc, 0.9 / nc) if kind == "cone_cyl" else g.DetFanLine(nc, 700 / nc)
    det = (row, g.DetFanLine(nr, npr / shift * 1100 / 600 * 1.3 / nr))
    params = g.ConeBeamProjGeomParams((nc - 1) / 2, rot, 1100.0, 600.0, (nr - 1) / 2)
    cg = g.SpiralCTGeom(det, g.ProjGeomFactory(*(type(d) for d in det)).create_all(params))
    zmid = -(npr / shift / (2 * math.pi)) * (2 * math.pi / npr) * (npr * turns - 1) / 2
    x = g.EqDistSampler(n, 300 / n)
    vg = g.ReconImgGeom(x, x, g.EqDistSampler(nz, 1.0), (0.0, 0.0, zmid))
    return g.FdkPlan(cg, vg, opts=g.FdkOptions(storage=storage, scan=g.SCAN_SPIRAL, z_per_thread=zpt))


@pytest.mark.parametrize("kind,npr,shift,n,nz,storage", [
    ("cone_flat", 360, 300, 256, 4, g.STORAGE_F32),   # four slices, windows hardly meet
    ("cone_cyl", 360, 12, 32, 64, g.STORAGE_F32),     # few columns
    ("cone_flat", 360, 12, 64, 3, g.STORAGE_F16),     # fewer slices than any depth
    ("cone_cyl", 360, 40, 128, 17, g.STORAGE_F16),
    ("cone_cyl", 360, 4, 256, 64, g.STORAGE_F32),     # dense
])
def test_default_depth_is_near_the_best(kind, npr, shift, n, nz, storage):
    import torch
    times, vols = {}, {}
    for zpt in (0, 1, 4, 8):
        with _plan(kind, npr, shift, n, nz, storage, zpt) as p:
            proj = torch.linspace(0.5, 1.5, p.cg.num_views * p.cg.num_rows * p.cg.num_cols, device="cuda")
            proj = torch.sin(proj * 4000).reshape(p.cg.num_views, p.cg.num_rows, p.cg.num_cols) + 2
            vol = torch.empty(p.vol_geom.shape, device="cuda")
            p.prepare(proj)
            p.backproject(vol)
            best = 1e9
            for _ in range(12):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record()
                p.backproject(vol)
                p.backproject(vol)
                e[1].record()
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]))
            times[zpt], vols[zpt] = best, vol.cpu().numpy()
    for zpt in (1, 4, 8):
        assert rel_rms(vols[zpt], vols[0]) <= (1e-5 if storage == g.STORAGE_F32 else 1e-3)
    assert times[0] <= 1.1 * times[1], times
    if shift <= 4:
        assert times[0] <= 1.1 * min(times.values()), times
