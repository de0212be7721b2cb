"""Forward projection of grids with an infinite voxel: a ray whose samples weight it is infinite of its sign
(a sum of weighted taps, not a difference), the others are what they are without it. Through copies of the
grid, the grid itself, a planar image and steps long enough for the range-checked path; the voxel in the
interior and at a face. Rays that graze the voxel's support (total weight below 1e-3) may go either way."""
import math

import numpy as np
import pytest

import gct_b200 as g
from test_forward_steps_gpu import _rays, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [math.inf, -math.inf])
@pytest.mark.parametrize("kind,n,vox,step", [("cone_flat", (33, 31, 37), 1.0, 0.5), ("cone_flat", (24, 22, 20), 1.4, 0.5),
                                             ("cone_flat", (40, 36, 32), 1.0, 2.5), ("fan_line", (151, 149, 1), 0.3, 0.5)])
@pytest.mark.parametrize("face", [False, True])
def test_infinite_voxel(kind, n, vox, step, face, value):
    import torch
    planar = kind == "fan_line"
    nv, nc, nr, du, dv, sid, sdd = 7, 36, 1 if planar else 12, 1.9, 2.3, 300.0, 500.0
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
    if planar:
        cg = g.AxialCTGeom.from_params((g.DetFanLine(nc, du),), g.FanBeamProjGeomParams((nc - 1) / 2, rot, sdd, sid))
    else:
        cg = g.AxialCTGeom.from_params((g.DetFanLine(nc, du), g.DetFanLine(nr, dv)),
                                       g.ConeBeamProjGeomParams((nc - 1) / 2, rot, sdd, sid, (nr - 1) / 2))
    s = [g.EqDistSampler(k, vox) for k in n]
    vg = g.ReconImgGeom(s[0], s[1]) if planar else g.ReconImgGeom(*s)
    vol = np.random.RandomState(5).rand(n[2], n[1], n[0]).astype(np.float32)
    at = (n[2] // 2, n[1] // 2 + 1, 0 if face else n[0] // 2)
    lo = [0.0 if planar and a == 2 else -(n[a] - 1) * vox / 2 for a in range(3)]
    o, d = _rays(kind, nv, nc, nr, du, dv, sid, sdd)
    one = np.zeros(vol.shape)
    one[at] = 1.0
    weight, _ = _reference(o, d, one, lo, (vox,) * 3, step, planar)
    vol[at] = 0.0
    rest, length = _reference(o, d, vol.astype(np.float64), lo, (vox,) * 3, step, planar)
    vol[at] = value
    out = torch.empty((nv, nr, nc), dtype=torch.float32, device="cuda")
    g.forward_project(cg, vg, torch.from_numpy(vol.reshape(vg.shape)).cuda(), out, step_vox=step)
    got = out.cpu().numpy().astype(np.float64)
    hit, miss = weight > 1e-3, weight == 0.0
    assert hit.sum() >= 2 and miss.sum() > hit.sum()
    assert (got[hit] == value).all()
    # a sample beside the support may land on its edge, where the voxel's weight is exactly zero: not a number
    ok = np.abs(got - rest) <= 5e-5 * (length + vox)
    assert (ok | ~np.isfinite(got))[miss].mean() == 1.0 and ok[miss].mean() > 0.99
