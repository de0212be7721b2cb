"""How exact the forward projector's sample positions are: through voxels that alternate between +1 and -1 along x
a sample's error is twice its position's, and the sum stays small. Whole-voxel steps on 32 voxels, where steps
in FP32 from a far point are at their worst.

Bound: FP64 positions rounded to FP32 (the best a position in FP32 voxel units can be) give these ray sums an rms
error of 4.7e-6 on 32 voxels, 3.8e-6 on 26 and 1.15e-6 on 12, by the same sums in numpy over 3000 such rays; on
12, where rays take the range-checked path, the products of its weights add 0.3e-6."""
import math

import numpy as np
import pytest

import gct_b200 as g
from test_forward_steps_gpu import _rays, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bound", [(32, 4.7e-6), (26, 3.8e-6), (12, 1.3e-6)])
def test_positions_are_as_good_as_rounded_exact_ones(n, bound):
    import torch
    nv, nc, nr = 360, 16, 2
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
    du = 0.4 * n / nc
    cg = g.AxialCTGeom.from_params((g.DetParallel(nc, du), g.DetParallel(nr, 1.0)),
                                   g.Parallel2DProjGeomParams((nc - 1) / 2, rot, (nr - 1) / 2))
    x, z = g.EqDistSampler(n, 1.0), g.EqDistSampler(8, 1.0)
    vg = g.ReconImgGeom(x, x, z, (0.0, 0.0, 0.0))
    vol = np.empty((8, n, n), np.float32)
    vol[:] = (-1.0) ** np.arange(n)
    out = torch.empty((nv, nr, nc), dtype=torch.float32, device="cuda")
    g.forward_project(cg, vg, torch.from_numpy(vol).cuda(), out, step_vox=1.0)
    got = out.cpu().numpy().astype(np.float64)
    o, d = _rays("parallel_2d", nv, nc, nr, du, 1.0, 0.0, 0.0)
    near = np.abs(d[0] + np.zeros((nv, nr, nc))) > 0.955  # within 17 degrees of x: through both x faces
    sub = lambda a: (a + np.zeros((nv, nr, nc)))[near]
    ref, _ = _reference([sub(a) for a in o], [sub(a) for a in d], vol.astype(np.float64),
                        [-(n - 1) / 2, -(n - 1) / 2, -3.5], (1.0, 1.0, 1.0), 1.0, False)
    rms = np.sqrt(np.mean((got[near] - ref) ** 2))
    assert near.sum() > 1000 and rms <= bound, rms
