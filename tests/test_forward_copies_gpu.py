"""Forward projections read the grid itself, an exchanged copy, or both orientations as pairs of planes, by what
the rays of the call are worth: a call of few rays through a large grid does not pay for copies of it (the kernels
a call launches show whether they are made). And each way gives the sum of the samples
(reference and tolerance of test_forward_steps_gpu.py) for grids above the size that is always copied."""
import math

import numpy as np
import pytest

import gct_b200 as g
from test_forward_steps_gpu import _rays, _reference

pytestmark = pytest.mark.gpu


def _scan(kind, nv, nc, nr, n, first=0.0):
    rot = g.RotationParams(g.RotDir.CW, first, 2 * math.pi / nv, nv)
    c0, r0 = (nc - 1) / 2, (nr - 1) / 2
    if kind == "parallel_2d":
        det, params = (g.DetParallel(nc, 300 / nc), g.DetParallel(nr, 300 / nr)), g.Parallel2DProjGeomParams(c0, rot, r0)
    else:
        det = (g.DetFanLine(nc, 480 / nc), g.DetFanLine(nr, 480 / nr))
        params = g.ConeBeamProjGeomParams(c0, rot, 1120.0, 700.0, r0)
    x = g.EqDistSampler(n, 300 / n)
    return g.AxialCTGeom.from_params(det, params), g.ReconImgGeom(x, x, x, (0.0, 0.0, 0.0))


def _kernels(cg, vg, vol, out):
    """Names of the kernels that one call launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    g.forward_project(cg, vg, vol, out)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        g.forward_project(cg, vg, vol, out)
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if "_kernel" in e.name]
    if not names:
        pytest.skip("no kernel records from the profiler")
    assert sum("forward_kernel" in n for n in names) == 1
    return names


@pytest.mark.parametrize("kind", ["cone_flat", "parallel_2d"])
@pytest.mark.parametrize("nv,nc,n,copied", [
    (2, 32, 384, False),     # few rays through a large grid
    (8, 64, 96, False),
    (180, 160, 96, True),    # many rays
    (4, 64, 48, True),       # copies of up to 2 MB cost nothing
    (4, 64, 24, False),      # a grid that the caches hold
])
def test_copies_are_made_for_enough_rays(kind, nv, nc, n, copied):
    import torch
    cg, vg = _scan(kind, nv, nc, nc, n)
    names = _kernels(cg, vg, torch.rand(vg.shape, device="cuda"), torch.empty((nv, nc, nc), device="cuda"))
    assert any("arrange_grid_kernel" in k for k in names) == copied


@pytest.mark.parametrize("kind,nv,nc,nr,step,n", [
    ("parallel_2d", 2, 24, 24, 0.5, (72, 70, 66)),     # the grid itself
    ("parallel_2d", 2, 700, 700, 0.25, (72, 70, 66)),  # rays along x: the exchanged grid
    ("cone_flat", 4, 700, 500, 0.25, (72, 70, 66)),    # half of the rays along x
    ("cone_flat", 90, 300, 200, 0.5, (72, 70, 66)),    # all around: pairs
])
def test_every_choice_sums_the_samples(kind, nv, nc, nr, step, n):
    import torch
    du = 90.0 / nc * (1.0 if kind == "parallel_2d" else 1.6)
    dv = 80.0 / nr * (1.0 if kind == "parallel_2d" else 1.6)
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
    c0, r0 = (nc - 1) / 2, (nr - 1) / 2
    if kind == "parallel_2d":
        det, params = (g.DetParallel(nc, du), g.DetParallel(nr, dv)), g.Parallel2DProjGeomParams(c0, rot, r0)
    else:
        det, params = (g.DetFanLine(nc, du), g.DetFanLine(nr, dv)), g.ConeBeamProjGeomParams(c0, rot, 500.0, 300.0, r0)
    cg = g.AxialCTGeom.from_params(det, params)
    x, y, z = (g.EqDistSampler(k, 1.0) for k in n)
    vg = g.ReconImgGeom(x, y, z, (0.0, 0.0, 0.0))
    vol = np.random.RandomState(7).rand(n[2], n[1], n[0]).astype(np.float32)
    out = torch.full((nv, nr, nc), float("nan"), dtype=torch.float32, device="cuda")
    g.forward_project(cg, vg, torch.from_numpy(vol).cuda(), out, step_vox=step)
    got = out.cpu().numpy().astype(np.float64)
    assert np.isfinite(got).all()
    # the reference takes its time per ray: a few hundred of them
    o, d = _rays(kind, nv, nc, nr, du, dv, 300.0, 500.0)
    pick = np.random.RandomState(3).choice(nv * nr * nc, 400, replace=False)
    sub = lambda a: (a + np.zeros((nv, nr, nc))).reshape(-1)[pick]
    lo = [-(k - 1) / 2 for k in n]
    ref, length = _reference([sub(a) for a in o], [sub(a) for a in d], vol.astype(np.float64), lo, (1.0, 1.0, 1.0),
                             step, False)
    err = np.abs(got.reshape(-1)[pick] - ref)
    assert (length > 0).mean() > 0.2
    assert (err <= 5e-5 * (length + 1.0)).all(), float((err / (length + 1.0)).max())
