"""Quarter-turn volumes in FP16 whose blocks fit one wave in the kernel's smaller register form take no second one:
400 x 400 x 16 voxels (1400 blocks) have 1.13 times the updates of 376 x 376 x 16 (1128, one wave in either form).
With a wave of the smaller form up to half slower, 1.7 times the time is the bound for arcs; parallel 1.13 and 4 %,
hence 1.25. Two waves of the larger form would take up to twice the time."""
import math

import pytest

import gct_b200 as g
from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _scan(kind, n, nz, nv, s):
    nc, nr = int(1.2 * n * s), int(1.2 * nz * s)
    rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
    c0, r0, dv = (nc - 1) / 2, (nr - 1) / 2, 1.2 * 300 * nz / n * 1.6 / nr
    if kind == "cone_cyl":
        det = (g.DetFanArc(nc, 0.5 / nc), g.DetFanLine(nr, dv))
    else:
        det = (g.DetParallel(nc, 360 / nc), g.DetFanLine(nr, dv))
    cg = g.AxialCTGeom.from_params(det, g.ConeBeamProjGeomParams(c0, rot, 1120.0, 700.0, r0))
    x = g.EqDistSampler(n, 300 / n)
    return cg, g.ReconImgGeom(x, x, g.EqDistSampler(nz, 300 / n), (0.0, 0.0, 0.0))


@pytest.mark.parametrize("kind,most", [("cone_parallel", 1.25), ("cone_cyl", 1.7)])
def test_blocks_of_one_wave_stay_one(kind, most):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sized for 148 SMs")
    times = []
    for n in (376, 400):
        cg, vg = _scan(kind, n, 16, 360, 2.5)
        proj, vol = torch.rand(360, cg.num_rows, cg.num_cols, device="cuda"), torch.empty(vg.shape, device="cuda")
        with g.FdkPlan(cg, vg, opts=g.FdkOptions(storage=g.STORAGE_F16)) as plan:
            assert plan.quarter_turn != 0
            plan.prepare(proj)
            plan.backproject(vol)
            best = 1e9
            for _ in range(12):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record()
                plan.backproject(vol)
                plan.backproject(vol)
                e[1].record()
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]))
        times.append(best)
    assert times[1] <= most * times[0], times


@pytest.mark.parametrize("kind", ["cone_parallel", "cone_cyl"])
def test_both_forms_agree(kind):
    # 400 x 400 x 16: the smaller form; as two halves of the views: the view-major kernel (its tolerance for FP16)
    import torch
    cg, vg = _scan(kind, 400, 16, 64, 1.3)
    proj = torch.rand(64, cg.num_rows, cg.num_cols, device="cuda") + 1
    whole, parts = (torch.full(vg.shape, float("nan"), device="cuda") for _ in range(2))
    with g.FdkPlan(cg, vg, opts=g.FdkOptions(storage=g.STORAGE_F16)) as plan:
        plan.prepare(proj)
        plan.backproject(whole)
        plan.backproject(parts, view_begin=0, view_count=32)
        plan.backproject(parts, view_begin=32, view_count=32, accumulate=True)
        plan.check()
    assert rel_rms(whole.cpu().numpy(), parts.cpu().numpy()) <= 1e-3
