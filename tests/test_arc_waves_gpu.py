"""FP32 arcs keep their blocks per SM: a volume whose blocks fit one wave at 16 blocks of 64 threads per SM does not
take a second one. 184 x 184 x 64 voxels (2208 blocks) have 1.32 times the updates of 160 x 160 x 64 (1600), which
fit at any rate; a second wave would make it 1.8 times the time."""
import math

import pytest

import gct_b200 as g

pytestmark = pytest.mark.gpu


def test_blocks_of_one_wave_stay_one():
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sized for 148 SMs")
    times = []
    for n in (160, 184):
        nv, nc, nr = 180, int(1.5 * n), 83
        rot = g.RotationParams(g.RotDir.CW, 0.0, 2 * math.pi / nv, nv)
        det = (g.DetFanArc(nc, 0.5 / nc), g.DetFanLine(nr, 1.2 * 64 * 300 / n * 1.6 / nr))
        cg = g.AxialCTGeom.from_params(det, g.ConeBeamProjGeomParams((nc - 1) / 2, rot, 1120.0, 700.0, (nr - 1) / 2))
        x = g.EqDistSampler(n, 300 / n)
        vg = g.ReconImgGeom(x, x, g.EqDistSampler(64, 300 / n), (0.0, 0.0, 0.0))
        proj, vol = torch.rand(nv, nr, nc, device="cuda"), torch.empty(vg.shape, device="cuda")
        with g.FdkPlan(cg, vg) as plan:
            plan.prepare(proj)
            plan.backproject(vol)
            best = 1e9
            for _ in range(15):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record()
                for _ in range(3):
                    plan.backproject(vol)
                e[1].record()
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]))
        times.append(best)
    assert times[1] <= 1.45 * times[0], times
