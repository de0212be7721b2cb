"""Images of few cells: several groups of threads share a block's views (one group, two, four or eight,
with view counts that leave them unequal or empty shares). Against the definition of test_rows_gpu.py with
its tolerances (the same sums, grouped otherwise), and against the same views added in calls of at most 15,
which run without clusters and groups: another order of the same FP32 terms, sqrt(n) x 6e-8, below 3e-6 for
1100 views."""
import pytest

import gct_b200 as g
from test_rows_gpu import _reference, _scan

pytestmark = pytest.mark.gpu

# kind, views, columns, nx, ny, pixel, centre, turn, storage
CASES = [
    ("parallel_1d", 63, 40, 32, 32, 1.0, (0.0, 0.0), 1, "f32"),     # seven or eight views a chunk: one group
    ("parallel_1d", 64, 40, 32, 32, 1.0, (0.0, 0.0), 1, "f32"),     # two groups of four
    ("parallel_1d", 515, 70, 33, 64, 1.0, (1.0, -2.0), -1, "f16"),
    ("fan_line", 131, 61, 40, 31, 1.0, (0.0, 3.0), 1, "f32"),       # four groups, uneven
    ("fan_line", 1025, 61, 30, 34, 1.0, (0.0, 0.0), 1, "f32"),      # eight groups, the last ones short
    ("fan_line", 258, 61, 64, 64, 1.0, (0.0, 0.0), 1, "f16"),       # no quarter turns
    ("fan_line", 260, 61, 64, 64, 1.0, (0.0, 0.0), 1, "f16"),       # quarter turns: 65 base views
    ("fan_line", 1096, 90, 130, 130, 1.0, (0.0, 0.0), -1, "f16"),   # four groups, 274 base views
    ("fan_line", 300, 50, 96, 96, 4.0, (0.0, 0.0), 1, "f16"),       # cells off and partly off the row
    ("fan_arc", 133, 61, 33, 31, 1.0, (0.0, 0.0), 1, "f32"),
    ("fan_arc", 777, 61, 64, 40, 1.0, (5.0, 3.0), -1, "f32"),
    ("fan_arc", 360, 41, 64, 64, 1.6, (0.0, 0.0), 1, "f32"),        # partly off the row, near the axis
    ("fan_arc", 240, 41, 64, 64, 9.0, (0.0, 0.0), 1, "f32"),        # around and behind the source
]


@pytest.mark.parametrize("kind,nv,nc,nx,ny,vox,mid,turn,storage", CASES)
def test_groups_share_a_chunks_views(kind, nv, nc, nx, ny, vox, mid, turn, storage):
    import numpy as np
    import torch
    cg, vg = _scan(kind, nv, nc, nx, ny, vox, mid, turn)
    p = torch.from_numpy(np.random.default_rng(5).uniform(0.0, 1.0, (nv, 1, nc)).astype(np.float32)).cuda()
    got, single, half = (torch.full(vg.shape, float("nan"), dtype=torch.float32, device="cuda") for _ in range(3))
    rows = torch.empty_like(p)
    with g.FdkPlan(cg, vg, opts=g.FdkOptions(storage=g.STORAGE_F16 if storage == "f16" else g.STORAGE_F32)) as plan:
        plan.filter(p, rows)
        plan.execute(p, got)
        plan.prepare(p)
        for v in range(0, nv, 15):
            plan.backproject(single, view_begin=v, view_count=min(15, nv - v), accumulate=v > 0)
        plan.backproject(half, view_begin=3, view_count=nv - 3)
        plan.backproject(half, view_begin=0, view_count=3, accumulate=True)
        plan.check()
    ref = _reference(kind, cg, rows.cpu().numpy()[:, 0].astype(np.float64), nx, ny, vox, mid, nv).reshape(vg.shape)
    scale = np.sqrt(np.mean(ref ** 2))
    got, single, half = (x.cpu().numpy() for x in (got, single, half))
    assert np.sqrt(np.mean((got - ref) ** 2)) <= (2e-5 if storage == "f32" else 1e-3) * scale
    # with quarter turns a whole scan evaluates the turned columns at their base views' forms, as the
    # single calls do for each of its views
    assert np.sqrt(np.mean((got - single) ** 2)) <= 3e-6 * scale
    assert np.sqrt(np.mean((got - half) ** 2)) <= 3e-6 * scale


@pytest.mark.parametrize("kind,storage,most", [("fan_arc", "f32", 0.65), ("fan_line", "f32", 0.85), ("fan_line", "f16", 0.85)])
def test_small_images_take_less_time(kind, storage, most):
    # 64 x 64 pixels against 256 x 256 with the same 1440 views: a sixteenth of the updates
    import torch
    times = []
    for n in (64, 256):
        cg, vg = _scan(kind, 1440, 97, n, n, 64.0 / n, (0.0, 0.0), 1)
        proj = torch.rand(1440, 1, 97, device="cuda")
        vol = torch.empty(vg.shape, device="cuda")
        with g.FdkPlan(cg, vg, opts=g.FdkOptions(storage=g.STORAGE_F16 if storage == "f16" else g.STORAGE_F32,
                                                 symmetry=g.SYMMETRY_OFF)) as plan:
            best = 1e9
            for _ in range(20):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                plan.execute(proj, vol)
                e[0].record()
                for _ in range(5):
                    plan.execute(proj, vol)
                e[1].record()
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]))
        times.append(best)
    assert times[0] <= most * times[1], times
