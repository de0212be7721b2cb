"""Planar items in the work queue of batches and of the server: a tile is one cell of 32 x 32 pixels whose views
two groups of threads share; stacks are view-major, and quarter-turn plans (FP16 lines at default
options, FP32 lines and arcs with the symmetry on) take every view's coordinates from its base view, so
that view chunks may begin and end in any quarter.

Against execute() of the same plan, with the bounds of the batch and server tests: a batch <= 1e-5
(chunks added atomically), a request <= 1e-6 of FP32 rounding where both evaluate the same forms, 1e-5
where execute() shares evaluations between partner views; a request alone and in a mix identical. The host
paths filter other pairs of views together than execute() does, so that entries may round to the neighbouring
half: the bound of FP16 storage, 1e-3."""
import numpy as np
import pytest

import gct_b200 as g
from cases import make_case
from conftest import rel_rms

pytestmark = pytest.mark.gpu

F32, F16 = g.STORAGE_F32, g.STORAGE_F16


def _item(kind, storage, sym, **kw):
    import torch
    case = make_case(kind, **kw)
    nv, nc = case.cg.num_views, case.cg.num_cols
    proj = np.random.default_rng(nv + nc).uniform(0.5, 1.5, (nv, 1, nc)).astype(np.float32)
    plan = g.FdkPlan(case.cg, case.vg, opts=g.FdkOptions(storage=storage, symmetry=sym))
    ref = torch.full(case.vg.shape, float("nan"), dtype=torch.float32, device="cuda")
    plan.execute(torch.from_numpy(proj).cuda(), ref)
    plan.check()
    return case, plan, proj, ref.cpu().numpy()


ITEMS = [  # kind, storage, symmetry, sizes
    ("fan_line", F16, g.SYMMETRY_AUTO, dict(nv=120, n=48)),
    ("fan_line", F16, g.SYMMETRY_AUTO, dict(nv=360, n=70, nc=121)),
    ("fan_line", F32, g.SYMMETRY_ON, dict(nv=100, n=66)),
    ("fan_arc", F32, g.SYMMETRY_ON, dict(nv=92, n=96)),
    ("fan_arc", F32, g.SYMMETRY_AUTO, dict(nv=67, n=33)),
    ("parallel_1d", F16, g.SYMMETRY_AUTO, dict(nv=61, n=31)),
    ("parallel_1d", F32, g.SYMMETRY_AUTO, dict(nv=1, n=64)),
]


@pytest.mark.parametrize("kind,storage,sym,kw", [i for i in ITEMS if i[3]["nv"] > 1])
def test_batch_of_one(kind, storage, sym, kw):
    import torch
    case, plan, proj, ref = _item(kind, storage, sym, **kw)
    turned = plan.quarter_turn != 0
    assert turned == (kw["nv"] % 4 == 0 and kw["n"] % 2 == 0 and kind != "parallel_1d" and sym != g.SYMMETRY_OFF
                      and (storage == F16 or sym == g.SYMMETRY_ON))
    vol = torch.full(case.vg.shape, float("nan"), dtype=torch.float32, device="cuda")
    with g.FdkBatch([(plan, torch.from_numpy(proj).cuda(), vol)]) as batch:
        if kw["nv"] >= 100:
            assert batch.item_config(0)["view_split"] > 1  # chunks added atomically, in any quarter
        batch.launch()
        torch.cuda.synchronize()
    assert rel_rms(vol.cpu().numpy(), ref) <= 1e-5
    plan.close()


def test_batch_of_all_and_its_tiles():
    import torch
    items = [_item(k, st, sym, **kw) for k, st, sym, kw in ITEMS if kw["nv"] > 1]
    vols = [torch.full(c.vg.shape, float("nan"), dtype=torch.float32, device="cuda") for c, *_ in items]
    with g.FdkBatch([(p, torch.from_numpy(pr).cuda(), v) for (_, p, pr, _), v in zip(items, vols)]) as batch:
        for _ in range(2):
            batch.launch()
        torch.cuda.synchronize()
    for (c, p, _, ref), v in zip(items, vols):
        assert rel_rms(v.cpu().numpy(), ref) <= 1e-5, c.name
        p.close()
    # views too few to split: one entry per cell
    case, plan, proj, _ = _item("fan_line", F32, g.SYMMETRY_OFF, nv=15, n=130)
    vol = torch.empty(case.vg.shape, dtype=torch.float32, device="cuda")
    with g.FdkBatch([(plan, torch.from_numpy(proj).cuda(), vol)]) as batch:
        assert batch.work()[0] == 25
    plan.close()


def test_requests_alone_and_in_mix():
    items = [_item(k, st, sym, **kw) for k, st, sym, kw in ITEMS if kw["nv"] > 1]
    with g.FdkServer(256 << 20, round_updates=1e5) as srv:  # rounds of 16 to 23 views
        alone = []
        for c, p, pr, _ in items:
            out = np.full(c.vg.shape, np.nan, np.float32)
            t = srv.submit(p, pr, out)
            srv.wait(t)
            assert (srv.info(t)["rounds"] > 1) == (c.cg.num_views > max(16, 1e5 // int(np.prod(c.vg.shape))))
            alone.append(out)
        mixed = [np.full(c.vg.shape, np.nan, np.float32) for c, *_ in items]
        for t in [srv.submit(p, pr, o) for (_, p, pr, _), o in zip(items, mixed)]:
            srv.wait(t)
    for (c, p, _, ref), a, m in zip(items, alone, mixed):
        assert np.array_equal(a, m), c.name
        assert rel_rms(a, ref) <= (1e-5 if p.quarter_turn else 1e-6), c.name
        p.close()


@pytest.mark.parametrize("kw", [dict(nv=240, n=64), dict(nv=76, n=50, nc=77), dict(nv=720, n=40)])
def test_host_paths_of_quarter_turn_lines(kw):
    # execute_host filters and backprojects chunks of base views with their partners into interleaved
    # stacks; execute_host_budget takes view-major chunks, here of one view, of 13 and of all
    case, plan, proj, ref = _item("fan_line", F16, g.SYMMETRY_AUTO, **kw)
    assert plan.quarter_turn != 0
    out = np.full(case.vg.shape, np.nan, np.float32)
    plan.execute_host(proj, out)
    assert rel_rms(out, ref) <= 1e-3
    per_view = 8 * case.cg.num_cols + 5 * (case.cg.num_cols + 4) * 8 + 12
    for views in (1, 13, kw["nv"]):
        out = np.full(case.vg.shape, np.nan, np.float32)
        plan.execute_host_budget(proj, out, 512 + views * per_view)
        assert rel_rms(out, ref) <= 1e-3, views
    plan.close()
