"""Spiral scans with several slices per thread: each slice has its own window of views, and the slices of
a thread meet windows that overlap nearly whole, barely and not at all, slices without a window beside
slices with one, a last group that is not full, columns that leave the detector on the way, and every
number of slices per thread. Against the FP64 oracle, with the bounds of the spiral tests (relative RMS
over the reconstructed slices: FP32 1e-4, FP16 1e-3; other slices exactly zero)."""
import numpy as np
import pytest

import gct_b200 as g
from cases import make_spiral_case, spiral_projections
from conftest import rel_rms
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

CASES = [  # kind, views per turn, turns, pitch, rows, side, slices, slices per thread
    ("cone_cyl", 60, 3, 1.0, 24, 33, 13, 0),
    ("cone_cyl", 48, 4, 3.0, 16, 20, 17, 4),
    ("cone_flat", 60, 5, 0.7, 24, 31, 9, 16),
    ("cone_flat", 37, 3, 4.0, 40, 24, 7, 8),
    ("cone_cyl", 30, 3, 6.0, 12, 16, 30, 1),
]


@pytest.mark.parametrize("storage", [g.STORAGE_F32, g.STORAGE_F16])
@pytest.mark.parametrize("kind,npr,turns,pitch,nr,n,nz,zpt", CASES)
def test_slices_take_their_own_views(kind, npr, turns, pitch, nr, n, nz, zpt, storage):
    import torch
    case = make_spiral_case(kind, npr=npr, turns=turns, pitch=pitch, nr=nr, n=n, nz=nz)
    proj = spiral_projections(case)
    opts = g.FdkOptions(storage=storage, scan=g.SCAN_SPIRAL, z_per_thread=zpt)
    vol = torch.full(case.vg.shape, float("nan"), dtype=torch.float32, device="cuda")
    with g.FdkPlan(case.cg, case.vg, opts=opts) as p:
        p.execute(torch.from_numpy(proj).cuda(), vol)
        p.check()
    got = vol.cpu().numpy()
    ref = orc.fdk_spiral(case.og, case.ov, proj)
    on = np.array([w is not None for w in orc.spiral_windows(case.og, case.ov)])
    assert on.any()
    assert np.all(got[~on] == 0.0)
    assert rel_rms(got[on], ref[on]) <= (1e-4 if storage == g.STORAGE_F32 else 1e-3)
