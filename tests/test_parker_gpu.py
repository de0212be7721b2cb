"""The Parker table that a plan computes on the device, through the weighted and filtered rows of white
projections, against the FP64 oracle: both turns, scans of just over half a turn, of three quarters and of
a whole one, flat and arc rows, off-centre columns (the window bounds come from the first view's fan
angles), and kinds whose weights are constant.

Tolerance: a transform of up to 1024 points in FP32 leaves about 10 x 6e-8 of the row's norm and the cosine
weights 2e-7; a weight in the wrong window would be off by up to 1. Bound 3e-6 relative RMS per view."""
import math

import numpy as np
import pytest

import gct_b200 as g
from cases import make_case
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("turn", [g.RotDir.CW, g.RotDir.CCW])
@pytest.mark.parametrize("kind,nv,nc,rng", [
    ("fan_line", 61, 97, 1.04 * math.pi), ("fan_line", 90, 64, 2 * math.pi), ("fan_arc", 77, 130, 1.5 * math.pi),
    ("cone_flat", 50, 45, 1.1 * math.pi), ("cone_cyl", 33, 52, 2 * math.pi), ("parallel_1d", 31, 40, math.pi),
    ("cone_parallel", 40, 36, 2 * math.pi)])
def test_weighted_rows(kind, nv, nc, rng, turn):
    import torch
    case = make_case(kind, nv=nv, nc=nc, nr=5, n=16, nz=4, rot_dir=turn, range_rad=rng)
    nr = case.cg.num_rows
    proj = np.random.default_rng(3).uniform(0.5, 1.5, (nv, nr, nc)).astype(np.float32)
    out = torch.empty((nv, nr, nc), device="cuda")
    with g.FdkPlan(case.cg, case.vg) as p:
        p.filter(torch.from_numpy(proj).cuda(), out)
        p.check()
    got = out.cpu().numpy().reshape(nv, -1)
    ref = orc.filter_stack(case.og, proj).reshape(nv, -1)
    norm = np.sqrt(np.mean(ref ** 2))
    assert np.all(np.sqrt(np.mean((got - ref) ** 2, axis=1)) <= 3e-6 * norm)
