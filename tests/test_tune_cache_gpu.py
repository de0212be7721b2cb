"""Tuned tile shapes are kept per process. Two FP16 fan-line plans of the same sizes, one with the FFT filter
(row pairs, a fixed tile) and one with a Toeplitz filter (quads, tuned), must not take each other's entry,
whichever a process makes first: an entry carries its measured rate, and two measurements do not agree to
the last bit. Each order takes sizes of its own, so that neither finds the other's entries."""
import pytest

import gct_b200 as g
from cases import make_case

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("n,rows_first", [(72, True), (88, False)])
@pytest.mark.parametrize("sym", [g.SYMMETRY_OFF, g.SYMMETRY_AUTO])
def test_row_and_quad_plans_keep_their_own_tiles(n, rows_first, sym):
    import torch
    case = make_case("fan_line", nv=60, n=n, nc=100)
    proj = torch.rand(60, 1, 100, device="cuda")
    got = {}
    for filt in [g.FILTER_FFT, g.FILTER_TOEPLITZ_BF16X4][::1 if rows_first else -1]:
        opts = g.FdkOptions(storage=g.STORAGE_F16, filter=filt, symmetry=sym)
        with g.FdkPlan(case.cg, case.vg, opts=opts) as plan:
            vol = torch.empty(case.vg.shape, dtype=torch.float32, device="cuda")
            with g.FdkBatch([(plan, proj, vol)]) as batch:
                got[filt] = batch.item_config(0)["tuned_gups"]
    assert min(got.values()) > 0.0
    assert got[g.FILTER_FFT] != got[g.FILTER_TOEPLITZ_BF16X4]
