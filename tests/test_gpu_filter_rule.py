"""The filter on both sides of the row count from which a plan of 129 to 256 channels takes the N = 2048 kernel
(below it, the shared-memory kernel of N = 512), in both layouts."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("YL", [129, 256])
@pytest.mark.parametrize("ZL,views", [(1, 1), (15, 273), (16, 256)])
def test_both_sides_of_the_row_rule(cuda, YL, ZL, views):
    lib = _lib.load()
    fa = G.replace(G.Scan(ZL=ZL), YL=YL).filter_args()
    rng = np.random.default_rng(YL + ZL)
    rows = rng.standard_normal((views, ZL, YL)).astype(np.float32)
    plan = ctypes.c_void_p()
    _lib.check(lib.hr_filter_plan_create(ctypes.byref(plan), YL, ZL, views, fa["PLC"], fa["ZLC"], fa["dYL"],
                                         fa["dZL"], fa["SO"]))
    d = torch.from_numpy(rows).to(cuda)
    outs = []
    for layout, src in ((_lib.HR_LAYOUT_ROWS, d), (_lib.HR_LAYOUT_REBIN, d.transpose(1, 2).contiguous())):
        out = torch.full((views, ZL, YL), float("nan"), device=cuda)
        _lib.check(lib.hr_filter_execute(plan, out.data_ptr(), src.data_ptr(), layout, 0, 0))
        outs.append(out.cpu().numpy())
    lib.hr_filter_plan_destroy(plan)
    assert np.array_equal(outs[0], outs[1])
    ref = oracle.filter_f64(rows.astype(np.float64), YL, ZL, views, fa["PLC"], fa["ZLC"], fa["dYL"], fa["dZL"],
                            fa["SO"])
    # FP32 transforms, at most 22 radix-2 steps of a few 2^-24 relative in the mean square: 22 x 4 x 6e-8 = 5e-6
    err = np.linalg.norm(outs[0] - ref, axis=-1) / np.linalg.norm(ref, axis=-1)
    assert err.max() < 5e-6, err.max()
