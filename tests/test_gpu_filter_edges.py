"""The register-resident filter at the edges of its pruned instances and of the range of lengths it takes, in both
input layouts: channels around 128, 512, 640, 896 and 1024, odd row counts (a last pair of one row), rows that are
no multiple of eight (not staged) and odd lengths (rows that start off 16-byte boundaries)."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("YL", [128, 129, 256, 512, 513, 640, 641, 896, 897, 1024])
@pytest.mark.parametrize("ZL,views", [(8, 2), (3, 1), (7, 90)])
def test_filter_edges_vs_fp64_oracle(cuda, YL, ZL, views):
    lib = _lib.load()
    fa = G.replace(G.Scan(ZL=ZL), YL=YL).filter_args()
    rng = np.random.default_rng(YL * 8 + ZL)
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
    assert np.array_equal(outs[0], outs[1])  # the same rows, paired the same way
    ref = oracle.filter_f64(rows.astype(np.float64), YL, ZL, views, fa["PLC"], fa["ZLC"], fa["dYL"], fa["dZL"],
                            fa["SO"])
    # FP32 transforms of 2048 points: eleven radix-2 steps each way of at most a few 2^-24 relative in the mean
    # square, white rows (no cancellation): 22 x 4 x 6e-8 = 5e-6
    err = np.linalg.norm(outs[0] - ref, axis=-1) / np.linalg.norm(ref, axis=-1)
    assert err.max() < 5e-6, err.max()
