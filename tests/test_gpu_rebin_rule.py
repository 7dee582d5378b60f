"""The rebinning on both sides of the launch size from which a thread walks four views: bit-identical to the reference's
arithmetic, with equal angle steps and with others."""
import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import api, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ZL,quads", [(8, 1), (12, 3)])
@pytest.mark.parametrize("more,ratio", [(0, 1.0), (1, 1.0), (2, 1.7), (3, 0.6)])
def test_walk_of_large_launches_is_bit_identical(cuda, ZL, quads, more, ratio):
    a = dict(G.Scan(ZL=ZL, N_2pi=36, rotations=2.0).rebin_args())  # every view is clamped somewhere
    ctas = -(-a["YL"] * quads // 256)  # per view; up to six per SM take one view each
    views = 6 * torch.cuda.get_device_properties(cuda).multi_processor_count // ctas + more
    a["ViewN"], a["DeltaTheta"] = views, a["DeltaFai"] * ratio
    rng = np.random.default_rng(more * 10 + ZL)
    fan = rng.standard_normal((views, a["YL"], ZL)).astype(np.float32)
    got = api.ParallelRebinningCBCurve(fan, a["YL"], ZL, views, a["YLC"] + 1, a["dYA"], a["DeltaTheta"], a["PLC"] + 1,
                                       a["DeltaT"], a["DeltaFai"], a["SO"], 1)
    ref = oracle.rebin_f32(fan, **a)
    assert np.array_equal(np.asarray(got).view(np.uint32), np.asarray(ref, dtype=np.float32).view(np.uint32))
