"""The rebinning kernel's walk over consecutive views, whose fan rows stay in registers: view counts around its
chunk, both row quads, angle steps that differ (the next view's lower fan view is then not always the last
one's upper), rows that are no multiple of four. Bit-identical to the reference's arithmetic."""
import numpy as np
import pytest

import oracle
from analyticalreconbigpatient_b200 import api, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ZL", [8, 12, 15])
@pytest.mark.parametrize("views,ratio", [(1, 1.0), (3, 1.0), (4, 1.7), (5, 1.0), (9, 0.6), (41, 1.0 + 2e-4)])
def test_view_chunks_are_bit_identical(cuda, ZL, views, ratio):
    a = dict(G.Scan(ZL=ZL, N_2pi=36, rotations=2.0).rebin_args())  # 10 degrees a view: every view is clamped somewhere
    a["ViewN"], a["DeltaTheta"] = views, a["DeltaFai"] * ratio
    rng = np.random.default_rng(views * 10 + ZL)
    fan = rng.standard_normal((views, a["YL"], ZL)).astype(np.float32)
    got = api.ParallelRebinningCBCurve(fan, a["YL"], ZL, views, a["YLC"] + 1, a["dYA"], a["DeltaTheta"], a["PLC"] + 1,
                                       a["DeltaT"], a["DeltaFai"], a["SO"], 1)
    ref = oracle.rebin_f32(fan, **a)
    assert np.array_equal(np.asarray(got).view(np.uint32), np.asarray(ref, dtype=np.float32).view(np.uint32))
