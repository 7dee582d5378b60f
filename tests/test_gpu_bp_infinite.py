"""Infinite samples in the filtered data: the voxels they reach are infinite with the sample's sign, NaN only where
samples of both signs meet, and every other voxel keeps its bits -- as from the reference's four weighted taps, which
the oracle evaluates."""
import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import StagePlans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "fp64"])
@pytest.mark.parametrize("geom", [dict(XN=21, YN=35, ZN=9, dz=0.7), dict(XN=10, YN=9, ZN=13, dz=1.9, dx=20.0)])
def test_infinite_samples(cuda, form, geom):
    double = form == "fp64"
    sc = G.tiny(delta=8, rotations=4, **geom)
    g = sc.bp_geom()
    rng = np.random.default_rng(sc.YN)
    fp = rng.standard_normal((g["PN"], g["ZL"], g["YL"])).astype(np.float32)
    w = oracle.weight_table(sc.N_2pi, sc.HSCoef, sc.delta)
    plans = StagePlans(sc, _lib.HR_FORM_FP64 if double else _lib.HR_FORM_PLAIN)
    d_fp = torch.tensor(fp, device=cuda, dtype=torch.float64 if double else torch.float32)
    clean = torch.empty((sc.YN, sc.XN, sc.ZN), device=cuda, dtype=d_fp.dtype)
    plans.backproject(clean, d_fp)
    for p in range(g["PN"] // 3, 2 * g["PN"] // 3, 1 if sc.dx > 15 else 9):
        v, u = int(rng.integers(g["ZL"])), int(rng.integers(30, g["YL"] - 30))
        fp[p, v, u] = np.inf if rng.random() < 0.7 else -np.inf
    vol = torch.empty_like(clean)
    plans.backproject(vol, torch.tensor(fp, device=cuda, dtype=d_fp.dtype))
    torch.cuda.synchronize()
    plans.close()
    mine, ref = vol.cpu().numpy().ravel(), oracle.bp_f64(fp.astype(np.float64), w, g)
    assert np.isposinf(ref).any() and np.isneginf(ref).any() and np.isnan(ref).any() and np.isfinite(ref).any()
    for cls in (np.isposinf, np.isneginf, np.isnan):
        assert np.array_equal(cls(mine), cls(ref)), cls
    keep = np.isfinite(ref)
    assert np.array_equal(mine[keep], clean.cpu().numpy().ravel()[keep])
