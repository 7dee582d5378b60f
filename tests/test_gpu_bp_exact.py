"""GPU tests of the table-weight backprojections (plain FP32 and FP64) where
their index estimates can go wrong: tile and z-block remainders, slices at and
beyond the scan's ends, detectors whose centre row is an integer (positions
that fall exactly on rows), and slices too thick for the per-block table.

Tolerances, from the arithmetic: FP32 sums of some 40..700 terms with relative
rounding of 6e-8 per operation stay below 1e-5 relative L2 (the plain form's
stated bound); the FP64 forms differ by rounding, below 1e-11. Index selection
is exact, so a voxel is zero exactly where the oracle's is."""

import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import StagePlans
from conftest import rel_l2

pytestmark = pytest.mark.gpu

CASES = {
    "one_voxel": dict(XN=1, YN=1, ZN=1),
    "tile_remainders": dict(XN=9, YN=33, ZN=9),
    "block_edges": dict(XN=8, YN=32, ZN=8, dx=20.0, dy=9.0),
    "integer_rows": dict(ZL=9, XN=17, YN=15, ZN=13, dx=10.0, dy=10.0, dz=0.75),
    "beyond_the_scan": dict(XN=12, YN=10, ZN=61, dz=2.0),
    "two_rows": dict(ZL=2, XN=13, YN=35, ZN=5, dz=0.5),
    "thick_slices": dict(XN=10, YN=9, ZN=7, dz=9.0, rotations=40),
    "table_too_large": dict(XN=10, YN=9, ZN=7, dz=20.0, rotations=40),
    "off_detector_columns": dict(XN=20, YN=20, ZN=6, dx=40.0, dy=40.0),
}


@pytest.mark.parametrize("form", ["plain", "fp64"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_table_weight_backprojection_vs_oracle(cuda, name, form):
    sc = G.tiny(delta=8, **CASES[name])
    g = sc.bp_geom()
    rng = np.random.default_rng(len(name))
    fp = rng.standard_normal((g["PN"], g["ZL"], g["YL"])).astype(np.float32)
    w = oracle.weight_table(sc.N_2pi, sc.HSCoef, sc.delta)
    double = form == "fp64"
    plans = StagePlans(sc, _lib.HR_FORM_FP64 if double else _lib.HR_FORM_PLAIN)
    d_fp = torch.tensor(fp, device=cuda, dtype=torch.float64 if double else torch.float32)
    vol = torch.full((sc.YN, sc.XN, sc.ZN), float("nan"), device=cuda, dtype=d_fp.dtype)
    plans.backproject(vol, d_fp)
    torch.cuda.synchronize()
    plans.close()
    mine = vol.cpu().numpy().astype(np.float64).ravel()
    ref = oracle.bp_f64(fp.astype(np.float64), w, g)
    assert np.array_equal(mine == 0, ref == 0)
    if np.count_nonzero(ref):
        assert rel_l2(mine, ref) < (1e-11 if double else 1e-5)


@pytest.mark.parametrize("form", ["plain", "fp64"])
def test_values_outside_a_slices_window_do_not_reach_it(cuda, form):
    """Views no slice's window holds, and rows off the detector, may hold
    anything (NaN, infinities) without reaching the volume; a NaN in a view of
    the window does."""
    sc = G.tiny(delta=8, XN=10, YN=12, ZN=3, dz=0.5, rotations=4)
    g = sc.bp_geom()
    s0 = [np.ceil((2 * G.PI_TRUNC * (z - g["ZNC"]) * g["dz"] / g["h"] - g["BetaS"]) / g["DeltaFai"] - 0.5)
          for z in range(sc.ZN)]
    half = int(np.ceil(g["N_pi"] * g["HSCoef"]))
    lo, hi = int(min(s0)) - half, int(max(s0)) + half
    assert 0 < lo and hi < sc.PN - 1
    double = form == "fp64"
    plans = StagePlans(sc, _lib.HR_FORM_FP64 if double else _lib.HR_FORM_PLAIN)
    fp = torch.ones((sc.PN, sc.ZL, sc.YL), device=cuda, dtype=torch.float64 if double else torch.float32)
    vol = torch.empty((sc.YN, sc.XN, sc.ZN), device=cuda, dtype=fp.dtype)
    plans.backproject(vol, fp)
    clean = vol.clone()
    fp[:lo] = float("nan")
    fp[hi + 1:] = float("inf")
    plans.backproject(vol, fp)
    assert torch.equal(vol, clean) and torch.isfinite(vol).all()
    fp[(lo + hi) // 2] = float("nan")
    plans.backproject(vol, fp)
    torch.cuda.synchronize()
    assert torch.isnan(vol).any()
    plans.close()
