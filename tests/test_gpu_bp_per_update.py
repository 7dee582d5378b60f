"""The per-update weight kernels of the plain and FP64 forms, which run where a block's weight table would not fit
(slices so thick that a block's union view window is some thousand views), against the oracle; describe() names the
kernel that runs: its weights and its tile.

Tolerances as for the table-weight kernels: 1e-5 relative L2 for FP32 sums, 1e-11 for FP64; index selection is exact."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import StagePlans
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "fp64"])
@pytest.mark.parametrize("dz,rotations,weights", [(1.5, 4, "per-block table"), (24.0, 56, "per update")])
def test_the_kernel_named_is_the_one_checked(cuda, form, dz, rotations, weights):
    sc = G.tiny(delta=8, XN=10, YN=33, ZN=9, dz=dz, rotations=rotations)
    g = sc.bp_geom()
    fp = np.random.default_rng(int(dz)).standard_normal((g["PN"], g["ZL"], g["YL"])).astype(np.float32)
    w = oracle.weight_table(sc.N_2pi, sc.HSCoef, sc.delta)
    double = form == "fp64"
    plans = StagePlans(sc, _lib.HR_FORM_FP64 if double else _lib.HR_FORM_PLAIN)
    buf = ctypes.create_string_buffer(256)
    _lib.check(_lib.load().hr_bp_describe(plans._bp, buf, 256))
    d = buf.value.decode()
    assert d.endswith("weights=" + weights) and d.startswith(form + " "), d
    assert ("tile=8x32" in d) == (weights == "per-block table"), d
    d_fp = torch.tensor(fp, device=cuda, dtype=torch.float64 if double else torch.float32)
    vol = torch.full((sc.YN, sc.XN, sc.ZN), float("nan"), device=cuda, dtype=d_fp.dtype)
    plans.backproject(vol, d_fp)
    torch.cuda.synchronize()
    plans.close()
    mine = vol.cpu().numpy().astype(np.float64).ravel()
    ref = oracle.bp_f64(fp.astype(np.float64), w, g)
    assert np.count_nonzero(ref) and np.array_equal(mine == 0, ref == 0)
    assert rel_l2(mine, ref) < (1e-11 if double else 1e-5)
