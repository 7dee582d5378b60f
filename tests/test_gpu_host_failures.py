"""A host-pointer call that fails after its helper threads have begun to make the output's pages resident (a volume of
more z blocks than one launch takes, found when the backprojection is launched) leaves every byte of the output, and
around it, as it was."""
import numpy as np
import pytest

import oracle
from analyticalreconbigpatient_b200 import _lib, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry,dtype,slices", [("hr_bp_host_float", np.float32, 8), ("hr_bp_host_double", np.float64, 4)])
@pytest.mark.parametrize("offset", [0, 3])
def test_a_call_that_fails_late_leaves_its_output_untouched(cuda, entry, dtype, slices, offset):
    sc = G.tiny(delta=8, XN=2, YN=2, ZN=slices * 65536, dz=1e-5)  # 65536 blocks: one more than a grid's z
    g = sc.bp_geom()
    n = sc.XN * sc.YN * sc.ZN
    assert n * np.dtype(dtype).itemsize >= 4 << 20  # smaller outputs start no helper threads
    rng = np.random.default_rng(offset)
    out = rng.integers(0, 256, (n + 64) * np.dtype(dtype).itemsize, dtype=np.uint8)
    keep = out.copy()
    fp = np.ones((g["PN"], g["ZL"], g["YL"]), dtype=dtype)
    w = np.asarray(oracle.weight_table(sc.N_2pi, sc.HSCoef, sc.delta), dtype=dtype)
    names = ("N_2pi XN YN ZN XNC YNC ZNC dx dy dz YL ZL PN YLC ZLC dYL dZL h BetaS DeltaFai N_pi HSCoef SO SD k1")
    with pytest.raises(_lib.HelixError, match="grid too large"):
        _lib.call(entry, out.ctypes.data + 16 * np.dtype(dtype).itemsize + offset, fp.ctypes.data, w.ctypes.data,
                  *[g[k] for k in names.split()])
    np.testing.assert_array_equal(out, keep)
