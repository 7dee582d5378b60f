"""GPU tests of the host-pointer entries at output sizes that make the output's
pages resident on helper threads: the result equals the device plan's, bytes
around the output stay as they are, pinned output works, and a call that fails
leaves its output untouched."""
import ctypes

import numpy as np
import pytest
import torch

from analyticalreconbigpatient_b200 import _lib, geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views,offset", [(7, 0), (300, 0), (301, 1)])
def test_rebin_host_output_pages(cuda, views, offset):
    sc = G.Scan(ZL=8, N_2pi=984, rotations=views / 984)
    ra = sc.rebin_args()
    n = views * sc.YL * sc.ZL  # 300 views: 8.5 MB
    rng = np.random.default_rng(views)
    proj = rng.random(n, dtype=np.float32)
    args = (ra["YL"], ra["ZL"], ra["ViewN"], ra["YLC"], ra["dYA"], ra["DeltaTheta"], ra["PLC"], ra["DeltaT"],
            ra["DeltaFai"], ra["SO"])
    big = np.full(n + 64, -3.0, dtype=np.float32)
    pinned = torch.empty(n, dtype=torch.float32, pin_memory=True)
    _lib.call("hr_rebin_host", big[16 + offset:].ctypes.data, proj.ctypes.data, *args)
    _lib.call("hr_rebin_host", pinned.data_ptr(), proj.ctypes.data, *args)
    plan = ctypes.c_void_p()
    lib = _lib.load()
    _lib.check(lib.hr_rebin_plan_create(ctypes.byref(plan), *args))
    d = torch.tensor(proj, device=cuda)
    o = torch.empty_like(d)
    _lib.check(lib.hr_rebin_execute(plan, o.data_ptr(), d.data_ptr(), 0))
    torch.cuda.synchronize()
    lib.hr_rebin_plan_destroy(plan)
    ref = o.cpu().numpy()
    np.testing.assert_array_equal(big[16 + offset:16 + offset + n], ref)
    np.testing.assert_array_equal(pinned.numpy(), ref)
    assert np.all(big[:16 + offset] == -3.0) and np.all(big[16 + offset + n:] == -3.0)


def test_a_failing_call_leaves_its_output_untouched(cuda):
    out = np.arange(2 * 2 * 600000, dtype=np.float32)
    keep = out.copy()
    with pytest.raises(_lib.HelixError):
        _lib.call("hr_filter_host", out.ctypes.data, out.ctypes.data, 3000, 16, 50, 1.0, 1.0, 1.0, 1.0, 541.0)
    np.testing.assert_array_equal(out, keep)
