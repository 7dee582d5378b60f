"""Plain and FP64 plans of different view windows (their weight tables take different amounts of shared memory)
executed at the same time by two host threads: no execution fails, and every volume is the one the plan gives
alone, bit for bit (each thread sums its own voxels in a fixed order)."""
import threading

import pytest
import torch

from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import StagePlans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "fp64"])
def test_plans_of_different_windows_from_two_threads(cuda, form):
    double = form == "fp64"
    work = []
    for dz in (0.05, 9.0):  # union windows of a z block: 73 and some 1700 views
        sc = G.tiny(delta=8, XN=9, YN=8, ZN=8, dz=dz, rotations=40 if dz > 1 else 4)
        plans = StagePlans(sc, _lib.HR_FORM_FP64 if double else _lib.HR_FORM_PLAIN)
        g = torch.Generator(device=cuda).manual_seed(int(dz))
        fp = torch.randn((sc.PN, sc.ZL, sc.YL), device=cuda, generator=g, dtype=torch.float64 if double else torch.float32)
        vol = torch.full((sc.YN, sc.XN, sc.ZN), float("nan"), device=cuda, dtype=fp.dtype)
        plans.backproject(vol, fp)
        work.append((plans, fp, vol.clone(), torch.cuda.Stream()))
    torch.cuda.synchronize()
    assert all(int(torch.count_nonzero(ref)) for _, _, ref, _ in work)
    start, failures = threading.Barrier(2), []

    def loop(plans, fp, ref, stream):
        out = torch.full_like(ref, float("nan"))
        start.wait()
        try:
            for _ in range(3000):
                plans.backproject(out, fp, stream.cuda_stream)
            stream.synchronize()
            if not torch.equal(out, ref):
                failures.append("the volume differs")
        except Exception as e:  # noqa: BLE001 (reported by the test's own thread)
            failures.append(str(e))

    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for plans, *_ in work:
        plans.close()
    assert not failures, failures
