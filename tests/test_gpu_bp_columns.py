"""The several-column texture backprojection, which only launches of at least two rounds of CTAs run: bit for bit the
one-column forms' volumes, on grids that end inside a tile, a warp and a thread's columns, at thin and thick
slices, and through a launch split into ranges of blocks (some too small for it)."""
import pytest
import torch

from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import HelicalRecon, StagePlans, project
from analyticalreconbigpatient_b200 import phantom as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("XN,YN,dz,ZN", [(509, 497, 0.6, 27), (512, 483, 4.0, 0), (403, 514, 1.0, 31)])
def test_several_columns_equal_one(cuda, XN, YN, dz, ZN):
    sc = G.Scan(ZL=16, pitch=0.9375, rotations=6 if ZN else 14, XN=XN, YN=YN, ZN=max(ZN, 1), dx=500.0 / XN,
                dy=500.0 / YN, dz=dz)
    if not ZN:
        sc = G.replace(sc, ZN=sc.fully_sampled_slices())
    # tiles of 16 x 32 columns, blocks of 4 and 8 slices: two rounds of 8 CTAs per SM
    tiles = -(-XN // 16) * -(-YN // 32)
    assert tiles * (sc.ZN // 4) >= 16 * torch.cuda.get_device_properties(cuda).multi_processor_count
    g = torch.Generator(device=cuda).manual_seed(XN)
    filt = torch.randn((sc.PN, sc.ZL, sc.YL), device=cuda, generator=g)
    fast = StagePlans(sc, _lib.HR_FORM_FAST)
    pairs = torch.empty((sc.PN, sc.ZL, sc.YL), dtype=torch.int32, device=cuda)
    fast.pack(pairs, filt)
    vols = {}
    for v in (16, 17, 18, 19, 21):
        _lib.check(_lib.load().hr_bp_select(fast._bp, v))
        vols[v] = torch.full((sc.YN, sc.XN, sc.ZN), float("nan"), device=cuda)
        fast.backproject(vols[v], pairs)
    torch.cuda.synchronize()
    fast.close()
    assert torch.isfinite(vols[16]).all() and int(torch.count_nonzero(vols[16])) > vols[16].numel() // 2
    for a, b in ((17, 16), (18, 16), (19, 17), (21, 17)):
        assert torch.equal(vols[a], vols[b]), (a, b)


@pytest.mark.parametrize("YL,ZL", [(104, 5), (100, 3), (101, 4)])
def test_texture_copy_by_rows(cuda, YL, ZL):
    """The copy's fill by eight, four and single channels, with row counts that are no multiple of four: an FP16
    copy blended in 1.8 fixed point against the FP32 copy blended the same, so FP16 rounding of BF16 data (none)."""
    sc = G.tiny(YL=YL, ZL=ZL, XN=24, YN=20, ZN=7, dx=4.0, dy=4.0, dz=1.0)
    g = torch.Generator(device=cuda).manual_seed(YL)
    filt = torch.randn((sc.PN, ZL, YL), device=cuda, generator=g)
    fast = StagePlans(sc, _lib.HR_FORM_FAST)
    pairs = torch.empty((sc.PN, ZL, YL), dtype=torch.int32, device=cuda)
    fast.pack(pairs, filt)
    vols = {}
    for v in (11, 14):  # eight slices per thread from the FP16 and the FP32 copy
        _lib.check(_lib.load().hr_bp_select(fast._bp, v))
        vols[v] = torch.zeros((sc.YN, sc.XN, sc.ZN), device=cuda)
        fast.backproject(vols[v], pairs)
    torch.cuda.synchronize()
    fast.close()
    assert int(torch.count_nonzero(vols[14])) > 0
    # the filter hardware may blend FP16 texels at less precision than FP32 ones: 2^-8 of a neighbour difference
    d = (vols[11].double() - vols[14].double()).norm() / vols[14].double().norm()
    assert float(d) < 1e-2, float(d)


def test_streamed_ranges_equal_the_whole(cuda, monkeypatch):
    monkeypatch.setenv("HELIXRECON_BP_VARIANT", "21")
    sc = G.Scan(ZL=16, N_2pi=492, pitch=0.9375, rotations=8, XN=300, YN=300, ZN=60, dx=500.0 / 300, dy=500.0 / 300,
                dz=0.8)
    fan = project(sc, P.random_ellipsoids(3, 8, (-30.0, 30.0)))
    rec = HelicalRecon(sc, form=_lib.HR_FORM_FAST)
    ref = rec.run(fan).clone()
    host = torch.empty(fan.shape, dtype=torch.float32, pin_memory=True)
    host.copy_(fan)
    out = torch.empty((sc.YN, sc.XN, sc.ZN), dtype=torch.float32, pin_memory=True)
    rec.run_host(host, out)
    rec.check()
    rec.close()
    # the streamed copy's FP16 scale differs by a power of two: the same but for subnormal FP16 samples
    d = (out.to(cuda).double() - ref.double()).norm() / ref.double().norm()
    assert float(d) < 1e-6, float(d)
