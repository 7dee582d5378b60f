"""Which form of the segmented texture kernels a plan times and runs: the autotuner's time of a variant is that of the
form (four columns per thread, or two views per iteration) that a launch over the plan's volume runs, and describe()
names it; four columns only where the launch has the CTAs, and, untuned, where the grid fills their threads."""
import ctypes
import re

import pytest
import torch

from analyticalreconbigpatient_b200 import _lib, geometry as G
from analyticalreconbigpatient_b200.pipeline import SlabRecon, StagePlans

pytestmark = pytest.mark.gpu


def _forms(plans, variants):
    """{variant: (timed with four columns, run with four columns)} from describe()."""
    buf = ctypes.create_string_buffer(1024)
    out = {}
    for v in variants:
        _lib.check(_lib.load().hr_bp_select(plans._bp, v))
        _lib.check(_lib.load().hr_bp_describe(plans._bp, buf, 1024))
        d = buf.value.decode()
        timed = re.search(rf" v{v}=[0-9.]+(x4)?[ )]", d)
        assert timed, d
        out[v] = (timed.group(1) == "x4", "four-columns" in d)
        assert ("two-views" in d) != ("four-columns" in d), d
        assert ("tile=16x32" in d) == ("four-columns" in d), d
    return out


# a band of 32 slices of 256 x 256 is 1024 CTAs of the four-column form, under two rounds on 148 SMs; 80 slices, 2560
@pytest.mark.parametrize("N,ZN,four", [(256, 80, True), (256, 32, False), (512, 40, True), (64, 80, False)])
def test_the_form_timed_is_the_form_run(cuda, N, ZN, four):
    sc = G.Scan(ZL=16, N_2pi=246, pitch=0.9375, rotations=10, XN=N, YN=N, ZN=ZN, dx=500.0 / N, dy=500.0 / N, dz=0.8)
    plans = StagePlans(sc, _lib.HR_FORM_FAST)
    pairs = torch.full((sc.PN, sc.ZL, sc.YL), 0x3f803f80, dtype=torch.int32, device=cuda)
    vol = torch.empty((sc.YN, sc.XN, sc.ZN), device=cuda)
    plans.autotune(vol, pairs)
    forms = _forms(plans, (18, 19, 21))
    plans.close()
    assert all(t == r for t, r in forms.values()), forms
    assert not forms[18][1] and (four or not any(r for _, r in forms.values())), forms


@pytest.mark.parametrize("N,ZN,four", [(512, 40, True), (509, 40, True), (256, 80, True), (256, 36, False),
                                       (130, 400, False), (165, 300, False)])
def test_the_form_of_an_untuned_plan(cuda, N, ZN, four):
    """130 and 165 rows of pixels leave 9 and 5 % of the lanes of four-column threads idle."""
    sc = G.Scan(ZL=8, N_2pi=246, pitch=0.9375, rotations=26, XN=N, YN=N, ZN=ZN, dx=500.0 / N, dy=500.0 / N, dz=0.25)
    plans = StagePlans(sc, _lib.HR_FORM_FAST)
    buf = ctypes.create_string_buffer(1024)
    for v in (18, 19, 21):
        _lib.check(_lib.load().hr_bp_select(plans._bp, v))
        _lib.check(_lib.load().hr_bp_describe(plans._bp, buf, 1024))
        assert ("four-columns" in buf.value.decode()) == (four and v != 18), (v, buf.value)
    plans.close()


@pytest.mark.parametrize("slab,four", [(80, True), (24, False)])
def test_slabs_settle_one_form(cuda, monkeypatch, slab, four):
    """Both buffers' captured graphs and the description use the form of the middle slab."""
    monkeypatch.setenv("HELIXRECON_BP_VARIANT", "21")
    sc = G.Scan(ZL=16, N_2pi=246, pitch=0.9375, rotations=20, XN=256, YN=256, ZN=170, dx=1.9, dy=1.9, dz=0.8)
    fan = torch.rand((sc.views, sc.YL, sc.ZL), device=cuda)
    vol = torch.empty((sc.YN, sc.XN, sc.ZN), device=cuda)
    rec = SlabRecon(sc, slab_slices=slab)
    rec.run(fan, vol)
    assert ("four-columns" in rec.describe()) == four, rec.describe()
    rec.close()
