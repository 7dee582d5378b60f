"""The work a user of the library has it do, as cases to time and to compare.

Every case goes through a public entry point (``api``, ``pipeline``, ``learned``) at the sizes of the
scanner the library is configured for: an 888-channel curved detector with 16, 32 or 64 rows, 984 (or, half
view, 492) views per rotation, grids of 128 to 512 pixels a side, slices from 0.18 to 4 mm.

* ``prepare(case, seed)`` makes what a program has in hand: the scan's projections (line integrals of a seeded
  phantom, with photon noise where ``I0`` is set) or volumes, and the plan or network it keeps.
* ``run(state)`` is one pass and returns its outputs whole.
* ``work(case)`` counts each input byte read once, each output byte written once, and the operations of the
  path's own arithmetic (per backprojection update 20: position, four-tap blend, weight, sum).
* ``exact(case, seed)`` is the same path in float64 with plain torch, from the same inputs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from analyticalreconbigpatient_b200 import _lib, api
from analyticalreconbigpatient_b200 import geometry as G
from analyticalreconbigpatient_b200 import phantom as P
from analyticalreconbigpatient_b200.learned import CIN, COUT, Corrector, init_params
from analyticalreconbigpatient_b200.pipeline import (BatchRecon, HelicalRecon, SlabRecon, StagePlans,
                                                     add_poisson_noise, project)

UPDATE_FLOPS = 20.0
DEV = "cuda:0"


# ---- the cases ----------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # one short segment through the three drop-in host calls, numpy arrays in and out, as the reference's
        # driver makes them: the smallest calls, where set-up and copies count beside the kernels
        dict(name="dropin_segment", kind="dropin", ZL=16, N_2pi=492, rotations=1.5, pitch=0.9375, N=128, ZN=8,
             dz=1.0, double=False),
        # fan -> parallel rebinning of a two-rotation scan on the full detector, a stage of its own
        dict(name="rebin_2rot", kind="rebin", ZL=64, N_2pi=984, rotations=2.0, pitch=0.984),
        # preweight + ramp filter of rows in the reference's layout (one rotation, odd view count)
        dict(name="filter_rows", kind="filter", YL=888, ZL=32, views=1023),
        # double-precision backprojection (the reference's CPU numerics), an odd grid
        dict(name="bp_double", kind="bp64", ZL=16, N_2pi=984, rotations=3.0, pitch=0.9375, N=186,
             YN=171, ZN=21, dz=1.0),
        # the drop-in numerics from fan data to volume on the device: two rotations of the full detector
        dict(name="plain_2rot", kind="chain", form="plain", ZL=64, N_2pi=984, rotations=2.0, pitch=0.984, N=512,
             ZN=48, dz=0.625, I0=0.0),
        # the fast form on a head scan: the smallest whole reconstruction
        dict(name="fast_head", kind="chain", form="fast", ZL=16, N_2pi=984, rotations=4.0, pitch=0.9375, N=256,
             ZN=32, dz=1.0, I0=0.0),
        # the fast form on the twenty-rotation scan of the full detector: the headline workload
        dict(name="fast_20rot", kind="chain", form="fast", ZL=64, N_2pi=984, rotations=20.0, pitch=0.984, N=512,
             ZN=0, dz=0.625, I0=0.0),
        # half-view scan from page-locked host memory to a host volume, streamed
        dict(name="host_halfview", kind="host", form="fast", ZL=64, N_2pi=492, rotations=6.0, pitch=0.984, N=512,
             ZN=0, dz=0.625, I0=1e5),
        # a long scan with thick slices, slab by slab on the device
        dict(name="slabs_thick", kind="slab", ZL=64, N_2pi=984, rotations=10.0, pitch=0.984, N=512, ZN=0, dz=3.92,
             slab=32, I0=0.0),
        # three noisy scans of uneven size in one batch
        dict(name="batch_uneven", kind="batch", scan_seed=20, scans=3, I0=2e5),
        # the correction network over a reconstructed volume
        dict(name="cnn_volume", kind="cnn", H=512, W=512, ZN=64),
        # one training step of the network on eight slices
        dict(name="cnn_train", kind="train", B=8, H=512, W=512),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(["dropin", "rebin", "filter", "bp64", "chain", "chain", "host", "slab", "batch", "cnn",
                       "train"])
    pitch = rng.choice([0.5, 0.9375, 0.984, 1.375])
    ZL = rng.choice([16, 32, 64])
    N_2pi = rng.choice([492, 984])
    N = rng.choice([256, 512]) if rng.random() < 0.5 else rng.randrange(128, 513)
    if kind == "dropin":
        return dict(kind=kind, ZL=rng.choice([7, 16, 32]), N_2pi=N_2pi, rotations=round(rng.uniform(1.2, 2.0), 2),
                    pitch=pitch, N=rng.randrange(64, 200), ZN=rng.randrange(3, 24), dz=round(rng.uniform(0.5, 1.5), 3),
                    double=rng.choice([False, True]))
    if kind == "rebin":
        return dict(kind=kind, ZL=rng.choice([15, 16, 20, 32, 64]), N_2pi=N_2pi, rotations=round(_log(rng, 1, 16), 2),
                    pitch=pitch)
    if kind == "filter":
        return dict(kind=kind, YL=rng.choice([888, 888, rng.randrange(300, 1025)]), ZL=rng.choice([7, 16, 32, 64]),
                    views=int(_log(rng, 100, 8000)))
    if kind == "bp64":
        return dict(kind=kind, ZL=ZL, N_2pi=N_2pi, rotations=round(rng.uniform(2.0, 4.0), 2), pitch=pitch,
                    N=rng.randrange(96, 257), YN=rng.randrange(96, 257), ZN=rng.randrange(3, 33), dz=round(rng.uniform(0.4, 2.0), 3))
    if kind == "chain":
        form = rng.choice(["plain", "fast"])
        rot = round(_log(rng, 2.0, 6.0 if form == "plain" else 16.0), 2)
        return dict(kind=kind, form=form, ZL=ZL, N_2pi=N_2pi, rotations=rot, pitch=pitch, N=N,
                    ZN=rng.randrange(16, 80) if form == "plain" else rng.randrange(24, 400),
                    dz=round(_log(rng, 0.2, 1.25), 4), I0=rng.choice([0.0, 2e5]))
    if kind == "host":
        return dict(kind=kind, form="fast", ZL=ZL, N_2pi=N_2pi, rotations=round(rng.uniform(3.0, 8.0), 2),
                    pitch=pitch, N=N, ZN=rng.randrange(40, 300), dz=0.625, I0=rng.choice([0.0, 1e5]))
    if kind == "slab":
        return dict(kind=kind, ZL=64, N_2pi=984, rotations=round(rng.uniform(6.0, 14.0), 2), pitch=0.984,
                    N=rng.choice([256, 512]), ZN=0, dz=round(rng.uniform(1.0, 4.0), 3), slab=rng.choice([24, 32, 64]),
                    I0=0.0)
    if kind == "batch":
        while True:
            c = dict(kind=kind, scan_seed=rng.randrange(1, 10000), scans=rng.choice([2, 3, 4]), I0=rng.choice([0.0, 2e5]))
            ss = _batch(c)
            if sum(s.updates() for s in ss) < 1e11 and sum(s.projection_bytes() for s in ss) < 8e9:
                return c
    if kind == "cnn":
        return dict(kind=kind, H=rng.randrange(128, 513), W=rng.choice([256, 512, rng.randrange(128, 513)]),
                    ZN=rng.randrange(5, 128))
    return dict(kind="train", B=rng.randrange(1, 9), H=rng.randrange(128, 513), W=rng.choice([128, 256, 512, 500]))


def _scan(c) -> G.Scan:
    N, ZN = c.get("N", 64), c.get("ZN", 1)
    s = G.Scan(ZL=c["ZL"], N_2pi=c["N_2pi"], rotations=c["rotations"], pitch=c["pitch"], XN=N, YN=c.get("YN", N),
               ZN=max(ZN, 1), dx=500.0 / N, dy=500.0 / N, dz=c.get("dz", 1.0))
    return s if ZN else s.with_full_z()


def _batch(c) -> list[G.Scan]:
    return G.batch_scans(c["scan_seed"], c["scans"])


# ---- inputs -----------------------------------------------------------------------------------------------
def _fan(scan: G.Scan, seed: int, I0: float) -> torch.Tensor:
    """Projections of a seeded phantom (an elliptic water body with 24 ellipsoids), device float32."""
    z = [scan.h * b / (2 * math.pi) for b in (scan.BetaS, scan.BetaS + scan.views * scan.dBeta)]
    fan = project(scan, P.random_ellipsoids(seed, 24, (min(z), max(z))))
    if I0 > 0:
        add_poisson_noise(fan, I0, seed)
    return fan


def _filter_scan(c) -> G.Scan:
    """A scan whose views left after the crop at both ends are the case's."""
    s = G.Scan(YL=c["YL"], ZL=c["ZL"], N_2pi=984, det_pitch=1.0239 * 888 / c["YL"])
    return G.replace(s, rotations=(c["views"] + 2 * s.seg_overlap + 0.25) / 984)


def _rows(c, seed: int) -> torch.Tensor:
    """Detector rows in the reference's layout [views][ZL][YL]: smooth projections with noise, float32."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = torch.linspace(-1.0, 1.0, c["YL"], device=DEV)
    v = torch.arange(c["views"], device=DEV, dtype=torch.float32).view(-1, 1, 1)
    r = torch.linspace(0.0, 1.0, c["ZL"], device=DEV).view(1, -1, 1)
    half = 0.55 + 0.1 * torch.cos(0.0128 * v + 0.3 * r)
    p = 6.0 * torch.sqrt(torch.clamp(half * half - u * u, min=0.0))
    p += 0.02 * torch.randn(p.shape, device=DEV, generator=g)
    return p.contiguous()


def _volume(H: int, W: int, n: int, seed: int) -> torch.Tensor:
    """A noisy water-like volume [H][W][n] with a few denser discs, float32."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    y = torch.linspace(-1, 1, H, device=DEV).view(-1, 1, 1)
    x = torch.linspace(-1, 1, W, device=DEV).view(1, -1, 1)
    z = torch.arange(n, device=DEV, dtype=torch.float32).view(1, 1, -1)
    v = (x * x / 0.52 + y * y / 0.31 < 1.0).float() * torch.ones(n, device=DEV)
    for k in range(6):
        c = torch.rand(3, device=DEV, generator=g) - 0.5
        v += 0.2 * ((x - c[0] - 0.002 * z) ** 2 + (y - 0.6 * c[1]) ** 2 < 0.01 + 0.02 * (c[2] + 0.5)).float()
    v += 0.05 * torch.randn(v.shape, device=DEV, generator=g)
    return (G.MU_WATER * v).contiguous()


def _params(seed: int) -> np.ndarray:
    """Network parameters with a last layer that is not zero, as after training."""
    p = init_params(seed)
    n = 9 * CIN[7] * COUT[7]
    o = p.size - COUT[7] - n
    p[o:o + 9 * CIN[7]] = np.random.default_rng(seed + 1).standard_normal(9 * CIN[7]) * 0.01
    return p


def _train_data(c, seed: int):
    vol = _volume(c["H"], c["W"], c["B"] + 4, seed)
    base = vol[:, :, 2:2 + c["B"]].permute(2, 0, 1).contiguous()
    g = torch.Generator(device=DEV).manual_seed(seed + 7)
    target = base + G.MU_WATER * 0.03 * torch.randn(base.shape, device=DEV, generator=g)
    return vol, base, target.contiguous()


def _bp_input(c, s: G.Scan, seed: int) -> torch.Tensor:
    """Filtered-like rows, double [PN][ZL][YL]."""
    g = torch.Generator(device=DEV).manual_seed(seed + 3)
    rows = _rows(dict(c, YL=s.YL, views=s.PN), seed).double()
    rows = 0.02 * (rows - rows.mean(dim=-1, keepdim=True))
    return rows + 0.01 * torch.randn(rows.shape, device=DEV, generator=g, dtype=torch.float64)


class _State:
    pass


def prepare(case: dict, seed: int):
    c, kind = case, case["kind"]
    st = _State()
    st.kind, st.case = kind, c
    if kind == "dropin":
        s = st.scan = _scan(c)
        st.fan = _fan(s, seed, 0.0).cpu().numpy()
        st.w = api.weight_table(s.N_2pi, s.HSCoef, s.delta)
        return st
    if kind == "rebin":
        s = st.scan = _scan(c)
        st.fan = _fan(s, seed, 0.0)
        st.plans = StagePlans(s)
        st.out = torch.empty_like(st.fan)
        return st
    if kind == "filter":
        st.rows = _rows(c, seed)
        st.out = torch.empty_like(st.rows)
        st.plans = StagePlans(_filter_scan(c))
        return st
    if kind == "bp64":
        s = st.scan = _scan(c)
        st.fp = _bp_input(c, s, seed)
        st.plans = StagePlans(s, _lib.HR_FORM_FP64)
        st.out = torch.empty((s.YN, s.XN, s.ZN), dtype=torch.float64, device=DEV)
        return st
    if kind in ("chain", "host"):
        s = st.scan = _scan(c)
        fan = _fan(s, seed, c["I0"])
        st.recon = HelicalRecon(s, form=_lib.HR_FORM_PLAIN if c["form"] == "plain" else _lib.HR_FORM_FAST)
        if kind == "host":
            st.fan = torch.empty(fan.shape, dtype=torch.float32, pin_memory=True)
            st.fan.copy_(fan)
            st.out = torch.empty((s.YN, s.XN, s.ZN), dtype=torch.float32, pin_memory=True)
        else:
            st.fan = fan
        return st
    if kind == "slab":
        s = st.scan = _scan(c)
        st.fan = _fan(s, seed, c["I0"])
        st.out = torch.empty((s.YN, s.XN, s.ZN), dtype=torch.float32, device=DEV)
        st.recon = SlabRecon(s, slab_slices=c["slab"])
        return st
    if kind == "batch":
        st.scans = _batch(c)
        st.fans = [_fan(s, seed + 1000 * i, c["I0"]) for i, s in enumerate(st.scans)]
        st.vols = [torch.empty((s.YN, s.XN, s.ZN), dtype=torch.float32, device=DEV) for s in st.scans]
        st.recon = BatchRecon(st.scans)
        return st
    st.net = Corrector(_params(seed))
    if kind == "cnn":
        st.vol = _volume(c["H"], c["W"], c["ZN"], seed)
        st.out = torch.empty_like(st.vol)
        return st
    vol, st.base, st.target = _train_data(c, seed)
    st.x = torch.empty((c["B"], c["H"], c["W"], 16), dtype=torch.int16, device=DEV)
    st.net.pack_input(st.x, vol, 2, c["B"])
    return st


# ---- one pass ------------------------------------------------------------------------------------------------
def run(st):
    kind = st.kind
    if kind == "dropin":
        s, ra, fa = st.scan, st.scan.rebin_args(), st.scan.filter_args()
        reb = api.ParallelRebinningCBCurve(st.fan, ra["YL"], ra["ZL"], ra["ViewN"], ra["YLC"] + 1, ra["dYA"],
                                           ra["DeltaTheta"], ra["PLC"] + 1, ra["DeltaT"], ra["DeltaFai"], ra["SO"], 1)
        rows = np.ascontiguousarray(reb[s.crop_front:s.views - s.crop_back].transpose(0, 2, 1))
        filt = api.reWeigAdFiltr_GPU(rows, fa["PLC"], fa["ZLC"], fa["dYL"], fa["dZL"], fa["SO"])
        bp = api.ParallekFDKHelical3DWeighting_GPU_double if st.case["double"] else \
            api.ParallekFDKHelical3DWeighting_GPU_float
        return {"rebinned": reb, "filtered": filt, "image": bp(filt, st.w, s.bp_geom())}
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "rebin":
        st.plans.rebin(st.out, st.fan, stream)
        return st.out
    if kind == "filter":
        st.plans.filter(st.out, st.rows, _lib.HR_LAYOUT_ROWS, 0, stream)
        return st.out
    if kind == "bp64":
        st.plans.backproject(st.out, st.fp, stream)
        return st.out
    if kind == "chain":
        return st.recon.run(st.fan)
    if kind == "host":
        return st.recon.run_host(st.fan, st.out)
    if kind == "slab":
        st.recon.run(st.fan, st.out)
        return st.out
    if kind == "batch":
        st.recon.run(st.fans, st.vols)
        return st.vols
    if kind == "cnn":
        return st.net.apply_volume(st.vol, st.out)
    loss = st.net.train_step(st.x, st.base, st.target, 1e-4)
    return {"loss": loss, "grads": st.net.grads(), "params": st.net.params()}


# ---- what a pass cannot do without ------------------------------------------------------------------------
def _fft_flops(YL: int) -> float:
    n = 1 << math.ceil(math.log2(2 * YL - 1))
    return 5.0 * n * math.log2(n)  # forward and inverse real transforms of one row


def _chain_work(s: G.Scan) -> dict:
    rows = s.PN * s.ZL
    return {"bytes": s.projection_bytes() + s.volume_bytes(),
            "flops": 8.0 * s.views * s.YL * s.ZL + rows * _fft_flops(s.YL) + UPDATE_FLOPS * s.updates()}


def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind in ("cnn", "train"):
        px = c["H"] * c["W"] * (c["ZN"] if kind == "cnn" else c["B"])
        macs = 9 * (5 * 32 + 6 * 32 * 32 + 32)  # five real input channels, one output channel
        if kind == "cnn":
            return {"bytes": 8.0 * px, "flops": 2.0 * macs * px}
        return {"bytes": (32.0 + 8.0) * px, "flops": 2.0 * px * (3 * macs - 9 * 5 * 32)}
    if kind == "filter":
        n = float(c["views"] * c["ZL"])
        return {"bytes": 8.0 * n * c["YL"], "flops": n * (_fft_flops(c["YL"]) + c["YL"])}
    if kind == "batch":
        parts = [_chain_work(s) for s in _batch(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    s = _scan(c)
    if kind == "rebin":
        return {"bytes": 2.0 * s.projection_bytes(), "flops": 8.0 * s.views * s.YL * s.ZL}
    if kind == "bp64":
        return {"bytes": 8.0 * s.PN * s.ZL * s.YL + 2.0 * s.volume_bytes(), "flops": UPDATE_FLOPS * s.updates()}
    w = _chain_work(s)
    if kind == "dropin":
        w["bytes"] += 3.0 * s.projection_bytes() + s.volume_bytes()
    return w


# ---- the same in float64, plain torch ----------------------------------------------------------------------
def _exact_rebin(fan: torch.Tensor, a: dict) -> torch.Tensor:
    """fan [views][YL][ZL] float32 -> float64, bilinear in (view, channel) at the parallel geometry."""
    V, YL = a["ViewN"], a["YL"]
    j = torch.arange(YL, device=DEV, dtype=torch.float64)
    t = (j - a["PLC"]) * a["DeltaT"]
    beta = torch.asin(t / a["SO"])
    ui = torch.atan(t / torch.sqrt(a["SO"] ** 2 - t * t)) / a["dYA"] + a["YLC"]
    U = torch.ceil(ui)
    cy = (U - ui).view(1, -1, 1)
    U = U.long()
    ub, uu = (U - 1).clamp(0, YL - 1), U.clamp(0, YL - 1)
    ub = torch.where(U > YL - 1, torch.full_like(ub, YL - 1), ub)
    out = torch.empty((V, YL, a["ZL"]), dtype=torch.float64, device=DEV)
    for i0 in range(0, V, 256):
        i = torch.arange(i0, min(V, i0 + 256), device=DEV, dtype=torch.float64)
        fi = (i.view(-1, 1) * a["DeltaTheta"] + beta.view(1, -1)) / a["DeltaFai"]
        F = torch.ceil(fi)
        cx = (F - fi).unsqueeze(-1)
        F = F.long()
        fb, fu = (F - 1).clamp(0, V - 1), F.clamp(0, V - 1)
        fb = torch.where(F > V - 1, torch.full_like(fb, V - 1), fb)
        lo = cx * fan[fb, ub.view(1, -1)].double() + (1 - cx) * fan[fu, ub.view(1, -1)].double()
        hi = cx * fan[fb, uu.view(1, -1)].double() + (1 - cx) * fan[fu, uu.view(1, -1)].double()
        out[i0:i0 + i.numel()] = cy * lo + (1 - cy) * hi
    return out


def _exact_filter(rows: torch.Tensor, a: dict) -> torch.Tensor:
    """rows [views][ZL][YL] -> float64: cosine preweight and the linear convolution with the ramp kernel."""
    YL, ZL, SO = a["YL"], a["ZL"], a["SO"]
    b = ((torch.arange(ZL, device=DEV, dtype=torch.float64) - a["ZLC"]) * a["dZL"]).view(-1, 1)
    t = ((torch.arange(YL, device=DEV, dtype=torch.float64) - a["PLC"]) * a["dYL"]).view(1, -1)
    wt = SO ** 2 / torch.sqrt(SO ** 2 * (SO ** 2 + b * b) - (b * t) ** 2)
    n = 1 << math.ceil(math.log2(2 * YL - 1))
    k = torch.arange(YL, device=DEV, dtype=torch.float64)
    hk = -2.0 / (math.pi ** 2 * (4 * k * k - 1)) / a["dYL"]
    h = torch.zeros(n, dtype=torch.float64, device=DEV)
    h[:YL] = hk
    h[n - YL + 1:] = hk[1:].flip(0)
    H = torch.fft.rfft(h)
    out = torch.empty(rows.shape, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 26) // (ZL * n))
    for v in range(0, rows.shape[0], step):
        out[v:v + step] = torch.fft.irfft(torch.fft.rfft(rows[v:v + step].double() * wt, n) * H, n)[..., :YL]
    return out


def _exact_weights(s: G.Scan) -> torch.Tensor:
    n_pi = s.N_2pi / 2.0
    half = math.ceil(n_pi * s.HSCoef)
    L, shift = 2 * half + 1, int(n_pi - half)
    w = torch.zeros(s.N_2pi, dtype=torch.float64)
    for k in range(L):
        v = 1.0
        if k < s.delta:
            v = math.cos(math.pi / 2 * (s.delta - k - 0.5) / s.delta) ** 2
        elif k >= L - s.delta:
            v = math.cos(math.pi / 2 * (k - (L - s.delta) + 0.5) / s.delta) ** 2
        if 0 <= k + shift < s.N_2pi:
            w[k + shift] = v
    return w.to(DEV)


def _exact_bp(fp: torch.Tensor, g: dict, w: torch.Tensor) -> torch.Tensor:
    """fp [PN][ZL][YL] float64 -> [YN][XN][ZN]: the 3D-weighted helical backprojection."""
    YL, ZL, PN = g["YL"], g["ZL"], g["PN"]
    f64 = dict(device=DEV, dtype=torch.float64)
    x = ((torch.arange(g["XN"], **f64) - g["XNC"]) * g["dx"]).view(1, 1, -1)
    y = ((torch.arange(g["YN"], **f64) - g["YNC"]) * g["dy"]).view(1, -1, 1)
    vol = torch.zeros((g["ZN"], g["YN"], g["XN"]), **f64)
    flat = fp.reshape(-1)
    half = math.ceil(g["N_pi"] * g["HSCoef"])
    SO, SD, k1 = g["SO"], g["SD"], g["k1"]
    step = max(1, (1 << 22) // (g["XN"] * g["YN"]))
    for zi in range(g["ZN"]):
        z = (zi - g["ZNC"]) * g["dz"]
        s0 = math.ceil((2 * G.PI_TRUNC * z / g["h"] - g["BetaS"]) / g["DeltaFai"] - 0.5)
        s1, s2 = s0 - half, s0 + half
        if s1 >= PN or s2 <= 0:
            continue
        for p0 in range(max(s1, 0), min(s2, PN - 1) + 1, step):
            p = torch.arange(p0, min(p0 + step, min(s2, PN - 1) + 1), device=DEV)
            view = (g["BetaS"] + p.double() * g["DeltaFai"]).view(-1, 1, 1)
            c, sn = torch.cos(view), torch.sin(view)
            UU, Yr = -x * c - y * sn, y * c - x * sn
            t1sq = SO * SO - Yr * Yr
            t1 = torch.sqrt(t1sq)
            t2 = z - g["h"] * view / (2 * math.pi)
            U1 = Yr / g["dYL"] + g["YLC"]
            V1 = t2 * (SO * SD) / (UU * t1 + t1sq) / g["dZL"] + g["ZLC"]
            U, V = torch.ceil(U1), torch.ceil(V1)
            ok = (U > 0) & (U < YL) & (V > 0) & (V < ZL)
            du, dv = U - U1, V - V1
            i = (p.view(-1, 1, 1) * ZL + (V.clamp(1, ZL - 1).long() - 1)) * YL + U.clamp(1, YL - 1).long() - 1
            tap = dv * (du * flat[i] + (1 - du) * flat[i + 1]) + (1 - dv) * (du * flat[i + YL] +
                                                                            (1 - du) * flat[i + YL + 1])
            before = p < s0
            d1 = (g["N_pi"] - (s0 - p).double()).long()
            d2 = torch.where(before, (d1 + g["N_pi"]).long(), (d1 - g["N_pi"]).long())
            w1, w2 = w[d1].view(-1, 1, 1), w[d2].view(-1, 1, 1)
            tc = torch.where(before.view(-1, 1, 1), t2 - 0.5, t2 + 0.5)
            m1 = (torch.abs(t2) / torch.abs(t1 + UU)) ** k1
            m2 = (torch.abs(tc) / torch.abs(t1 - UU)) ** k1
            vol[zi] += (torch.where(ok, tap, torch.zeros_like(tap)) * (w1 * m2 / (w2 * m1 + w1 * m2))).sum(0)
    return (vol * g["DeltaFai"]).permute(1, 2, 0).contiguous()


def _exact_chain(s: G.Scan, fan: torch.Tensor) -> torch.Tensor:
    reb = _exact_rebin(fan, s.rebin_args())[s.crop_front:s.views - s.crop_back]
    filt = _exact_filter(reb.transpose(1, 2), s.filter_args())
    del reb
    return _exact_bp(filt, s.bp_geom(), _exact_weights(s))


def _exact_net(p: torch.Tensor, u: torch.Tensor) -> torch.Tensor:
    """u [B][16][H][W] float64 -> the residual channel; p: the parameters, per layer W[co][tap][ci] then b[co]."""
    o, a = 0, u
    for l, (ci, co) in enumerate(zip(CIN, COUT)):
        n = 9 * ci * co
        k = p[o:o + n].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        if l == 7:  # one output channel is used
            return torch.nn.functional.conv2d(a, k[:1], p[o + n:o + n + 1], padding=1)[:, 0]
        a = torch.relu(torch.nn.functional.conv2d(a, k, p[o + n:o + n + co], padding=1))
        o += n + co


def exact(case: dict, seed: int):
    c, kind = case, case["kind"]
    if kind == "dropin":
        s = _scan(c)
        reb = _exact_rebin(_fan(s, seed, 0.0), s.rebin_args())
        filt = _exact_filter(reb[s.crop_front:s.views - s.crop_back].transpose(1, 2), s.filter_args())
        return {"rebinned": reb, "filtered": filt,
                "image": _exact_bp(filt, s.bp_geom(), _exact_weights(s))}
    if kind == "rebin":
        s = _scan(c)
        return _exact_rebin(_fan(s, seed, 0.0), s.rebin_args())
    if kind == "filter":
        return _exact_filter(_rows(c, seed), _filter_scan(c).filter_args())
    if kind == "bp64":
        s = _scan(c)
        return _exact_bp(_bp_input(c, s, seed), s.bp_geom(), _exact_weights(s))
    if kind in ("chain", "host", "slab"):
        s = _scan(c)
        if s.updates() > 1.2e11:  # about half a minute of plain float64
            return None
        return _exact_chain(s, _fan(s, seed, c["I0"]))
    if kind == "batch":
        ss = _batch(c)
        if sum(s.updates() for s in ss) > 1.2e11:
            return None
        return [_exact_chain(s, _fan(s, seed + 1000 * i, c["I0"])) for i, s in enumerate(ss)]
    p = torch.from_numpy(_params(seed)).to(DEV).double()
    if kind == "cnn":
        vol = _volume(c["H"], c["W"], c["ZN"], seed)
        out = torch.empty(vol.shape, dtype=torch.float64, device=DEV)
        for z in range(c["ZN"]):
            at = torch.arange(z - 2, z + 3, device=DEV).clamp(0, c["ZN"] - 1)
            u = torch.zeros((1, 16, c["H"], c["W"]), dtype=torch.float64, device=DEV)
            u[0, :5] = vol[:, :, at].double().permute(2, 0, 1) / G.MU_WATER - 1.0
            out[:, :, z] = vol[:, :, z].double() + G.MU_WATER * _exact_net(p, u)[0]
        return out
    vol, base, target = _train_data(c, seed)
    p.requires_grad_(True)
    px = base.numel()
    loss = 0.0
    for b in range(c["B"]):
        u = torch.zeros((1, 16, c["H"], c["W"]), dtype=torch.float64, device=DEV)
        u[0, :5] = vol[:, :, b:b + 5].double().permute(2, 0, 1) / G.MU_WATER - 1.0
        pred = base[b].double() + G.MU_WATER * _exact_net(p, u)[0]
        e = (((pred - target[b].double()) / G.MU_WATER) ** 2).sum() / px
        e.backward()
        loss += float(e)
    g = p.grad
    step = 1e-4 * g / (g.abs() + 1e-8)  # the first Adam step: both moments are the gradient's own
    return {"loss": loss, "grads": g, "params": (p - step).detach()}
