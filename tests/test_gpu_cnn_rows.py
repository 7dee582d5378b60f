"""The convolution kernel's shares of output rows and ring of accumulators, and the whole-volume entry, bit for
bit against smaller calls (which the oracle tests cover).

Sizes where the dispatch can go wrong: shares that cross from one image to the next, of more rows than the
ring has accumulators, single rows, column strips with a remainder; volumes whose pixel and slice counts are
not multiples of the residual kernel's 32 x 32 tiles, below and above one chunk.
"""
import numpy as np
import pytest
import torch

from analyticalreconbigpatient_b200 import learned as L
from analyticalreconbigpatient_b200.geometry import MU_WATER
from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(3, 1000, 24), (7, 5, 129), (2, 1, 257), (5, 700, 8)])
def test_forward_does_not_depend_on_the_row_shares(cuda, B, H, W):
    """A batch equals its images alone bit for bit: the shares differ (on 148 SMs 3000 rows are cut into 592
    shares of five or six rows, 1000 rows into 250 of four), the order of every pixel's sums does not."""
    rng = np.random.default_rng(B * 1000 + W)
    u = np.zeros((B, H, W, 16), dtype=np.float32)
    u[..., :5] = rng.standard_normal((B, H, W, 5)).astype(np.float32) * 0.3
    x = torch.from_numpy(u).to(torch.bfloat16).view(torch.int16).to(cuda)
    base = torch.from_numpy((1.0 + rng.standard_normal((B, H, W)) * 0.05).astype(np.float32)).to(cuda)
    net = L.Corrector(C.init_params(B, zero_last=False))
    both = net.forward(x, base)
    alone = torch.cat([net.forward(x[b:b + 1].contiguous(), base[b:b + 1].contiguous()) for b in range(B)])
    net.check()
    net.close()
    assert float((both - base).abs().max()) > 0.0
    assert torch.equal(both, alone)


@pytest.mark.parametrize("H,W,ZN,chunk", [(9, 33, 37, 32), (5, 130, 3, 32), (4, 32, 70, 33), (3, 7, 1, 8)])
def test_volume_equals_its_slices(cuda, H, W, ZN, chunk):
    g = torch.Generator(device=cuda).manual_seed(ZN)
    vol = (MU_WATER * (1.0 + 0.1 * torch.randn((H, W, ZN), device=cuda, generator=g))).contiguous()
    net = L.Corrector(C.init_params(2, zero_last=False))
    out = net.apply_volume(vol, chunk=chunk)
    x = torch.empty((ZN, H, W, 16), dtype=torch.int16, device=cuda)
    net.pack_input(x, vol, 0, ZN)
    ref = net.forward(x, vol.permute(2, 0, 1).contiguous())
    net.check()
    assert torch.equal(out.permute(2, 0, 1), ref)  # the same sums and one fused multiply-add per pixel
    net.close()


def test_volume_under_graph_capture(cuda):
    """The kernels are launched as programmatic dependents of one another: captured and replayed, they wait for
    one another as in a stream (two chunks, so that every buffer is written twice)."""
    g = torch.Generator(device=cuda).manual_seed(9)
    vol = (MU_WATER * (1.0 + 0.1 * torch.randn((40, 150, 12), device=cuda, generator=g))).contiguous()
    net = L.Corrector(C.init_params(3, zero_last=False))
    ref = net.apply_volume(vol, chunk=7).clone()
    out = torch.zeros_like(vol)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        net.apply_volume(vol, out, chunk=7)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    net.check()
    del graph
    net.close()
