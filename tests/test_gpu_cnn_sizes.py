"""The correction network at sizes its launches and buffers could limit: images of more rows than a grid holds, and the
device memory a network takes for widths around its 128-pixel tiles, inputs on any byte boundary."""
import pytest
import torch

from analyticalreconbigpatient_b200 import _lib, learned as L
from analyticalreconbigpatient_b200.geometry import MU_WATER
from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu


def test_volume_of_more_rows_than_a_grid(cuda):
    """Bit for bit the slices' own corrections (the entry that takes the network's input)."""
    H, W, ZN = 65535 + 6, 3, 2
    g = torch.Generator(device=cuda).manual_seed(5)
    vol = (MU_WATER * (1.0 + 0.1 * torch.randn((H, W, ZN), device=cuda, generator=g))).contiguous()
    net = L.Corrector(C.init_params(2, zero_last=False))
    out = net.apply_volume(vol)
    x = torch.empty((ZN, H, W, 16), dtype=torch.int16, device=cuda)
    net.pack_input(x, vol, 0, ZN)
    ref = net.forward(x, vol.permute(2, 0, 1).contiguous())
    net.check()
    net.close()
    assert torch.equal(out.permute(2, 0, 1), ref)
    assert float((out - vol).abs().max()) > 0.0


@pytest.mark.parametrize("W", [16, 64, 130])
@pytest.mark.parametrize("call", ["forward", "train_step", "apply_volume"])
def test_buffers_are_no_larger_than_unpadded_planes(cuda, call, W):
    """At most 304 channels of two bytes per pixel, the input's 16, seven activations and two gradients of 32, in
    rows of two pixels more than the image's: narrow images must not be padded to whole tiles in memory."""
    H = (1 << 22) // W
    base = torch.full((1, H, W), MU_WATER, device=cuda)
    vol = base.reshape(H, W, 1).contiguous()
    out = torch.empty_like(vol)
    x = torch.zeros((1, H, W, 16), dtype=torch.int16, device=cuda)
    small = L.Corrector(seed=1)  # the kernels' own first-launch memory is not the network's
    for n in (1, 2):
        small.forward(x[:, :n].contiguous(), base[:, :n].contiguous())
        small.train_step(x[:, :n].contiguous(), base[:, :n].contiguous(), base[:, :n].contiguous(), lr=0.0)
        small.apply_volume(vol[:n].contiguous())
    small.close()
    net = L.Corrector(seed=1)
    pred = torch.empty_like(base)  # what forward() allocates for its result comes from torch's pool
    del pred
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    if call == "forward":
        net.forward(x, base)
    elif call == "train_step":
        net.train_step(x, base, base, lr=0.0)
    else:
        net.apply_volume(vol, out)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    net.check()
    net.close()
    assert 0 < used <= 304 * 2 * H * (W + 2) + (32 << 20), used / (H * W)


@pytest.mark.parametrize("shift", [1, 2, 3, 8])
def test_input_on_any_byte_boundary(cuda, shift):
    """forward() takes an input that starts anywhere, as the copy it is brought in by may."""
    B, H, W = 2, 3, 131
    g = torch.Generator(device=cuda).manual_seed(shift)
    x = (0.3 * torch.randn((B, H, W, 16), device=cuda, generator=g)).to(torch.bfloat16).view(torch.int16)
    base = torch.full((B, H, W), MU_WATER, device=cuda)
    raw = torch.zeros(x.numel() * 2 + 16, dtype=torch.uint8, device=cuda)
    raw[shift:shift + x.numel() * 2] = x.reshape(-1).view(torch.uint8)
    net = L.Corrector(C.init_params(3, zero_last=False))
    ref = net.forward(x, base)
    out = torch.full_like(base, float("nan"))
    _lib.check(_lib.load().hr_cnn_forward(net._net, out.data_ptr(), raw.data_ptr() + shift, base.data_ptr(), H * W, 1,
                                          B, H, W, MU_WATER, torch.cuda.current_stream().cuda_stream))
    net.check()
    net.close()
    assert torch.equal(out, ref)
