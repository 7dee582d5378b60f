"""The correction network at sizes its launches and buffers could limit: images of more rows than a grid holds."""
import pytest
import torch

from analyticalreconbigpatient_b200 import learned as L
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
