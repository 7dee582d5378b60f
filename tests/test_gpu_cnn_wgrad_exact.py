"""The weight-gradient contractions by themselves: a network whose layers pass BF16 values on unchanged (one weight of
1 per channel, exact sums in FP32), so that every layer's operands are known bit for bit and its gradients can be
compared with a float64 contraction of the same operands. All terms are positive, so nothing cancels.

Tolerance: a tensor-core accumulator truncates; over 32 steps (four tiles of eight 16-pixel steps) of a sum that
grows evenly from 0, that is at most 32 x 2^-23 / 2 = 1.9e-6 of the sum. The FP32 sums after it round to nearest
(some 16 flushes and 148 CTAs: below 3e-7). 2.5e-6 together; an accumulator left to run over a CTA's whole share of the
largest image here (55 tiles) loses 1.1e-5."""
import numpy as np
import pytest
import torch

from analyticalreconbigpatient_b200 import learned as L

pytestmark = pytest.mark.gpu
TOL = 2.5e-6


def _pass_on_params():
    """Layer 1 copies its 16 inputs to channels 0..15 and, from the pixel up and left, to 16..31; layers 2..7 copy;
    layer 8 adds the channels' values times powers of two. W[co][tap][ci], then the biases."""
    parts = []
    for l, (ci, co) in enumerate(zip(L.CIN, L.COUT)):
        w = np.zeros((co, 9, ci), dtype=np.float32)
        for c in range(co):
            if l == 0:
                w[c, 4 if c < 16 else 0, c % 16] = 1.0
            elif l < 7:
                w[c, 4, c] = 1.0
        if l == 7:
            w[0, 4, :] = 2.0 ** -(np.arange(ci) % 4)
        parts += [w.ravel(), np.zeros(co, dtype=np.float32)]
    return np.concatenate(parts)


def gradient_errors(cuda, B, H, W, seed):
    """Relative L2 error of each layer's weight and bias gradients."""
    g = torch.Generator(device=cuda).manual_seed(seed)
    u = torch.randint(1, 128, (B, H, W, 16), device=cuda, generator=g).float() / 64  # eight significant bits
    base = torch.randint(0, 64, (B, H, W), device=cuda, generator=g).float() / 64
    act = torch.zeros((B, H, W, 32), device=cuda)
    act[..., :16] = u
    act[:, 1:, 1:, 16:] = u[:, :-1, :-1, :]
    w8 = (2.0 ** -(torch.arange(32, device=cuda) % 4)).float()
    resid = (act * w8).sum(-1)  # exact: multiples of 2^-9 below 2^6
    target = base - torch.randint(1, 64, (B, H, W), device=cuda, generator=g).float() / 64  # every error is positive
    net = L.Corrector(_pass_on_params())
    net.train_step(u.to(torch.bfloat16).view(torch.int16), base, target, lr=0.0, mu_w=1.0)
    got = net.grads()
    net.check()
    net.close()
    # output gradient: two FP32 operations and the rounding to BF16, as the kernel's
    d = (float(np.float32(2.0) / np.float32(B * H * W)) * (base + resid - target)).to(torch.bfloat16).double()
    d7 = d[..., None] * w8.double() * (act > 0)
    errors, o = [], 0
    refs = {}
    for l, (ci, co) in enumerate(zip(L.CIN, L.COUT)):
        key = (ci, co)
        if key not in refs:
            x = torch.nn.functional.pad(u if l == 0 else act, (0, 0, 1, 1, 1, 1))
            grad = torch.zeros((B, H, W, co), device=cuda, dtype=torch.float64)
            if l == 7:
                grad[..., 0] = d
            else:
                grad[:] = d7
            ref = torch.zeros((co, 9, ci), dtype=torch.float64, device=cuda)
            for b in range(B):
                gt = grad[b].reshape(-1, co).T
                for tap in range(9):
                    ref[:, tap] += gt @ x[b, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W].reshape(-1, ci).double()
            refs[key] = (ref.cpu().numpy(), grad.sum((0, 1, 2)).cpu().numpy())
        rw, rb = refs[key]
        n = 9 * ci * co
        w, bias = got[o:o + n].reshape(co, 9, ci).astype(np.float64), got[o + n:o + n + co].astype(np.float64)
        errors.append((np.linalg.norm(w - rw) / np.linalg.norm(rw), np.linalg.norm(bias - rb) / np.linalg.norm(rb)))
        o += n + co
    return errors


@pytest.mark.parametrize("B,H,W", [(1, 3, 5), (2, 37, 200), (1, 64, 129), (3, 301, 500), (8, 512, 512)])
def test_weight_gradients_of_known_operands(cuda, B, H, W):
    errors = gradient_errors(cuda, B, H, W, H)
    assert all(w < TOL and b < TOL for w, b in errors), errors


def test_sums_of_a_cta_are_added_once(cuda):
    """The last additions, one per CTA and one after another in FP32, each round by 0.3 of half a unit of the sum so
    far on average: 2.5e-8 sqrt(N / 3) of the whole for N additions. 64 CTAs (32 pairs of rows, two strips) give
    1.15e-7 for the 9216 weights of a layer together, two additions per CTA 1.63e-7: the limit is 1.4e-7. 148 CTAs
    give 1.8e-7 for the biases, of which few differ, so the limit is 6e-7, over three times that; with one per warp
    (eight per CTA) they are expected 5e-7 off and come out beyond it in one of eight layers."""
    for seed in (1, 2):
        assert all(w < 1.4e-7 for w, _ in gradient_errors(cuda, 1, 64, 129, seed)[1:7])
        assert all(b < 6e-7 for _, b in gradient_errors(cuda, 8, 512, 512, seed))
