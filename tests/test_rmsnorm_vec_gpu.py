"""RMSNorm forward and backward against 64 bits at the edges of the lane and vector split."""
import pytest
import torch

from chaoscontrol_b200.kernels import fused_rms_norm

pytestmark = pytest.mark.gpu

EPS = 1e-6


# widths: one vector, below / at / above each lanes-per-row and vectors-per-lane step, and 70 (not a whole number
# of 16-byte vectors: the general kernel); rows: one, fewer than a block's, ragged, more than one row per warp
@pytest.mark.parametrize("R,D", [(1, 8), (3, 64), (33, 72), (17, 128), (4801, 136), (9, 256), (257, 264), (20001, 64),
                                 (70, 512), (7, 520), (100, 768), (41, 1000), (6000, 1024), (65, 1536), (129, 70)])
@pytest.mark.parametrize("shift", [0, 2])
def test_rmsnorm_against_64_bits(R, D, shift):
    """``shift`` > 0 offsets the input by that many elements, so that it is 4- but not 16-byte aligned."""
    g = torch.Generator(device="cuda").manual_seed(R + D)
    x = torch.randn(R * D + shift, generator=g, device="cuda").bfloat16()[shift:].view(R, D).requires_grad_(True)
    w = (torch.rand(D, generator=g, device="cuda") + 0.5).bfloat16().requires_grad_(True)
    go = torch.randn(R, D, generator=g, device="cuda").bfloat16()
    y = fused_rms_norm(x, w, EPS)
    gx, gw = torch.autograd.grad(y, (x, w), go)
    x64, w64, g64 = x.detach().double(), w.detach().double(), go.double()
    inv = torch.rsqrt(x64.square().mean(-1, keepdim=True) + EPS)
    xh, gwt = x64 * inv, g64 * w64
    rnd = 2.0 ** -8                                   # half a unit in the last place of bf16
    fp = (D + 16) * 2.0 ** -24                        # fp32: a row sum and a few products
    assert ((y.double() - xh * w64).abs() <= (rnd + fp) * (xh * w64).abs() + 1e-30).all()
    dot = (gwt * xh).mean(-1, keepdim=True)
    mag = inv * (gwt.abs() + xh.abs() * (gwt * xh).abs().mean(-1, keepdim=True))
    assert ((gx.double() - inv * (gwt - xh * dot)).abs() <= rnd * (inv * (gwt - xh * dot)).abs() + fp * mag).all()
    ref = (g64 * xh).sum(0)
    assert ((gw.double() - ref).abs() <= rnd * ref.abs() + (R + 16) * 2.0 ** -24 * (g64 * xh).abs().sum(0)).all()


# one row more than two rounds of 256-row blocks on 148 SMs, and several rounds; whole vectors and not
@pytest.mark.parametrize("R,D", [(2 * 296 * 256 + 1, 64), (400003, 66)])
def test_rmsnorm_backward_of_many_rows(R, D):
    """The weight gradient over several rounds of blocks against 64 bits (R fp32 products and additions at most, rounded
    to bf16), and the same bits on every run."""
    from chaoscontrol_b200.kernels import fused_rms_norm
    g = torch.Generator(device="cuda").manual_seed(R)
    x = torch.randn(R, D, generator=g, device="cuda").bfloat16()
    w = torch.ones(D, device="cuda").bfloat16().requires_grad_(True)
    go = torch.randn(R, D, generator=g, device="cuda").bfloat16()
    (gw,) = torch.autograd.grad(fused_rms_norm(x, w), (w,), go)
    xd = x.double()
    terms = go.double() * xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6)
    ref, mag = terms.sum(0), terms.abs().sum(0)
    assert ((gw.double() - ref).abs() <= R * 2.0 ** -24 * mag + 2.0 ** -8 * ref.abs()).all()
    assert torch.equal(gw, torch.autograd.grad(fused_rms_norm(x, w), (w,), go)[0])
