"""Block-scaled e4m3 linear: quantisers, GEMM and the autograd layer against fp32 statements."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from chaoscontrol_b200.ops import fp8_block as FB
from chaoscontrol_b200.precision import maybe_promote_linears_to_fused_fp8


def _rel(a, b):
    a, b = a.detach().float().cpu(), b.detach().float().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-12))


def test_quantisers_round_trip_cpu():
    torch.manual_seed(0)
    x = (torch.randn(37, 256) * torch.logspace(-2, 2, 37)[:, None]).bfloat16()
    qr, inv, y = FB.quant_rows(x)
    assert qr.q.shape == (37, 256) and qr.s_t.shape == (2, 37) and inv is None and y is None
    assert _rel(qr.dequant(), x) < 0.04           # e4m3: 3 mantissa bits, per-row-block scale
    w = torch.randn(200, 256).bfloat16()
    q, qt, s = FB.quant_blocks(w)
    assert q.shape == (200, 256) and qt.shape == (256, 200) and s.shape == (2, 2)
    assert torch.equal(q.t().contiguous().view(torch.uint8), qt.view(torch.uint8))
    assert _rel(FB._dequant_t(qt, s, 200, 256).t(), w) < 0.04
    # fused RMSNorm variant
    wn = torch.rand(256) + 0.5
    qn, inv, yn = FB.quant_rows(x, norm_weight=wn, want_normed=True)
    ref = F.rms_norm(x.float(), (256,), eps=1e-6) * wn.bfloat16().float()
    assert _rel(yn, ref) < 1e-2 and _rel(qn.dequant(), ref) < 0.04
    with pytest.raises(ValueError):
        FB.quant_rows(torch.randn(4, 100).bfloat16())


def test_block_gemm_emulation_matches_dequantised_matmul():
    torch.manual_seed(1)
    x, w = torch.randn(50, 384).bfloat16(), (torch.randn(200, 384) * 0.1).bfloat16()
    qa = FB.quant_rows(x)[0]
    q, qt, s = FB.quant_blocks(w)
    out = FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), out_dtype=torch.float32)
    ref = FB.block_linear_reference(x, w)
    assert _rel(out, ref) < 1e-5
    assert _rel(out, x.float() @ w.float().t()) < 0.05


def test_layer_forward_backward_cpu():
    torch.manual_seed(2)
    lin = nn.Linear(256, 128, bias=True)
    layer = FB.BlockFP8Linear.from_nn_linear(lin)
    x = torch.randn(3, 9, 256, requires_grad=True)
    xr = x.detach().clone().requires_grad_(True)
    out = layer(x)
    ref = lin(xr)
    assert out.shape == ref.shape and _rel(out, ref) < 0.06
    g = torch.randn_like(ref)
    out.backward(g)
    gw, gb = lin.weight.grad.clone(), lin.bias.grad.clone()
    lin.weight.grad = lin.bias.grad = None
    ref.backward(g)
    assert _rel(x.grad, xr.grad) < 0.08
    assert _rel(gw, lin.weight.grad) < 0.02 and _rel(gb, lin.bias.grad) < 0.02


def test_promotion_block_mode():
    m = nn.Sequential(nn.Linear(128, 64), nn.Linear(64, 128), nn.Linear(256, 256))
    n = maybe_promote_linears_to_fused_fp8(m, True, scaling="block")
    assert n == 2 and isinstance(m[0], FB.BlockFP8Linear) and isinstance(m[1], nn.Linear)
    with pytest.raises(ValueError):
        maybe_promote_linears_to_fused_fp8(m, True, scaling="nope")


# ---------------------------------------------------------------- GPU
@pytest.mark.gpu
@pytest.mark.parametrize("R,K,N", [(128, 128, 128), (1000, 256, 384), (4096, 512, 256), (777, 2048, 512)])
def test_block_gemm_gpu(R, K, N):
    from chaoscontrol_b200.ops import _lib
    torch.manual_seed(3)
    x = (torch.randn(R, K, device="cuda") * torch.logspace(-1, 1, R, device="cuda")[:, None]).bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    qa, _, _ = FB.quant_rows(x)
    qc, _, _ = FB.quant_rows(x.cpu())
    # the kernel multiplies by a reciprocal, the emulation divides: a code may differ by one step, rarely
    assert (qa.q.cpu().view(torch.uint8) != qc.q.view(torch.uint8)).float().mean() < 2e-3
    assert torch.allclose(qa.s_t.cpu(), qc.s_t, rtol=1e-6)
    q, qt, s = FB.quant_blocks(w)
    q_c, qt_c, s_c = FB.quant_blocks(w.cpu())
    assert (q.cpu().view(torch.uint8) != q_c.view(torch.uint8)).float().mean() < 2e-3
    assert torch.equal(q.t().contiguous().view(torch.uint8), qt.view(torch.uint8))
    assert torch.allclose(s.cpu(), s_c, rtol=1e-6)
    out = FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), out_dtype=torch.float32)
    _lib.assert_ok()
    # exact statement on the kernel's own quantised operands
    ref = FB.QuantRows(qa.q.cpu(), qa.s_t.cpu()).dequant() @ FB._dequant_t(qt.cpu(), s.cpu(), N, K)
    assert _rel(out.cpu(), ref) < 1e-4, _rel(out.cpu(), ref)
    assert _rel(out.cpu(), x.float().cpu() @ w.float().cpu().t()) < 0.05
    bias = torch.randn(N, device="cuda").bfloat16()
    outb = FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), bias=bias)
    assert _rel(outb.cpu(), ref + bias.cpu().float()) < 1e-2
    assert torch.equal(outb, FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), bias=bias))


@pytest.mark.gpu
def test_layer_and_fused_norm_gpu():
    from chaoscontrol_b200.models.core import RMSNorm
    from chaoscontrol_b200.ops import _lib
    torch.manual_seed(4)
    norm = RMSNorm(256).cuda().to(torch.bfloat16)
    with torch.no_grad():
        norm.weight.uniform_(0.5, 1.5)
    lin = nn.Linear(256, 512, bias=False).cuda().to(torch.bfloat16)
    layer = FB.BlockFP8Linear.from_nn_linear(lin)
    x = torch.randn(6, 100, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    xr = x.detach().clone().float().requires_grad_(True)
    norm.emit_fp8_blocks = True
    h = norm(x)
    assert hasattr(h, "_ccb_quant")
    out = layer(h)
    ref = F.linear(F.rms_norm(xr, (256,), eps=norm.eps) * norm.weight.float(), lin.weight.float())
    _lib.assert_ok()
    assert _rel(out, ref) < 0.06
    g = torch.randn_like(ref)
    out.backward(g.to(out.dtype))
    gw, gn = lin.weight.grad.clone().float(), norm.weight.grad.clone().float()
    lin.weight.grad = norm.weight.grad = None
    ref.backward(g)
    _lib.assert_ok()
    assert _rel(x.grad, xr.grad) < 0.08
    assert _rel(gw, lin.weight.grad.float()) < 0.03 and _rel(gn, norm.weight.grad.float()) < 0.05
    # without the producer tag the layer quantises on its own and agrees
    out2 = layer(h.detach().clone())
    assert _rel(out2, out) < 3e-2   # re-quantising the bf16-rounded row moves a few codes


@pytest.mark.gpu
@pytest.mark.parametrize("R,K", [(1, 128), (17, 128), (9, 256), (33, 384), (8, 512), (5, 640), (100, 1024), (7, 2048)])
@pytest.mark.parametrize("norm", [False, True])
def test_quant_rows_segments(R, K, norm):
    """Row quantiser at the edges of its lane and segment split: scales to rounding, codes within one step of the exact
    quotient (e4m3 keeps 3 fraction bits: half a step is 2^-4 of the value, or 2^-10 below the smallest normal)."""
    g = torch.Generator(device="cuda").manual_seed(R + K)
    x = torch.randn(R, K, generator=g, device="cuda").bfloat16()
    w = (torch.rand(K, generator=g, device="cuda") + 0.5).bfloat16() if norm else None
    qa, inv, y = FB.quant_rows(x, norm_weight=w, want_normed=norm)
    v = x.double()
    if norm:
        ri = torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-6)
        v = v * ri * w.double()
        assert torch.allclose(inv.double(), ri.squeeze(1), rtol=1e-5)
        assert ((y.double() - v).abs() <= (2.0 ** -8 + 1e-5) * v.abs()).all()
    scale = v.view(R, K // 128, 128).abs().amax(-1).clamp_min(1e-12) / 448.0
    assert torch.allclose(qa.s_t.double().t(), scale, rtol=2e-5)
    quo = (v.view(R, K // 128, 128) / scale.unsqueeze(-1)).view(R, K)
    assert ((qa.q.double() - quo).abs() <= (2.0 ** -4 + 1e-4) * quo.abs() + 2.0 ** -10 * 1.001).all()


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(8, 128), (130, 128), (129, 100), (256, 200), (384, 264), (7, 9)])
def test_quant_blocks_edges(N, K):
    """Ragged blocks, sizes in eights (vector kernel) and not: the transposed codes are the codes, and each is within
    half a step of the exact quotient."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    q, qt, s = FB.quant_blocks(w)
    assert torch.equal(q.t().contiguous().view(torch.uint8), qt.view(torch.uint8))
    nb, kb = s.shape
    pad = torch.nn.functional.pad(w.double(), (0, kb * 128 - K, 0, nb * 128 - N)).view(nb, 128, kb, 128)
    assert torch.allclose(s.double(), pad.abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0, rtol=1e-6)
    quo = (pad / s.double()[:, None, :, None]).view(nb * 128, kb * 128)[:N, :K]
    assert ((q.double() - quo).abs() <= (2.0 ** -4 + 1e-4) * quo.abs() + 2.0 ** -10 * 1.001).all()


# more tiles than SMs: resident weights.  One, two, four and eight column tiles to a CTA, a last group that is not
# full, a ragged last row and column tile, the deepest resident contraction and the first that streams
@pytest.mark.gpu
@pytest.mark.parametrize("R,K,N", [(19000, 128, 384), (40000, 256, 1024), (20011, 256, 640), (39000, 512, 264),
                                   (26000, 384, 520), (19100, 1024, 256), (19100, 1152, 136)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_block_gemm_resident_weights(R, K, N, out_dtype):
    """Against 64-bit products of the same 8-bit operands: products of e4m3 values are exact in fp32, so the
    difference is K fp32 additions (and the rounding of a bf16 result)."""
    g = torch.Generator(device="cuda").manual_seed(K + N)
    qa, _, _ = FB.quant_rows(torch.randn(R, K, generator=g, device="cuda").bfloat16())
    q, _, s = FB.quant_blocks((torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16())
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    out = FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), bias=bias, out_dtype=out_dtype)
    from chaoscontrol_b200.ops import _lib
    _lib.assert_ok()
    a = (qa.q.double().view(R, K // 128, 128) * qa.s_t.double().t().unsqueeze(-1)).view(R, K)
    nb = s.shape[0]
    pad = torch.nn.functional.pad(q.double(), (0, 0, 0, nb * 128 - N)).view(nb, 128, K // 128, 128)
    w = (pad * s.double()[:, None, :, None]).view(nb * 128, K)[:N]
    ref, mag = a @ w.t() + bias.double(), a.abs() @ w.abs().t() + bias.double().abs()
    rnd = 2.0 ** -8 if out_dtype is torch.bfloat16 else 0.0
    assert ((out.double() - ref).abs() <= (K + 8) * 2.0 ** -24 * mag + rnd * ref.abs()).all()
    assert torch.equal(out, FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1), bias=bias, out_dtype=out_dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("R,N", [(1, 8), (31, 256), (33, 264), (4097, 1024), (70001, 136), (50, 12)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_bias_gradient_column_sums(R, N, dt):
    """R fp32 additions a column in a fixed order, rounded once (N = 12: the PyTorch statement)."""
    g = torch.Generator(device="cuda").manual_seed(R + N)
    x = torch.randn(R, N, generator=g, device="cuda").bfloat16()
    got = FB._bias_grad(x, dt)
    ref, mag = x.double().sum(0), x.double().abs().sum(0)
    rnd = 2.0 ** -8 if dt is torch.bfloat16 else 0.0
    assert got.dtype == dt and ((got.double() - ref).abs() <= (R + 1) * 2.0 ** -24 * mag + rnd * ref.abs()).all()
    assert torch.equal(got, FB._bias_grad(x, dt))


@pytest.mark.gpu
@pytest.mark.parametrize("R,N", [(8000, 512), (64095, 1024), (2001, 128)])
def test_bias_gradient_error_is_no_larger_than_that_of_the_fp32_reduction(R, N):
    """fp32 column sums against 64 bits, next to PyTorch's reduction of an fp32 copy, which they take the place of."""
    x = torch.randn(R, N, generator=torch.Generator(device="cuda").manual_seed(R), device="cuda").bfloat16()
    ref = x.double().sum(0)
    rms = lambda s: float((s.double() - ref).square().mean().sqrt())
    assert rms(FB._bias_grad(x, torch.float32)) <= rms(x.float().sum(0))


def _plan(M, N, K, sms=148):
    from chaoscontrol_b200.ops import _lib
    if not _lib._LIB_PATH.exists():
        pytest.skip("the kernel library is not built")
    return int(_lib.lib().ccb_fp8_block_plan(M, N, K, sms))


def _work(M, N, K, nt, sms=148):
    """Tiles of the busiest CTA: of the resident kernel with ``nt`` column tiles to a CTA, of the streaming kernel."""
    tm, tn = -(-M // 128), -(-N // 128)
    if nt == 0:
        return -(-tm * tn // sms)
    return -(-tm // min(sms // -(-tn // nt), tm)) * min(nt, tn)


@pytest.mark.parametrize("K", [128, 256, 384, 512, 640, 1024, 1152])
def test_resident_weights_keep_the_sms_busy(K):
    """Over the sizes of a layer and far beyond: the resident kernel is taken only while its busiest CTA has little more
    to do than the streaming kernel's."""
    limit = 7 / 6 if K == 128 else (4 / 3 if K <= 512 else 17 / 16)
    taken = 0
    for M in (100, 2560, 9000, 18944, 20000, 65536, 300001):
        for N in list(range(128, 2049, 128)) + [136, 2500, 3200, 6400, 9600, 12800, 18944, 19200, 50304]:
            nt = _plan(M, N, K)
            if nt:
                taken += 1
                assert K <= 1024 and nt * (K // 128) <= 8 and (nt == 1 or K <= 512)
                assert _work(M, N, K, nt) <= limit * _work(M, N, K, 0), (M, N)
    assert (taken > 0) == (K <= 1024)


@pytest.mark.parametrize("M,N,K,resident", [(65536, 1024, 256, True), (65536, 1024, 1024, True), (65536, 896, 1024, True),
                                            (65536, 640, 384, True), (65536, 9600, 1024, False), (65536, 6400, 1024, False),
                                            (65536, 19200, 512, False), (65536, 18944, 512, True), (128, 1024, 256, False)])
def test_resident_weights_at_measured_sizes(M, N, K, resident):
    assert (_plan(M, N, K) > 0) == resident


# four column tiles to a CTA with a last group of three, two with a last group of one, eight; ragged last row and column
# tiles; wide results that stream
@pytest.mark.gpu
@pytest.mark.parametrize("R,K,N,nt", [(37838, 256, 888, 4), (37627, 512, 520, 2), (75700, 128, 1024, 8),
                                      (2500, 1024, 9600, 0), (2500, 512, 19000, 0)])
def test_block_gemm_column_groups(R, K, N, nt):
    """As the resident-weight test above, against 64-bit products."""
    from chaoscontrol_b200.ops import _lib
    assert _plan(R, N, K, _lib.lib().ccb_num_sms()) == nt
    g = torch.Generator(device="cuda").manual_seed(K + N)
    qa, _, _ = FB.quant_rows(torch.randn(R, K, generator=g, device="cuda").bfloat16())
    q, _, s = FB.quant_blocks((torch.randn(N, K, generator=g, device="cuda") * 0.1).bfloat16())
    out = FB.block_gemm(qa, q, s, sb_strides=(s.shape[1], 1))
    _lib.assert_ok()
    a = (qa.q.double().view(R, K // 128, 128) * qa.s_t.double().t().unsqueeze(-1)).view(R, K)
    nb = s.shape[0]
    pad = torch.nn.functional.pad(q.double(), (0, 0, 0, nb * 128 - N)).view(nb, 128, K // 128, 128)
    w = (pad * s.double()[:, None, :, None]).view(nb * 128, K)[:N]
    ref, mag = a @ w.t(), a.abs() @ w.abs().t()
    assert ((out.double() - ref).abs() <= (K + 8) * 2.0 ** -24 * mag + 2.0 ** -8 * ref.abs()).all()
