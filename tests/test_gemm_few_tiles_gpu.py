"""GEMMs that would leave half of the SMs without a 256-wide tile run in 128-wide ones: every epilogue that does."""
import pytest
import torch

from chaoscontrol_b200.ops import _lib
from chaoscontrol_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


# one row to several row tiles; columns below, at and off 128 and 256; a contraction that is not whole k-blocks
@pytest.mark.parametrize("M,N,K", [(1, 136, 64), (127, 256, 72), (130, 384, 256), (512, 1024, 256), (300, 520, 328)])
@pytest.mark.parametrize("epi", [G.EPI_STORE, G.EPI_ROWSCALE, G.EPI_ROWSCALE_SILU, G.EPI_DSILU])
def test_few_tiles_epilogues(M, N, K, epi):
    """Against the fp32 statement: K fp32 additions of bf16 products, then one (SiLU: two) bf16 rounding."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    b_mn = epi == G.EPI_DSILU
    a, b = rnd(M, K).bfloat16(), (rnd(K, N) if b_mn else rnd(N, K)).bfloat16()
    ss = torch.rand(M, generator=g, device="cuda") * K + 0.5
    kw = dict(rowss=ss, inv_dim=1.0 / K, eps=1e-6) if epi != G.EPI_STORE else dict(alpha=0.5, beta=-2.0, cin=rnd(M, N).bfloat16())
    if epi == G.EPI_DSILU:
        kw["r1"] = rnd(M, N).bfloat16()
    c2 = torch.empty(M, N, dtype=torch.bfloat16, device="cuda") if epi == G.EPI_ROWSCALE_SILU else None
    out = G.gemm(a, b, b_mn=b_mn, epi=epi, c2=c2, **kw)
    _lib.assert_ok()
    ref = G.gemm_reference(a, b, b_mn=b_mn, epi=epi, **kw)
    pairs = [(out, ref)] if c2 is None else [(out, ref[0]), (c2, ref[1])]
    for got, want in pairs:
        tol = 2.0 ** -7 * want.abs() + 2e-3 * want.abs().max()      # the sigmoid of the SiLU pair is a fast one (1e-3)
        assert ((got.float() - want).abs() <= tol).all()
    assert torch.equal(out, G.gemm(a, b, b_mn=b_mn, epi=epi, c2=c2, **kw))


@pytest.mark.parametrize("G_,M,N,K", [(1, 256, 256, 256), (5, 72, 264, 136), (16, 256, 256, 256)])
def test_few_tiles_batches_and_layouts(G_, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    for a_mn, b_mn in ((False, False), (False, True), (True, True)):
        a = rnd(G_, K, M) if a_mn else rnd(G_, M, K)
        b = rnd(G_, K, N) if b_mn else rnd(G_, N, K)
        for dt in (torch.bfloat16, torch.float32):
            out = G.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=dt)
            ref = G.gemm_reference(a, b, a_mn=a_mn, b_mn=b_mn)
            _lib.assert_ok()
            tol = (2.0 ** -8 if dt is torch.bfloat16 else 0.0) * ref.abs() + 1e-5 * ref.abs().max()
            assert ((out.float() - ref).abs() <= tol).all()


# contractions just above the line where a weight gradient takes 256-row tiles; ragged columns and k-blocks
@pytest.mark.parametrize("M,N,K", [(1024, 256, 58000), (512, 248, 114000), (256, 256, 227400), (1536, 384, 19003)])
def test_tall_weight_gradient_tiles(M, N, K):
    """dW = A^T B over K rows against 64 bits: K fp32 additions of exact products, spread over the splits."""
    S = G.wgrad_splits(M, N, K)
    assert S == _lib.lib().ccb_gemm_wgrad_splits(M, N, K, 1) and S >= 4
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = (torch.randn(K, n, generator=g, device="cuda").bfloat16() for n in (M, N))
    part = G.gemm(a, b, a_mn=True, b_mn=True, splits=S, out_dtype=torch.float32)
    _lib.assert_ok()
    ref, mag = a.double().t() @ b.double(), a.double().abs().t() @ b.double().abs()
    per = (K + S - 1) // S
    assert ((part.double().sum(0) - ref).abs() <= per * 2.0 ** -24 * mag).all()
    assert torch.equal(part, G.gemm(a, b, a_mn=True, b_mn=True, splits=S, out_dtype=torch.float32))
    assert G.wgrad_splits(M, N, K // 2) == G.pick_splits(M, N, K // 2)      # below the line: 128-row tiles
