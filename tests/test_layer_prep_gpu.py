"""One-launch weight preparation and row statistics against their PyTorch statements."""
import pytest
import torch

from chaoscontrol_b200.ops import trunk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,F", [(8, 8), (64, 128), (72, 40), (384, 768), (512, 2048)])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
def test_layer_fold(D, F, packed, shift):
    """``shift``: a feed-forward weight that is not 16-byte aligned takes the separate launches."""
    g = torch.Generator(device="cuda").manual_seed(D + F)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    Wp, wn1, wn2, log_a = rnd(4 * D, D), rnd(D), rnd(D), rnd(D)
    fc = rnd(F * D + shift)[shift:].view(F, D)
    rest = dict(Wo=rnd(D, D), Wfc=fc, Wproj=rnd(D, F), wn1=wn1, wn2=wn2, log_a=log_a)
    if packed:
        w = trunk.LayerWeights(Wp=Wp, **rest).prepare()
    else:
        w = trunk.LayerWeights.from_parts(*(t.clone() for t in Wp.split(D, 0)), **rest)
    assert torch.equal(w.Wp, Wp)
    assert torch.equal(w.Wp_f, (Wp.float() * wn1.float()).bfloat16())
    assert torch.equal(w.Wfc_f, (fc.float() * wn2.float()).bfloat16())
    assert torch.equal(w.log_a32, log_a.float())


@pytest.mark.parametrize("R,D", [(1, 8), (5, 64), (33, 128), (1001, 192), (7, 256), (300, 520), (9, 1536), (4, 70)])
def test_row_ss(R, D):
    g = torch.Generator(device="cuda").manual_seed(R * D)
    a, b = (torch.randn(R, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    tol = (D + 1) * 2.0 ** -24                       # D products added in fp32, all of one sign
    ref = a.double().square().sum(-1)
    assert ((trunk.row_ss(a).double() - ref).abs() <= tol * ref).all()
    s, ss = trunk.add_row_ss(a, b)
    assert torch.equal(s, a + b)
    ref = (a + b).double().square().sum(-1)
    assert ((ss.double() - ref).abs() <= tol * ref).all()


@pytest.mark.parametrize("B,T,D,F", [(1, 1, 64, 128), (3, 70, 128, 256), (2, 65, 192, 768), (5, 200, 256, 512),
                                     (2, 129, 320, 640), (1, 300, 512, 1024)])
@pytest.mark.parametrize("state", [False, True])
def test_native_layer_matches_separate_launches(B, T, D, F, state, monkeypatch):
    """One native call issues the launches of the step-by-step sequence: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(D + T)
    rnd = lambda *s, k=1.0: (torch.randn(*s, generator=g, device="cuda") * k)
    w = _weights(rnd, D, F)
    x, dx3 = rnd(B * T, D).bfloat16(), rnd(B * T, D).bfloat16()
    h0, dhT = (rnd(B, D), rnd(B, D)) if state else (None, None)
    ss = trunk.row_ss(x)
    res = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(trunk, "_layer_forward_native", lambda *a, **k: None)
        x3, ss3, hT, c = trunk.layer_forward(x, ss, w, B, T, h0)
        assert isinstance(c, trunk.PackedCtx) == native
        x3n, ss3n, hTn, none = trunk.layer_forward(x, ss, w, B, T, h0, save=False)
        assert none is None and torch.equal(x3, x3n) and torch.equal(hT, hTn)
        row = [x3, ss3, hT]
        for dt in (torch.float32, torch.bfloat16):
            dx, gr = trunk.layer_backward(dx3, c, w, B, T, dhT, want_dh0=state, grad_dtype=dt)
            row += [dx, gr.dWp, gr.dWo, gr.dWfc, gr.dWproj, gr.dwn1, gr.dwn2, gr.dlog_a.to(dt)]
            row += [gr.dh0] if state else []
        outs = {k: torch.empty_like(getattr(gr, k), dtype=torch.float32)
                for k in ("dWp", "dWo", "dWfc", "dWproj", "dwn1", "dwn2", "dlog_a")}
        trunk.layer_backward(dx3, c, w, B, T, dhT, outs=outs)
        res.append(row + list(outs.values()))
    assert len(res[0]) == len(res[1])
    for i, (a, b) in enumerate(zip(*res)):
        assert a.dtype == b.dtype and torch.equal(a, b), i


def _weights(rnd, D, F):
    lin = lambda n, k: rnd(n, k, k=k ** -0.5).bfloat16()
    return trunk.LayerWeights(Wp=lin(4 * D, D), Wo=lin(D, D), Wfc=lin(F, D), Wproj=lin(D, F), wn1=rnd(D).bfloat16(),
                          wn2=rnd(D).bfloat16(), log_a=rnd(D).bfloat16()).prepare()


# tokens in one chunk, in sixteen and in seventeen (one warp / all warps of a block), vocabularies on both sides of
# 16-bit keys, and ids outside the table, which no gradient takes
@pytest.mark.parametrize("V,dt", [(31, torch.int64), (33, torch.int32), (32767, torch.int64), (32768, torch.int64),
                                  (40000, torch.int32)])
@pytest.mark.parametrize("D", [256, 512])
def test_embed_bwd_token_widths(V, dt, D):
    g = torch.Generator(device="cuda").manual_seed(V + D)
    runs = [(0, 1), (1, 31), (2, 32 * 14), (5, 32 * 15 + 3), (7, 32 * 16 + 5), (V - 1, 2000), (-3, 40), (V, 33), (V + 70000, 9)]
    tok = torch.cat([torch.full((n,), t, dtype=torch.int64) for t, n in runs]).cuda()
    tok = tok[torch.randperm(tok.numel(), generator=g, device="cuda")].to(dt)
    dx = torch.randn(tok.numel(), D, generator=g, device="cuda").bfloat16()
    got = trunk.embed_bwd(tok, dx, V)
    ok = (tok >= 0) & (tok < V)
    ref = torch.zeros(V, D, dtype=torch.float64, device="cuda").index_add_(0, tok[ok].long(), dx[ok].double())
    mag = torch.zeros(V, D, dtype=torch.float64, device="cuda").index_add_(0, tok[ok].long(), dx[ok].double().abs())
    assert ((got.double() - ref).abs() <= 2048 * 2.0 ** -24 * mag).all()          # at most 2000 fp32 additions a row
    assert torch.equal(got, trunk.embed_bwd(tok, dx, V, sort_cache=torch.sort(tok.long(), stable=True)))


@pytest.mark.parametrize("B,T,D,F", [(1, 3, 64, 128), (5, 200, 256, 512), (2, 129, 320, 640)])
def test_split_projection_gradients(B, T, D, F, monkeypatch):
    """The four projections' gradients as tensors of their own: the rows of the packed one, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s, k=1.0: (torch.randn(*s, generator=g, device="cuda") * k)
    w = _weights(rnd, D, F)
    x, dx3 = rnd(B * T, D).bfloat16(), rnd(B * T, D).bfloat16()
    for native in (True, False):
        if not native:
            monkeypatch.setattr(trunk, "_layer_forward_native", lambda *a, **k: None)
        c = trunk.layer_forward(x, trunk.row_ss(x), w, B, T)[3]
        for dt in (torch.float32, torch.bfloat16):
            one = trunk.layer_backward(dx3, c, w, B, T, grad_dtype=dt)[1]
            four = trunk.layer_backward(dx3, c, w, B, T, grad_dtype=dt, split_wp=True)[1]
            assert [t.dtype for t in four.dWp] == [dt] * 4 and torch.equal(torch.cat(four.dWp), one.dWp)
            assert all(torch.equal(getattr(four, k), getattr(one, k)) for k in ("dWo", "dWfc", "dWproj", "dwn1", "dwn2"))


def test_parameter_gradients_own_their_memory():
    """No two gradients of a block share an allocation or a version counter."""
    from chaoscontrol_b200.models.core_fused import FusedCareSSMBlock
    blk = FusedCareSSMBlock(64).cuda().bfloat16()
    x = torch.randn(2, 9, 64, device="cuda").bfloat16()
    grads = torch.autograd.grad(blk(x).float().square().sum(), list(blk.parameters()))
    assert len({t.untyped_storage().data_ptr() for t in grads}) == len(grads)
    assert all(t.untyped_storage().nbytes() == t.numel() * t.element_size() for t in grads)
    seen = [t._version for t in grads]
    grads[0].zero_()
    assert [t._version for t in grads[1:]] == seen[1:]


# tokens of a join block: 1, 2 and 7 (four blocks to an SM), then 32; the block's share that is not full
@pytest.mark.parametrize("V", [256, 600, 4100, 20000])
def test_embed_bwd_join_blocks(V):
    """Every word joined, long and short runs side by side, against 64-bit sums (at most 9000 fp32 additions a row)."""
    g = torch.Generator(device="cuda").manual_seed(V)
    tok = torch.cat([torch.randint(0, V, (60000,), generator=g, device="cuda"),
                     torch.full((8000,), V - 1, device="cuda"), torch.full((700,), V // 2, device="cuda")])
    dx = torch.randn(tok.numel(), 256, generator=g, device="cuda").bfloat16()
    got = trunk.embed_bwd(tok, dx, V)
    ref = torch.zeros(V, 256, dtype=torch.float64, device="cuda").index_add_(0, tok, dx.double())
    mag = torch.zeros(V, 256, dtype=torch.float64, device="cuda").index_add_(0, tok, dx.double().abs())
    assert ((got.double() - ref).abs() <= 9000 * 2.0 ** -24 * mag).all()
