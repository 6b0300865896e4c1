"""Fused LM-head kernels (lse / train / dW) vs the fp32 PyTorch statement."""
import pytest
import torch

from chaoscontrol_b200.ops import _lib
from chaoscontrol_b200.ops import lm_head as LH

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[(4, 0), (2, 0), (2, 1), (4, 1)], ids=["epi16warps", "epi8warps", "epi8warps-deep", "epi16warps-deep"])
def epilogue_parts(request):
    """Run a test with both widths of the fused head's epilogue (sixteen or eight warps) and with
    both ring layouts of the one-sweep training kernel (two stages with X in shared memory, three
    stages with X in tensor memory)."""
    L = _lib.lib()
    parts, deep = request.param
    old = L.ccb_lmhead_epilogue_parts(parts)
    old_deep = L.ccb_lmhead_deep_ring(deep)
    yield request.param
    L.ccb_lmhead_epilogue_parts(old)
    L.ccb_lmhead_deep_ring(old_deep)


def _mk(R, V, seed=0, wscale=0.08):
    torch.manual_seed(seed)
    x = torch.randn(R, 256, device="cuda").bfloat16()
    W = (torch.randn(V, 256, device="cuda") * wscale).bfloat16()
    t = torch.randint(0, V, (R,), device="cuda")
    ss = (x.float() ** 2).sum(-1)
    return x, W, t, ss


@pytest.mark.parametrize("R,V", [(128, 128), (256, 512), (1000, 1024), (4096, 16384)])
def test_lmhead_lse(R, V, epilogue_parts):
    x, W, t, ss = _mk(R, V)
    loss, lse = LH.lm_head_lse(x, ss, W, t)
    _lib.assert_ok()
    rl, rlse, _, _ = LH.lm_head_reference(x, ss, W, t, want_grads=False)
    assert torch.allclose(lse, rlse, rtol=1e-3, atol=2e-2), (lse - rlse).abs().max()
    assert torch.allclose(loss, rl, rtol=1e-3, atol=3e-2), (loss - rl).abs().max()


@pytest.mark.parametrize("R,V,chunks,norm", [(128, 128, 1, True), (384, 512, 3, True),
                                             (1000, 1024, 2, False), (2048, 16384, 4, True)])
def test_lmhead_train(R, V, chunks, norm, epilogue_parts):
    x, W, t, ss = _mk(R, V, seed=1)
    w = torch.rand(R, device="cuda")
    gscale = 1.0 / R
    rowss = ss if norm else None
    loss, lse, dX, part = LH.lm_head_train(x, rowss, W, t, gscale=gscale, rowweight=w,
                                           row_chunks=chunks)
    _lib.assert_ok()
    rl, rlse, rdX, rdW = LH.lm_head_reference(x, rowss, W, t, gscale=gscale, rowweight=w)
    assert torch.allclose(lse, rlse, rtol=1e-3, atol=2e-2)
    assert torch.allclose(loss, rl, rtol=1e-3, atol=3e-2), (loss - rl).abs().max()
    sx = rdX.abs().max().item()
    assert (dX.float() - rdX).abs().max().item() <= 0.03 * sx + 1e-7, \
        ((dX.float() - rdX).abs().max().item(), sx)
    dW = part.sum(0)
    sw = rdW.abs().max().item()
    assert (dW - rdW).abs().max().item() <= 0.03 * sw + 1e-7, ((dW - rdW).abs().max().item(), sw)


def test_lmhead_train_deterministic(epilogue_parts):
    x, W, t, ss = _mk(1024, 2048, seed=2)
    a = LH.lm_head_train(x, ss, W, t, gscale=1e-3)
    b = LH.lm_head_train(x, ss, W, t, gscale=1e-3)
    _lib.assert_ok()
    for u, v in zip(a, b):
        assert torch.equal(u, v)


def _mk_d(R, V, D, seed=0, wscale=0.08):
    torch.manual_seed(seed)
    x = torch.randn(R, D, device="cuda").bfloat16()
    W = (torch.randn(V, D, device="cuda") * wscale).bfloat16()
    t = torch.randint(0, V, (R,), device="cuda")
    return x, W, t, (x.float() ** 2).sum(-1)


@pytest.mark.parametrize("R,V,D,norm", [(300, 1000, 512, True), (1024, 16384, 512, True),
                                        (515, 520, 128, False), (20000, 2048, 384, True)])
def test_lmhead_general_dims(R, V, D, norm):
    """Model dims other than 256 go through the GEMM-epilogue LM head."""
    x, W, t, ss = _mk_d(R, V, D, seed=3)
    assert not LH.fused_supported(x, W) and LH.general_supported(x, W)
    rowss = ss if norm else None
    loss, lse = LH.lm_head_lse(x, rowss, W, t)
    rl, rlse, _, _ = LH.lm_head_reference(x, rowss, W, t, want_grads=False)
    _lib.assert_ok()
    assert torch.allclose(lse, rlse, rtol=1e-3, atol=2e-2), (lse - rlse).abs().max()
    assert torch.allclose(loss, rl, rtol=1e-3, atol=3e-2), (loss - rl).abs().max()
    w = torch.rand(R, device="cuda")
    gscale = 1.0 / R
    loss2, lse2, dX, part = LH.lm_head_train(x, rowss, W, t, gscale=gscale, rowweight=w)
    _lib.assert_ok()
    _, _, rdX, rdW = LH.lm_head_reference(x, rowss, W, t, gscale=gscale, rowweight=w)
    assert torch.allclose(loss2, rl, rtol=1e-3, atol=3e-2), (loss2 - rl).abs().max()
    assert torch.equal(lse2, lse)
    sx = rdX.abs().max().item()
    assert (dX.float() - rdX).abs().max().item() <= 0.03 * sx + 1e-7, ((dX.float() - rdX).abs().max().item(), sx)
    dW = part.sum(0)
    sw = rdW.abs().max().item()
    assert (dW - rdW).abs().max().item() <= 0.03 * sw + 1e-7, ((dW - rdW).abs().max().item(), sw)
    again = LH.lm_head_train(x, rowss, W, t, gscale=gscale, rowweight=w)
    for u, v in zip((loss2, lse2, dX, part), again):
        assert torch.equal(u, v)


@pytest.mark.parametrize("wscale,peak", [(0.08, 0.0), (1.5, 0.0), (0.3, 40.0)])
def test_lmhead_one_sweep_matches_two_sweeps_and_the_reference(wscale, peak, epilogue_parts):
    """The single-sweep training kernel (fixed per-row reference instead of the true row maximum)
    against the two-sweep kernel and the fp32 statement: ordinary logits, logits spread over tens of
    nats, and a target column that towers over the row's first 32 logits."""
    R, V = 1024, 4096
    x, W, t, ss = _mk(R, V, seed=3, wscale=wscale)
    if peak:
        # make each row's target logit ~`peak` nats larger than the rest: align W[t] with x
        xn = torch.nn.functional.normalize(x.float(), dim=-1)
        Wf = W.float()
        Wf[t] = Wf[t] + xn * (peak / 16.0)
        W = Wf.bfloat16()
    w = torch.rand(R, device="cuda") + 0.5
    kw = dict(gscale=1.0 / R, rowweight=w, row_chunks=2)
    l1, lse1, dX1, p1 = LH.lm_head_train(x, ss, W, t, one_sweep=True, **kw)
    l2, lse2, dX2, p2 = LH.lm_head_train(x, ss, W, t, one_sweep=False, **kw)
    _lib.assert_ok()
    rl, rlse, rdX, rdW = LH.lm_head_reference(x, ss, W, t, gscale=1.0 / R, rowweight=w)
    assert torch.isfinite(dX1.float()).all() and torch.isfinite(lse1).all()
    assert torch.allclose(lse1, rlse, rtol=1e-3, atol=3e-2), (lse1 - rlse).abs().max()
    assert torch.allclose(l1, rl, rtol=2e-3, atol=5e-2), (l1 - rl).abs().max()

    def rel(a, b):
        return float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12))
    assert rel(dX1, rdX) < 2e-2 and rel(dX1, dX2) < 2e-2, (rel(dX1, rdX), rel(dX1, dX2))
    assert rel(p1.sum(0), rdW) < 2e-2 and rel(p1.sum(0), p2.sum(0)) < 1e-2


@pytest.mark.parametrize("R,D,V", [(4096 + 77, 256, 512), (130, 256, 1024), (301, 384, 640)])
@pytest.mark.parametrize("up", [1.0, -0.37, 3e-6, 0.0])
def test_upstream_gradient_scales_inside_the_kernels(R, D, V, up):
    """Both gradients of ``up * loss`` against autograd through 32-bit logits.  The gradient tile of a row is rounded to
    bf16 once (relative 2^-8 an element) and so are the results; the sums over the vocabulary and the rows average the
    first out, so the 2-norm differs by less than 1e-2."""
    from chaoscontrol_b200.kernels import fused_linear_cross_entropy
    g = torch.Generator(device="cuda").manual_seed(R)
    x = torch.randn(R, D, generator=g, device="cuda").bfloat16().requires_grad_(True)
    W = (torch.randn(V, D, generator=g, device="cuda") * 0.1).bfloat16().requires_grad_(True)
    t = torch.randint(0, V, (R,), generator=g, device="cuda")
    gx, gW = torch.autograd.grad(fused_linear_cross_entropy(x, W, t, reduction="sum") * up, (x, W))
    (only,) = torch.autograd.grad(fused_linear_cross_entropy(x, W.detach(), t, reduction="sum") * up, (x,))
    xf, Wf = x.detach().float().requires_grad_(True), W.detach().float().requires_grad_(True)
    rx, rW = torch.autograd.grad(torch.nn.functional.cross_entropy(xf @ Wf.t(), t, reduction="sum") * up, (xf, Wf))
    assert torch.equal(only, gx)
    for a, b in ((gx, rx), (gW, rW)):
        assert (a.float() - b).norm() <= 1e-2 * b.norm()


@pytest.mark.parametrize("nparts", [1, 15, 16, 17, 64, 65, 130])
@pytest.mark.parametrize("M", [1, 31, 33, 300])
def test_lse_combine_partials(nparts, M):
    """Merging (max, sum) pairs, empty ones (sum 0 under any maximum) among them, against 64 bits: each merge rounds the
    sum and a power of two, and log2 of the sum is taken once."""
    g = torch.Generator(device="cuda").manual_seed(nparts * M)
    part = torch.stack([torch.randn(nparts, M, generator=g, device="cuda") * 30,
                        torch.rand(nparts, M, generator=g, device="cuda") * 100 + 1e-3], -1).contiguous()
    if nparts > 1:
        part[::3, ::2, 1] = 0.0
        part[::3, ::2, 0] = 1e4
        part[1, :, 1] = 5.0                      # never all empty
    zt = torch.randn(M, generator=g, device="cuda")
    lse, loss = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
    _lib.check(_lib.lib().ccb_lse_combine(part.data_ptr(), nparts, M, zt.data_ptr(), lse.data_ptr(), loss.data_ptr(),
                                          _lib.stream_ptr()), "lse_combine")
    p64 = part.double()
    ln2 = 0.6931471805599453
    z = torch.where(p64[..., 1] > 0, p64[..., 0] * ln2 + p64[..., 1].clamp_min(1e-300).log(), float("-inf"))
    ref = torch.logsumexp(z, 0)
    tol = (nparts + 8) * 2.0 ** -23 + 2.0 ** -23 * ref.abs()
    assert ((lse.double() - ref).abs() <= tol).all()
    assert ((loss.double() - (ref - zt.double())).abs() <= tol + 2.0 ** -23 * zt.abs().double()).all()


# row tiles: fewer than SMs, one more, several waves; vocabularies whose tiles divide the shares and not; a last row
# tile that is not full
@pytest.mark.parametrize("R,V", [(4096, 4096), (9000, 4352), (18944 + 60, 4096), (18944 + 128, 2304), (40000, 2560)])
@pytest.mark.parametrize("norm", [False, True])
def test_evenly_dealt_sweeps_match_whole_tiles(R, V, norm):
    """The split walk against whole row tiles, kernel by kernel.  lse, loss and entropy differ by the order of fp32
    sums; dX by that and one bf16 rounding."""
    x, W, t, ss = _mk_d(R, V, 256, wscale=0.3, seed=7)
    rowss = ss if norm else None
    w = torch.rand(R, device="cuda")
    L = _lib.lib()
    assert L.ccb_lmhead_work(R, V, 256, 1) > 0
    res = []
    real = LH._split_work
    for split in (True, False):
        LH._split_work = real if split else (lambda *a: None)
        try:
            row = list(LH.lm_head_lse(x, rowss, W, t, want_entropy=True))
            for kw in (dict(lse=row[1]), dict(one_sweep=True)):
                l, z, dX, _ = LH.lm_head_train(x, rowss, W, t, gscale=0.5, rowweight=w, want_dw=False, **kw)
                row += [l, z, dX]
        finally:
            LH._split_work = real
        res.append(row)
    _lib.assert_ok()
    for i, (a, b) in enumerate(zip(*res)):
        a, b = a.float(), b.float()
        if a.dim() == 1:
            assert (a - b).abs().max().item() <= 2e-4 * (1.0 + b.abs().max().item()), i
        else:
            assert (a - b).abs().max().item() <= 2.0 ** -7 * b.abs().max().item(), i
            assert (a - b).norm() <= 2e-3 * b.norm(), i
    again = LH.lm_head_train(x, rowss, W, t, gscale=0.5, rowweight=w, want_dw=False, one_sweep=True)
    assert torch.equal(again[2], res[0][8])


@pytest.mark.parametrize("nparts", [2, 17, 130])
@pytest.mark.parametrize("bad", [(float("inf"), float("nan")), (3.0, float("nan")), (float("-inf"), float("nan"))])
def test_lse_combine_lets_a_broken_partial_through(nparts, bad):
    """A tile that held an infinite or NaN logit arrives with a NaN sum: the row's lse and loss are NaN, wherever the
    partial stands and whether or not the others are empty; rows without one are untouched."""
    M = nparts + 40
    g = torch.Generator(device="cuda").manual_seed(nparts)
    part = torch.stack([torch.randn(nparts, M, generator=g, device="cuda"),
                        torch.rand(nparts, M, generator=g, device="cuda") + 0.5], -1).contiguous()
    clean = part.clone()
    for i in range(nparts):
        part[i, i] = torch.tensor(bad)           # row i: the i-th partial
    part[:, nparts, 1] = 0.0                     # only the broken one is not empty
    part[nparts // 2, nparts] = torch.tensor(bad)
    zt = torch.zeros(M, device="cuda")

    def combine(p):
        lse, loss = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
        _lib.check(_lib.lib().ccb_lse_combine(p.data_ptr(), nparts, M, zt.data_ptr(), lse.data_ptr(), loss.data_ptr(),
                                              _lib.stream_ptr()), "lse_combine")
        return lse, loss
    for a, b in zip(combine(part), combine(clean)):
        assert a[: nparts + 1].isnan().all()
        assert b.isfinite().all() and torch.equal(a[nparts + 1:], b[nparts + 1:])


@pytest.mark.parametrize("R,D", [(511, 256), (300, 384)])
def test_infinite_logits_reach_the_loss(R, D):
    """Scoring with a damaged head: a vocabulary row whose logit is +inf makes every loss non-finite, a whole tile of
    -inf logits has probability zero and changes nothing else (against 32-bit logits of the other columns; tolerance of
    the scoring tests)."""
    V = 1024
    g = torch.Generator(device="cuda").manual_seed(D)
    x = (torch.rand(R, D, generator=g, device="cuda") + 0.5).bfloat16()          # positive: the overflow has one sign
    W = (torch.randn(V, D, generator=g, device="cuda") * 0.05).bfloat16()
    t = torch.randint(0, 256, (R,), generator=g, device="cuda")
    up, down = W.clone(), W.clone()
    up[700] = 3e38
    down[256:512] = -3e38
    loss, lse = LH.lm_head_lse(x, None, up, t)
    assert not loss.isfinite().any() and not lse.isfinite().any()
    loss, lse = LH.lm_head_lse(x, None, down, t)
    _lib.assert_ok()
    keep = torch.cat([W[:256], W[512:]])
    rl, rlse, _, _ = LH.lm_head_reference(x, None, keep, t, want_grads=False)
    assert torch.allclose(lse, rlse, rtol=1e-3, atol=2e-2) and torch.allclose(loss, rl, rtol=1e-3, atol=3e-2)


@pytest.mark.parametrize("R,D", [(1020, 256), (4080, 256), (1020, 384), (4080, 384)])
def test_mean_loss_gradients_keep_their_precision_at_every_row_count(R, D):
    """1/1020 and 1/4080 lie almost half a unit in the last place from the next bf16 value.  Rounding a result to bf16
    leaves a 2-norm error of about 0.42 * 2^-8 = 0.0016 (uniform in the unit, mantissas spread over their logarithm), the
    gradient tile's own rounding a little more; a scale rounded in every row alike would add 0.0035."""
    from chaoscontrol_b200.kernels import fused_linear_cross_entropy
    V = 2048
    g = torch.Generator(device="cuda").manual_seed(R + D)
    x = torch.randn(R, D, generator=g, device="cuda").bfloat16().requires_grad_(True)
    W = (torch.randn(V, D, generator=g, device="cuda") * 0.1).bfloat16().requires_grad_(True)
    t = torch.randint(0, V, (R,), generator=g, device="cuda")
    gx, gW = torch.autograd.grad(fused_linear_cross_entropy(x, W, t), (x, W))
    xd, Wd = x.detach().double().requires_grad_(True), W.detach().double().requires_grad_(True)
    rx, rW = torch.autograd.grad(torch.nn.functional.cross_entropy(xd @ Wd.t(), t), (xd, Wd))
    for a, b in ((gx, rx), (gW, rW)):
        assert float((a.double() - b).norm() / b.norm()) <= 0.0025


@pytest.mark.parametrize("R,D,norm", [(300, 256, True), (300, 384, True), (300, 384, False), (4096 + 77, 256, True),
                                      (18944 + 60, 256, True)])
def test_device_scale_is_applied_to_dx_and_left_out_of_the_partials(R, D, norm):
    """``gscale_dev`` against the same call without it: a power of two commutes with every rounding, so dX is exactly that
    much larger; the weight partials are the same bits.  Every path: few rows, general, whole row tiles, split sweep."""
    x, W, t, ss = _mk_d(R, 1024, D, wscale=0.3, seed=11)
    rowss = ss if norm else None
    _, lse = LH.lm_head_lse(x, rowss, W, t)
    up = torch.full((), 0.25, device="cuda")
    for kw in (dict(lse=lse), dict()):
        a = LH.lm_head_train(x, rowss, W, t, gscale=0.5, **kw)
        b = LH.lm_head_train(x, rowss, W, t, gscale=0.5, gscale_dev=up, **kw)
        _lib.assert_ok()
        assert torch.equal(b[2].float(), a[2].float() * 0.25) and torch.equal(b[3], a[3])


@pytest.mark.parametrize("R,V", [(4096, 4096), (18944 + 128, 2304)])
def test_split_one_sweep_keeps_the_rows_own_reference(R, V, epilogue_parts):
    """Bands of logits 200 nats below the rest wherever a piece of a row tile may begin (the first 32 words of every
    vocabulary tile but the first).  The row's reference, the maximum of its first 32 logits, is ordinary; every piece
    has to use it.  lse and loss as in the other one-sweep test, dX against whole row tiles."""
    x, W, t, _ = _mk_d(R, V, 256, wscale=0.05, seed=13)
    x[:, 0] = 8.0
    W[:, 0] = 0.0
    low = torch.arange(V, device="cuda").view(-1, 128)[1:, :32].reshape(-1)
    W[low, 0] = -25.0
    t = torch.where((t >= 128) & (t % 128 < 32), t + 32, t)
    assert _lib.lib().ccb_lmhead_work(R, V, 256, 1) > 0
    kw = dict(gscale=0.5, want_dw=False, one_sweep=True)
    loss, lse, dX, _ = LH.lm_head_train(x, None, W, t, **kw)
    real = LH._split_work
    LH._split_work = lambda *a: None
    try:
        wloss, wlse, wdX, _ = LH.lm_head_train(x, None, W, t, **kw)
    finally:
        LH._split_work = real
    _lib.assert_ok()
    rl, rlse, _, _ = LH.lm_head_reference(x, None, W, t, want_grads=False)
    assert torch.allclose(lse, rlse, rtol=1e-3, atol=2e-2) and torch.allclose(loss, rl, rtol=1e-3, atol=3e-2)
    assert torch.allclose(lse, wlse, rtol=0, atol=2e-4) and torch.allclose(loss, wloss, rtol=0, atol=2e-4)
    assert (dX.float() - wdX.float()).norm() <= 2e-3 * wdX.float().norm()


# one warp to a row (at most 8 partials), four, and sixteen (more than 32 partials, at most 16 384 rows)
@pytest.mark.parametrize("nparts,M", [(8, 513), (9, 129), (32, 127), (33, 33), (33, 16384), (33, 16385)])
def test_lse_combine_warps_to_a_row(nparts, M):
    """Against 64 bits, tolerance as above; and the same bits on every run."""
    g = torch.Generator(device="cuda").manual_seed(nparts + M)
    part = torch.stack([torch.randn(nparts, M, generator=g, device="cuda") * 30,
                        torch.rand(nparts, M, generator=g, device="cuda") * 100 + 1e-3], -1).contiguous()
    zt = torch.randn(M, generator=g, device="cuda")
    res = []
    for _ in range(2):
        lse, loss = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
        _lib.check(_lib.lib().ccb_lse_combine(part.data_ptr(), nparts, M, zt.data_ptr(), lse.data_ptr(), loss.data_ptr(),
                                              _lib.stream_ptr()), "lse_combine")
        res.append((lse, loss))
    ref = torch.logsumexp(part[..., 0].double() * 0.6931471805599453 + part[..., 1].double().log(), 0)
    tol = (nparts + 8) * 2.0 ** -23 + 2.0 ** -23 * ref.abs()
    assert ((res[0][0].double() - ref).abs() <= tol).all()
    assert all(torch.equal(a, b) for a, b in zip(*res))
