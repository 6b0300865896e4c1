"""Split-K reduction against 64-bit sums, at the edges of its tiles and of its split groups."""
import pytest
import torch

from chaoscontrol_b200.ops.trunk import splitk_reduce

pytestmark = pytest.mark.gpu


# S: one below, at and above each group rule (4, 8, 24); N: below, at and off the 8-row tile; K: off the 64-column
# tile, and 10 (not a multiple of 4: the any-width kernel)
@pytest.mark.parametrize("S,N,K", [(1, 1, 4), (4, 8, 64), (5, 9, 68), (8, 31, 256), (9, 64, 128), (24, 7, 60),
                                   (25, 256, 256), (74, 257, 264), (3, 20, 10), (30, 5, 10)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fold", [False, True])
def test_splitk_reduce(S, N, K, dt, fold):
    g = torch.Generator(device="cuda").manual_seed(S * 1000 + N)
    part = torch.randn(S, N, K, generator=g, device="cuda")
    W = torch.randn(N, K, generator=g, device="cuda").bfloat16() if fold else None
    cs = torch.randn(K, generator=g, device="cuda").bfloat16() if fold else None
    out, dcol = splitk_reduce(part, colscale=cs, W=W, out_dtype=dt)
    p64 = part.double()
    c64 = cs.double() if fold else torch.ones(K, device="cuda", dtype=torch.float64)
    ref = p64.sum(0) * c64
    # S + 3 roundings of fp32 on the sum of magnitudes, then the rounding of the stored type: half a unit in the
    # last place is 2^-8 of the value for bf16's 8 significant bits
    rnd = 2.0 ** -8 if dt is torch.bfloat16 else 2.0 ** -24
    bound = (S + 3) * 2.0 ** -24 * (p64.abs().sum(0) * c64).abs() + rnd * ref.abs()
    assert out.dtype == dt and ((out.double() - ref).abs() <= bound + 1e-30).all()
    if fold:
        terms = p64.sum(0) * W.double()
        mag = (p64.abs().sum(0) * W.double().abs()).sum(0)
        assert ((dcol.double() - terms.sum(0)).abs() <=
                (S + N + 4) * 2.0 ** -24 * mag + rnd * terms.sum(0).abs() + 1e-30).all()
    else:
        assert dcol is None


@pytest.mark.parametrize("S,N,K", [(1, 8, 64), (30, 64, 256), (30, 5, 10)])
def test_splitk_reduce_scale(S, N, K):
    """A device scale multiplies the fp32 sums before anything is rounded: exact for a power of two."""
    g = torch.Generator(device="cuda").manual_seed(S)
    part = torch.randn(S, N, K, generator=g, device="cuda")
    W = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    up = torch.full((), -0.5, device="cuda")
    for dt in (torch.float32, torch.bfloat16):
        for a, b in zip(splitk_reduce(part, W=W, out_dtype=dt, scale=up), splitk_reduce(part, W=W, out_dtype=dt)):
            assert torch.equal(a, b * -0.5)


# blocks of the result on both sides of the group rule (about 1000 blocks times groups), every group count
@pytest.mark.parametrize("S,N,K", [(30, 64, 256), (30, 584, 256), (30, 1192, 256), (30, 2376, 256), (12, 1200, 256),
                                   (6, 2400, 256), (15, 4096, 512)])
def test_splitk_reduce_group_rule(S, N, K):
    """fp32 sums against 64 bits: at most S roundings on the sum of magnitudes; the same bits on every run."""
    part = torch.randn(S, N, K, generator=torch.Generator(device="cuda").manual_seed(N), device="cuda")
    out, _ = splitk_reduce(part)
    p64 = part.double()
    assert ((out.double() - p64.sum(0)).abs() <= S * 2.0 ** -24 * p64.abs().sum(0) + 1e-30).all()
    assert torch.equal(out, splitk_reduce(part)[0])


@pytest.mark.parametrize("S,N,K", [(5, 8192, 256), (15, 4096, 512), (37, 1024, 256), (74, 256, 256), (40, 4096, 256)])
def test_splitk_reduce_error_is_below_that_of_a_serial_sum(S, N, K):
    """fp32 sums of random partials against 64 bits, next to adding them one after the other in fp32."""
    part = torch.randn(S, N, K, generator=torch.Generator(device="cuda").manual_seed(S), device="cuda")
    serial = torch.zeros(N, K, device="cuda")
    for p in part:
        serial += p
    ref = part.double().sum(0)
    assert (splitk_reduce(part)[0].double() - ref).norm() <= 0.98 * (serial.double() - ref).norm()
