"""One-launch weight preparation and row statistics against their PyTorch statements."""
import pytest
import torch

from chaoscontrol_b200.ops import trunk as T

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
        w = T.LayerWeights(Wp=Wp, **rest).prepare()
    else:
        w = T.LayerWeights.from_parts(*(t.clone() for t in Wp.split(D, 0)), **rest)
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
    assert ((T.row_ss(a).double() - ref).abs() <= tol * ref).all()
    s, ss = T.add_row_ss(a, b)
    assert torch.equal(s, a + b)
    ref = (a + b).double().square().sum(-1)
    assert ((ss.double() - ref).abs() <= tol * ref).all()
