"""Operands whose shapes do not fit together never reach the native layer calls (host logic, no GPU)."""
import pytest
import torch

from chaoscontrol_b200.ops import trunk as T

B, TN, D, F = 2, 3, 16, 32


class _FakeLib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 0
        return call


@pytest.fixture
def lib(monkeypatch):
    fake = _FakeLib()
    monkeypatch.setattr(T, "_plain_bf16", lambda *a: True)      # CPU tensors stand in for bf16 CUDA ones
    monkeypatch.setattr(T, "_plain_f32", lambda *a: True)
    monkeypatch.setattr(T._lib, "lib", lambda: fake)
    monkeypatch.setattr(T._lib, "stream_ptr", lambda: 0)
    return fake


def _weights(**other):
    shapes = dict(Wp=(4 * D, D), Wo=(D, D), Wfc=(F, D), Wproj=(D, F), wn1=(D,), wn2=(D,), log_a=(D,),
                  Wp_f=(4 * D, D), Wfc_f=(F, D), log_a32=(D,))
    return T.LayerWeights(**{k: torch.zeros(other.get(k, s)) for k, s in shapes.items()})


BAD = [dict(Wp_f=(3 * D, D)), dict(Wo=(D, D - 8)), dict(Wo=(D - 8, D)), dict(Wproj=(D, F - 8)), dict(Wproj=(D - 8, F)),
       dict(Wfc_f=(F, D - 8)), dict(log_a32=(B, D))]


@pytest.mark.parametrize("bad", [{}] + BAD + [dict(ss1=(TN,))], ids=str)
def test_forward(lib, bad):
    bad = dict(bad)
    ss1 = torch.zeros(bad.pop("ss1", (B * TN,)))
    res = T._layer_forward_native(torch.zeros(B * TN, D), ss1, _weights(**bad), B, TN, None, True)
    fits = not bad and ss1.numel() == B * TN
    assert (res is not None) == fits and lib.calls == (["ccb_layer_forward"] if fits else [])


@pytest.mark.parametrize("bad", [{}] + BAD + [dict(Wp=(D, D)), dict(Wfc=(F - 8, D)), dict(wn1=(1,)), dict(wn2=(D - 8,)),
                                              dict(dWo=(D, D - 8)), dict(dlog_a=(1,))], ids=str)
def test_backward(lib, monkeypatch, bad):
    monkeypatch.setattr(_FakeLib, "ccb_layer_bwd_ws16", lambda *a: 8, raising=False)
    monkeypatch.setattr(_FakeLib, "ccb_layer_bwd_ws32", lambda *a: 8, raising=False)
    grads = dict(dWp=(4 * D, D), dWo=(D, D), dWfc=(F, D), dWproj=(D, F), dwn1=(D,), dwn2=(D,), dlog_a=(D,))
    outs = {k: torch.zeros(bad.get(k, s)) for k, s in grads.items()}
    w = _weights(**{k: v for k, v in bad.items() if k not in grads})
    R = B * TN
    ctx = T.PackedCtx(torch.zeros(R, D), torch.zeros(R), torch.zeros(R * (7 * D + 2 * F)), torch.zeros(R), None, F)
    res = T._layer_backward_native(torch.zeros(R, D), ctx, w, B, TN, None, False, outs, torch.float32)
    assert (res is not None) == (not bad) and lib.calls == ([] if bad else ["ccb_layer_backward"])


@pytest.mark.parametrize("bad", [{}, dict(log_a=(B, D)), dict(wn1=(1,)), dict(wn2=(1,)), dict(Wp=(3 * D, D)),
                                 dict(Wp=(4 * D, D - 8))], ids=str)
def test_fold_packed(lib, bad):
    """A decay vector per batch row, among others, keeps its shape: it is not read as one of [D]."""
    assert _weights(**bad)._fold_launch() == (not bad) and lib.calls == ([] if bad else ["ccb_layer_fold"])


@pytest.mark.parametrize("i", [None, 0, 3])
def test_fold_parts(lib, i):
    parts = [torch.zeros(D - 8 if k == i else D, D) for k in range(4)]
    assert _weights()._fold_launch(parts) == (i is None) and lib.calls == (["ccb_layer_fold"] if i is None else [])


@pytest.mark.parametrize("save", [True, False])
def test_activation_buffer(lib, monkeypatch, save):
    """The parts of the packed activations tile the buffer without gaps, and the states, which only backward reads, are
    neither allocated nor passed without ``save``."""
    got = {}
    monkeypatch.setattr(_FakeLib, "ccb_layer_forward", lambda self, a, s: got.setdefault("a", a._obj) and 0, raising=False)
    sizes = []
    real = torch.empty

    def empty(*a, **k):
        t = real(*a, **k)
        sizes.append((t.data_ptr(), t.numel() * t.element_size()))
        return t
    monkeypatch.setattr(T.torch, "empty", empty)
    R = B * TN
    res = T._layer_forward_native(torch.zeros(R, D), torch.zeros(R), _weights(), B, TN, None, save)
    a = got["a"]
    spans = [(a.P, 8 * R * D), (a.y, 2 * R * D), (a.x2, 2 * R * D), (a.u, 2 * R * F), (a.f, 2 * R * F)]
    spans += [(a.h, 2 * R * D)] if save else []
    assert save or not a.h
    spans.sort()
    assert all(p + n == q for (p, n), (q, _) in zip(spans, spans[1:]))
    assert (spans[0][0], sum(n for _, n in spans)) in sizes
    if save:
        ctx = res[3]
        assert [ctx.P.data_ptr(), ctx.y.data_ptr(), ctx.x2.data_ptr(), ctx.u.data_ptr(), ctx.f.data_ptr(),
                ctx.h.data_ptr()] == [a.P, a.y, a.x2, a.u, a.f, a.h]
