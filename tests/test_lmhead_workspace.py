"""Host logic of the LM head, no GPU: the sweep workspace belongs to the caller until the native call has returned; the
number of row chunks of the weight gradient."""
import weakref

import pytest
import torch

from chaoscontrol_b200.ops import lm_head as LH


class _FakeLib:
    """Stands in for the native library: remembers whether the workspace was alive inside each call."""

    def __init__(self):
        self.work, self.alive = None, []

    def __getattr__(self, name):
        def call(*args):
            if name in ("ccb_lmhead_lse", "ccb_lmhead_train"):
                w = self.work()
                self.alive.append(w is not None and w.data_ptr() in args)
            return 0
        return call


@pytest.mark.parametrize("train", [False, True])
def test_split_workspace_outlives_the_native_call(monkeypatch, train):
    lib = _FakeLib()

    def work(*_):
        w = torch.empty(64)
        lib.work = weakref.ref(w)
        return w
    monkeypatch.setattr(LH._lib, "lib", lambda: lib)
    monkeypatch.setattr(LH._lib, "stream_ptr", lambda: 0)
    monkeypatch.setattr(LH, "fused_supported", lambda *a: True)
    monkeypatch.setattr(LH, "_few_rows", lambda R: False)
    monkeypatch.setattr(LH, "_split_work", work)
    x, W, t = torch.zeros(8, 256), torch.zeros(128, 256), torch.zeros(8, dtype=torch.long)
    if train:
        LH.lm_head_train(x, None, W, t, gscale=1.0, want_dw=False)
    else:
        LH.lm_head_lse(x, None, W, t)
    assert lib.alive == [True]


@pytest.mark.parametrize("R,V,chunks", [(5000, 4096, 4), (4096, 8192, 2), (9000, 16384, 1), (32768, 1024, 18),
                                        (65536, 512, 37), (131072, 16384, 8)])
def test_row_chunks_weigh_partials_against_even_shares(R, V, chunks):
    """The counts that measured fastest (or within 2 % of it); an even deal alone would take 40 for the first."""
    assert LH.default_row_chunks(R, V) == chunks
