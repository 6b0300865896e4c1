"""Hand-scheduled forward and backward of the diagonal-SSM trunk.

One layer is four GEMMs and one scan kernel in each direction; every
elementwise op of the block (both RMSNorms, the gate nonlinearities, SiLU, the
two residual adds) lives in a GEMM epilogue or in the scan kernel, so no
``[rows, dim]`` tensor is ever touched by a standalone elementwise pass:

forward (x: residual stream, ss = row sum of squares of x)::

    P   = rs1 * (x  @ Wp'^T)          Wp' = [select;in;gate;delta] * w_input_norm   (EPI_ROWSCALE)
    y,h = scan(P, log_a, h0)
    x2  = x  + y @ Wo^T , ss2         (EPI_RESID_SS)
    u,f = rs2 * (x2 @ Wfc'^T), silu   Wfc' = fc * w_ff_norm                         (EPI_ROWSCALE_SILU)
    x3  = x2 + f @ Wproj^T , ss3      (EPI_RESID_SS)

The RMSNorm weight is folded into the following linear's weight (tiny, once
per step) and the row scale ``rs = rsqrt(ss/D + eps)`` is applied to the GEMM
output, which is algebraically the reference block
(src/chaoscontrol/model.py:111-140, core.py:492-507, core.py:322-335).

backward mirrors it with the RMSNorm backward fused into the input-gradient
GEMM epilogue (EPI_RMSBWD) and weight gradients from split-K MN-major GEMMs.
Everything here also runs on CPU tensors (fp32) through the op stand-ins, which
is how the algebra is tested against autograd of the plain module.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass, field
from typing import Optional

import torch

from . import _lib
from .gemm import (EPI_DSILU, EPI_RESID_SS, EPI_RMSBWD, EPI_ROWSCALE, EPI_ROWSCALE_SILU,
                   EPI_STORE, gemm, wgrad_splits)
from .scan import scan_fused_bwd, scan_fused_fwd, scan_fused_reference

EPS = 1e-6


# ---------------------------------------------------------------------------
# small op wrappers with CPU stand-ins
# ---------------------------------------------------------------------------
def fold_colscale(W: torch.Tensor, wn: torch.Tensor) -> torch.Tensor:
    """``W * wn[None, :]`` in the activation dtype (RMSNorm weight folded into W)."""
    if W.is_cuda and W.dtype == torch.bfloat16 and wn.dtype == torch.bfloat16 and W.is_contiguous():
        out = torch.empty_like(W)
        _lib.check(_lib.lib().ccb_fold_colscale(W.data_ptr(), wn.data_ptr(), out.data_ptr(),
                                                W.shape[0], W.shape[1], _lib.stream_ptr()), "fold")
        return out
    return (W.float() * wn.float()[None, :]).to(W.dtype)


def row_ss(x: torch.Tensor) -> torch.Tensor:
    """fp32 ``[R]`` row sums of squares of a contiguous ``[R, D]``."""
    if x.is_cuda and x.dtype == torch.bfloat16:
        ss = torch.empty(x.shape[0], dtype=torch.float32, device=x.device)
        rc = _lib.lib().ccb_row_ss(x.data_ptr(), None, None, ss.data_ptr(), x.shape[0], x.shape[1], _lib.stream_ptr())
        if rc <= 0:
            _lib.check(rc, "row_ss")
            return ss
    return x.float().square().sum(-1)


def add_row_ss(a: torch.Tensor, b: torch.Tensor):
    """``(a + b, its row sums of squares)`` of two ``[R, D]`` tensors."""
    if a.is_cuda and a.dtype == b.dtype == torch.bfloat16 and a.is_contiguous() and b.is_contiguous():
        out = torch.empty_like(a)
        ss = torch.empty(a.shape[0], dtype=torch.float32, device=a.device)
        rc = _lib.lib().ccb_row_ss(a.data_ptr(), b.data_ptr(), out.data_ptr(), ss.data_ptr(), a.shape[0], a.shape[1],
                                   _lib.stream_ptr())
        if rc <= 0:
            _lib.check(rc, "row_ss")
            return out, ss
    x = (a + b).contiguous()
    return x, x.float().square().sum(-1)


def embed_fwd(tokens: torch.Tensor, E: torch.Tensor):
    """Gather rows of ``E`` and their sums of squares.  Returns ``(x [R,D], ss [R])``."""
    flat = tokens.reshape(-1)
    R, D = flat.numel(), E.shape[1]
    if E.is_cuda:
        assert E.dtype == torch.bfloat16 and E.is_contiguous()
        if flat.dtype not in (torch.int32, torch.int64):
            flat = flat.long()
        flat = flat.contiguous()
        x = torch.empty(R, D, dtype=E.dtype, device=E.device)
        ss = torch.empty(R, dtype=torch.float32, device=E.device)
        _lib.check(_lib.lib().ccb_embed_fwd(flat.data_ptr(), int(flat.dtype == torch.int64),
                                            E.data_ptr(), x.data_ptr(), ss.data_ptr(), R, D,
                                            E.shape[0], _lib.stream_ptr()), "embed_fwd")
        return x, ss
    x = E[flat.long()]
    return x, (x.float() ** 2).sum(-1)


EMBED_BWD_DIMS = (256, 512, 1024)      # widths of the sorted embedding-backward kernel


def token_sort(tokens: torch.Tensor, V: int):
    """``(sorted tokens, stable permutation)`` for :func:`embed_bwd`.  On the GPU 16-bit keys where the table allows."""
    flat = tokens.reshape(-1)
    if flat.is_cuda and V < 32768 and flat.dtype in (torch.int32, torch.int64) and flat.numel() > 0:
        flat = flat.contiguous()
        key = torch.empty(flat.numel(), dtype=torch.int16, device=flat.device)
        _lib.check(_lib.lib().ccb_token_keys(flat.data_ptr(), int(flat.dtype == torch.int64), key.data_ptr(),
                                             flat.numel(), V, _lib.stream_ptr()), "token_keys")
        flat = key
    else:
        flat = flat.long()
    return torch.sort(flat, stable=True)


def embed_bwd(tokens: torch.Tensor, dx: torch.Tensor, V: int,
              sort_cache: Optional[tuple] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """fp32 ``[V, D]`` gradient of the embedding table (sum of the ``dx`` rows of each token).

    On the GPU the rows are added in a fixed order derived from the stably sorted token array, so
    the same batch gives the same bits on every run and on every replica."""
    D = dx.shape[1]
    if out is not None:
        dE = out.zero_()
    else:
        dE = torch.zeros(V, D, dtype=torch.float32, device=dx.device)
    if dx.is_cuda and D in EMBED_BWD_DIMS:
        if sort_cache is None:
            sort_cache = token_sort(tokens, V)
        st, perm = sort_cache
        L = _lib.lib()
        R = st.numel()
        slots = torch.empty(int(L.ccb_embed_bwd_slots(R, D, V)), dtype=torch.float32, device=dx.device)
        _lib.check(L.ccb_embed_bwd_sorted_as(st.data_ptr(), st.element_size(), perm.data_ptr(), dx.data_ptr(),
                                             dE.data_ptr(), slots.data_ptr(), R, D, V, _lib.stream_ptr()),
                   "embed_bwd")
        return dE
    dE.index_add_(0, tokens.reshape(-1).long(), dx.float())
    return dE


def splitk_reduce(part: torch.Tensor, *, colscale: Optional[torch.Tensor] = None,
                  W: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
                  dcol_out: Optional[torch.Tensor] = None, out_dtype: torch.dtype = torch.float32,
                  scale: Optional[torch.Tensor] = None):
    """Sum split-K partials ``[S, N, K]`` (or ``[N, K]``).

    Returns ``(dW [N,K], dcol [K] or None)`` with
    ``dW = colscale * sum`` and ``dcol = sum_n sum[n,k] * W[n,k]`` -- the
    gradients of ``W`` and of the RMSNorm weight folded into it.  Results are fp32;
    ``out_dtype=torch.bfloat16`` rounds them once, as they are stored.  ``scale``, a one-element
    fp32 tensor, multiplies the fp32 sums.
    """
    if part.dim() == 2:
        part = part.unsqueeze(0)
    S, N, K = part.shape
    if part.is_cuda and (colscale is None or colscale.dtype == torch.bfloat16) and (
            W is None or (W.dtype == torch.bfloat16 and W.is_contiguous())) and (
            out_dtype in (torch.float32, torch.bfloat16)):
        if out is None:
            out = torch.empty(N, K, dtype=out_dtype, device=part.device)
        assert out.dtype == out_dtype and out.is_contiguous()
        nb = (N + 7) // 8
        colpart = torch.empty(nb, K, dtype=torch.float32, device=part.device) if W is not None else None
        dcol = None
        if W is not None:
            dcol = dcol_out if dcol_out is not None else torch.empty(K, dtype=out_dtype, device=part.device)
            assert dcol.dtype == out_dtype
        _lib.check(_lib.lib().ccb_splitk_reduce_as(part.data_ptr(), S, part.stride(0), N, K,
                                                   _lib.ptr(colscale), _lib.ptr(W), _lib.ptr(scale), out.data_ptr(),
                                                   int(out_dtype == torch.bfloat16), 0,
                                                   _lib.ptr(colpart), _lib.ptr(dcol), 0,
                                                   _lib.stream_ptr()), "splitk_reduce")
        return out, dcol
    s = part.float().sum(0)
    if scale is not None:
        s = s * scale
    dcol = (s * W.float()).sum(0).to(out_dtype) if W is not None else None
    if colscale is not None:
        s = s * colscale.float()[None, :]
    s = s.to(out_dtype)
    if out is not None:
        out.copy_(s)
        s = out
    if dcol is not None and dcol_out is not None:
        dcol_out.copy_(dcol)
        dcol = dcol_out
    return s, dcol


def _wgrad(dy: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """Split-K partials of ``dy^T @ x`` (``[S, N, K]`` fp32)."""
    M, N = dy.shape
    K = x.shape[1]
    S = wgrad_splits(N, K, M) if dy.is_cuda else 1
    out = gemm(dy, x, a_mn=True, b_mn=True, splits=S, out_dtype=torch.float32)
    return out if out.dim() == 3 else out.unsqueeze(0)


# ---------------------------------------------------------------------------
# per-layer weights as the kernels want them
# ---------------------------------------------------------------------------
@dataclass
class LayerWeights:
    Wp: torch.Tensor        # [4D, D]  select | in | gate | delta  (unscaled)
    Wo: torch.Tensor        # [D, D]
    Wfc: torch.Tensor       # [F, D]
    Wproj: torch.Tensor     # [D, F]
    wn1: torch.Tensor       # [D] input_norm.weight
    wn2: torch.Tensor       # [D] ff_norm.weight
    log_a: torch.Tensor     # [D]
    # derived per step
    Wp_f: torch.Tensor = field(default=None)     # Wp * wn1
    Wfc_f: torch.Tensor = field(default=None)    # Wfc * wn2
    log_a32: torch.Tensor = field(default=None)

    @classmethod
    def from_parts(cls, sel, inp, gate, delta, *, Wo, Wfc, Wproj, wn1, wn2, log_a) -> "LayerWeights":
        """Packed and prepared from four separate ``[D, D]`` projections."""
        rest = dict(Wo=Wo.contiguous(), Wfc=Wfc.contiguous(), Wproj=Wproj.contiguous(), wn1=wn1.contiguous(),
                    wn2=wn2.contiguous(), log_a=log_a)
        w = cls(Wp=None, **rest)
        if not w._fold_launch([t.contiguous() for t in (sel, inp, gate, delta)]):
            w.Wp = torch.cat([sel, inp, gate, delta], 0)
            w.prepare()
        return w

    def _fold_launch(self, parts: Optional[list] = None) -> bool:
        """:meth:`prepare` as one kernel launch; False (nothing done) for operands it does not take.
        ``parts``: the four projections, to be packed as well."""
        ops = [self.Wfc, self.wn1, self.wn2, self.log_a, *(parts if parts is not None else [self.Wp])]
        if not _plain_bf16(*ops):
            return False
        F_, D = self.Wfc.shape
        sq = (D, D)
        if not (self.wn1.shape == (D,) and self.wn2.shape == (D,) and self.log_a.shape == (D,) and
                (self.Wp.shape == (4 * D, D) if parts is None else
                 parts[0].shape == sq and parts[1].shape == sq and parts[2].shape == sq and parts[3].shape == sq)):
            return False
        dev = self.Wfc.device
        Wp = torch.empty(4 * D, D, dtype=torch.bfloat16, device=dev) if parts is not None else None
        Wp_f = torch.empty(4 * D, D, dtype=torch.bfloat16, device=dev)
        Wfc_f = torch.empty_like(self.Wfc)
        la = torch.empty(D, dtype=torch.float32, device=dev)
        src = ([t.data_ptr() for t in parts] if parts is not None else
               [self.Wp.data_ptr() + 2 * i * D * D for i in range(4)])
        rc = _lib.lib().ccb_layer_fold(*src, self.wn1.data_ptr(), self.Wfc.data_ptr(), self.wn2.data_ptr(),
                                       self.log_a.data_ptr(), _lib.ptr(Wp), Wp_f.data_ptr(), Wfc_f.data_ptr(),
                                       la.data_ptr(), D, F_, _lib.stream_ptr())
        if rc > 0:
            return False
        _lib.check(rc, "layer_fold")
        if Wp is not None:
            self.Wp = Wp
        self.Wp_f, self.Wfc_f, self.log_a32 = Wp_f, Wfc_f, la
        return True

    def prepare(self) -> "LayerWeights":
        if self._fold_launch():
            return self
        self.Wp_f = fold_colscale(self.Wp, self.wn1)
        self.Wfc_f = fold_colscale(self.Wfc, self.wn2)
        self.log_a32 = self.log_a.float().contiguous()
        return self


@dataclass
class LayerCtx:
    x: torch.Tensor
    ss1: torch.Tensor
    P: torch.Tensor
    h: torch.Tensor
    y: torch.Tensor
    x2: torch.Tensor
    ss2: torch.Tensor
    u: torch.Tensor
    f: torch.Tensor
    h0: Optional[torch.Tensor]


@dataclass
class PackedCtx:
    """The same activations of a layer that ran as one native call: all bf16 ones in ``acts``."""
    x: torch.Tensor
    ss1: torch.Tensor
    acts: torch.Tensor      # P [R,4D] | y [R,D] | x2 [R,D] | u [R,F] | f [R,F] | h [R,D] (last: evaluation goes without)
    ss2: torch.Tensor
    h0: Optional[torch.Tensor]
    F: int

    def _part(self, start: int, width: int) -> torch.Tensor:
        R = self.x.shape[0]
        return self.acts[start * R:(start + width) * R].view(R, width)

    P = property(lambda c: c._part(0, 4 * c.x.shape[1]))
    y = property(lambda c: c._part(4 * c.x.shape[1], c.x.shape[1]))
    x2 = property(lambda c: c._part(5 * c.x.shape[1], c.x.shape[1]))
    u = property(lambda c: c._part(6 * c.x.shape[1], c.F))
    f = property(lambda c: c._part(6 * c.x.shape[1] + c.F, c.F))
    h = property(lambda c: c._part(6 * c.x.shape[1] + 2 * c.F, c.x.shape[1]))


@dataclass
class LayerGrads:
    dWp: torch.Tensor       # [4D, D] fp32 (or the grad_dtype asked for), or four [D, D] (split_wp)
    dWo: torch.Tensor
    dWfc: torch.Tensor
    dWproj: torch.Tensor
    dwn1: torch.Tensor
    dwn2: torch.Tensor
    dlog_a: torch.Tensor
    dh0: Optional[torch.Tensor] = None


def _scan_fwd(P, log_a32, h0, B, T, D, save_h):
    if P.is_cuda:
        return scan_fused_fwd(P, log_a32, h0, B, T, D, save_h=save_h)
    y, h, hT = scan_fused_reference(P, log_a32, h0, B, T, D)
    return y.to(P.dtype), h.to(P.dtype), hT


def _scan_bwd(P, log_a32, h0, h, dy, dhT, rowss, inv_dim, eps, B, T, D, want_dh0):
    if P.is_cuda:
        return scan_fused_bwd(P, log_a32, h0, h, dy, dhT, rowss, inv_dim, eps, B, T, D,
                              want_dh0=want_dh0)
    with torch.enable_grad():
        Pr = P.detach().float().requires_grad_(True)
        la = log_a32.detach().clone().requires_grad_(True)
        h0r = h0.detach().clone().requires_grad_(True) if h0 is not None else None
        y, _, hT = scan_fused_reference(Pr, la, h0r, B, T, D)
        obj = (y * dy.float()).sum()
        if dhT is not None:
            obj = obj + (hT * dhT.float()).sum()
        ins = [Pr, la] + ([h0r] if (h0r is not None and want_dh0) else [])
        grads = torch.autograd.grad(obj, ins)
    dP = grads[0]
    if rowss is not None:
        dP = dP * torch.rsqrt(rowss.float() * inv_dim + eps)[:, None]
    return dP.to(P.dtype), grads[1], (grads[2] if len(grads) > 2 else None)


def _plain_bf16(*ts, dtype=torch.bfloat16) -> bool:
    for t in ts:                                # loops: half the time of a generator, on every layer call
        if not (t.is_cuda and t.dtype is dtype and t.is_contiguous()):
            return False
    return True


def _layer_shaped(w: "LayerWeights", D: int, F_: int) -> bool:
    """The native layer calls take addresses and the sizes of one layer: every operand's shape has to be as they say.
    Anything else goes through the step-by-step form, whose operations check (or broadcast) what they are given.
    (Written out: a layer's host time is part of a small batch's.)"""
    return (w.Wp_f.shape == (4 * D, D) and w.Wfc_f.shape == (F_, D) and w.Wo.shape == (D, D) and
            w.Wproj.shape == (D, F_) and w.log_a32.shape == (D,))


def _plain_f32(*ts, dtype=torch.float32) -> bool:
    for t in ts:
        if t is not None and not (t.is_cuda and t.dtype is dtype and t.is_contiguous()):
            return False
    return True


def _layer_args(w: LayerWeights, B: int, T: int, D: int, F_: int, x, ss1, h0, acts, ss2) -> "_lib.LayerArgs":
    a = _lib.LayerArgs()
    a.B, a.T, a.D, a.F, a.eps = B, T, D, F_, EPS
    a.Wp_f, a.Wfc_f, a.Wo, a.Wproj = w.Wp_f.data_ptr(), w.Wfc_f.data_ptr(), w.Wo.data_ptr(), w.Wproj.data_ptr()
    a.log_a, a.h0 = w.log_a32.data_ptr(), _lib.ptr(h0)
    a.x, a.ss1, a.ss2 = x.data_ptr(), ss1.data_ptr(), ss2.data_ptr()
    rd = 2 * x.numel()
    a.P = p = acts.data_ptr()
    rf = 2 * x.shape[0] * F_
    a.y, a.x2, a.u = p + 4 * rd, p + 5 * rd, p + 6 * rd
    a.f, a.h = p + 6 * rd + rf, p + 6 * rd + 2 * rf
    return a


def _layer_forward_native(x, ss1, w, B, T, h0, save):
    """:func:`layer_forward` as one native call; None when an operand is not plain."""
    R, D = x.shape
    F_ = w.Wfc.shape[0]
    if not (R == B * T and R > 0 and D % 8 == 0 and F_ % 8 == 0 and _layer_shaped(w, D, F_) and
            ss1.shape == (R,) and
            _plain_bf16(x, w.Wp_f, w.Wfc_f, w.Wo, w.Wproj) and _plain_f32(ss1, w.log_a32, h0)):
        return None
    dev = x.device
    acts = torch.empty(R * ((7 if save else 6) * D + 2 * F_), dtype=torch.bfloat16, device=dev)
    x3 = torch.empty_like(x)
    ss2 = torch.empty(R, dtype=torch.float32, device=dev)
    ss3 = torch.empty(R, dtype=torch.float32, device=dev)
    hT = torch.empty(B, D, dtype=torch.float32, device=dev)
    a = _layer_args(w, B, T, D, F_, x, ss1, h0, acts, ss2)
    if not save:
        a.h = None
    a.x3, a.ss3, a.hT = x3.data_ptr(), ss3.data_ptr(), hT.data_ptr()
    _lib.check(_lib.lib().ccb_layer_forward(C.byref(a), _lib.stream_ptr()), "layer_forward")
    return x3, ss3, hT, (PackedCtx(x, ss1, acts, ss2, h0, F_) if save else None)


_GRAD_KEYS = ("dWp", "dWo", "dWfc", "dWproj", "dwn1", "dwn2", "dlog_a")


def _layer_backward_native(dx3, ctx, w, B, T, dhT, want_dh0, outs, grad_dtype, split_wp=False):
    """:func:`layer_backward` as one native call; None when an operand is not plain."""
    R, D = ctx.x.shape
    F_ = ctx.F
    if not (_plain_bf16(dx3, w.Wp_f, w.Wfc_f, w.Wo, w.Wproj, w.Wp, w.Wfc, w.wn1, w.wn2) and
            _plain_f32(w.log_a32, dhT) and dx3.shape == ctx.x.shape and _layer_shaped(w, D, F_) and
            w.Wp.shape == (4 * D, D) and w.Wfc.shape == (F_, D) and w.wn1.shape == (D,) and w.wn2.shape == (D,)):
        return None
    dev = dx3.device
    if outs:
        if grad_dtype != torch.float32 or any(k not in outs for k in _GRAD_KEYS):
            return None
        g = [outs[k] for k in _GRAD_KEYS]
        if not (_plain_f32(*g) and g[0].shape == (4 * D, D) and g[1].shape == (D, D) and g[2].shape == (F_, D) and
                g[3].shape == (D, F_) and g[4].shape == g[5].shape == g[6].shape == (D,)):
            return None
    elif grad_dtype in (torch.float32, torch.bfloat16):
        # an allocation each: a gradient that is kept, saved or changed in place leaves the others alone
        new, Wo, wn1 = torch.empty_like, w.Wo, w.wn1
        if grad_dtype == torch.bfloat16:
            g = [new(Wo), new(w.Wfc), new(w.Wproj), new(wn1), new(wn1), new(wn1)]
            g.insert(0, (new(Wo), new(Wo), new(Wo), new(Wo)) if split_wp else new(w.Wp))
        else:
            g = [new(t, dtype=grad_dtype) for t in (Wo, w.Wfc, w.Wproj, wn1, wn1, wn1)]
            g.insert(0, tuple(new(Wo, dtype=grad_dtype) for _ in range(4)) if split_wp else new(w.Wp, dtype=grad_dtype))
    else:
        return None
    L = _lib.lib()
    ws16 = torch.empty(L.ccb_layer_bwd_ws16(R, D, F_), dtype=torch.bfloat16, device=dev)
    ws32 = torch.empty(L.ccb_layer_bwd_ws32(B, T, D, F_), dtype=torch.float32, device=dev)
    dx = torch.empty_like(dx3)
    dh0 = torch.empty(B, D, dtype=torch.float32, device=dev) if want_dh0 else None
    a = _layer_args(w, B, T, D, F_, ctx.x, ctx.ss1, ctx.h0, ctx.acts, ctx.ss2)
    a.grad_bf16 = int(grad_dtype == torch.bfloat16)
    a.Wp, a.Wfc, a.wn1, a.wn2 = w.Wp.data_ptr(), w.Wfc.data_ptr(), w.wn1.data_ptr(), w.wn2.data_ptr()
    a.dx3, a.dhT, a.ws16, a.ws32 = dx3.data_ptr(), _lib.ptr(dhT), ws16.data_ptr(), ws32.data_ptr()
    a.dx, a.dh0 = dx.data_ptr(), _lib.ptr(dh0)
    if split_wp:
        a.dWp, a.dWp1, a.dWp2, a.dWp3 = (t.data_ptr() for t in g[0])
    else:
        a.dWp = g[0].data_ptr()
    a.dWo, a.dWfc, a.dWproj, a.dwn1, a.dwn2, a.dlog_a = (t.data_ptr() for t in g[1:])
    _lib.check(L.ccb_layer_backward(C.byref(a), _lib.stream_ptr()), "layer_backward")
    return dx, LayerGrads(*g, dh0)


def layer_forward(x: torch.Tensor, ss1: torch.Tensor, w: LayerWeights, B: int, T: int,
                  h0: Optional[torch.Tensor] = None, *, save: bool = True):
    """One block.  Returns ``(x3, ss3, hT, ctx)``; ``ctx`` is None when ``save`` is False."""
    if x.is_cuda:
        res = _layer_forward_native(x, ss1, w, B, T, h0, save)
        if res is not None:
            return res
    R, D = x.shape
    F_ = w.Wfc.shape[0]
    inv_d = 1.0 / D
    P = gemm(x, w.Wp_f, epi=EPI_ROWSCALE, rowss=ss1, inv_dim=inv_d, eps=EPS)
    y, h, hT = _scan_fwd(P, w.log_a32, h0, B, T, D, save)
    ss2 = torch.empty(R, dtype=torch.float32, device=x.device)
    x2 = gemm(y, w.Wo, epi=EPI_RESID_SS, r1=x, ss_out=ss2)
    f = torch.empty(R, F_, dtype=x.dtype, device=x.device)
    u = gemm(x2, w.Wfc_f, epi=EPI_ROWSCALE_SILU, rowss=ss2, inv_dim=inv_d, eps=EPS, c2=f)
    ss3 = torch.empty(R, dtype=torch.float32, device=x.device)
    x3 = gemm(f, w.Wproj, epi=EPI_RESID_SS, r1=x2, ss_out=ss3)
    ctx = LayerCtx(x, ss1, P, h, y, x2, ss2, u, f, h0) if save else None
    return x3, ss3, hT, ctx


def layer_backward(dx3: torch.Tensor, ctx: LayerCtx, w: LayerWeights, B: int, T: int,
                   dhT: Optional[torch.Tensor] = None, *, want_dh0: bool = False,
                   outs: Optional[dict] = None, grad_dtype: torch.dtype = torch.float32, split_wp: bool = False):
    """Backward of :func:`layer_forward`.  Returns ``(dx, LayerGrads)``.

    Weight gradients are fp32, or rounded once to ``grad_dtype`` as they are stored.  ``split_wp`` (without
    ``outs``): the gradients of the four packed projections as four tensors of their own.
    ``outs`` may map ``dWp / dWo / dWfc / dWproj / dwn1 / dwn2`` to preallocated
    fp32 tensors (views of a flat gradient buffer) that receive the results.
    """
    if outs and split_wp:
        raise ValueError("layer_backward: split_wp allocates the gradients; it takes no outs")
    if isinstance(ctx, PackedCtx):
        res = _layer_backward_native(dx3, ctx, w, B, T, dhT, want_dh0, outs, grad_dtype, split_wp)
        if res is not None:
            return res
    R, D = ctx.x.shape
    inv_d = 1.0 / D
    o = outs or {}
    gd = grad_dtype
    # feed-forward half
    du = gemm(dx3, w.Wproj, b_mn=True, epi=EPI_DSILU, r1=ctx.u, rowss=ctx.ss2, inv_dim=inv_d, eps=EPS)
    dWproj, _ = splitk_reduce(_wgrad(dx3, ctx.f), out=o.get("dWproj"), out_dtype=gd)
    dx2 = gemm(du, w.Wfc_f, b_mn=True, epi=EPI_RMSBWD, r1=ctx.x2, r2=dx3, rowss=ctx.ss2,
               inv_dim=inv_d, eps=EPS)
    dWfc, dwn2 = splitk_reduce(_wgrad(du, ctx.x2), colscale=w.wn2, W=w.Wfc, out=o.get("dWfc"),
                               dcol_out=o.get("dwn2"), out_dtype=gd)
    # recurrence half
    dy = gemm(dx2, w.Wo, b_mn=True)
    dWo, _ = splitk_reduce(_wgrad(dx2, ctx.y), out=o.get("dWo"), out_dtype=gd)
    dP, dlog_a, dh0 = _scan_bwd(ctx.P, w.log_a32, ctx.h0, ctx.h, dy, dhT, ctx.ss1, inv_d, EPS, B, T,
                                D, want_dh0)
    dx = gemm(dP, w.Wp_f, b_mn=True, epi=EPI_RMSBWD, r1=ctx.x, r2=dx2, rowss=ctx.ss1, inv_dim=inv_d,
              eps=EPS)
    dWp, dwn1 = splitk_reduce(_wgrad(dP, ctx.x), colscale=w.wn1, W=w.Wp, out=o.get("dWp"),
                              dcol_out=o.get("dwn1"), out_dtype=gd)
    if "dlog_a" in o:
        o["dlog_a"].copy_(dlog_a)
    if split_wp:
        dWp = tuple(t.clone() for t in dWp.split(D, 0))
    return dx, LayerGrads(dWp, dWo, dWfc, dWproj, dwn1, dwn2, dlog_a, dh0)
