"""Timed workloads of the framework's public entry points on one GPU.

Seven families, each the call that a user's program makes:

``scan``    ``kernels.ssm_scan`` forward and backward (the public recurrence op)
``norm``    ``kernels.fused_rms_norm`` forward and backward
``block``   ``models.core_fused.FusedCareSSMBlock``: a training pass (forward and backward, with or
            without a carried state) or an evaluation pass that takes and returns the state
``head``    RMSNorm + linear + cross-entropy over the vocabulary: a training pass
            (``kernels.fused_rms_linear_cross_entropy``) or per-token scoring without gradients
``fp8``     ``ops.fp8_block.BlockFP8Linear`` forward and backward
``ns``      ``optim.muon.newton_schulz_orthogonalize`` on one shape group of gradients
``train``   ``train_ssm.train_ssm_step``: a whole training step of a small language model

Sizes: width 256, 4 layers, vocabulary 16 384 and sequence 512 are the benchmark's trunk; widths 384
and 512 are the wider configurations; widths 64 and 128 and short sequences are the tests'.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from chaoscontrol_b200.kernels import (fused_linear_cross_entropy_with_ce, fused_rms_linear_cross_entropy,
                                       fused_rms_norm, ssm_scan)
from chaoscontrol_b200.models.core_fused import FusedCareSSMBlock
from chaoscontrol_b200.models.model import CareStudentLM
from chaoscontrol_b200.ops.fp8_block import BlockFP8Linear
from chaoscontrol_b200.optim.muon import newton_schulz_orthogonalize
from chaoscontrol_b200.train_ssm import train_ssm_step
from chaoscontrol_b200.utils.arena import ParamArena

DEV = "cuda"
BF16 = torch.bfloat16
_DT = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
#: (decay, update) dtype pairs the public scan accepts
_SCAN_PAIRS = [("bf16", "bf16"), ("bf16", "fp16"), ("fp16", "fp16"), ("fp32", "fp32"), ("fp32", "bf16"),
               ("fp32", "fp16")]
EPS = 1e-6


def listed():
    return [
        # one short odd-sized sequence pair through the public recurrence: launches and latency
        {"name": "scan_small", "op": "scan", "B": 2, "T": 129, "D": 96, "decay": "fp32", "update": "fp32"},
        # the recurrence of one layer of a large training batch
        {"name": "scan_train", "op": "scan", "B": 256, "T": 512, "D": 256, "decay": "bf16", "update": "bf16"},
        # normalisation of a wide model's activations (a row count that no tile divides)
        {"name": "norm_train", "op": "norm", "R": 100001, "D": 512},
        # evaluation of one document, chunk by chunk with the state carried over
        {"name": "block_chunk", "op": "block", "B": 1, "T": 512, "D": 256, "ff": 2, "state": True, "grad": False},
        # a block of the benchmark's trunk at a large batch
        {"name": "block_train", "op": "block", "B": 256, "T": 512, "D": 256, "ff": 2, "state": False, "grad": True},
        # a block of a wider model on a small ragged batch with a carried state (truncated backpropagation)
        {"name": "block_wide", "op": "block", "B": 37, "T": 300, "D": 384, "ff": 2, "state": True, "grad": True},
        # per-token scoring of one chunk of a document
        {"name": "head_score", "op": "head", "R": 511, "D": 256, "V": 16384, "grad": False},
        # loss and gradients of the benchmark's vocabulary
        {"name": "head_train", "op": "head", "R": 65536, "D": 256, "V": 16384, "grad": True},
        # the same at a wider model, a smaller vocabulary and a row count that no tile divides
        {"name": "head_wide", "op": "head", "R": 9000, "D": 384, "V": 8192, "grad": True},
        # the packed projection of a trunk layer in 8-bit floats
        {"name": "fp8_linear", "op": "fp8", "R": 65536, "K": 256, "N": 1024, "bias": False},
        # the optimizer's orthogonalisation of the trunk's square projections (4 layers x 4)
        {"name": "muon_ns", "op": "ns", "G": 16, "r": 256, "c": 256},
        # a whole training step of the benchmark's model at a small batch
        {"name": "train_step", "op": "train", "B": 64, "T": 512, "D": 256, "L": 4, "V": 16384},
    ]


# ---------------------------------------------------------------------------
# drawn cases: the same families over their ranges
# ---------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(["scan", "norm", "block", "block", "head", "head", "fp8", "ns", "train"])
    if op == "scan":
        dt, ut = rng.choice(_SCAN_PAIRS)
        T, D = _log_int(rng, 8, 2048), _log_int(rng, 16, 512)
        fits = (1 << 24) // (T * D)          # as many elements as the listed 32-bit equivalent allows
        return {"op": op, "B": _log_int(rng, 1, max(1, min(256, fits))), "T": T, "D": D, "decay": dt, "update": ut}
    if op == "norm":
        D = 2 * rng.randint(32, 512)
        return {"op": op, "R": _log_int(rng, 1, 50_000_000 // D), "D": D}
    if op == "block":
        D, T = 64 * rng.randint(1, 8), _log_int(rng, 16, 1024)
        fits = (1 << 23) // (T * D)
        return {"op": op, "B": _log_int(rng, 1, max(1, min(256, fits))), "T": T, "D": D,
                "ff": rng.choice([2, 2, 4]) if D <= 256 else 2, "state": rng.random() < 0.5,
                "grad": rng.random() < 0.6}
    if op == "head":
        D = rng.choice([64, 128, 192, 256, 256, 320, 384, 512])
        V = 128 * _log_int(rng, 4, 128)
        fits = (65536 * 256 * 16384) // (2 * D * V)
        return {"op": op, "R": _log_int(rng, 16, min(65536, fits)), "D": D, "V": V, "grad": rng.random() < 0.6}
    if op == "fp8":
        K, N = 128 * rng.randint(1, 8), 128 * rng.randint(1, 8)
        return {"op": op, "R": _log_int(rng, 16, min(65536, (65536 * 1024) // max(K, N))), "K": K, "N": N,
                "bias": rng.random() < 0.5}
    if op == "ns":
        r, c = 8 * _log_int(rng, 8, 64), 8 * _log_int(rng, 8, 64)
        return {"op": op, "G": rng.randint(1, 16), "r": r, "c": c}
    D = 64 * rng.randint(2, 6)
    T = _log_int(rng, 32, 512)
    return {"op": op, "B": _log_int(rng, 1, max(1, 8192 // T)), "T": T, "D": D, "L": rng.randint(1, 4),
            "V": 128 * _log_int(rng, 8, 64)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, dtype=BF16, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _zipf_tokens(g, V, *shape):
    """Token ids whose frequencies fall off like natural text's (rank^-1)."""
    u = torch.rand(*shape, generator=g, device=DEV)
    return (V ** u - 1.0).long().clamp_(0, V - 1)


def _linear(g, n, k):
    return _randn(g, n, k, scale=k ** -0.5)


def _block_weights(g, D, ff):
    """Parameters of one block under the block's own state-dict names."""
    w = {"core." + n + "_proj.weight": _linear(g, D, D) for n in ("select", "in", "gate", "delta", "out")}
    w["ff.fc.weight"] = _linear(g, ff * D, D)
    w["ff.proj.weight"] = _linear(g, D, ff * D)
    w["input_norm.weight"] = (1.0 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(BF16)
    w["ff_norm.weight"] = (1.0 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(BF16)
    w["core.log_a"] = torch.randn(D, generator=g, device=DEV).sub_(1.0).to(BF16)
    return w


def _draw_inputs(case, seed):
    """The tensors of a case, from its seed alone (the 64-bit statement starts from the same ones)."""
    g = _gen(seed)
    op = case["op"]
    if op == "scan":
        B, T, D = case["B"], case["T"], case["D"]
        return {"decay": torch.sigmoid(torch.randn(B, T, D, generator=g, device=DEV) + 2.0).to(_DT[case["decay"]]),
                "update": _randn(g, B, T, D, dtype=_DT[case["update"]], scale=0.5),
                "go": _randn(g, B, T, D, dtype=_DT[case["update"]])}
    if op == "norm":
        R, D = case["R"], case["D"]
        return {"x": _randn(g, R, D, scale=1.5), "go": _randn(g, R, D),
                "w": (1.0 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(BF16)}
    if op == "block":
        B, T, D = case["B"], case["T"], case["D"]
        d = {"w": _block_weights(g, D, case["ff"]), "x": _randn(g, B, T, D)}
        if case["state"]:
            d["h0"] = _randn(g, B, D, dtype=torch.float32, scale=0.5)
        if case["grad"]:
            d["go"] = _randn(g, B, T, D)
        return d
    if op == "head":
        R, D, V = case["R"], case["D"], case["V"]
        return {"x": _randn(g, R, D), "nw": (1.0 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(BF16),
                "W": _linear(g, V, D), "t": _zipf_tokens(g, V, R)}
    if op == "fp8":
        R, K, N = case["R"], case["K"], case["N"]
        d = {"x": _randn(g, R, K), "W": _linear(g, N, K), "go": _randn(g, R, N)}
        if case["bias"]:
            d["b"] = _randn(g, N, scale=0.1)
        return d
    if op == "ns":
        # a gradient: few strong directions on a flat background
        G, r, c = case["G"], case["r"], case["c"]
        low = _randn(g, G, r, 8, dtype=torch.float32) @ _randn(g, G, 8, c, dtype=torch.float32)
        return {"g": (low + _randn(g, G, r, c, dtype=torch.float32)).to(BF16)}
    if op == "train":
        B, T, D, V = case["B"], case["T"], case["D"], case["V"]
        sd = {"embed.weight": _randn(g, V, D), "lm_head.weight": _linear(g, V, D),
              "final_norm.weight": (1.0 + 0.1 * torch.randn(D, generator=g, device=DEV)).to(BF16)}
        for i in range(case["L"]):
            sd.update({f"layers.{i}.{k}": v for k, v in _block_weights(g, D, 2).items()})
        return {"sd": sd, "tok": _zipf_tokens(g, V, B, T + 1)}
    raise ValueError(op)


def prepare(case, seed):
    op = case["op"]
    d = _draw_inputs(case, seed)
    d["case"] = dict(case)
    if op == "scan":
        d["decay"].requires_grad_(True)
        d["update"].requires_grad_(True)
    elif op == "norm":
        d["x"].requires_grad_(True)
        d["w"].requires_grad_(True)
    elif op == "block":
        blk = FusedCareSSMBlock(case["D"], case["ff"]).to(DEV).to(BF16)
        blk.load_state_dict(d.pop("w"), strict=True)
        d["blk"] = blk
        if case["grad"]:
            d["x"].requires_grad_(True)
            if "h0" in d:
                d["h0"].requires_grad_(True)
    elif op == "head":
        if case["grad"]:
            for k in ("x", "nw", "W"):
                d[k].requires_grad_(True)
    elif op == "fp8":
        lin = BlockFP8Linear(case["K"], case["N"], bias=case["bias"], device=DEV)
        with torch.no_grad():
            lin.weight.copy_(d.pop("W"))
            if case["bias"]:
                lin.bias.copy_(d.pop("b"))
        d["lin"] = lin
        d["x"].requires_grad_(True)
    elif op == "train":
        model = CareStudentLM(vocab_size=case["V"], dim=case["D"], num_layers=case["L"]).to(DEV).to(BF16)
        model.load_state_dict(d.pop("sd"), strict=True)
        ParamArena.install(model)
        model.train()
        d["model"] = model
        tok = d.pop("tok")
        d["inputs"], d["targets"] = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
    return d


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "scan":
        out = ssm_scan(state["decay"], state["update"])
        gd, gu = torch.autograd.grad(out, (state["decay"], state["update"]), state["go"])
        return {"states": out.detach(), "g_decay": gd, "g_update": gu}
    if op == "norm":
        y = fused_rms_norm(state["x"], state["w"], EPS)
        gx, gw = torch.autograd.grad(y, (state["x"], state["w"]), state["go"])
        return {"y": y.detach(), "gx": gx, "gw": gw}
    if op == "block":
        blk, h0 = state["blk"], state.get("h0")
        if not case["grad"]:
            with torch.no_grad():
                y, hT = blk(state["x"], initial_state=h0, return_final_state=True)
            return {"y": y, "hT": hT}
        y, hT = blk(state["x"], initial_state=h0, return_final_state=True)
        names, ps = zip(*blk.named_parameters())
        wrt = [state["x"]] + ([h0] if h0 is not None else []) + list(ps)
        grads = torch.autograd.grad(y, wrt, state["go"])
        out = {"y": y.detach(), "hT": hT.detach()}
        labels = ["x"] + (["h0"] if h0 is not None else []) + list(names)
        out.update({"g:" + n: g for n, g in zip(labels, grads)})
        return out
    if op == "head":
        if not case["grad"]:
            with torch.no_grad():
                loss, rows = fused_linear_cross_entropy_with_ce(fused_rms_norm(state["x"], state["nw"], EPS),
                                                                state["W"], state["t"])
            return {"loss": loss, "rows": rows}
        loss = fused_rms_linear_cross_entropy(state["x"], state["nw"], state["W"], state["t"], eps=EPS)
        gx, gn, gW = torch.autograd.grad(loss, (state["x"], state["nw"], state["W"]))
        return {"loss": loss.detach(), "gx": gx, "gn": gn, "gW": gW}
    if op == "fp8":
        lin = state["lin"]
        y = lin(state["x"])
        wrt = [state["x"], lin.weight] + ([lin.bias] if lin.bias is not None else [])
        grads = torch.autograd.grad(y, wrt, state["go"])
        out = {"y": y.detach(), "gx": grads[0], "gW": grads[1]}
        if lin.bias is not None:
            out["gb"] = grads[2]
        return out
    if op == "ns":
        return newton_schulz_orthogonalize(state["g"])
    model = state["model"]
    for p in model.parameters():
        p.grad = None
    loss = train_ssm_step(model, state["inputs"], state["targets"], 64, lm_head_backward_mode="fused_streaming_cached",
                          lm_head_tile_size=8192)
    out = {"loss": loss}
    out.update({"g:" + n: p.grad for n, p in model.named_parameters()})
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _block_work(B, T, D, ff, grad, state):
    R = B * T
    w = (5 + 2 * ff) * D * D
    flops = 2.0 * R * w * (3 if grad else 1)
    data = 2 * R * D * (2 + (3 if grad else 0)) + 4 * B * D * (1 + (1 if state else 0))
    # forward and backward are two calls: the block's input is read by both, its weights too
    return data + 2 * w * (3 if grad else 1), flops


def work(case):
    op = case["op"]
    if op == "scan":
        n = case["B"] * case["T"] * case["D"]
        d, u = (4 if case[k] == "fp32" else 2 for k in ("decay", "update"))
        # forward: decay, update -> states; backward: decay, states, go -> two gradients
        return {"bytes": n * (d + u + u + d + u + u + d + u), "flops": 6.0 * n}
    if op == "norm":
        n = case["R"] * case["D"]
        return {"bytes": n * 2 * 5, "flops": 14.0 * n}
    if op == "block":
        b, f = _block_work(case["B"], case["T"], case["D"], case["ff"], case["grad"], case["state"])
        return {"bytes": b, "flops": f}
    if op == "head":
        R, D, V = case["R"], case["D"], case["V"]
        if not case["grad"]:
            return {"bytes": 2 * R * D + 2 * V * D + 12 * R, "flops": 2.0 * R * D * V}
        # logits, hidden gradient, weight gradient, and the logits once more: they do not fit in memory traffic
        return {"bytes": 2 * R * D * 3 + 2 * V * D * 3 + 8 * R, "flops": 2.0 * R * D * V * 4}
    if op == "fp8":
        R, K, N = case["R"], case["K"], case["N"]
        return {"bytes": 2 * R * (3 * K + 2 * N) + 2 * N * K * 3, "flops": 2.0 * R * K * N * 3}
    if op == "ns":
        G, r, c = case["G"], case["r"], case["c"]
        k = min(r, c)
        return {"bytes": 4 * G * r * c, "flops": 5 * 2.0 * G * (2.0 * k * r * c + k ** 3)}
    B, T, D, L, V = (case[k] for k in ("B", "T", "D", "L", "V"))
    R = B * T
    params = L * 9 * D * D + 2 * V * D
    # every layer's input is kept for the backward: written once, read once
    return {"bytes": 2 * params * 3 + L * 2 * R * D * 2 + 16 * R,
            "flops": 2.0 * R * (3 * L * 9 * D * D + 4 * V * D)}


# ---------------------------------------------------------------------------
# tolerances
# ---------------------------------------------------------------------------
def tolerance(case):
    op = case["op"]
    if op == "scan":
        # 32-bit recurrences differ by the order of their sums; 16-bit results by one rounding
        return {"rel": 1e-5 if (case["decay"], case["update"]) == ("fp32", "fp32") else 4e-3}
    if op == "norm":
        return {"rel": 4e-3}
    if op == "block":
        return {"rel": 1.5e-2 if case["grad"] else 8e-3}
    if op == "head":
        return {"rel": 1e-2 if case["grad"] else 2e-3}
    if op == "fp8":
        return {"rel": 1e-2}
    if op == "ns":
        # five bf16 iterations of a polynomial that amplifies small singular values
        return {"rel": 3e-2}
    return {"rel": 2.5e-2}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _norm64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _block64(x, w, h0):
    """One block in 64 bits: ``(output, final state)``; ``w`` holds doubles under the state-dict names."""
    B, T, D = x.shape
    n = _norm64(x, w["input_norm.weight"])
    s, c, gt, dl = (n @ w["core." + k + "_proj.weight"].t() for k in ("select", "in", "gate", "delta"))
    decay = torch.exp(-F.softplus(dl).clamp_min(1e-4) * torch.sigmoid(w["core.log_a"]))
    update = torch.sigmoid(s) * torch.tanh(c)
    h = torch.zeros(B, D, dtype=x.dtype, device=x.device) if h0 is None else h0
    hs = []
    for dt, ut in zip(decay.unbind(1), update.unbind(1)):
        h = dt * h + ut
        hs.append(h)
    x = x + (torch.sigmoid(gt) * torch.stack(hs, 1)) @ w["core.out_proj.weight"].t()
    u = _norm64(x, w["ff_norm.weight"]) @ w["ff.fc.weight"].t()
    return x + F.silu(u) @ w["ff.proj.weight"].t(), h


def _head64(x, W, t, grad, chunk=4096):
    """``(rows, gx, gW)`` of the mean cross-entropy of already normalised rows, in row chunks."""
    R = x.shape[0]
    rows, gx = torch.empty(R, dtype=x.dtype, device=x.device), torch.empty_like(x) if grad else None
    gW = torch.zeros_like(W) if grad else None
    for i in range(0, R, chunk):
        xc, tc = x[i:i + chunk], t[i:i + chunk, None]
        z = xc @ W.t()
        lse = torch.logsumexp(z, -1, keepdim=True)
        rows[i:i + chunk] = (lse - z.gather(1, tc)).squeeze(1)
        if grad:
            p = z.sub_(lse).exp_()
            p.scatter_add_(1, tc, torch.full_like(lse, -1.0))
            p /= R
            gx[i:i + chunk] = p @ W
            gW += p.t() @ xc
    return rows, gx, gW


def exact(case, seed):
    op = case["op"]
    d = _draw_inputs(case, seed)
    if op == "scan":
        dec, upd, go = (d[k].double() for k in ("decay", "update", "go"))
        T = case["T"]
        h, s = torch.empty_like(upd), torch.zeros_like(upd[:, 0])
        for t in range(T):
            s = dec[:, t] * s + upd[:, t]
            h[:, t] = s
        gd, gu, carry = torch.empty_like(dec), torch.empty_like(upd), torch.zeros_like(s)
        for t in reversed(range(T)):
            g = go[:, t] + carry
            gu[:, t] = g
            gd[:, t] = g * h[:, t - 1] if t > 0 else 0.0
            carry = g * dec[:, t]
        return {"states": h, "g_decay": gd, "g_update": gu}
    if op == "norm":
        x, w, go = (d[k].double() for k in ("x", "w", "go"))
        inv = torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
        xh, gw_ = x * inv, go * w
        return {"y": xh * w, "gx": inv * (gw_ - xh * (gw_ * xh).mean(-1, keepdim=True)), "gw": (go * xh).sum(0)}
    if op == "block":
        names = [n for n, _ in FusedCareSSMBlock(64, 2).named_parameters()]
        w = {n: d["w"][n].double().requires_grad_(case["grad"]) for n in names}
        x = d["x"].double().requires_grad_(case["grad"])
        h0 = d["h0"].double().requires_grad_(case["grad"]) if "h0" in d else None
        with torch.set_grad_enabled(case["grad"]):
            y, hT = _block64(x, w, h0)
        out = {"y": y.detach(), "hT": hT.detach()}
        if case["grad"]:
            labels = ["x"] + (["h0"] if h0 is not None else []) + names
            grads = torch.autograd.grad(y, [x] + ([h0] if h0 is not None else []) + [w[n] for n in names],
                                        d["go"].double())
            out.update({"g:" + n: g for n, g in zip(labels, grads)})
        return out
    if op == "head":
        x, nw, W, t = d["x"].double(), d["nw"].double(), d["W"].double(), d["t"]
        if not case["grad"]:
            rows, _, _ = _head64(_norm64(x, nw), W, t, False)
            return {"loss": rows.mean(), "rows": rows}
        x.requires_grad_(True)
        nw.requires_grad_(True)
        xn = _norm64(x, nw)
        rows, gxn, gW = _head64(xn.detach(), W, t, True)
        gx, gn = torch.autograd.grad(xn, (x, nw), gxn)
        return {"loss": rows.mean(), "gx": gx, "gn": gn, "gW": gW}
    if op == "fp8":
        x, W, go = (d[k].double() for k in ("x", "W", "go"))
        y = x @ W.t()
        out = {"y": y + d["b"].double() if case["bias"] else y, "gx": go @ W, "gW": go.t() @ x}
        if case["bias"]:
            out["gb"] = go.sum(0)
        return out
    if op == "ns":
        a, b, c = 3.4445, -4.7750, 2.0315
        X = d["g"].double()
        X = X / (X.norm(dim=(-2, -1), keepdim=True) + 1e-7)
        tall = X.size(-2) > X.size(-1)
        X = X.mT if tall else X
        for _ in range(5):
            A = X @ X.mT
            X = a * X + (b * A + c * (A @ A)) @ X
        return X.mT if tall else X
    # the whole step, one layer at a time
    sd = {k: v.double().requires_grad_(True) for k, v in d["sd"].items()}
    tok = d["tok"]
    inputs, targets = tok[:, :-1], tok[:, 1:].reshape(-1)
    x = F.embedding(inputs, sd["embed.weight"])
    for i in range(case["L"]):
        pre = f"layers.{i}."
        x, _ = _block64(x, {k[len(pre):]: v for k, v in sd.items() if k.startswith(pre)}, None)
    xn = _norm64(x.reshape(-1, case["D"]), sd["final_norm.weight"])
    rows, gxn, gW = _head64(xn.detach(), sd["lm_head.weight"].detach(), targets, True)
    rest = [k for k in sd if k != "lm_head.weight"]
    grads = dict(zip(rest, torch.autograd.grad(xn, [sd[k] for k in rest], gxn)))
    grads["lm_head.weight"] = gW
    out = {"loss": rows.mean()}
    out.update({"g:" + n: grads[n] for n in sd})
    return out
