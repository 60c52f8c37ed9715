"""The workloads by which this framework's speed is followed.

Each case is a dict of plain values.  `prepare` makes what a program holds before the call (inputs, weights, a trainer),
`run` is one pass through the public entry points, `exact` the same outputs in 64-bit floating point by plain torch,
`work` the bytes and operations one pass cannot do without, `tolerance` how far another correct implementation at the
same precision may be from it.

Kinds:
  attention  the attention operator, causal with rotary embedding (decoder) or without a mask (image encoder)
  mlp        the decoder's feed-forward half: norm, gate|up, SwiGLU, down
  head       final norm's output to vocabulary logits and the mean cross-entropy
  mlp_fp8    the feed-forward half in the 8-bit (E4M3) forward option
  vit_block  one block of the image encoder
  block      one decoder block as a module, optionally with grouped key / value heads and QKV biases
  step       a whole optimizer step of the trainer
`train` selects forward and backward (else forward only).
"""
from __future__ import annotations

import math

import torch
import torch.utils.checkpoint

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
THETA, EPS = 10000.0, 1e-5


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # attention of the 12-layer / 768-wide decoder, one layer of its training step
        dict(name="attn_flagship", kind="attention", B=16, T=1024, H=12, hd=64, causal=True, train=True),
        # attention of the 24-layer / 2048-wide decoder (head size 128, the sharded configuration)
        dict(name="attn_wide", kind="attention", B=8, T=2048, H=16, hd=128, causal=True, train=True),
        # the image encoder's attention: 196 patches of a 224 x 224 image and the class token, every token sees every token
        dict(name="attn_image", kind="attention", B=32, T=197, H=12, hd=64, causal=False, train=True),
        # evaluation of sequences whose length is no multiple of anything
        dict(name="attn_ragged", kind="attention", B=3, T=1000, H=12, hd=64, causal=True, train=False),
        # feed-forward half of the 2048-wide decoder
        dict(name="mlp_wide", kind="mlp", rows=16384, C=2048, I=5504, train=True),
        # feed-forward half of the 768-wide decoder on a small, odd number of tokens (fine-tuning on a few samples)
        dict(name="mlp_ragged", kind="mlp", rows=1003, C=768, I=2048, train=True),
        # vocabulary head of the 768-wide decoder in its training step
        dict(name="head_flagship", kind="head", rows=16384, C=768, V=50304, train=True),
        # feed-forward half of the 768-wide decoder with the 8-bit forward switched on
        dict(name="mlp_fp8", kind="mlp_fp8", rows=16384, C=768, I=2048, train=False),
        # one block of the image encoder with LayerNorm, training
        dict(name="vit_block", kind="vit_block", B=16, T=197, C=768, H=12, I=2048, train=True),
        # one 2048-wide decoder block with grouped key / value heads and biases, training
        dict(name="block_gqa", kind="block", B=2, T=2048, C=2048, H=16, Hkv=4, I=5504, bias=True, train=True),
        # the whole optimizer step of the 12-layer / 768-wide decoder, as the benchmark and the training mode take it
        dict(name="step_flagship", kind="step", B=16, T=1024, C=768, H=12, I=2048, L=12, V=50304, train=True),
        # the smallest call: the step of the overfitting mode (head size 32), bound by launches
        dict(name="step_tiny", kind="step", B=4, T=64, C=128, H=4, I=256, L=4, V=256, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "mlp", "head", "mlp_fp8", "vit_block", "block", "step"])
    if kind == "attention":
        causal = rng.random() < 0.65
        hd = rng.choice([64, 64, 128]) if rng.random() < 0.85 else 32
        T = _log(rng, 16, 256 if hd == 32 else 2048) if causal else _log(rng, 17, 600)
        H = rng.choice([1, 2, 3, 4, 6, 8, 12, 16])
        B = _log(rng, 1, max(1, min(64, 16384 // T)))
        return dict(kind=kind, B=B, T=T, H=H, hd=hd, causal=causal, train=rng.random() < 0.7)
    if kind == "mlp":
        C, I = rng.choice([(128, 256), (128, 384), (768, 2048), (768, 2048), (1024, 2816), (2048, 5504)])
        return dict(kind=kind, rows=_log(rng, 16, 16384), C=C, I=I, train=rng.random() < 0.7)
    if kind == "head":
        C = rng.choice([128, 768, 768, 2048])
        V = rng.choice([256, 512, 32768, 50304])
        return dict(kind=kind, rows=_log(rng, 16, 16384 if C <= 768 else 4096), C=C, V=V, train=rng.random() < 0.7)
    if kind == "mlp_fp8":
        C, I = rng.choice([(768, 2048), (768, 2048), (1024, 2816), (2048, 5504)])
        # (the 8-bit product takes more than 128 rows; below, a model falls back to the bf16 weights)
        return dict(kind=kind, rows=_log(rng, 160, 16384), C=C, I=I, train=False)
    if kind == "vit_block":
        T = rng.choice([17, 50, 65, 145, 197, 197, 257, 577])      # (image / patch)^2 + 1
        H = rng.choice([4, 6, 12, 12, 16])
        return dict(kind=kind, B=_log(rng, 1, max(1, min(48, 8192 // T))), T=T, C=64 * H, H=H,
                    I=rng.choice([128 * H, 2048]), train=rng.random() < 0.7)
    if kind == "block":
        C, H, I = rng.choice([(768, 12, 2048), (1024, 16, 2816), (2048, 16, 5504), (2048, 32, 5504)])
        T = _log(rng, 64, 2048)
        return dict(kind=kind, B=_log(rng, 1, max(1, 4096 // T)), T=T, C=C, H=H, Hkv=rng.choice([2, 4, H]) if H % 4 == 0 else H, I=I,
                    bias=rng.random() < 0.5, train=rng.random() < 0.7)
    C, H, I = rng.choice([(128, 4, 256), (128, 4, 384), (256, 4, 512), (768, 12, 2048)])
    T = _log(rng, 32, 256) if C == 128 else _log(rng, 64, 1024)
    return dict(kind="step", B=_log(rng, 1, max(1, min(16, (2048 if C == 128 else 8192) // T))), T=T, C=C, H=H, I=I, L=rng.randint(1, 4),
                V=rng.choice([256, 512, 32768]), train=True)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=F32) * std).to(dtype)


def _inputs(case, seed):
    """Tensors by name; grads_of names those whose gradients a training pass returns."""
    g, k = _gen(seed), case["kind"]
    if k == "attention":
        n, C = case["B"] * case["T"], case["H"] * case["hd"]
        return dict(qkv=_randn(g, n, 3 * C), dout=_randn(g, n, C))
    if k in ("mlp", "mlp_fp8"):
        n, C, I = case["rows"], case["C"], case["I"]
        return dict(x=_randn(g, n, C), w=1 + _randn(g, C, std=0.1), gate_up=_randn(g, 2 * I, C, std=0.5 / math.sqrt(C)),
                    down=_randn(g, C, I, std=0.5 / math.sqrt(I)), dout=_randn(g, n, C))
    if k == "head":
        n, C, V = case["rows"], case["C"], case["V"]
        return dict(x=_randn(g, n, C), lm=_randn(g, V, C, std=0.02),
                    tgt=torch.randint(0, V, (n,), generator=g, device="cuda", dtype=torch.int32))
    if k == "vit_block":
        n, C, I = case["B"] * case["T"], case["C"], case["I"]
        b = lambda m: _randn(g, m, std=0.1)
        return dict(x=_randn(g, n, C), n1_w=1 + b(C), n1_b=b(C), qkv_w=_randn(g, 3 * C, C, std=1 / math.sqrt(C)), qkv_b=b(3 * C),
                    o_w=_randn(g, C, C, std=0.5 / math.sqrt(C)), o_b=b(C), n2_w=1 + b(C), n2_b=b(C),
                    gu_w=_randn(g, 2 * I, C, std=0.5 / math.sqrt(C)), gu_b=b(2 * I), down_w=_randn(g, C, I, std=0.5 / math.sqrt(I)),
                    down_b=b(C), dout=_randn(g, n, C))
    if k == "block":
        n, C, I = case["B"] * case["T"], case["C"], case["I"]
        q = (case["H"] + 2 * case["Hkv"]) * (C // case["H"])
        d = dict(x=_randn(g, n, C), ln1=1 + _randn(g, C, std=0.1), qkv=_randn(g, q, C, std=1 / math.sqrt(C)),
                 o=_randn(g, C, C, std=0.5 / math.sqrt(C)), ln2=1 + _randn(g, C, std=0.1),
                 gate_up=_randn(g, 2 * I, C, std=0.5 / math.sqrt(C)), down=_randn(g, C, I, std=0.5 / math.sqrt(I)), dout=_randn(g, n, C))
        if case["bias"]:
            d["qkv_bias"] = _randn(g, q, std=0.1)
        return d
    n, V = case["B"] * case["T"], case["V"]
    r = lambda: torch.randint(0, V, (n,), generator=g, device="cuda", dtype=torch.int32)
    C, I, L, std = case["C"], case["I"], case["L"], 0.02
    # flat parameters in the layout's order: wte, per layer (ln1 qkv o ln2 gate up down), final norm, head
    so = std / math.sqrt(2 * L)
    parts = [_randn(g, V * C, std=std, dtype=F32)]
    for _ in range(L):
        parts += [torch.ones(C, device="cuda"), _randn(g, 3 * C * C, std=std, dtype=F32), _randn(g, C * C, std=so, dtype=F32),
                  torch.ones(C, device="cuda"), _randn(g, 2 * I * C, std=std, dtype=F32), _randn(g, C * I, std=so, dtype=F32)]
    parts += [torch.ones(C, device="cuda"), _randn(g, V * C, std=std, dtype=F32)]
    return dict(ids=r(), tgt=r(), master=torch.cat(parts))


def _rope(T, hd, dtype=F64):
    f = 1.0 / (THETA ** (torch.arange(0, hd, 2, dtype=F64, device="cuda") / hd))
    a = torch.arange(T, dtype=F64, device="cuda")[:, None] * f[None, :]
    return a.cos().to(dtype), a.sin().to(dtype)


def prepare(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    s = {"case": case, "in": d}
    if k == "attention":
        from ml_b200 import ops
        s["cos"], s["sin"] = ops.rope_tables(case["T"], case["hd"], THETA, torch.device("cuda"))
        d["qkv"].requires_grad_(case["train"])
    elif k in ("mlp", "head"):
        for n in ("x", "w", "gate_up", "down", "lm"):
            if n in d:
                d[n].requires_grad_(case["train"])
    elif k == "mlp_fp8":
        from ml_b200 import ops
        # the optimizer keeps the E4M3 copies of the weights; the activations' buffers belong to the model
        n, C, I = case["rows"], case["C"], case["I"]
        e = lambda *sh, dt=BF16: torch.empty(*sh, dtype=dt, device="cuda")
        u8 = torch.uint8
        s["gate_up8"], s["down8"] = e(2 * I, C, dt=u8), e(C, I, dt=u8)
        ops.native_module().cast_bf16_fp8(s["gate_up8"], d["gate_up"], 16.0)
        ops.native_module().cast_bf16_fp8(s["down8"], d["down"], 16.0)
        s.update(ln=e(n, C), ln8=e(n, C, dt=u8), rstd=e(n, dt=F32), gu=e(n, 2 * I), sw=e(n, I), sw8=e(n, I, dt=u8), y=e(n, C))
    elif k == "vit_block":
        from ml_b200.models.vit import ViTBlock
        m = ViTBlock(case["C"], case["H"], case["I"], "layer", EPS, BF16, "cuda")
        s["module"] = _load(m, d, case["train"])
    elif k == "block":
        from ml_b200 import Config, ops
        from ml_b200.models.modules import Block
        cfg = Config(V=256, C=case["C"], L=1, H=case["H"], I=case["I"], T=case["T"])
        s["cos"], s["sin"] = ops.rope_tables(cfg.T, cfg.hd, cfg.rope_theta, torch.device("cuda"))
        s["module"] = _load(Block(cfg, BF16, "cuda", case["Hkv"], case["bias"]), d, case["train"])
    else:
        from ml_b200 import Config, RunConfig
        from ml_b200.trainer import Trainer
        cfg = Config(V=case["V"], C=case["C"], L=case["L"], H=case["H"], I=case["I"], T=case["T"])
        tr = _trainer(Trainer, cfg, case["B"], RunConfig())
        tr.model.master.copy_(d["master"])
        tr.model.sync_params()
        tr.set_batch(d["ids"], d["tgt"])
        s["trainer"] = tr
    return s


def _trainer(Trainer, cfg, B, run):
    """The trainer without its host-side random initialisation (seconds at 163 M parameters): the weights are set afterwards, as
    from a checkpoint."""
    from ml_b200.models import GPT
    init = GPT.init_weights
    GPT.init_weights = lambda self, seed=0: None
    try:
        return Trainer(cfg, B, "cuda", run=run, lr=1e-4, wd=0.1)
    finally:
        GPT.init_weights = init


def _load(m, d, train):
    with torch.no_grad():
        for n, p in m.named_parameters():
            p.copy_(d[n])
            p.requires_grad_(train)
    d["x"].requires_grad_(train)
    return m


# ------------------------------------------------------------------ one pass
def _grads(out, dout, named):
    names = list(named)
    gs = torch.autograd.grad(out, [named[n] for n in names], dout)
    return {"out": out.detach(), **{"d_" + n: g for n, g in zip(names, gs)}}


def run(state):
    case, d = state["case"], state["in"]
    k = case["kind"]
    if k == "attention":
        from ml_b200.ops import autograd as F
        B, T, H, hd = case["B"], case["T"], case["H"], case["hd"]
        with torch.set_grad_enabled(case["train"]):
            if case["causal"]:
                out = F.rope_causal_attention(d["qkv"], state["cos"], state["sin"], B, T, H, hd)
            else:
                out = F.bidir_attention(d["qkv"], B, T, H, hd)
        return _grads(out, d["dout"], {"qkv": d["qkv"]}) if case["train"] else {"out": out}
    if k == "mlp":
        from ml_b200.ops import autograd as F
        with torch.set_grad_enabled(case["train"]):
            h = F.rmsnorm(d["x"], d["w"], EPS)
            out = F.linear(F.swiglu(F.linear(h, d["gate_up"])), d["down"])
        return _grads(out, d["dout"], {n: d[n] for n in ("x", "w", "gate_up", "down")}) if case["train"] else {"out": out}
    if k == "head":
        from ml_b200.ops import autograd as F
        if not case["train"]:
            with torch.no_grad():
                logits = F.linear(d["x"], d["lm"])
                return {"logits": logits, "loss": F.cross_entropy(logits, d["tgt"])}
        logits = F.linear(d["x"], d["lm"])
        loss = F.cross_entropy(logits, d["tgt"])
        gx, gw = torch.autograd.grad(loss, [d["x"], d["lm"]])
        return {"loss": loss.detach(), "d_x": gx, "d_lm": gw}
    if k == "mlp_fp8":
        from ml_b200 import ops
        nat, s = ops.native_module(), state
        nat.rmsnorm_fwd_fp8(s["ln"], s["ln8"], s["rstd"], d["x"], d["w"], EPS, 1.0)
        if not nat.linear_fwd_fp8(s["gu"], s["ln8"], s["gate_up8"], 1.0 / 16.0):
            ops.linear_fwd(s["gu"], s["ln"], d["gate_up"])
        nat.swiglu_fwd_fp8(s["sw"], s["sw8"], s["gu"], 1.0)
        if not nat.linear_fwd_fp8(s["y"], s["sw8"], s["down8"], 1.0 / 16.0):
            ops.linear_fwd(s["y"], s["sw"], d["down"])
        return {"ln": s["ln"], "rstd": s["rstd"], "gu": s["gu"], "sw": s["sw"], "y": s["y"]}
    if k in ("vit_block", "block"):
        m = state["module"]
        with torch.set_grad_enabled(case["train"]):
            if k == "vit_block":
                out = m(d["x"], case["B"], case["T"])
            else:
                out = m(d["x"], state["cos"], state["sin"], case["B"])
        return _grads(out, d["dout"], {"x": d["x"], **dict(m.named_parameters())}) if case["train"] else {"out": out}
    tr = state["trainer"]
    tr.step()
    return {"losses": tr.model.losses, "grads": tr.model.grads, "weights": tr.model.master}


# ------------------------------------------------------------------ what a pass cannot do without
def _attn_flops(B, T, H, hd, causal, train):
    pairs = T * (T + 1) / 2 if causal else T * T
    return B * H * pairs * hd * 4 * (3.5 if train else 1.0)      # two products forward, five backward


def work(case):
    k, tr = case["kind"], case["train"]
    f3 = 3.0 if tr else 1.0
    if k == "attention":
        n, C = case["B"] * case["T"], case["H"] * case["hd"]
        return {"bytes": 2.0 * n * C * ((3 + 1 + 1 + 3) if tr else 4), "flops": _attn_flops(case["B"], case["T"], case["H"], case["hd"], case["causal"], tr)}
    if k in ("mlp", "mlp_fp8"):
        n, C, I = case["rows"], case["C"], case["I"]
        w = 3.0 * C * I + C
        if k == "mlp_fp8":
            return {"bytes": 3.0 * C * I + 2.0 * n * (C + C + 2 * I + I + C) + 4.0 * n, "flops": 6.0 * n * C * I}
        return {"bytes": 2.0 * (w * (2 if tr else 1) + n * C * (4 if tr else 2)), "flops": 6.0 * n * C * I * f3}
    if k == "head":
        n, C, V = case["rows"], case["C"], case["V"]
        b = 2.0 * (2 * V * C + 2 * n * C) if tr else 2.0 * (V * C + n * C + n * V)
        return {"bytes": b + 4.0 * n, "flops": 2.0 * n * C * V * f3}
    if k in ("vit_block", "block"):
        n, C, I, H = case["B"] * case["T"], case["C"], case["I"], case["H"]
        qkv = 3 * C if k == "vit_block" else (H + 2 * case["Hkv"]) * (C // H)
        w = qkv * C + C * C + 3 * C * I
        return {"bytes": 2.0 * (w * (2 if tr else 1) + n * C * (4 if tr else 2)),
                "flops": 2.0 * n * w * f3 + _attn_flops(case["B"], case["T"], H, C // H, k == "block", tr)}
    n, C, I, V, L = case["B"] * case["T"], case["C"], case["I"], case["V"], case["L"]
    w = L * (4 * C * C + 3 * C * I + 2 * C) + 2 * V * C + C
    return {"bytes": w * (3 * 4 * 2 + 4 + 2 + 2.0) + 8.0 * n,
            "flops": 6.0 * n * (w - V * C) + L * _attn_flops(case["B"], case["T"], case["H"], C // case["H"], True, True)}


def tolerance(case):
    # about four times what the path shows against `exact` on a B200: bf16 outputs alone are 0.0017 off, a chain of layers more,
    # the 8-bit option's second product 0.014 (a bf16 input that rounds to the neighbouring E4M3 value)
    return {"rel": {"attention": 0.014, "mlp": 0.017, "head": 0.007, "mlp_fp8": 0.03, "vit_block": 0.026, "block": 0.028, "step": 0.022}[case["kind"]]}


# ------------------------------------------------------------------ the same in 64 bits
def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _ln64(x, w, b):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, EPS)


def _swiglu64(gu):
    g, u = gu.chunk(2, dim=-1)
    return torch.nn.functional.silu(g) * u


def _rot64(t, cos, sin):
    a, b = t.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _attn64(q, k, v, causal):
    """[heads, T, hd] each."""
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    return torch.softmax(s, -1) @ v


def _mha64(qkv, B, T, H, Hkv, hd, causal):
    """qkv [B*T, (H + 2 Hkv) hd] -> [B*T, H hd], one sample at a time."""
    cos, sin = _rope(T, hd) if causal else (None, None)
    outs = []
    for b in range(B):
        x = qkv[b * T:(b + 1) * T].view(T, H + 2 * Hkv, hd).transpose(0, 1)
        q, k, v = x[:H], x[H:H + Hkv], x[H + Hkv:]
        if causal:
            q, k = _rot64(q, cos, sin), _rot64(k, cos, sin)
        k, v = k.repeat_interleave(H // Hkv, 0), v.repeat_interleave(H // Hkv, 0)
        o = torch.utils.checkpoint.checkpoint(_attn64, q, k, v, causal, use_reentrant=False)
        outs.append(o.transpose(0, 1).reshape(T, H * hd))
    return torch.cat(outs)


def _e4m3(x, scale=1.0):
    return (x * scale).float().clamp(-448, 448).to(torch.float8_e4m3fn).to(F64)


def exact(case, seed):
    k, tr = case["kind"], case["train"]
    d = {n: (t.to(F64) if t.is_floating_point() else t) for n, t in _inputs(case, seed).items()}
    with torch.set_grad_enabled(tr):
        if k == "step":
            return _exact_step(case, d)
        leaves = {n: t.requires_grad_(tr) for n, t in d.items() if t.is_floating_point() and n != "dout"}
        if k == "attention":
            out = _mha64(d["qkv"], case["B"], case["T"], case["H"], case["H"], case["hd"], case["causal"])
        elif k == "mlp":
            out = _swiglu64(_rms64(d["x"], d["w"]) @ d["gate_up"].T) @ d["down"].T
        elif k == "head":
            logits = d["x"] @ d["lm"].T
            loss = torch.nn.functional.cross_entropy(logits, d["tgt"].long())
            if not tr:
                return {"logits": logits, "loss": loss}
            gx, gw = torch.autograd.grad(loss, [d["x"], d["lm"]])
            return {"loss": loss.detach(), "d_x": gx, "d_lm": gw}
        elif k == "mlp_fp8":
            r = torch.rsqrt(d["x"].pow(2).mean(-1) + EPS)
            ln = d["x"] * r[:, None] * d["w"]
            gu = _e4m3(ln) @ (_e4m3(d["gate_up"], 16.0) / 16.0).T
            sw = _swiglu64(gu)
            return {"ln": ln, "rstd": r, "gu": gu, "sw": sw, "y": _e4m3(sw) @ (_e4m3(d["down"], 16.0) / 16.0).T}
        elif k == "vit_block":
            B, T, H = case["B"], case["T"], case["H"]
            x = d["x"]
            qkv = _ln64(x, d["n1_w"], d["n1_b"]) @ d["qkv_w"].T + d["qkv_b"]
            x = x + _mha64(qkv, B, T, H, H, case["C"] // H, False) @ d["o_w"].T + d["o_b"]
            gu = _ln64(x, d["n2_w"], d["n2_b"]) @ d["gu_w"].T + d["gu_b"]
            out = x + _swiglu64(gu) @ d["down_w"].T + d["down_b"]
        else:
            x = d["x"]
            qkv = _rms64(x, d["ln1"]) @ d["qkv"].T
            if case["bias"]:
                qkv = qkv + d["qkv_bias"]
            x = x + _mha64(qkv, case["B"], case["T"], case["H"], case["Hkv"], case["C"] // case["H"], True) @ d["o"].T
            out = x + _swiglu64(_rms64(x, d["ln2"]) @ d["gate_up"].T) @ d["down"].T
        return _grads(out, d["dout"], leaves) if tr else {"out": out}


def _exact_step(case, d):
    """First AdamW step (lr 1e-4, betas 0.9 / 0.95, eps 1e-8, decay 0.1) on the bf16-rounded weights.  The rounding of the
    weights is part of the computation: master weights stay in 32 bits, products read their bf16 copy."""
    B, T, C, H, I, L, V = (case[n] for n in ("B", "T", "C", "H", "I", "L", "V"))
    n = B * T
    if n * (V + 12 * C * L) > 4e8:
        return None                      # more than twenty seconds, or more memory than the 64-bit activations have
    flat = d["master"].float().to(BF16).to(F64).requires_grad_(True)
    off = [0]

    def take(*shape):
        m = math.prod(shape)
        off[0] += m
        return flat[off[0] - m:off[0]].view(*shape)

    x = take(V, C)[d["ids"].long()]
    for _ in range(L):
        ln1, qkv, o, ln2, gu, down = take(C), take(3 * C, C), take(C, C), take(C), take(2 * I, C), take(C, I)
        x = x + _mha64(_rms64(x, ln1) @ qkv.T, B, T, H, H, C // H, True) @ o.T
        x = x + _swiglu64(_rms64(x, ln2) @ gu.T) @ down.T
    logits = _rms64(x, take(C)) @ take(V, C).T
    losses = torch.nn.functional.cross_entropy(logits, d["tgt"].long(), reduction="none")
    (g,) = torch.autograd.grad(losses.mean(), [flat])
    w = d["master"]
    return {"losses": losses.detach(), "grads": g, "weights": w - 1e-4 * (g / (g.abs() + 1e-8) + 0.1 * w)}
