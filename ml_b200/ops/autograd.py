"""torch.autograd wiring of the fused ops.

The trainer itself drives forward and backward explicitly (flat gradient buffer, bucket hooks), but every op is also
available as a differentiable function so that the kernels can be composed into ordinary `nn.Module`s
(`ml_b200.models.modules`).  Each Function allocates its outputs, calls the same op entry points as the engine
(`ml_b200.ops`: sm_100a kernels for CUDA tensors, the fp32 oracle for CPU tensors) and saves exactly what the
backward kernels need.
"""
from __future__ import annotations

import torch

from .. import ops


def _like(x, *shape, dtype=None):
    return x.new_empty(*shape) if dtype is None else x.new_empty(*shape, dtype=dtype)


class Linear(torch.autograd.Function):
    """y[M,N] = x[M,K] @ W[N,K]^T (+ b[N], added to the fp32 accumulators); dW is summed in fp32 and rounded once to W's dtype."""

    @staticmethod
    def forward(ctx, x, W, b=None):
        ctx.save_for_backward(x, W)
        ctx.bias = None if b is None else b.dtype
        out = _like(x, x.shape[0], W.shape[0])
        if b is None:
            ops.linear_fwd(out, x.contiguous(), W.contiguous())
        else:
            ops.linear_bias_fwd(out, x.contiguous(), W.contiguous(), b.contiguous())
        return out

    @staticmethod
    def backward(ctx, dout):
        x, W = ctx.saved_tensors
        dout = dout.contiguous()
        dx = _like(x, *x.shape)
        ops.linear_dx(dx, dout, W.contiguous())
        dW = _like(W, *W.shape)
        ops.linear_dw_cast(dW, dout, x.contiguous())
        db = None
        if ctx.bias is not None:
            db = _like(dout, dout.shape[1], dtype=ctx.bias)
            ops.colsum(db, dout)
        return dx, dW, db


class RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        out = _like(x, *x.shape)
        rstd = _like(x, x.shape[0], dtype=torch.float32)
        ops.rmsnorm_fwd(out, rstd, x.contiguous(), w, eps)
        ctx.save_for_backward(x, w, rstd)
        return out

    @staticmethod
    def backward(ctx, dy):
        x, w, rstd = ctx.saved_tensors
        dx, dw = _like(x, *x.shape), _like(w, *w.shape)
        ops.rmsnorm_bwd_cast(dx, dw, dy.contiguous(), x.contiguous(), w, rstd)
        return dx, dw, None


class SwiGLU(torch.autograd.Function):
    """out[M,I] = silu(gu[:, :I]) * gu[:, I:]"""

    @staticmethod
    def forward(ctx, gu):
        ctx.save_for_backward(gu)
        out = _like(gu, gu.shape[0], gu.shape[1] // 2)
        ops.swiglu_fwd(out, gu.contiguous())
        return out

    @staticmethod
    def backward(ctx, dout):
        (gu,) = ctx.saved_tensors
        dgu = _like(gu, *gu.shape)
        ops.swiglu_bwd(dgu, dout.contiguous(), gu.contiguous())
        return dgu


class RopeCausalAttention(torch.autograd.Function):
    """qkv[B*T, (H + 2 Hkv) hd] -> out[B*T, H hd]: rotate-half RoPE on Q and K, then causal attention (scale 1/sqrt(hd)); every key /
    value head serves H / Hkv consecutive query heads (Hkv None: one each).  Rows behind the B*T are left alone."""

    @staticmethod
    def forward(ctx, qkv, cos, sin, B, T, H, hd, Hkv=None):
        heads = H if Hkv is None else Hkv
        width = (H + 2 * heads) * hd
        if heads < 1 or H % heads or qkv.numel() < B * T * width or qkv.numel() % width:
            raise ValueError(f"qkv {tuple(qkv.shape)} does not hold {B * T} rows of {H} query and 2 x {heads} key / value heads of {hd}")
        qkv = qkv.contiguous()
        q = _like(qkv, B * T, 3 * H * hd)
        ops.rope_copy(q, qkv.view(-1, width)[:B * T], cos, sin, B, T, H, hd, Hkv)
        out = _like(qkv, B * T, H * hd)
        lse = _like(qkv, B, H, T, dtype=torch.float32)
        ops.attn_fwd(out, lse, q, B, T, H, hd)
        ctx.save_for_backward(q, out, lse, cos, sin)
        ctx.dims = (B, T, H, hd)
        ctx.Hkv, ctx.shape = Hkv, qkv.shape
        return out

    @staticmethod
    def backward(ctx, dout):
        q, out, lse, cos, sin = ctx.saved_tensors
        B, T, H, hd = ctx.dims
        dqkv = _like(q, *q.shape)
        fused = ops.attn_bwd(dqkv, dout.contiguous(), q, out, lse, B, T, H, hd, rope=(cos, sin))
        if not fused:
            ops.rope_bwd(dqkv, cos, sin, B, T, H, hd)
        if ctx.Hkv not in (None, H):
            full, dqkv = dqkv, _like(q, B * T, (H + 2 * ctx.Hkv) * hd)
            ops.kv_group_sum(dqkv, full, B, T, H, hd, ctx.Hkv)
        if ctx.shape.numel() != dqkv.numel():
            used, dqkv = dqkv, dqkv.new_zeros(ctx.shape)
            dqkv.view(-1, used.shape[1])[:B * T] = used
        return dqkv.view(ctx.shape), None, None, None, None, None, None, None


class BidirAttention(torch.autograd.Function):
    """qkv[B*T, 3C] -> out[B*T, C]: attention without a mask (every token sees every token), scale 1/sqrt(hd)."""

    @staticmethod
    def forward(ctx, qkv, B, T, H, hd):
        q = qkv.contiguous()
        out = _like(qkv, B * T, H * hd)
        lse = _like(qkv, B, H, T, dtype=torch.float32)
        ops.attn_bidir_fwd(out, lse, q, B, T, H, hd)
        ctx.save_for_backward(q, out, lse)
        ctx.dims = (B, T, H, hd)
        return out

    @staticmethod
    def backward(ctx, dout):
        q, out, lse = ctx.saved_tensors
        B, T, H, hd = ctx.dims
        dqkv = _like(q, *q.shape)
        ops.attn_bidir_bwd(dqkv, dout.contiguous(), q, out, lse, B, T, H, hd)
        return dqkv, None, None, None, None


class LayerNorm(torch.autograd.Function):
    """y = (x - mean) * rstd * w + b over the last dimension (b may be None)."""

    @staticmethod
    def forward(ctx, x, w, b, eps):
        x = x.contiguous()
        out = _like(x, *x.shape)
        mean = _like(x, x.shape[0], dtype=torch.float32)
        rstd = _like(x, x.shape[0], dtype=torch.float32)
        ops.layernorm_fwd(out, mean, rstd, x, w, b, eps)
        ctx.save_for_backward(x, w, mean, rstd)
        ctx.has_b = b is not None
        return out

    @staticmethod
    def backward(ctx, dy):
        x, w, mean, rstd = ctx.saved_tensors
        dx, dw = _like(x, *x.shape), _like(w, *w.shape)
        db = _like(w, *w.shape) if ctx.has_b else None
        ops.layernorm_bwd_cast(dx, dw, db, dy.contiguous(), x, w, mean, rstd)
        return dx, dw, db, None


class CrossEntropy(torch.autograd.Function):
    """Mean loss over rows with tgt >= 0.  The gradient is computed here, in the same kernel, when it will be asked for."""

    @staticmethod
    def forward(ctx, logits, tgt):
        logits = logits.contiguous()
        losses = _like(logits, logits.shape[0], dtype=torch.float32)
        loss = _like(logits, (), dtype=torch.float32)
        grad = _like(logits, *logits.shape) if ctx.needs_input_grad[0] else None
        ops.ce_mean(loss, losses, grad, logits, tgt)
        if grad is not None:
            ctx.save_for_backward(grad)
        return loss

    @staticmethod
    def backward(ctx, g):
        (dlogits,) = ctx.saved_tensors
        out = _like(dlogits, *dlogits.shape)      # (not in place: a program can get at a Python node's saved tensors, or put a hook on them)
        ops.scale_dev(out, dlogits, g.float().contiguous())
        return out, None


class Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, wte, ids, T):
        out = _like(wte, ids.numel(), wte.shape[1])
        ops.embed_fwd(out, wte, ids)
        ctx.save_for_backward(ids)
        ctx.shape, ctx.T, ctx.dtype = wte.shape, T, wte.dtype
        return out

    @staticmethod
    def backward(ctx, dout):
        (ids,) = ctx.saved_tensors
        dw = torch.zeros(ctx.shape, dtype=torch.float32, device=dout.device)
        ops.embed_bwd(dw, dout.contiguous(), ids, ctx.T, 0)
        return dw.to(ctx.dtype), None, None


# What programs call.  Plain calls on CUDA tensors go through the extension module (csrc/torch/bridge.cpp), which runs the same kernels
# on the same saved tensors without the interpreter; it declines what is not plain, and that takes the Functions above.
def _plain(name, x, *args):
    if not getattr(x, "is_cuda", False):
        return NotImplemented
    b = ops.native_module().bridge()
    return NotImplemented if b is None else getattr(b, name)(x, *args)


def linear(x, W, b=None):
    y = _plain("linear", x, W, b)
    return Linear.apply(x, W, b) if y is NotImplemented else y


def rmsnorm(x, w, eps):
    y = _plain("rmsnorm", x, w, eps)
    return RMSNorm.apply(x, w, eps) if y is NotImplemented else y


def swiglu(gu):
    y = _plain("swiglu", gu)
    return SwiGLU.apply(gu) if y is NotImplemented else y


def rope_causal_attention(qkv, cos, sin, B, T, H, hd, Hkv=None):
    y = _plain("rope_causal_attention", qkv, cos, sin, B, T, H, hd, Hkv)
    return RopeCausalAttention.apply(qkv, cos, sin, B, T, H, hd, Hkv) if y is NotImplemented else y


def cross_entropy(logits, tgt):
    y = _plain("cross_entropy", logits, tgt)
    return CrossEntropy.apply(logits, tgt) if y is NotImplemented else y


def bidir_attention(qkv, B, T, H, hd):
    y = _plain("bidir_attention", qkv, B, T, H, hd)
    return BidirAttention.apply(qkv, B, T, H, hd) if y is NotImplemented else y


def layer_norm(x, w, b, eps):
    y = _plain("layer_norm", x, w, b, eps)
    return LayerNorm.apply(x, w, b, eps) if y is NotImplemented else y


embedding = Embedding.apply
