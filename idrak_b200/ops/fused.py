"""Layer-level fused autograd functions used by the decoder on the GPU.

``qkv_attention``  packed QKV buffer -> (RoPE in place) -> flash attention; the backward pass writes
                   dQ, dK, dV straight into one d(QKV) buffer (strided outputs) and un-rotates in place.
``mlp_gelu``       x -> GELU(x W1^T + b1) W2^T + b2 (+ residual) with the GELU and its derivative (one tanh for
                   both) inside the first GEMM's epilogue and the multiplication by that derivative inside the
                   epilogue of the backward GEMM
                   (the reference's gemm_tc_nn_gelu / gemm_tc_nt_gelugrad pair,
                   src/Idrak.Gpu/Cuda/PtxKernels.TensorCore.cs:80-144).
``mlp_gated``      x -> act(x Wg^T) * (x Wu^T) -> W2 (+ residual) with gate and up in one GEMM.

CPU tensors take the plain PyTorch statement of the same math.
"""
from __future__ import annotations

import math

import torch

from .. import _native
from . import rowops
from ._util import stream_ptr
from .attention import attention_reference, flash_backward, flash_forward
from .gemm import gemm, weight_bias_grad, weight_grad
from .rowops import GATE_KINDS, _gate_ref, colsum, rope_, rope_reference


def _split_qkv(qkv, H, Hkv, D):
    B, S, _ = qkv.shape
    q = qkv[..., : H * D].unflatten(-1, (H, D))
    k = qkv[..., H * D: (H + Hkv) * D].unflatten(-1, (Hkv, D))
    v = qkv[..., (H + Hkv) * D:].unflatten(-1, (Hkv, D))
    return q, k, v


def _query_key_heads(qkv, heads, D):
    """The query and key heads of a packed projection as one ``[tokens, heads, D]`` view."""
    return qkv[..., : heads * D].unflatten(-1, (heads, D)).flatten(0, 1)


class _QkvAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, H, Hkv, D, causal, scale, rope_theta, rope_dim, rope_scale, positions, window=None,
                row_start=None, softcap=None):
        B, S, _ = qkv.shape
        q, k, v = _split_qkv(qkv, H, Hkv, D)
        if rope_theta is not None:
            # the projection output is ours to overwrite: rotate q and k (neighbouring heads) where they lie
            rope_(_query_key_heads(qkv, H + Hkv, D), positions, rope_theta, rope_dim, rope_scale, False)
        out, lse = flash_forward(q, k, v, causal, scale, window, row_start, softcap)
        ctx.save_for_backward(qkv, out, lse, positions)
        ctx.cfg = (H, Hkv, D, causal, scale, rope_theta, rope_dim, rope_scale)
        ctx.modes = (window, row_start, softcap)
        # qkv was rotated through its raw pointer; its producer (a projection) does not need it again
        return out.reshape(B, S, H * D)

    @staticmethod
    def backward(ctx, dout):
        qkv, out, lse, positions = ctx.saved_tensors
        H, Hkv, D, causal, scale, rope_theta, rope_dim, rope_scale = ctx.cfg
        B, S, _ = qkv.shape
        q, k, v = _split_qkv(qkv, H, Hkv, D)
        dqkv = torch.empty_like(qkv)
        dq, dk, dv = _split_qkv(dqkv, H, Hkv, D)
        window, row_start, softcap = ctx.modes
        flash_backward(dout.reshape(B, S, H, D), q, k, v, out, lse, causal, scale, (dq, dk, dv), window, row_start,
                       softcap)
        if rope_theta is not None:
            rope_(_query_key_heads(dqkv, H + Hkv, D), positions, rope_theta, rope_dim, rope_scale, True)
        return (dqkv,) + (None,) * 12


def _small_attention_grad(qkv, dout, H, Hkv, D, causal, scale):
    """d(qkv) of ``attention_reference`` over a packed projection in plain operations (fp32): differentiable once more, and over
    several upstream gradients at once."""
    B, S, _ = qkv.shape
    q, k, v = (t.float().transpose(1, 2) for t in _split_qkv(qkv, H, Hkv, D))
    G = H // Hkv
    k, v = k.repeat_interleave(G, dim=1), v.repeat_interleave(G, dim=1)
    do = dout.reshape(B, S, H, D).float().transpose(1, 2)
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=qkv.device).triu(1), float("-inf"))
    p = torch.softmax(s, dim=-1)
    dp = torch.matmul(do, v.transpose(-1, -2))
    ds = p * (dp - (p * dp).sum(-1, keepdim=True)) * scale
    dq, dk, dv = torch.matmul(ds, k), torch.matmul(ds.transpose(-1, -2), q), torch.matmul(p.transpose(-1, -2), do)
    dk, dv = (t.reshape(B, Hkv, G, S, D).sum(2) for t in (dk, dv))
    return torch.cat([t.transpose(1, 2).reshape(B, S, -1) for t in (dq, dk, dv)], -1).to(qkv.dtype)


class _SmallQkvAttention(torch.autograd.Function):
    """Attention over a packed projection with heads below 64 on the fp32 kernels (``csrc/small_attn.cu``)."""

    @staticmethod
    def forward(ctx, qkv, H, Hkv, D, causal, scale):
        B, S, _ = qkv.shape
        out = torch.empty(B, S, H * D, dtype=qkv.dtype, device=qkv.device)
        o32 = torch.empty(B, S, H * D, dtype=torch.float32, device=qkv.device)
        lse = torch.empty(B, H, S, dtype=torch.float32, device=qkv.device)
        rc = _native.lib().idrak_small_attention(qkv.data_ptr(), None, out.data_ptr(), None, o32.data_ptr(), lse.data_ptr(), B, S,
                                                 H, Hkv, D, int(causal), float(scale), stream_ptr())
        _native.check(rc, "idrak_small_attention")
        ctx.save_for_backward(qkv, o32, lse)
        ctx.cfg = (H, Hkv, D, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv, o32, lse = ctx.saved_tensors
        H, Hkv, D, causal, scale = ctx.cfg
        if torch.is_grad_enabled() or not torch._C._has_storage(dout) or dout.dtype != torch.bfloat16:
            return (_small_attention_grad(qkv, dout, H, Hkv, D, causal, scale),) + (None,) * 5
        B, S, _ = qkv.shape
        qkv, dout = _whole(qkv), _whole(dout)               # a hook may hand the saved tensor back in another place
        dqkv = torch.empty_like(qkv)
        rc = _native.lib().idrak_small_attention(qkv.data_ptr(), dout.data_ptr(), None, dqkv.data_ptr(), o32.contiguous().data_ptr(),
                                                 lse.contiguous().data_ptr(), B, S, H, Hkv, D, int(causal),
                                                 float(scale), stream_ptr())
        _native.check(rc, "idrak_small_attention")
        return (dqkv,) + (None,) * 5


def _whole(t):
    return t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _plain_call(t: torch.Tensor) -> bool:
    """Whether an operation on this tensor just runs: no transform, trace, forward-mode derivative or dispatch mode around it and
    an ordinary tensor. Everything else goes through torch's own operations, which take part in all of those."""
    return (type(t) in (torch.Tensor, torch.nn.Parameter) and torch._C._has_storage(t)
            and not torch._C._are_functorch_transforms_active() and torch._C._get_tracing_state() is None
            and not torch.compiler.is_compiling() and torch.autograd.forward_ad._current_level < 0
            and torch._C._len_torch_dispatch_stack() == 0)


def qkv_attention(qkv: torch.Tensor, heads: int, kv_heads: int, head_dim: int, causal: bool = True,
                  scale: float | None = None, rope_theta: float | None = None, rope_dim: int | None = None,
                  rope_scale: float = 1.0, positions: torch.Tensor | None = None, window: int | None = None,
                  row_start: torch.Tensor | None = None, softcap: float | None = None) -> torch.Tensor:
    """Self-attention over a packed ``[B, S, (H + 2*Hkv) * D]`` projection; returns ``[B, S, H*D]``.

    On the GPU the buffer is rotated in place (it must be a fresh projection output). ``window``, ``row_start``
    (``[B, S]`` first visible key per position: sequences packed into one row) and ``softcap`` as in
    ``ops.attention``."""
    B, S, _ = qkv.shape
    if qkv.is_cuda and qkv.dtype == torch.bfloat16 and head_dim in (64, 128):
        if positions is None and rope_theta is not None:
            positions = (torch.arange(S, device=qkv.device, dtype=torch.int32).repeat(B))
        return _QkvAttention.apply(qkv, heads, kv_heads, head_dim, causal, scale, rope_theta, rope_dim,
                                   rope_scale, positions, window, row_start, softcap)
    q, k, v = _split_qkv(qkv, heads, kv_heads, head_dim)
    if rope_theta is not None:
        pos = positions if positions is not None else torch.arange(S, device=qkv.device).repeat(B)
        q = rope_reference(q.reshape(B * S, heads, head_dim), pos, rope_theta, rope_dim, rope_scale).reshape(q.shape)
        k = rope_reference(k.reshape(B * S, kv_heads, head_dim), pos, rope_theta, rope_dim, rope_scale).reshape(k.shape)
    if (qkv.is_cuda and qkv.dtype == torch.bfloat16 and head_dim < 64 and head_dim % 8 == 0 and qkv.numel() > 0
            and not (window or row_start is not None or softcap) and heads % kv_heads == 0 and max(heads, B) <= 65535
            and _plain_call(qkv)):
        packed = qkv if rope_theta is None else torch.cat([t.flatten(2) for t in (q, k, v)], -1)
        return _SmallQkvAttention.apply(_whole(packed), heads, kv_heads, head_dim, causal,
                                        scale if scale is not None else 1.0 / math.sqrt(head_dim))
    return attention_reference(q, k, v, causal, scale, window, row_start, softcap).reshape(B, S, heads * head_dim)


class _MlpGelu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, residual):
        shape = x.shape
        x2 = x.reshape(-1, shape[-1])
        r2 = residual.reshape(-1, w2.shape[0]) if residual is not None else None
        h, dact = gemm(x2, w1, bias=b1, act="gelu_d")          # dact = gelu'(pre-activation), saved instead of it
        y = gemm(h, w2, bias=b2, residual=r2)
        ctx.save_for_backward(x2, w1, w2, dact, h)
        ctx.params = (w1, b1, w2, b2)
        ctx.flags = (b1 is not None, b2 is not None, residual is not None)
        return y.reshape(*shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w1, w2, dact, h = ctx.saved_tensors
        has_b1, has_b2, has_res = ctx.flags
        dy2 = dy.reshape(-1, w2.shape[0])
        if dy2.stride(1) != 1 or dy2.stride(0) != dy2.shape[1]:
            dy2 = dy2.contiguous()
        p_w1, p_b1, p_w2, p_b2 = ctx.params
        dw2, db2 = weight_bias_grad(dy2, h, p_w2, p_b2, dy) if has_b2 else (weight_grad(dy2, h, p_w2), None)
        dpre = gemm(dy2, w2, b_mn=True, act="mul_aux", aux=dact)
        dw1, db1 = weight_bias_grad(dpre, x2, p_w1, p_b1) if has_b1 else (weight_grad(dpre, x2, p_w1), None)
        dx = gemm(dpre, w1, b_mn=True).reshape(*dy.shape[:-1], w1.shape[1])
        return dx, dw1, db1, dw2, db2, (dy if has_res else None)


def mlp_gelu(x, w1, b1, w2, b2, residual=None):
    """``GELU(x W1^T + b1) W2^T + b2 (+ residual)``; weights in ``nn.Linear`` layout."""
    if x.is_cuda and x.dtype == torch.bfloat16:
        return _MlpGelu.apply(x, w1, b1, w2, b2, residual)
    h = torch.nn.functional.gelu(torch.nn.functional.linear(x, w1, b1), approximate="tanh")
    y = torch.nn.functional.linear(h, w2, b2)
    return y + residual if residual is not None else y


class _MlpGated(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, wgu, bgu, w2, b2, residual, kind):
        shape = x.shape
        x2 = x.reshape(-1, shape[-1])
        r2 = residual.reshape(-1, w2.shape[0]) if residual is not None else None
        gu = gemm(x2, wgu, bias=bgu)
        Hd = gu.shape[1] // 2
        act = torch.empty((gu.shape[0], Hd), dtype=gu.dtype, device=gu.device)
        from .. import _native
        from ._util import stream_ptr
        _native.check(_native.lib().idrak_gated_fwd(gu.data_ptr(), act.data_ptr(), gu.shape[0], Hd, kind,
                                                    stream_ptr()), "gated_fwd")
        y = gemm(act, w2, bias=b2, residual=r2)
        ctx.save_for_backward(x2, wgu, w2, gu, act)
        ctx.params = (wgu, bgu, w2, b2)
        ctx.flags = (bgu is not None, b2 is not None, residual is not None, kind)
        return y.reshape(*shape[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        from .. import _native
        from ._util import stream_ptr
        x2, wgu, w2, gu, act = ctx.saved_tensors
        has_bgu, has_b2, has_res, kind = ctx.flags
        dy2 = dy.reshape(-1, w2.shape[0])
        if dy2.stride(1) != 1 or dy2.stride(0) != dy2.shape[1]:
            dy2 = dy2.contiguous()
        p_wgu, p_bgu, p_w2, p_b2 = ctx.params
        dw2, db2 = weight_bias_grad(dy2, act, p_w2, p_b2, dy) if has_b2 else (weight_grad(dy2, act, p_w2), None)
        dact = gemm(dy2, w2, b_mn=True)
        dgu = torch.empty_like(gu)
        Hd = gu.shape[1] // 2
        _native.check(_native.lib().idrak_gated_bwd(gu.data_ptr(), dact.data_ptr(), dgu.data_ptr(), gu.shape[0], Hd,
                                                    kind, stream_ptr()), "gated_bwd")
        dwgu, dbgu = weight_bias_grad(dgu, x2, p_wgu, p_bgu) if has_bgu else (weight_grad(dgu, x2, p_wgu), None)
        dx = gemm(dgu, wgu, b_mn=True).reshape(*dy.shape[:-1], wgu.shape[1])
        return dx, dwgu, dbgu, dw2, db2, (dy if has_res else None), None


def mlp_gated(x, w_gate_up, b_gate_up, w_down, b_down, residual=None, kind: str = "silu"):
    """``down(act(gate(x)) * up(x)) (+ residual)`` with ``w_gate_up = [gate; up]`` stacked on the output dim."""
    k = GATE_KINDS[kind]
    if x.is_cuda and x.dtype == torch.bfloat16 and (w_gate_up.shape[0] // 2) % 8 == 0:
        return _MlpGated.apply(x, w_gate_up, b_gate_up, w_down, b_down, residual, k)
    gu = torch.nn.functional.linear(x, w_gate_up, b_gate_up)
    Hd = gu.shape[-1] // 2
    y = torch.nn.functional.linear(_gate_ref(gu[..., :Hd], k) * gu[..., Hd:], w_down, b_down)
    return y + residual if residual is not None else y
