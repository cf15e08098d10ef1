"""The blocks of a prefill as one native call (``csrc/prefill.cpp``).

``run`` collects the pointers of a model's layers anew for every call - nothing is kept from one call for the next - and
refuses (returns ``None``) whatever the native loop does not cover, which the caller then runs launch by launch.

Reference: the prefill step of TextGenerator (src/Idrak/Generation/TextGenerator.cs:569-623).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from .. import _native
from ..ops._util import scratch, stream_ptr
from ..ops.rowops import GATE_KINDS

_POINTERS = ("attn_norm_w", "attn_norm_b", "qkv_w", "qkv_b", "q_norm", "k_norm", "o_w", "o_b", "mlp_norm_w", "mlp_norm_b", "up_w",
             "up_b", "down_w", "down_b", "k_cache", "v_cache", "k_scale", "v_scale")
_ROW = np.dtype([(n, np.uint64) for n in _POINTERS] + [(n, np.float64) for n in ("attn_norm_eps", "mlp_norm_eps", "scale", "theta")]
                + [("rot_dim", np.int64)])


class _Args(C.Structure):
    _fields_ = ([(n, C.c_void_p) for n in ("positions", "slots", "prompts", "x", "y", "normed", "qkv", "attn", "up", "act", "mean", "rstd",
                                           "lse", "workspace")]
                + [(n, C.c_longlong) for n in ("tokens", "dim", "heads", "kv_heads", "head_dim", "ff", "count", "attn_rms", "mlp_rms",
                                               "gate_kind", "kv_int8")] + [("qk_eps", C.c_double)])


def _bind():
    vp, i = C.c_void_p, C.c_int
    _native.bind("idrak_prefill_workspace", C.c_longlong, [i] * 5)
    _native.bind("idrak_prefill_blocks", i, [vp, i, vp, vp, vp])


def _pointer(t, shape, keep) -> int:
    """The address of a whole bf16 matrix or vector of this shape, 0 for none; raises ``ValueError`` for anything else."""
    if t is None:
        return 0
    if t.dtype != torch.bfloat16 or tuple(t.shape) != shape or not t.is_contiguous() or not t.is_cuda:
        raise ValueError
    at = t.data_ptr()
    if at % 16:
        raise ValueError
    keep.append(t)
    return at


def _layers(runner, keep) -> np.ndarray:
    s, blocks = runner.spec, runner.model.blocks
    dim, out, qkv, ff = s.dim, s.heads * s.head_dim, (s.heads + 2 * s.kv_heads) * s.head_dim, s.ff_dim
    rows = np.zeros(len(blocks), dtype=_ROW)
    for li, blk in enumerate(blocks):
        attn, mlp = blk.attn, blk.mlp
        if s.is_windowed(attn.layer) and s.sliding_window:
            raise ValueError
        rope = attn.rope
        vals = [_pointer(t, shape, keep) for t, shape in (
            (blk.attn_norm.effective_weight(), (dim,)), (blk.attn_norm.bias, (dim,)), (attn.qkv_weight, (qkv, dim)),
            (attn.qkv_bias, (qkv,)), (attn.q_norm.effective_weight() if s.qk_norm else None, (s.head_dim,)),
            (attn.k_norm.effective_weight() if s.qk_norm else None, (s.head_dim,)), (attn.o_weight, (dim, out)), (attn.o_bias, (dim,)),
            (blk.mlp_norm.effective_weight(), (dim,)), (blk.mlp_norm.bias, (dim,)), (mlp.up_weight, (2 * ff, dim)),
            (mlp.up_bias, (2 * ff,)), (mlp.down_weight, (dim, ff)), (mlp.down_bias, (dim,)))]
        if not (vals[2] and vals[6] and vals[10] and vals[12]):       # packed weights
            raise ValueError
        caches = [t.data_ptr() if t is not None else 0 for t in (runner.k_cache[li], runner.v_cache[li], runner.k_scale[li],
                                                                 runner.v_scale[li])]
        rows[li] = (*vals, *caches, blk.attn_norm.eps, blk.mlp_norm.eps, attn.scale, rope.theta if rope is not None else 10000.0,
                    (rope.rotary_dim or s.head_dim) if rope is not None else 0)
    return rows


def run(runner, x, positions, slots, bounds, runs):
    """``x [tokens, dim]`` (overwritten with the result) through every block; ``runs`` are ``(first, count, length)`` of the items
    that are attended together, an item each otherwise. ``None``: not covered."""
    s = runner.spec
    H, Hkv, D, T = s.heads, s.kv_heads, s.head_dim, x.shape[0]
    from ..runtime.tuning import tuner
    t = tuner()
    if (T == 0 or D not in (64, 128) or x.dtype != torch.bfloat16 or not x.is_contiguous() or t.enabled or t.entries()
            or any(blk.attn.rope is not None and (blk.attn.rope.rotary_dim or D) % 64 for blk in runner.model.blocks)):
        return None
    if s.dim % 8 or s.ff_dim % 8 or runner.k_cache[0].dtype not in (torch.bfloat16, torch.int8):
        return None
    keep = []
    try:
        layers = _layers(runner, keep)
    except ValueError:
        return None
    _bind()
    lib = _native.lib()
    # items of one length side by side are one batch
    prompts, done = [], {}
    for first, count, length in runs:
        done[first] = (count, length)
    i = 0
    while i < len(bounds) - 1:
        count, length = done.get(i, (1, bounds[i + 1] - bounds[i]))
        if length:
            prompts.append((bounds[i], count, length))
        i += count
    table = np.asarray(prompts, dtype=np.int64).reshape(-1, 3)
    dim, out, qkv, ff = s.dim, H * D, (H + 2 * Hkv) * D, s.ff_dim
    # y, normed, and one region that holds first qkv and attention, then gate, up and activation
    half = torch.empty(2 * T * dim + T * max(qkv + out, 3 * ff), dtype=torch.bfloat16, device=x.device)
    stats = torch.empty(2 * T + T * H, dtype=torch.float32, device=x.device)
    ws_elems = lib.idrak_prefill_workspace(T, dim, qkv, out, ff)
    ws = scratch("gemm_splitk", ws_elems, torch.float32, x.device) if ws_elems else None
    at, st = half.data_ptr(), stats.data_ptr()
    big = at + 4 * T * dim
    blk = runner.model.blocks[0]
    args = _Args(positions.data_ptr(), slots.data_ptr(), table.ctypes.data, x.data_ptr(), at, at + 2 * T * dim, big, big + 2 * T * qkv, big,
                 big + 4 * T * ff, st, st + 4 * T, st + 8 * T, ws.data_ptr() if ws is not None else None, T, dim, H, Hkv, D, ff,
                 len(table), int(blk.attn_norm.kind != "layer"), int(blk.mlp_norm.kind != "layer"), GATE_KINDS[s.activation],
                 int(runner.kv_int8), s.norm_epsilon)
    failed = C.c_int(0)
    rc = lib.idrak_prefill_blocks(layers.ctypes.data, len(layers), C.byref(args), C.byref(failed), stream_ptr())
    _native.check(rc, f"idrak_prefill_blocks (layer {failed.value})")
    return x
