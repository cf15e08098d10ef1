"""Runs a decoder over the paged KV cache: packed prefill of several prompts, and batched one-token decode.

Prefill packs the uncached tokens of every admitted prompt into one ``[1, T, dim]`` activation so each
projection is a single GEMM; attention then runs per prompt (flash kernel over that prompt's keys) and the
keys / values go to the prompt's cache blocks. Decode advances every running sequence by one token: one
GEMM per projection over ``[n, dim]``, in-place RoPE at each sequence's position, a paged cache write, the
split-KV decode-attention kernel over the block tables, the head GEMM, and the device sampler - the host
reads one int per sequence and nothing else.

Model features outside the kernels' fast path (attention soft-capping, scaled RoPE tables, query/key norms)
are composed from primitives around the same cache; numerics equal the training forward.

Reference: TextGenerator's prefill / decode loop (src/Idrak/Generation/TextGenerator.cs:569-623), KeyValueCache and
decode primitives (src/Idrak.Abstraction/Generation/Decoding.cs:243, Tensors/Tensor.Decoding.cs).
"""
from __future__ import annotations

import os
import weakref

from dataclasses import dataclass
from typing import List, Optional, Sequence

import numpy as np
import torch
from torch.nn.modules.module import _has_any_global_hook

from .. import ops
from ..models.decoder import Decoder, FeedForward, Norm, apply_rope_table, masked_attention, project
from ..ops import decode as dops


@dataclass
class PrefillItem:
    tokens: List[int]          # the tokens to compute (positions start .. start + len - 1)
    start: int                 # number of leading tokens already in the cache (shared prefix)
    blocks: List[int]          # block table covering positions 0 .. start + len


def fold_norms_into_projections(model: Decoder) -> bool:
    """Rewrites an inference copy of a pre-norm decoder so that every RMS norm's weight lives in the projection that
    follows it (query/key/value, gate/up, the head) and the norm itself has unit weight: ``norm(x) W^T`` becomes
    ``(x rstd) (W diag(w))^T``. Same function up to bf16 rounding of the folded weights, for every path (prefill, decode,
    training forward), and it lets the few-row decode kernel apply ``rstd`` in its epilogue instead of a norm launch.
    Returns False (and changes nothing) for models it does not cover: LayerNorm, post-norms, parallel blocks, experts,
    adapters or packed weights, tied embeddings (the head shares the embedding matrix)."""
    s = model.spec
    if getattr(model, "_norms_folded", False):
        return True
    if s.norm != "rms" or s.post_norms or s.parallel_blocks or s.experts > 0 or model.head is None:
        return False
    from ..ops.skinny import fold_norm
    blocks = list(model.blocks)
    for blk in blocks:
        if any(getattr(m, "adapters", None) is not None or getattr(m, "packed", None) for m in (blk.attn, blk.mlp)):
            return False
    with torch.no_grad():
        def fold(weight: torch.nn.Parameter, norm) -> None:
            weight.copy_(fold_norm(weight, norm.effective_weight()))
            norm.weight.fill_(1.0 - (s.norm_offset or 0.0))          # effective weight 1 from here on
        for blk in blocks:
            fold(blk.attn.qkv_weight, blk.attn_norm)
            fold(blk.mlp.up_weight, blk.mlp_norm)
        fold(model.head, model.norm)
    model._norms_folded = True
    return True


def _plain(module, cls) -> bool:
    """Whether calling ``module`` runs ``cls.forward`` and nothing besides (but for hooks on every module there is)."""
    if type(module) is not cls:
        return False
    d = module.__dict__
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or "forward" in d)


class ModelRunner:
    def __init__(self, model: Decoder, num_blocks: int, block_size: int = 16, max_batch: int = 256,
                 cache_dtype: Optional[torch.dtype] = None):
        self.model = model.eval()
        self.spec = model.spec
        p = next(model.parameters())
        self.device, self.dtype = p.device, p.dtype
        self.block_size, self.num_blocks, self.max_batch = block_size, num_blocks, max_batch
        s = self.spec
        cd = cache_dtype or self.dtype
        # one block more than the scheduler hands out: padding rows of a graph-replayed decode batch write there
        self.k_cache = [torch.zeros(num_blocks + 1, block_size, s.kv_heads, s.head_dim, dtype=cd, device=self.device)
                        for _ in range(s.layers)]
        self.v_cache = [torch.zeros_like(k) for k in self.k_cache]
        # an int8 cache keeps one fp32 scale per (slot, kv head) beside the codes
        self.kv_int8 = cd == torch.int8
        self.k_scale = self.v_scale = [None] * s.layers
        if self.kv_int8:
            self.k_scale = [torch.zeros(num_blocks + 1, block_size, s.kv_heads, dtype=torch.float32, device=self.device)
                            for _ in range(s.layers)]
            self.v_scale = [torch.zeros_like(k) for k in self.k_scale]
        self.trash_block = num_blocks
        self.max_blocks_per_seq = (s.max_positions + block_size - 1) // block_size
        self._graphs = {}
        self._graph_pool = None
        self._few_rows_ok = None
        self._state = self._model_state()
        self.graph_replays = 0

    # ------------------------------------------------------------------ sizing
    @staticmethod
    def blocks_that_fit(spec, bytes_available: int, block_size: int = 16, elem_bytes: int = 2) -> int:
        per_block = 2 * spec.layers * block_size * spec.kv_heads * (spec.head_dim * elem_bytes + (4 if elem_bytes == 1 else 0))
        return max(int(bytes_available // per_block), 1)

    # ------------------------------------------------------------------ shared pieces
    def _embed(self, ids: torch.Tensor, positions: torch.Tensor) -> torch.Tensor:
        m, s = self.model, self.spec
        x = ops.embedding(ids.view(1, -1), m.embed, None)
        if m.pos is not None:
            x = x + m.pos[positions.long()][None]
        if s.embedding_scale is not None:
            x = x * s.embedding_scale
        return x

    def _qkv(self, attn, x):
        adapters = getattr(attn, "adapters", None)
        packed = getattr(attn, "packed", {})
        if adapters is not None:
            from ..adapters.lora import _slices_attention, project_with_adapters
            qkv = project_with_adapters(x, attn.qkv_weight, attn.qkv_bias, adapters, _slices_attention(self.spec),
                                        packed=packed.get("qkv"))
            return qkv.contiguous()
        return project(x, attn.qkv_weight, packed.get("qkv"), attn.qkv_bias)

    def _out(self, attn, a, residual):
        adapters = getattr(attn, "adapters", None)
        packed = getattr(attn, "packed", {})
        if adapters is not None and "o" in adapters:
            from ..adapters.lora import project_with_adapters
            return project_with_adapters(a, attn.o_weight, attn.o_bias, adapters, {"o": (0, self.spec.dim)}, residual,
                                         packed=packed.get("o"))
        return project(a, attn.o_weight, packed.get("o"), attn.o_bias, residual)

    def _rotate_and_cache(self, attn, qkv2, positions, slots, li: int) -> None:
        """Query / key norms, RoPE (both in place on the packed projection) and the cache write of the new keys and
        values: one fused launch where the kernel covers the model's settings, the separate steps otherwise."""
        s = self.spec
        rope = attn.rope
        if rope is None or rope.scaling is None:
            qn = attn.q_norm.effective_weight() if s.qk_norm else None
            kn = attn.k_norm.effective_weight() if s.qk_norm else None
            dops.norm_rope_kv(qkv2, s.heads, s.kv_heads, s.head_dim, positions, slots, self.k_cache[li], self.v_cache[li],
                              self.k_scale[li], self.v_scale[li], qn, kn, s.norm_epsilon,
                              rope.theta if rope is not None else None, rope.rotary_dim if rope is not None else None)
            return
        self._rotate(attn, qkv2, positions)
        dops.norm_rope_kv(qkv2, s.heads, s.kv_heads, s.head_dim, None, slots, self.k_cache[li], self.v_cache[li],
                          self.k_scale[li], self.v_scale[li])

    def _cached_kv(self, li: int, blocks: torch.Tensor, total: int, dtype):
        """Keys and values of positions ``0 .. total`` of one sequence read back from its blocks: ``[1, total, Hkv, D]``."""
        s = self.spec
        k = self.k_cache[li][blocks].reshape(-1, s.kv_heads, s.head_dim)[:total]
        v = self.v_cache[li][blocks].reshape(-1, s.kv_heads, s.head_dim)[:total]
        if self.kv_int8:
            k = k.float() * self.k_scale[li][blocks].reshape(-1, s.kv_heads)[:total, :, None]
            v = v.float() * self.v_scale[li][blocks].reshape(-1, s.kv_heads)[:total, :, None]
        return k[None].to(dtype), v[None].to(dtype)

    def _rotate(self, attn, qkv2, positions):
        """RoPE (and query / key norms) in place on the packed ``[T, (H + 2 Hkv) D]`` projection."""
        s = self.spec
        H, Hkv, D = s.heads, s.kv_heads, s.head_dim
        T = qkv2.shape[0]
        qk = qkv2[:, : (H + Hkv) * D].unflatten(-1, (H + Hkv, D))
        if s.qk_norm:
            q = attn.q_norm(qk[:, :H].contiguous())
            k = attn.k_norm(qk[:, H:].contiguous())
            qk[:, :H].copy_(q)
            qk[:, H:].copy_(k)
        rope = attn.rope
        if rope is None:
            return
        if rope.scaling is None:
            ops.rope_(qk, positions, rope.theta, rope.rotary_dim, 1.0)
        else:
            r = apply_rope_table(qk[None], rope, positions[None])
            qk.copy_(r[0])

    def _block(self, blk, x, attend):
        """One decoder block around ``attend(attn_module, normed_x, residual_or_None)``; mirrors DecoderBlock.forward."""
        s = self.spec
        if s.parallel_blocks:
            h = blk.attn_norm(x)
            return x + attend(blk.attn, h, None) + blk.mlp(h)
        if s.post_norms:
            a = blk.post_attn_norm(attend(blk.attn, blk.attn_norm(x), None))
            x = x + a
            return x + blk.post_mlp_norm(blk.mlp(blk.mlp_norm(x)))
        x = attend(blk.attn, blk.attn_norm(x), x)
        return blk.mlp(blk.mlp_norm(x), x)

    def _logits(self, h: torch.Tensor) -> torch.Tensor:
        """``[rows, padded vocabulary]`` logits of already-normalised hidden rows."""
        m, s = self.model, self.spec
        logits = ops.linear(h, m.head_weight(), m.head_bias)
        if s.logit_softcap:
            c = s.logit_softcap
            logits = torch.tanh(logits.float() / c).mul(c).to(logits.dtype)
        return logits.reshape(-1, logits.shape[-1])

    # ------------------------------------------------------------------ prefill
    @torch.no_grad()
    def prefill(self, items: Sequence[PrefillItem], all_logits: bool = False) -> torch.Tensor:
        """Computes the listed tokens of every item, fills the cache, and returns the logits of each item's last
        token ``[len(items), padded vocabulary]`` (or of every computed token, packed, when ``all_logits``)."""
        s, dev = self.spec, self.device
        H, Hkv, D = s.heads, s.kv_heads, s.head_dim
        ids_t, pos_t, slots_t, last, bounds = self._pack(items)
        tables = [torch.tensor(it.blocks, dtype=torch.long, device=dev) if it.start > 0 else None for it in items]
        x = self._embed(ids_t, pos_t)
        runs = []                                  # (first item, count, length) of >= 2 fresh prompts of equal length
        i = 0
        while i < len(items):
            j = i
            while (j + 1 < len(items) and items[j + 1].start == 0 and items[i].start == 0
                   and len(items[j + 1].tokens) == len(items[i].tokens)):
                j += 1
            if j > i and len(items[i].tokens) % 8 == 0:
                runs.append((i, j - i + 1, len(items[i].tokens)))
            i = j + 1

        def attention(attn, qkv2, li):
            """Attention of every item over its own keys: ``[T, H D]`` from the packed projection."""
            q = qkv2[:, : H * D].unflatten(-1, (H, D))
            k = qkv2[:, H * D: (H + Hkv) * D].unflatten(-1, (Hkv, D))
            v = qkv2[:, (H + Hkv) * D:].unflatten(-1, (Hkv, D))
            window = s.sliding_window if s.is_windowed(attn.layer) else None
            fast = window is None and s.attention_softcap is None
            out = None
            done = set()

            def put(a, b, o):
                nonlocal out
                if (a, b) == (0, qkv2.shape[0]):
                    out = o.reshape(b - a, H * D)
                    return
                if out is None:
                    out = torch.empty(qkv2.shape[0], H * D, dtype=qkv2.dtype, device=dev)
                out[a:b] = o.reshape(b - a, H * D)

            if fast:
                # runs of fresh prompts of one length are contiguous in the pack: one batched attention launch
                for first, count, length in runs:
                    a, b = bounds[first], bounds[first + count]
                    put(a, b, self._flash(q[a:b].unflatten(0, (count, length)), k[a:b].unflatten(0, (count, length)),
                                          v[a:b].unflatten(0, (count, length)), attn.scale))
                    done.update(range(first, first + count))
            for i, it in enumerate(items):
                if i in done:
                    continue
                a, b = bounds[i], bounds[i + 1]
                qi = q[a:b][None]
                if it.start > 0:     # queries see the shared prefix too: read keys / values back from the cache
                    ki, vi = self._cached_kv(li, tables[i], it.start + (b - a), qkv2.dtype)
                else:
                    ki, vi = k[a:b][None], v[a:b][None]
                put(a, b, self._flash(qi, ki, vi, attn.scale) if fast
                    else masked_attention(qi, ki, vi, attn.scale, window, s.attention_softcap))
            return out if out is not None else qkv2.new_empty(qkv2.shape[0], H * D)

        if self._direct_prefill():
            # the kernels of the modules' forwards, in their order, without the modules: a short prompt is bound by the host
            x = x.view(ids_t.shape[0], -1)
            done = self._native_blocks(x, pos_t, slots_t, bounds, runs) if all(it.start == 0 for it in items) else None
            x = done if done is not None else self._row_blocks(x, pos_t, slots_t, attention, self._dense)
            return self._logits(self._norm(self.model.norm, x if all_logits else x[last]))

        layer_index = {id(blk.attn): i for i, blk in enumerate(self.model.blocks)}

        def attend(attn, h, residual):
            li = layer_index[id(attn)]
            qkv = self._qkv(attn, h)
            qkv2 = qkv.view(-1, qkv.shape[-1])
            self._rotate_and_cache(attn, qkv2, pos_t, slots_t, li)
            return self._out(attn, attention(attn, qkv2, li)[None], residual)

        for blk in self.model.blocks:
            x = self._block(blk, x, attend)
        if all_logits:
            return self._logits(self.model.norm(x))
        h = self.model.norm(x[0, last][None])
        return self._logits(h)

    @staticmethod
    def _flash(q, k, v, scale):
        """Causal attention of a prefill: the kernel without an autograd node where it takes the call."""
        if q.is_cuda and q.dtype == torch.bfloat16 and q.shape[-1] in (64, 128):
            return ops.flash_forward(q, k, v, True, scale)[0]
        return ops.attention(q, k, v, True, scale)

    def _pack(self, items: Sequence[PrefillItem]):
        """Token ids, positions and cache slots of the packed items (int32, on the device), the index of every item's last
        token, and the items' bounds in the pack. One copy from pinned memory that the host does not wait for: a copy per
        list from pageable memory made the GPU wait for the host before every prefill."""
        bs = self.block_size
        counts = [len(it.tokens) for it in items]
        bounds = [0]
        for n in counts:
            bounds.append(bounds[-1] + n)
        T = bounds[-1]
        meta = torch.empty(3 * T + len(items), dtype=torch.int32, pin_memory=self.device.type == "cuda")
        m = meta.numpy()
        for it, a, n in zip(items, bounds, counts):
            p = np.arange(it.start, it.start + n)
            m[a: a + n] = it.tokens
            m[T + a: T + a + n] = p
            m[2 * T + a: 2 * T + a + n] = np.asarray(it.blocks, dtype=np.int64)[p // bs] * bs + p % bs
        m[3 * T:] = np.asarray(bounds[1:]) - 1
        dev = meta.to(self.device, non_blocking=True)
        return dev[:T], dev[T: 2 * T], dev[2 * T: 3 * T], dev[3 * T:], bounds

    # ------------------------------------------------------------------ decode
    @torch.no_grad()
    def decode(self, tokens: torch.Tensor, positions: torch.Tensor, block_table: torch.Tensor,
               max_len_hint: Optional[int] = None) -> torch.Tensor:
        """One new token per sequence. ``tokens`` / ``positions`` int32 ``[n]`` (position = index of the new
        token), ``block_table`` int32 ``[n, max_blocks]``. Returns logits ``[n, padded vocabulary]``."""
        s, dev, bs = self.spec, self.device, self.block_size
        H, Hkv, D = s.heads, s.kv_heads, s.head_dim
        n = tokens.shape[0]
        slots, lens = dops.decode_slots(positions, block_table, bs)
        x = self._embed(tokens, positions)
        if n <= 64 and self._few_row_path():
            return self._decode_few_rows(x.view(n, -1), positions, slots, block_table, lens, max_len_hint)
        layer_index = {id(blk.attn): i for i, blk in enumerate(self.model.blocks)}

        def attend(attn, h, residual):
            li = layer_index[id(attn)]
            qkv = self._qkv(attn, h)
            qkv2 = qkv.view(-1, qkv.shape[-1])
            self._rotate_and_cache(attn, qkv2, positions, slots, li)
            q = qkv2[:, : H * D].unflatten(-1, (H, D))
            window = s.sliding_window if s.is_windowed(attn.layer) else 0
            if s.attention_softcap is None:
                o = dops.paged_decode(q, self.k_cache[li], self.v_cache[li], block_table, lens,
                                      attn.scale, window or 0, max_len_hint=max_len_hint,
                                      k_scale=self.k_scale[li], v_scale=self.v_scale[li])
            else:
                o = self._decode_softcap(q, li, block_table, lens, attn.scale, window or None)
            return self._out(attn, o.reshape(1, n, H * D), residual)

        for blk in self.model.blocks:
            x = self._block(blk, x, attend)
        return self._logits(self.model.norm(x))

    # ------------------------------------------------------------------ what the model holds at the moment
    def _model_state(self) -> list:
        """What the choice of path and a recorded decode step depend on and a program may change between calls: the blocks'
        modules, their adapters and packed weights, folded norms. Weak references, equal only while it is the same living
        object."""
        ref = weakref.ref
        state: list = [getattr(self.model, "_norms_folded", False)]
        for blk in self.model.blocks:
            for name in ("attn", "mlp"):
                m = blk._modules.get(name) or getattr(blk, name)      # a block may be wrapped
                state.append(ref(m))
                adapters = m._modules.get("adapters", m.__dict__.get("adapters"))
                state.append(adapters if adapters is None else ref(adapters))
                state += [ref(w) for w in (m.__dict__.get("packed") or {}).values()]
        return state

    def _follow_model(self) -> None:
        """Forgets the choice of path and the recorded decode steps when the model no longer holds what they were made for."""
        state = self._model_state()
        if state != self._state:
            self._state, self._few_rows_ok = state, None
            self._graphs, self._graph_pool = {}, None

    # ------------------------------------------------------------------ decode of at most 64 rows: fused projections
    def _few_row_path(self) -> bool:
        """Whether decode steps of up to 64 sequences run on the few-row kernels: one launch per projection with bias,
        residual add, gated activation and (with folded norms) the RMS norm inside it."""
        self._follow_model()
        if self._few_rows_ok is not None:
            return self._few_rows_ok
        from ..ops import skinny
        from .. import _native
        s = self.spec
        ok = (self.device.type == "cuda" and self.dtype == torch.bfloat16 and _native.has("idrak_skinny_gemm")
              and os.environ.get("IDRAK_FEW_ROW_DECODE", "1") != "0"
              and not s.parallel_blocks and not s.post_norms and s.experts == 0 and s.attention_softcap is None
              and s.gated and s.activation in skinny._KINDS and s.dim % 8 == 0 and s.ff_dim % 8 == 0
              and not s.logit_softcap)
        for blk in self.model.blocks:
            if not ok or not isinstance(blk.mlp, FeedForward):
                ok = False
                break
            rope = blk.attn.rope
            packed = [w for m in (blk.attn, blk.mlp) for w in (getattr(m, "packed", None) or {}).values()]
            dense = [w for w in (blk.attn.qkv_weight, blk.attn.o_weight, blk.mlp.up_weight, blk.mlp.down_weight) if w is not None]
            ok = (not any(getattr(m, "adapters", None) is not None for m in (blk.attn, blk.mlp))
                  and (rope is None or rope.scaling is None)
                  and (not packed or (self.few_row_packed and len(packed) == 4 and not dense
                                      and all(self._streams(w, "silu" if w is blk.mlp.packed["up"] else None) for w in packed))))
        self._few_rows_ok = bool(ok)
        return self._few_rows_ok

    few_row_packed = True          # the few-row path takes int8 / int4 weights too (a subclass with its own path may not)

    def _streams(self, w, gate) -> bool:
        """Whether the few-row kernels take a packed weight as it is stored (``ops.skinny.packed_supported``)."""
        from ..ops.skinny import packed_supported
        return (w.bits in (4, 8) and getattr(w, "kind", "int") == "int"
                and packed_supported(torch.empty(1, w.rows, dtype=self.dtype, device=self.device), w, gate))

    @staticmethod
    def _few(x, owner, name, residual=None, gate=None, norm_eps=None):
        """One few-row projection of a block: ``name`` in qkv / o / up / down of an attention or feed-forward module."""
        from ..ops.skinny import packed_linear, skinny_linear
        w, bias = getattr(owner, name + "_weight"), getattr(owner, name + "_bias")
        if w is None:
            assert norm_eps is None, "no norm inside a product over packed weights"
            return packed_linear(x, owner.packed[name], bias, residual, gate)
        return skinny_linear(x, w, bias, residual, gate, norm_eps)

    @staticmethod
    def _dense(x, owner, name, residual=None, gate=None):
        """The same projection of any number of rows on the dense (or unpacking) product, as the modules' forwards run it."""
        from ..ops.rowops import GATE_KINDS, gated_forward
        from ..quant.weights import qgemm
        w, bias = getattr(owner, name + "_weight"), getattr(owner, name + "_bias")
        if w is None:
            y = qgemm(x, owner.packed[name], False, bias, residual)
        else:
            y = ops.gemm(x, w, bias=bias, residual=residual)
        return y if gate is None else gated_forward(y, GATE_KINDS[gate])

    def _direct_prefill(self) -> bool:
        """Whether prefill calls the kernels of the modules' forwards itself: the few-row path's models, as long as the modules
        would run nothing else and the runner's own steps are the library's."""
        cls = type(self)
        if not (cls._block is ModelRunner._block and cls._qkv is ModelRunner._qkv and cls._out is ModelRunner._out
                and self._few_row_path() and _plain(self.model.norm, Norm)) or _has_any_global_hook():
            return False
        for blk in self.model.blocks:
            mods = blk._modules
            if not (_plain(mods.get("attn_norm"), Norm) and _plain(mods.get("mlp_norm"), Norm)
                    and _plain(mods.get("mlp"), FeedForward)):
                return False
        return True

    def _native_blocks(self, x, positions, slots, bounds, runs):
        """The blocks over fresh prompts as one native call, or ``None`` where the runner's own steps are a subclass's, or the call
        is not covered."""
        cls = type(self)
        if any(n in self.__dict__ or getattr(cls, n) is not getattr(ModelRunner, n) for n in ("_row_blocks", "_rotate_and_cache", "_dense", "_flash", "_norm")):
            return None
        from . import native_prefill
        return native_prefill.run(self, x, positions, slots, bounds, runs)

    @staticmethod
    def _norm(layer, t):
        """A norm layer's forward without an autograd node."""
        if not _plain(layer, Norm) or _has_any_global_hook():
            return layer(t)
        from ..ops.rowops import norm_forward
        return norm_forward(t, layer.effective_weight(), layer.bias, layer.eps, layer.kind != "layer")[0]

    def _row_blocks(self, x, positions, slots, attention, project, norm_eps=None):
        """The blocks over rows ``x [n, dim]``: (norm |) qkv | norms of q, k + RoPE + cache write | attention | out + residual
        | (norm |) gate/up, activation | down + residual. ``attention(attn, qkv, layer)`` gives ``[n, H D]`` from the packed
        projection; ``project`` is ``_few`` (at most 64 rows) or ``_dense``. With ``norm_eps`` the norms run inside the
        projections (folded weights, ``_few`` only) of the blocks whose weights are not packed."""
        for li, blk in enumerate(self.model.blocks):
            attn, mlp = blk.attn, blk.mlp
            fold = {"norm_eps": norm_eps} if norm_eps is not None and attn.qkv_weight is not None else {}
            qkv = project(x if fold else self._norm(blk.attn_norm, x), attn, "qkv", **fold)
            self._rotate_and_cache(attn, qkv, positions, slots, li)
            x = project(attention(attn, qkv, li), attn, "o", residual=x)
            g = project(x if fold else self._norm(blk.mlp_norm, x), mlp, "up", gate=self.spec.activation, **fold)
            x = project(g, mlp, "down", residual=x)
        return x

    def _decode_few_rows(self, x, positions, slots, block_table, lens, max_len_hint):
        s = self.spec
        H, D = s.heads, s.head_dim

        def attention(attn, qkv, li):
            window = s.sliding_window if s.is_windowed(attn.layer) else 0
            o = dops.paged_decode(qkv[:, : H * D].unflatten(-1, (H, D)), self.k_cache[li], self.v_cache[li], block_table, lens,
                                  attn.scale, window or 0, max_len_hint=max_len_hint, k_scale=self.k_scale[li],
                                  v_scale=self.v_scale[li])
            return o.reshape(-1, H * D)

        from ..ops.skinny import few_row_linear
        m = self.model
        eps = s.norm_epsilon if getattr(m, "_norms_folded", False) else None
        x = self._row_blocks(x, positions, slots, attention, self._few, eps)
        logits = few_row_linear(x if eps is not None else self._norm(m.norm, x), m.head_weight(), m.head_bias, norm_eps=eps)
        return logits.reshape(-1, logits.shape[-1])

    # ------------------------------------------------------------------ decode as a replayed CUDA graph
    BATCH_BUCKETS = (1, 2, 4, 8, 16, 32, 64, 96, 128, 160, 192, 224, 256)     # above 64 a row that is padded costs as any other

    @torch.no_grad()
    def decode_graphed(self, tokens: torch.Tensor, positions: torch.Tensor, block_table: torch.Tensor,
                       longest: int) -> torch.Tensor:
        """``decode`` recorded once per (batch bucket, context bucket) as a CUDA graph and replayed: a decode step is
        hundreds of small launches, and replaying them removes the host's share of the step. The batch is padded to
        the bucket with rows that write to a spare cache block; the context bucket fixes the key split of the
        attention kernel. Returns logits ``[n, padded vocabulary]`` (a view of the graph's output buffer)."""
        n = tokens.shape[0]
        bucket = next((b for b in self.BATCH_BUCKETS if b >= n), None)
        if bucket is None or self.device.type != "cuda" or self.spec.attention_softcap is not None:
            return self.decode(tokens, positions, block_table, max_len_hint=longest)
        ctx = 256
        while ctx < longest:
            ctx *= 2
        width = self.max_blocks_per_seq
        key = (bucket, ctx)
        self._follow_model()
        entry = self._graphs.get(key)
        if entry is None:
            tok = torch.zeros(bucket, dtype=torch.int32, device=self.device)
            pos = torch.zeros(bucket, dtype=torch.int32, device=self.device)
            tab = torch.full((bucket, width), self.trash_block, dtype=torch.int32, device=self.device)
            side = torch.cuda.Stream(device=self.device)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):                   # warm-up: lazy buffers and kernel attributes get created
                for _ in range(2):
                    self.decode(tok, pos, tab, max_len_hint=ctx)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, pool=self._graph_pool):
                out = self.decode(tok, pos, tab, max_len_hint=ctx)
            if self._graph_pool is None:
                self._graph_pool = graph.pool()
            entry = self._graphs[key] = (graph, tok, pos, tab, out)
        graph, tok, pos, tab, out = entry
        tok[:n].copy_(tokens, non_blocking=True)
        pos[:n].copy_(positions, non_blocking=True)
        if n < bucket:
            tok[n:].zero_()
            pos[n:].zero_()
            tab[n:].fill_(self.trash_block)
        w = block_table.shape[1]
        tab[:n, :w].copy_(block_table, non_blocking=True)
        graph.replay()
        self.graph_replays += 1
        return out[:n]

    def _decode_softcap(self, q, li, block_table, lens, scale, window):
        """Soft-capped scores (Gemma-2 style) composed from primitives, one sequence at a time."""
        s = self.spec
        out = torch.empty_like(q)
        for i in range(q.shape[0]):
            n = int(lens[i])
            blocks = block_table[i, : (n + self.block_size - 1) // self.block_size].long()
            k, v = self._cached_kv(li, blocks, n, q.dtype)
            out[i] = masked_attention(q[i][None, None], k, v, scale, window, s.attention_softcap)[0, 0]
        return out

    # ------------------------------------------------------------------ embeddings endpoint
    @torch.no_grad()
    def embed_text(self, tokens: Sequence[int], pooling: str = "mean") -> torch.Tensor:
        """A sentence vector from the final hidden states (mean over tokens, or the last token), L2-normalised."""
        ids = torch.tensor([list(tokens)], dtype=torch.int32, device=self.device)
        h = self.model.hidden(ids).float()[0]
        v = h.mean(0) if pooling == "mean" else h[-1]
        return torch.nn.functional.normalize(v, dim=0)
