"""Serving-side ops: paged KV cache writes, decode attention over block tables, device-side sampling.

Each op runs the sm_100a kernel on CUDA tensors and a plain PyTorch statement of the same math on CPU
tensors (the oracle of the GPU tests and the engine's CPU path).

Reference: Tensor.AttentionRows / KeyValueWrite / SampleRows (src/Idrak.Abstraction/Tensors/Tensor.Decoding.cs),
KeyValueCache (src/Idrak.Abstraction/Generation/Decoding.cs:243), TokenSampler (TokenSamplers.cs).
"""
from __future__ import annotations

import ctypes as C
import math
from typing import Optional

import torch

from .. import _native
from ._util import ptr, scratch, stream_ptr

_BOUND = False


def _bind():
    global _BOUND
    if _BOUND:
        return
    vp, i, f, ll = C.c_void_p, C.c_int, C.c_float, C.c_longlong
    _native.bind("idrak_decode_partial_floats", ll, [i, i, i, i])
    _native.bind("idrak_paged_decode_kv", i, [vp, C.c_longlong, vp, vp, vp, vp, vp, vp, vp, vp, i, i, i, i, i, i, ll, i, i, f, i, vp])
    _native.bind("idrak_norm_rope_kv", i, [vp, ll, vp, vp, vp, vp, vp, vp, vp, vp, f, f, f, i, i, i, i, i, i, vp])
    _native.bind("idrak_decode_slots", i, [vp, vp, i, ll, i, i, vp, vp, vp])
    _native.bind("idrak_kv_write_paged", i, [vp, vp, ll, vp, vp, vp, i, i, vp])
    _native.bind("idrak_argmax_rows", i, [vp, i, i, i, ll, vp, vp])
    _native.bind("idrak_sample_rows", i, [vp, i, i, i, ll, vp, vp, vp, vp, vp, vp, vp, i, vp, vp, vp, vp, C.c_uint, vp])
    _BOUND = True


# --------------------------------------------------------------------------- KV cache
def decode_slots(positions: torch.Tensor, block_table: torch.Tensor, block_size: int):
    """``(slots, lens)`` int32 of a decode step: the cache slot of every sequence's new token (at ``positions``, looked up in
    ``block_table [n, width]``) and the sequence's length with it. On the GPU a position outside the table's row gives slot
    -1, which cache writes skip, and a bad argument in the status word."""
    if positions.is_cuda and block_table.dim() == 2 and block_table.shape[0] < positions.shape[0]:
        raise IndexError(f"{positions.shape[0]} positions for a block table of {block_table.shape[0]} rows")
    if (positions.is_cuda and positions.dtype == torch.int32 and block_table.dtype == torch.int32
            and block_table.device == positions.device and positions.dim() == 1 and block_table.dim() == 2
            and positions.is_contiguous() and block_table.stride(1) == 1 and block_table.shape[1] > 0):
        _bind()
        out = torch.empty((2, positions.shape[0]), dtype=torch.int32, device=positions.device)
        rc = _native.lib().idrak_decode_slots(positions.data_ptr(), block_table.data_ptr(), positions.shape[0],
                                              block_table.stride(0), block_table.shape[1], block_size, out[0].data_ptr(),
                                              out[1].data_ptr(), stream_ptr())
        _native.check(rc, "idrak_decode_slots")
        return out[0], out[1]
    rows = torch.arange(positions.shape[0], device=positions.device)
    slots = block_table[rows, (positions // block_size).long()] * block_size + positions % block_size
    return slots.to(torch.int32), (positions + 1).to(torch.int32)


def kv_write_paged(k_src: torch.Tensor, v_src: torch.Tensor, slots: torch.Tensor, k_cache: torch.Tensor,
                   v_cache: torch.Tensor) -> None:
    """Write the new tokens' keys / values (``[tokens, Hkv, D]`` views with packed heads) into cache slots
    ``slots[t] = block * block_size + offset`` (negative = skip)."""
    tokens, Hkv, D = k_src.shape
    row = Hkv * D
    if not k_src.is_cuda:
        flat_k, flat_v = k_cache.view(-1, row), v_cache.view(-1, row)
        keep = slots >= 0
        flat_k[slots[keep].long()] = k_src.reshape(tokens, row)[keep]
        flat_v[slots[keep].long()] = v_src.reshape(tokens, row)[keep]
        return
    _bind()
    assert k_src.stride(2) == 1 and k_src.stride(1) == D and v_src.stride(0) == k_src.stride(0)
    assert slots.dtype == torch.int32
    rc = _native.lib().idrak_kv_write_paged(k_src.data_ptr(), v_src.data_ptr(), k_src.stride(0), slots.data_ptr(),
                                            k_cache.data_ptr(), v_cache.data_ptr(), tokens, row, stream_ptr())
    _native.check(rc, "idrak_kv_write_paged")


def quantize_kv_reference(x: torch.Tensor):
    """int8 codes and one fp32 scale per (token, head) of ``[tokens, heads, D]``: scale = max|x| / 127."""
    xf = x.float()
    mx = xf.abs().amax(-1)
    scale = torch.where(mx > 0, mx / 127.0, torch.ones_like(mx))
    q = torch.round(xf / scale[..., None]).clamp(-127, 127).to(torch.int8)
    return q, scale


def norm_rope_kv(qkv: torch.Tensor, heads: int, kv_heads: int, head_dim: int, positions: Optional[torch.Tensor],
                 slots: Optional[torch.Tensor], k_cache: Optional[torch.Tensor], v_cache: Optional[torch.Tensor],
                 k_scale: Optional[torch.Tensor] = None, v_scale: Optional[torch.Tensor] = None,
                 q_norm_weight: Optional[torch.Tensor] = None, k_norm_weight: Optional[torch.Tensor] = None,
                 eps: float = 1e-6, theta: Optional[float] = None, rot_dim: Optional[int] = None,
                 freq_scale: float = 1.0) -> None:
    """In place on the packed projection ``[T, (H + 2 Hkv) D]``: per-head RMS norm of queries and keys (when weights
    are given), RoPE of both (when ``theta`` is given), and the write of keys / values into the paged cache rows
    ``slots`` - bf16, or int8 codes with one scale per (slot, kv head) when ``k_scale`` / ``v_scale`` are given. One
    kernel launch on the GPU; the CPU path composes the same steps."""
    T = qkv.shape[0]
    H, Hkv, D = heads, kv_heads, head_dim
    rot = (rot_dim or D) if theta is not None else 0
    fused = (qkv.is_cuda and qkv.dtype == torch.bfloat16 and D in (64, 128, 256) and rot % 64 == 0
             and qkv.stride(1) == 1)
    if fused:
        _bind()
        int8 = k_scale is not None
        rc = _native.lib().idrak_norm_rope_kv(
            qkv.data_ptr(), qkv.stride(0), ptr(positions), ptr(slots), ptr(k_cache), ptr(v_cache), ptr(k_scale),
            ptr(v_scale), ptr(q_norm_weight), ptr(k_norm_weight), float(eps), float(theta or 10000.0), float(freq_scale),
            int(rot), T, H, Hkv, D, int(int8), stream_ptr())
        _native.check(rc, "idrak_norm_rope_kv")
        return
    from .rowops import rope_
    qk = qkv[:, : (H + Hkv) * D].unflatten(-1, (H + Hkv, D))

    def rms(x, w):
        xf = x.float()
        return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()).to(x.dtype)
    if q_norm_weight is not None:
        qk[:, :H].copy_(rms(qk[:, :H], q_norm_weight))
    if k_norm_weight is not None:
        qk[:, H:].copy_(rms(qk[:, H:], k_norm_weight))
    if theta is not None:
        rope_(qk, positions, theta, rot_dim, freq_scale)
    if slots is None:
        return
    k = qkv[:, H * D: (H + Hkv) * D].unflatten(-1, (Hkv, D))
    v = qkv[:, (H + Hkv) * D:].unflatten(-1, (Hkv, D))
    if k_scale is None:
        kv_write_paged(k, v, slots, k_cache, v_cache)
        return
    keep = slots >= 0
    idx = slots[keep].long()
    for src, cache, scales in ((k, k_cache, k_scale), (v, v_cache, v_scale)):
        q8, sc = quantize_kv_reference(src[keep])
        cache.view(-1, Hkv, D)[idx] = q8
        scales.view(-1, Hkv)[idx] = sc


def paged_decode_reference(q, k_cache, v_cache, block_table, seq_lens, scale=None, window: int = 0,
                           k_scale=None, v_scale=None):
    if k_scale is not None:
        k_cache = (k_cache.float() * k_scale.view(*k_cache.shape[:3], 1)).to(q.dtype)
        v_cache = (v_cache.float() * v_scale.view(*v_cache.shape[:3], 1)).to(q.dtype)
    seqs, H, D = q.shape
    _, bs, Hkv, _ = k_cache.shape
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    out = torch.zeros_like(q, dtype=torch.float32)
    for s in range(seqs):
        n = int(seq_lens[s])
        if n == 0:
            continue
        blocks = block_table[s, : (n + bs - 1) // bs].long()
        k = k_cache[blocks].reshape(-1, Hkv, D)[:n].float()
        v = v_cache[blocks].reshape(-1, Hkv, D)[:n].float()
        if window and n > window:
            k, v = k[n - window:], v[n - window:]
        k = k.repeat_interleave(H // Hkv, dim=1)
        v = v.repeat_interleave(H // Hkv, dim=1)
        sc = torch.einsum("hd,nhd->hn", q[s].float(), k) * scale
        out[s] = torch.einsum("hn,nhd->hd", torch.softmax(sc, -1), v)
    return out.to(q.dtype)


DECODE_TILE, DECODE_CTAS = 16, 16384


def key_shares(seqs: int, kv_heads: int, longest: int, window: int = 0, sms: int = 148):
    """``(splits, min_keys)`` of a decode step: by how many CTAs per KV head a sequence's keys are shared at most, and how many
    keys a share has at least, from a bound on the lengths alone (a power of two above the longest).

    A share costs a CTA's set-up and a partial result to merge, a long one is a long chain. With the machine idle the best share
    grows like the square root of the length (128 keys below 4096, then 256, 512 from 16384 on), as long as the CTAs are there
    together, three to an SM: a second round costs as much as the first. With sequences x KV heads from a quarter of the SMs on,
    each has few shares and unequal lengths weigh more: 1024 CTAs if every sequence had the bound, and 256 keys at least from
    half of the SMs, 512 from all of them on. From two CTAs per SM on shares only even out a batch: 1024 keys, 2048 from five per
    SM on. Measured over 476 batches of 50 to 32000 keys, equal, mixed, or one long one among short ones, head sizes 64 and 128:
    4, 4 and 10 % above the best choice for each on average, where two CTAs per SM and none beyond are 9, 11 and 145 % above it.
    us, shares of 128 / 256 / 512 / 1024 keys: one sequence of 4000, 8 KV heads 17 / 15 / 18 / 29, of 32000 53 / 52 / 53 / 44;
    64 of 100 to 4000 192 / 143 / 122 / 115 (unsplit 128), 200 of 300 115 / 97 / 69 unsplit.

    At most 64 shares, and 16384 CTAs in all: each has a partial result in HBM and is launched whether its sequence reaches it or
    not. 256 sequences of 8 KV heads under a bound of 32768, us, unsplit / 8 / 32 shares: one of 32000 tokens and the others of
    300 717 / 212 / 199, all of 300 94 / 110 / 161 (136 MB of partial results at 32 query heads of 128, 34 at 8 shares)."""
    if window > 0:
        longest = min(longest, window + DECODE_TILE)       # a window may start inside a tile
    if longest <= 256:
        return 1, 128
    heads = max(seqs * kv_heads, 1)
    share = 128 << max(0, (longest.bit_length() - 11) // 2)
    if heads > sms // 4:
        if heads > 2 * sms:
            share = max(share, 1024 if heads <= 5 * sms else 2048)
        elif heads > sms and longest <= 1024:
            share = max(share, 1024)
        else:
            least = 128 if heads <= sms // 2 else 256 if heads <= sms else 512
            share = max(share, least, min(1024, -(-longest * heads // 1024 // 128) * 128))
        # to the nearest: a window may leave a share of one tile
        return max(1, min((longest + share // 2) // share, 64, DECODE_CTAS // heads)), share
    splits, together = min(-(-longest // share), 64), 3 * sms // heads
    if splits > together:
        splits = together if longest <= 8192 or together >= 16 else max(together, min(splits, longest // 1024))
    return splits, share


def paged_decode(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, block_table: torch.Tensor,
                 seq_lens: torch.Tensor, scale: Optional[float] = None, window: int = 0,
                 splits: Optional[int] = None, max_len_hint: Optional[int] = None,
                 k_scale: Optional[torch.Tensor] = None, v_scale: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One query token per sequence against its cached keys / values. q: ``[seqs, H, D]``. With ``k_scale`` /
    ``v_scale`` (``[blocks, block_size, Hkv]`` fp32) the caches hold int8 codes."""
    if not q.is_cuda:
        return paged_decode_reference(q, k_cache, v_cache, block_table, seq_lens, scale, window, k_scale, v_scale)
    _bind()
    seqs, H, D = q.shape
    _, bs, Hkv, _ = k_cache.shape
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    lib = _native.lib()
    min_keys = 0
    if splits is None:
        longest = max_len_hint if max_len_hint is not None else block_table.shape[1] * bs
        splits, min_keys = key_shares(seqs, Hkv, longest, window, lib.idrak_sm_count())
    out = torch.empty(seqs, H, D, dtype=q.dtype, device=q.device)
    part = None
    if splits > 1:
        part = scratch("decode_partial", lib.idrak_decode_partial_floats(seqs, H, D, splits), torch.float32, q.device)
    if q.stride(2) != 1 or q.stride(1) != D or q.stride(0) % 8 or q.data_ptr() % 16:
        q = q.contiguous()                     # heads must be packed; sequences may be a strided view
    assert block_table.dtype == torch.int32 and seq_lens.dtype == torch.int32
    rc = lib.idrak_paged_decode_kv(q.data_ptr(), q.stride(0), k_cache.data_ptr(), v_cache.data_ptr(), ptr(k_scale),
                                   ptr(v_scale), block_table.data_ptr(), seq_lens.data_ptr(), out.data_ptr(), ptr(part),
                                   seqs, H, Hkv, D, bs, block_table.shape[1], k_cache.shape[0] * bs, splits, min_keys, float(scale), int(window),
                                   stream_ptr())
    _native.check(rc, "idrak_paged_decode_kv")
    return out


# --------------------------------------------------------------------------- sampling
def argmax_rows(logits: torch.Tensor, vocab: Optional[int] = None) -> torch.Tensor:
    """Greedy token per row (lowest id among ties). logits: ``[rows, ld]`` bf16 or fp32."""
    rows, ld = logits.shape
    vocab = vocab or ld
    if not logits.is_cuda:
        return logits[:, :vocab].float().argmax(-1).to(torch.int32)
    _bind()
    assert logits.stride(1) == 1 and logits.dtype in (torch.bfloat16, torch.float32)
    ids = torch.empty(rows, dtype=torch.int32, device=logits.device)
    rc = _native.lib().idrak_argmax_rows(logits.data_ptr(), int(logits.dtype == torch.float32), rows, vocab,
                                         logits.stride(0), ids.data_ptr(), stream_ptr())
    _native.check(rc, "idrak_argmax_rows")
    return ids


def sample_rows_reference(logits, vocab, temperature, top_k, top_p, min_p, uniforms):
    """Same filtering as the kernel; ``uniforms[row]`` in [0,1) picks along the kept, sorted candidates."""
    out = []
    for r in range(logits.shape[0]):
        v = logits[r, :vocab].float() / max(float(temperature[r]), 1e-6)
        k = int(top_k[r]) if int(top_k[r]) > 0 else 64
        k = min(k, 64, vocab)
        vals, idx = torch.sort(v, descending=True, stable=True)
        vals, idx = vals[:k], idx[:k]
        pr = torch.exp(vals - vals[0])
        keep = k
        if float(min_p[r]) > 0:
            keep = max(int((pr >= float(min_p[r]) * pr[0]).sum()), 1)
        if float(top_p[r]) < 1:
            cum = torch.cumsum(pr[:keep] / pr.sum(), 0)
            c = int((cum < float(top_p[r])).sum()) + 1
            keep = max(min(c, keep), 1)
        cum = torch.cumsum(pr[:keep], 0)
        u = float(uniforms[r]) * float(cum[-1])
        pick = int((cum <= u).sum())
        out.append(int(idx[min(pick, keep - 1)]))
    return torch.tensor(out, dtype=torch.int32)


def penalise_reference(logits, vocab, history, repeat_penalty=None, presence_penalty=None, frequency_penalty=None):
    """The kernel's penalties: tokens seen in ``history`` (-1 = empty) are divided / multiplied by the repeat
    penalty (positive / negative logits), then lose the presence penalty and count x the frequency penalty."""
    out = logits[:, :vocab].float().clone()
    for r in range(out.shape[0]):
        h = history[r][history[r] >= 0].long()
        if h.numel() == 0:
            continue
        ids, counts = torch.unique(h, return_counts=True)
        v = out[r, ids]
        rp = float(repeat_penalty[r]) if repeat_penalty is not None else 1.0
        if rp != 1.0:
            v = torch.where(v > 0, v / rp, v * rp)
        if presence_penalty is not None:
            v = v - float(presence_penalty[r])
        if frequency_penalty is not None:
            v = v - float(frequency_penalty[r]) * counts.float()
        out[r, ids] = v
    return out


def sample_rows(logits: torch.Tensor, vocab: int, temperature: torch.Tensor, top_k: torch.Tensor,
                top_p: torch.Tensor, min_p: torch.Tensor, seeds: torch.Tensor, step: int,
                history: Optional[torch.Tensor] = None, repeat_penalty: Optional[torch.Tensor] = None,
                presence_penalty: Optional[torch.Tensor] = None, frequency_penalty: Optional[torch.Tensor] = None,
                return_logprobs: bool = False):
    """Sample one token per row on the device. Per-row settings are tensors on the logits' device
    (float32 / int32; ``seeds`` int64)."""
    rows = logits.shape[0]
    if not logits.is_cuda:
        u = torch.empty(rows)
        for r in range(rows):      # one stream per row, so a row's draw does not depend on its batch neighbours
            g = torch.Generator().manual_seed((int(seeds[r]) * 1000003 + step) & 0x7FFFFFFFFFFFFFFF)
            u[r] = torch.rand(1, generator=g)[0]
        if history is not None:
            logits = penalise_reference(logits, vocab, history, repeat_penalty, presence_penalty, frequency_penalty)
        ids = sample_rows_reference(logits, vocab, temperature, top_k, top_p, min_p, u)
        return (ids, torch.zeros(rows)) if return_logprobs else ids
    _bind()
    ids = torch.empty(rows, dtype=torch.int32, device=logits.device)
    lp = torch.empty(rows, dtype=torch.float32, device=logits.device) if return_logprobs else None
    rc = _native.lib().idrak_sample_rows(
        logits.data_ptr(), int(logits.dtype == torch.float32), rows, vocab, logits.stride(0), ids.data_ptr(), ptr(lp),
        temperature.data_ptr(), top_k.data_ptr(), top_p.data_ptr(), min_p.data_ptr(), ptr(history),
        history.shape[1] if history is not None else 0, ptr(repeat_penalty), ptr(presence_penalty),
        ptr(frequency_penalty), seeds.data_ptr(), int(step), stream_ptr())
    _native.check(rc, "idrak_sample_rows")
    return (ids, lp) if return_logprobs else ids
