"""Few-row projections for decoding (at most 64 token rows): one launch per projection with its epilogue inside.

``skinny_linear(x, w, ...)`` computes ``x @ w.T`` on the cluster split-K kernel (``csrc/skinny_gemm.cu``) and, in the
same launch, any of: a folded RMS norm of ``x`` (``norm_eps``: ``w`` must carry the norm weight in its columns, see
``fold_norm``), a bias, a residual add, and - with ``gate`` - the gated activation of a stacked ``[gate; up]`` matrix.
``skinny_reference`` is the fp32 statement of the same thing and the CPU path.

Reference: the fused few-row GEMV family (src/Idrak.Gpu/Cuda/PtxKernels.Quantized.cs:454-495).
"""
from __future__ import annotations

from typing import Optional

import torch

from .. import _native
from ._util import ptr, stream_ptr
from .rowops import GATE_KINDS, _gate_ref

MAX_ROWS = 64
_KINDS = {"silu": 0, "swiglu": 0, "gelu": 1, "geglu": 1, "relu": 2, "reglu": 2}


def fold_norm(weight: torch.Tensor, norm_weight: torch.Tensor) -> torch.Tensor:
    """``weight * norm_weight[None, :]``: the projection that, applied to ``x * rstd``, equals ``norm(x) @ weight.T``."""
    return (weight.float() * norm_weight.float()[None, :]).to(weight.dtype)


def skinny_reference(x, w, bias=None, residual=None, gate: Optional[str] = None, norm_eps: Optional[float] = None):
    xf = x.float()
    if norm_eps is not None:
        xf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + norm_eps)
    y = xf @ w.float().t()
    if bias is not None:
        y = y + bias.float()
    if gate is not None:
        ff = y.shape[-1] // 2
        y = _gate_ref(y[..., :ff], GATE_KINDS[gate]) * y[..., ff:]
    if residual is not None:
        y = y + residual.float()
    return y.to(x.dtype)


def supported(x: torch.Tensor, w: torch.Tensor, gate: Optional[str] = None) -> bool:
    return (x.is_cuda and _native.has("idrak_skinny_gemm") and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.dim() == 2
            and x.shape[0] <= MAX_ROWS and x.shape[1] % 8 == 0 and x.stride(1) == 1 and w.stride(1) == 1
            and x.stride(0) % 8 == 0 and w.stride(0) % 8 == 0 and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0
            and (gate is None or (gate in _KINDS and (w.shape[0] // 2) % 8 == 0)))


def _readable(M: int, N: int, outputs: int, bias, residual, out) -> bool:
    """Whether the few-row kernels read this bias and residual and write this result: bf16, whole, rows of unit stride."""
    bf16 = torch.bfloat16
    return ((bias is None or (bias.dtype == bf16 and bias.numel() == outputs))
            and all(t is None or (t.dtype == bf16 and t.shape == (M, N) and t.stride(1) == 1) for t in (residual, out)))


def skinny_linear(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
                  residual: Optional[torch.Tensor] = None, gate: Optional[str] = None,
                  norm_eps: Optional[float] = None, out: Optional[torch.Tensor] = None, one_pass: bool = False) -> torch.Tensor:
    """``x [M <= 64, K]``, ``w [N, K]`` (or ``[2 ff, K]`` with ``gate``) -> ``[M, N]`` (``[M, ff]``). With ``one_pass`` K is not cut:
    the bits of the dense kernel's uncut sum."""
    if not supported(x, w, gate):
        y = skinny_reference(x, w, bias, residual, gate, norm_eps)
        return y if out is None else out.copy_(y)
    M, K = x.shape
    N = w.shape[0] // 2 if gate is not None else w.shape[0]
    assert _readable(M, N, w.shape[0], bias, residual, out), "bias, residual and out are bf16 matrices of the result's shape"
    if out is None:
        out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    rc = _native.lib().idrak_skinny_gemm(
        x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), M, N, K, ptr(bias),
        ptr(residual), residual.stride(0) if residual is not None else 0, _KINDS[gate] if gate is not None else -1,
        float(norm_eps) if norm_eps is not None else -1.0, int(one_pass), stream_ptr())
    _native.check(rc, "idrak_skinny_gemm")
    return out


def wide_linear(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None,
                out: Optional[torch.Tensor] = None, one_pass: bool = False) -> torch.Tensor:
    """``x [M <= 256, K]`` times ``w [N, K]`` on the kernel for some more rows (``csrc/skinny_wide.cu``); operands as ``supported``
    asks of the few-row kernel's."""
    M, K = x.shape
    N = w.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=x.dtype, device=x.device)
    rc = _native.lib().idrak_skinny_wide(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), M, N, K,
                                         ptr(bias), ptr(residual), residual.stride(0) if residual is not None else 0, int(one_pass),
                                         stream_ptr())
    _native.check(rc, "idrak_skinny_wide")
    return out


# From this many weight rows on, and with more than 32 activation rows, the dense GEMM is level with the few-row kernel or
# ahead of it: many waves of tiles hide its split-K, and the few-row kernel reads the activations once per 128 weight rows.
# Measured at 32 / 64 activation rows, us, few-row against dense: 28672 x 4096 41 / 45 against 47 / 48, 50304 x 768 21.5 / 25.2
# against 22.7 / 23.5, 128256 x 4096 165 / 181 against 177 / 179.
DENSE_FROM_ROWS, DENSE_ABOVE_ROWS = 49152, 32
# From this many weight rows on, a call that the few-row kernel does not take (more than 64 rows, another gate, an fp32 result)
# runs on the dense GEMM, and below it as the fp32 statement, whose gated pair is not rounded before the activation.
WIDE_ROWS = 12288


def few_row_linear(x: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
                   residual: Optional[torch.Tensor] = None, gate: Optional[str] = None,
                   norm_eps: Optional[float] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """A decode-sized product on whichever of the two kernels measured faster for the weight's size: the few-row cluster
    kernel (fused epilogues) or, for a very wide plain product of more rows, the dense GEMM. The dense GEMM (and the activation
    kernel) also take a wide product that the few-row kernel does not. A folded norm (``norm_eps``) exists only in the few-row
    kernel."""
    M, rows = x.shape[0], w.shape[0]
    N = rows // 2 if gate is not None else rows
    if (norm_eps is None and rows >= WIDE_ROWS and supported(x[:MAX_ROWS], w) and (gate is None or N % 8 == 0)
            and (M > (DENSE_ABOVE_ROWS if gate is None and rows >= DENSE_FROM_ROWS else MAX_ROWS)
                 or not supported(x, w, gate) or not _readable(M, N, rows, bias, residual, out))):
        from .gemm import gemm
        if gate is None:
            return gemm(x, w, bias=bias, residual=residual, out=out)
        from .rowops import gated_activation
        y = gated_activation(gemm(x, w, bias=bias), gate)
        if residual is not None:
            y = y + residual
        return y if out is None else out.copy_(y)
    return skinny_linear(x, w, bias, residual, gate, norm_eps, out)


def skinny8_reference(x, w8, bias=None, residual=None, gate: Optional[str] = None):
    """fp32 statement of ``skinny8_linear``; ``w8`` is an ``Int8Weight`` ([in, out]; gated: out = [gate | up])."""
    y = x.float() @ w8.dequantize().to(x.device)
    if bias is not None:
        y = y + bias.float()
    if gate is not None:
        g, u = y.chunk(2, -1)
        act = {"silu": torch.nn.functional.silu, "swiglu": torch.nn.functional.silu, "relu": torch.relu, "reglu": torch.relu,
               "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh"),
               "geglu": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[gate]
        y = act(g) * u
    if residual is not None:
        y = y + residual.float()
    return y.to(x.dtype)


def packed_supported(x: torch.Tensor, w, gate: Optional[str] = None) -> bool:
    """Whether the few-row kernels take ``x @ W`` over this int8 / int4 weight: at most 64 bf16 rows, whole 16-byte chunks of
    inputs (int8) or whole groups of 32 (int4), and a gated weight's up half on a 16-byte boundary of the codes."""
    n_out = w.cols // 2 if gate is not None else w.cols
    step = 16 if w.bits == 8 else 32
    return (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.shape[0] <= MAX_ROWS and x.shape[1] == w.rows
            and w.rows % step == 0 and _native.has("idrak_skinny_packed") and w.codes.is_cuda
            and (w.bits == 8 or (w.ld % 4 == 0 and w.codes.data_ptr() % 16 == 0 and w.scale_ld % 8 == 0
                                 and w.scales.data_ptr() % 16 == 0))
            and (gate is None or (gate in _KINDS and w.cols % 2 == 0 and n_out % step == 0)))


def packed_linear(x: torch.Tensor, w, bias: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None,
                  gate: Optional[str] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x [M <= 64, K]`` times a packed int8 or int4 weight ``[K, N]`` (``packed_supported``) -> ``[M, N]``; with ``gate``
    the outputs are ``[gate | up]`` and the result is ``act(gate) * up`` ``[M, N / 2]``. The kernels stream the codes as
    they are stored and expand them on the way to the tensor cores."""
    M, K = x.shape
    n_out = w.cols // 2 if gate is not None else w.cols
    codes, up_col = w.codes, n_out
    if w.bits == 8:
        codes, up_col = w.gate_codes() if gate is not None else (w.tma_codes(), 0)
    if x.stride(1) != 1 or x.stride(0) % 8 or x.data_ptr() % 16:
        x = x.clone(memory_format=torch.contiguous_format)
    if out is None:
        out = torch.empty((M, n_out), dtype=torch.bfloat16, device=x.device)
    assert out.dtype == torch.bfloat16 and out.shape == (M, n_out) and out.stride(1) == 1
    if bias is not None:
        assert bias.dtype == torch.bfloat16 and bias.numel() == w.cols
    if residual is not None:
        assert residual.dtype == torch.bfloat16 and residual.shape == (M, n_out) and residual.stride(1) == 1
    rc = _native.lib().idrak_skinny_packed(x.data_ptr(), x.stride(0), codes.data_ptr(), codes.stride(0) * codes.element_size(),
                                           w.scales.data_ptr(), w.scale_ld, w.bits, out.data_ptr(), out.stride(0), M, n_out, K,
                                           ptr(bias), ptr(residual), residual.stride(0) if residual is not None else 0,
                                           _KINDS[gate] if gate is not None else -1, up_col, stream_ptr())
    _native.check(rc, "idrak_skinny_packed")
    return out


def skinny8_linear(x: torch.Tensor, w8, bias: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None,
                   gate: Optional[str] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``packed_linear`` over an int8 weight - also a gated one whose up half starts between 16-byte boundaries (a multiple of
    8 outputs), from a padded copy of the codes - or its fp32 statement where the kernels do not take the call."""
    if packed_supported(x, w8, gate) or (gate in _KINDS and w8.cols % 16 == 0 and packed_supported(x, w8)):
        return packed_linear(x, w8, bias, residual, gate, out)
    res = skinny8_reference(x, w8, bias, residual, gate)
    if out is not None:
        out.copy_(res)
        return out
    return res
