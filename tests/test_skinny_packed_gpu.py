"""The few-row products over packed weights (int8 and int4, both kernels) against the de-quantised product in 64 bits.

Bound per value: the result is rounded to bf16 once (relative 2^-9; the gated epilogue adds two roundings' worth of fp32
activation error), sums are fp32 over K terms (K 2^-24 of the sum of magnitudes), and int4 weights above 16 rows are rounded
to bf16 (2^-9 of the sum of magnitudes)."""
import pytest
import torch

from idrak_b200 import _native
from idrak_b200.ops.skinny import packed_linear, packed_supported
from idrak_b200.quant import qgemm, quantize_weight
from idrak_b200.quant.weights import Int8Weight

pytestmark = pytest.mark.gpu


def _inputs(kind, M, N, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + M * 7 + N)
    w = quantize_weight(torch.randn(K, N, generator=g, device="cuda") * 0.05, kind)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    return mk(M, K), w, mk(N), mk(M, N)


def _check(got, x, w, M, K, bias=None, residual=None, gate=False):
    wd = w.dequantize().double()
    y, mag = x.double() @ wd, x.double().abs() @ wd.abs()
    slack = mag * (K * 2.0 ** -24 + (2.0 ** -9 if w.bits == 4 and M > 16 else 0.0))
    if bias is not None:
        y = y + bias.double()
    if gate:
        (a, u), (sa, su) = y.chunk(2, -1), slack.chunk(2, -1)
        act = torch.nn.functional.silu(a)
        y = act * u
        slack = 1.1 * sa * u.abs() + act.abs() * su + sa * su + 2.0 ** -20 * y.abs()      # |silu'| < 1.1
    if residual is not None:
        y = y + residual.double()
    assert ((got.double() - y).abs() <= 2.0 ** -8 * y.abs() + slack + 1e-6).all()
    _native.check_status("packed few-row product")


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(136, 64), (1000, 1056), (4096, 512)])
def test_plain_bias_residual(kind, M, N, K):
    x, w, b, r = _inputs(kind, M, N, K)
    if not packed_supported(x, w):
        pytest.skip("outputs do not start on 16-byte boundaries of the codes")
    a = packed_linear(x, w)
    _check(a, x, w, M, K)
    assert torch.equal(a, packed_linear(x, w))                    # fixed order of the sums
    _check(packed_linear(x, w, b, r), x, w, M, K, b, r)


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(160, 64), (1056, 1056)])
def test_widths_that_end_inside_a_tile(kind, M, N, K):
    test_plain_bias_residual(kind, M, N, K)       # of the ragged widths above int4 takes none


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("M", [3, 16, 40])
@pytest.mark.parametrize("ff", [96, 1792])
def test_gated(kind, M, ff):
    x, w, b, _ = _inputs(kind, M, 2 * ff, 256)
    _check(packed_linear(x, w, b, gate="silu"), x, w, M, 256, b, gate=True)


@pytest.mark.parametrize("K", [16, 48, 1040])
def test_int8_inputs_that_end_inside_a_block(K):
    x, w, _, _ = _inputs("int8", 5, 256, K)
    _check(packed_linear(x, w), x, w, 5, K)
    x, w, _, _ = _inputs("int8", 20, 256, K)
    _check(packed_linear(x, w), x, w, 20, K)


def test_strided_rows_short_code_rows_and_routing():
    x_full, w, _, _ = _inputs("int8", 12, 200, 512)
    wide = torch.cat([torch.full_like(x_full, float("nan")), x_full], 1)
    x = wide[:, 512:]                                             # rows 1024 apart, NaN beside them
    ref = packed_linear(x_full, w)
    assert torch.equal(packed_linear(x, w), ref)
    assert torch.equal(qgemm(x, w), ref)
    short = Int8Weight(w.codes[:, :200].contiguous(), w.scales, 512, 200)      # rows of 200 bytes, as older files have
    assert short.ld % 16 and torch.equal(packed_linear(x, short), ref)
