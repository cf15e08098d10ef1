"""``few_row_linear``, ``skinny_linear`` and ``skinny8_linear`` outside the few-row kernels' own range: which kernel answers, and what is refused."""
import pytest
import torch

from idrak_b200 import _native
from idrak_b200.ops import gemm
from idrak_b200.ops.rowops import gated_activation
from idrak_b200.ops.skinny import few_row_linear, skinny8_linear, skinny_linear
from idrak_b200.quant.weights import Int8Weight

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("M,N", [(65, 12288), (300, 12800), (65, 49152)])
def test_more_rows_than_the_few_row_kernel_takes_go_to_the_dense_one(M, N):
    x, w, b, r = _rand(M, 64, seed=1), _rand(N, 64, seed=2), _rand(N, seed=3), _rand(M, N, seed=4)
    assert torch.equal(few_row_linear(x, w, b, r), gemm(x, w, bias=b, residual=r))
    assert torch.equal(few_row_linear(x[:9], w, b, gate="tanh"), gated_activation(gemm(x[:9], w, bias=b), "tanh"))
    gated = gated_activation(gemm(x, w, bias=b), "silu")
    half = r[:, : N // 2].contiguous()
    assert torch.equal(few_row_linear(x, w, b, gate="silu"), gated)
    out = torch.empty_like(half)
    assert few_row_linear(x, w, b, half, "silu", out=out) is out and torch.equal(out, gated + half)


@pytest.mark.parametrize("N", [264, 12288])
def test_results_go_where_they_were_asked_for(N):
    """fp32 results of a wide product as the dense kernel gives them, a destination also where the kernel does not take the
    call, and types that the kernels do not read are refused."""
    x, w = _rand(5, 64, seed=1), _rand(N, 64, seed=2)
    want = x.float() @ w.float().t()
    out = torch.full((5, N), float("nan"), device="cuda")
    if N >= 12288:
        few_row_linear(x, w, out=out)
        assert (out - want).abs().max() <= 1e-4
    else:
        with pytest.raises(AssertionError):
            skinny_linear(x, w, out=out)
    odd = _rand(5, 67, seed=3)[:, 1:65]                        # rows that start on two-byte boundaries
    dst = torch.zeros(5, N, dtype=torch.bfloat16, device="cuda")
    assert skinny_linear(odd, w, out=dst) is dst
    assert (dst.float() - odd.float() @ w.float().t()).abs().max() <= 2.0 ** -8 * 64
    for bad in ({"bias": torch.zeros(N, device="cuda")}, {"bias": _rand(N - 1)}, {"residual": torch.zeros(5, N, device="cuda")},
                {"residual": _rand(4, N)}):
        with pytest.raises(AssertionError):
            few_row_linear(x, w, **bad)


@pytest.mark.parametrize("M", [3, 20])
@pytest.mark.parametrize("ff", [24, 1000])
def test_int8_gate_whose_halves_start_between_16_byte_boundaries(M, ff):
    """The up half of the codes starts 8 bytes past a 16-byte boundary: the kernel answers all the same."""
    x, b, r = _rand(M, 128, seed=1), _rand(2 * ff, seed=2), _rand(M, ff, seed=3)
    w = Int8Weight.quantize(torch.randn(128, 2 * ff, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda") * 0.05)
    skinny8_linear(x, w, b, r, "silu")
    before = _native.lib().idrak_launch_count()
    got = skinny8_linear(x, w, b, r, "silu")
    assert _native.lib().idrak_launch_count() == before + 1
    y = x.double() @ w.dequantize().double() + b.double()
    a, u = y.chunk(2, -1)
    want = torch.nn.functional.silu(a) * u + r.double()
    # one rounding to bf16, fp32 sums of 128 terms and the fp32 activation
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-3).all()
    _native.check_status("gated int8 product")


@pytest.mark.parametrize("gate,cols", [(None, 200), ("silu", 208)])
def test_codes_padded_while_a_graph_is_recorded_are_not_kept(gate, cols):
    """The first use of a weight whose codes need another layout may be inside a recording: eager calls before the replay, the
    replay, and eager calls after the graph is gone all see the codes."""
    x = _rand(5, 128, seed=1)
    w = Int8Weight.quantize(torch.randn(128, cols, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda"))
    want = skinny8_linear(x, Int8Weight(w.codes[:, :cols].clone(), w.scales, 128, cols), gate=gate)
    fresh = Int8Weight(w.codes[:, :cols].contiguous() if gate is None else w.codes, w.scales, 128, cols)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        recorded = skinny8_linear(x, fresh, gate=gate)
    assert torch.equal(skinny8_linear(x, fresh, gate=gate), want)
    graph.replay()
    assert torch.equal(recorded, want)
    del graph, recorded
    torch.cuda.synchronize()
    assert torch.equal(skinny8_linear(x, fresh, gate=gate), want)
