"""Row-wise kernels (norms, activations, RoPE, embedding, column sums) vs plain PyTorch fp32."""
import pytest
import torch

from idrak_b200 import ops

pytestmark = pytest.mark.gpu


def _rand(shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _close(a, b, tol=2e-2):
    a, b = a.float(), b.float()
    err = (a - b).abs().max().item()
    assert err <= tol * (b.abs().max().item() + 1e-3), f"err {err}"


@pytest.mark.parametrize("rows,C", [(7, 64), (300, 768), (129, 1024), (33, 4096), (5, 8192)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_forward_backward(rows, C, rms):
    x = _rand((rows, C), 1.0, 1).requires_grad_()
    w = (_rand((C,), 0.2, 2).float() + 1).to(torch.bfloat16).requires_grad_()
    b = None if rms else _rand((C,), 0.2, 3).requires_grad_()
    y = ops.rms_norm(x, w, 1e-5) if rms else ops.layer_norm(x, w, b, 1e-5)
    dy = _rand((rows, C), 1.0, 4)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    br = None if rms else b.detach().float().requires_grad_()
    if rms:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    else:
        yr = torch.nn.functional.layer_norm(xr, (C,), wr, br, 1e-5)
    yr.backward(dy.float())
    _close(y, yr)
    _close(x.grad, xr.grad)
    _close(w.grad, wr.grad, 3e-2)
    if not rms:
        _close(b.grad, br.grad, 3e-2)


@pytest.mark.parametrize("rows,C", [(64, 64), (1000, 768), (4099, 1024), (16384, 768), (70, 256), (40, 4096)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_branch_adds_the_residual_gradient_and_leaves_column_sums(rows, C, rms):
    """``(norm(x), x)``: one backward kernel gives d(norm) + d(residual), the norm's parameter gradients and - where
    the row length fits the pipelined kernel - the column sums of that dx, which a following bias gradient reuses."""
    x = _rand((rows, C), 1.0, 1).requires_grad_()
    w = (_rand((C,), 0.2, 2).float() + 1).to(torch.bfloat16).requires_grad_()
    b = None if rms else _rand((C,), 0.2, 3).requires_grad_()
    y, xr_out = ops.norm_branch(x, w, b, 1e-5, rms)
    dy, dres = _rand((rows, C), 1.0, 4), _rand((rows, C), 1.0, 5)
    got = {}
    x.register_hook(lambda g: got.setdefault("dx", g))
    torch.autograd.backward([y, xr_out], [dy, dres])
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    br = None if rms else b.detach().float().requires_grad_()
    if rms:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    else:
        yr = torch.nn.functional.layer_norm(xr, (C,), wr, br, 1e-5)
    torch.autograd.backward([yr, xr], [dy.float(), dres.float()])
    _close(y, yr)
    _close(x.grad, xr.grad)
    _close(w.grad, wr.grad, 3e-2)
    if not rms:
        _close(b.grad, br.grad, 3e-2)
    tagged = getattr(got["dx"], "_idrak_colsum", None)
    from idrak_b200 import _native
    if _native.lib().idrak_norm_bwd_sums_dx(rows, C):
        assert 256 <= C <= 1024
        assert tagged is not None and tagged[1] == got["dx"]._version
        want = got["dx"].float().sum(0)
        assert (tagged[0] - want).abs().max().item() <= 1e-3 * max(1.0, want.abs().max().item())
        # deterministic: a second pass gives the same bits
        x2 = x.detach().clone().requires_grad_()
        y2, r2 = ops.norm_branch(x2, w.detach().requires_grad_(), None if rms else b.detach().requires_grad_(), 1e-5, rms)
        again = {}
        x2.register_hook(lambda g: again.setdefault("dx", g))
        torch.autograd.backward([y2, r2], [dy, dres])
        assert torch.equal(again["dx"], got["dx"]) and torch.equal(again["dx"]._idrak_colsum[0], tagged[0])


def test_bias_gradient_reuses_the_sums_left_by_the_norm_backward():
    """linear (with bias) -> pre-norm block input: the bias gradient must equal the one computed by a column-sum pass,
    and an in-place change of the gradient tensor must make the stale sums unusable."""
    from idrak_b200.ops.gemm import bias_grad
    dy = _rand((512, 768), 1.0, 7)
    ref = ops.colsum(dy)
    dy._idrak_colsum = (dy.float().sum(0), dy._version)
    got = bias_grad(dy.reshape(-1, 768), None, dy)
    _close(got, ref, 1e-2)
    dy.add_(1.0)                                    # version moves on: the attached sums no longer describe dy
    got = bias_grad(dy.reshape(-1, 768), None, dy)
    _close(got, dy.float().sum(0), 1e-2)


def test_norm_with_residual_sum():
    x, r = _rand((64, 768), 1.0, 1), _rand((64, 768), 1.0, 2)
    w, b = _rand((768,), 1.0, 3), _rand((768,), 1.0, 4)
    out, mean, rstd, summed = ops.norm_forward(x, w, b, 1e-5, False, residual=r)
    s_ref = (x.float() + r.float()).to(torch.bfloat16)
    assert torch.equal(summed, s_ref)
    _close(out, torch.nn.functional.layer_norm(s_ref.float(), (768,), w.float(), b.float(), 1e-5))


def test_gelu_and_gated():
    x = _rand((128, 3072), 2.0, 1).requires_grad_()
    y = ops.gelu(x)
    dy = _rand(x.shape, 1.0, 2)
    y.backward(dy)
    xr = x.detach().float().requires_grad_()
    yr = torch.nn.functional.gelu(xr, approximate="tanh")
    yr.backward(dy.float())
    _close(y, yr)
    _close(x.grad, xr.grad)
    for kind in ("silu", "gelu", "relu", "tanh"):
        gu = _rand((96, 2 * 1024), 1.5, 3).requires_grad_()
        o = ops.gated_activation(gu, kind)
        do = _rand(o.shape, 1.0, 4)
        o.backward(do)
        gr = gu.detach().float().requires_grad_()
        from idrak_b200.ops.rowops import _gate_ref, GATE_KINDS
        orf = _gate_ref(gr[:, :1024], GATE_KINDS[kind]) * gr[:, 1024:]
        orf.backward(do.float())
        _close(o, orf)
        _close(gu.grad, gr.grad)


def test_rope_matches_reference_and_inverts():
    x = _rand((50, 8, 64), 1.0, 1)
    pos = torch.arange(50, device="cuda", dtype=torch.int32) + 3
    y = x.clone()
    ops.rope_(y, pos, 10000.0)
    _close(y, ops.rope_reference(x, pos, 10000.0))
    ops.rope_(y, pos, 10000.0, inverse=True)
    _close(y, x)


def test_embedding_forward_backward():
    V, C, B, S = 1000, 256, 4, 64
    wte, wpe = _rand((V, C), 1.0, 1).requires_grad_(), _rand((S, C), 1.0, 2).requires_grad_()
    g = torch.Generator(device="cuda").manual_seed(3)
    ids = torch.randint(0, 50, (B, S), generator=g, device="cuda")   # many repeats
    out = ops.embedding(ids, wte, wpe)
    do = _rand(out.shape, 1.0, 4)
    out.backward(do)
    wr, pr = wte.detach().float().requires_grad_(), wpe.detach().float().requires_grad_()
    outr = wr[ids] + pr[None, :S]
    outr.backward(do.float())
    _close(out, outr)
    _close(wte.grad, wr.grad)
    _close(wpe.grad, pr.grad)


def test_colsum():
    x = _rand((1000, 200), 1.0, 1)
    _close(ops.colsum(x), x.float().sum(0), 1e-2)


@pytest.mark.parametrize("tokens,heads,D,rot", [(1, 1, 64, 64), (3, 5, 128, 128), (7, 40, 128, 64), (2000, 40, 128, 128),
                                                (1500, 33, 64, 64), (50, 3, 64, 32), (9, 4, 256, 128)])
@pytest.mark.parametrize("inverse", [False, True])
def test_rope_of_a_packed_projection(tokens, heads, D, rot, inverse):
    """A strided view of a packed projection, positions given: runs of heads per warp, partial rotary widths, and the
    general kernel (rot 32). One bf16 rounding (2^-8 of the pair's magnitude covers it and the angle's fp32 error)."""
    buf = _rand((tokens, heads * D + 2 * D), 1.0, 1)
    keep = buf.clone()
    x = buf[:, D: D + heads * D].unflatten(-1, (heads, D))
    pos = torch.randint(0, 5000, (tokens,), device="cuda", dtype=torch.int32, generator=torch.Generator(device="cuda").manual_seed(2))
    want = ops.rope_reference(x.clone(), pos, 10000.0, rot, 1.0, inverse).float()
    ops.rope_(x, pos, 10000.0, rot, 1.0, inverse)
    assert ((x.float() - want).abs() <= 2.0 ** -8 * 6 + 2e-3).all()
    assert torch.equal(buf[:, :D], keep[:, :D]) and torch.equal(buf[:, D + heads * D:], keep[:, D + heads * D:])
    assert torch.equal(x[..., rot:], keep[:, D: D + heads * D].unflatten(-1, (heads, D))[..., rot:])


@pytest.mark.parametrize("rows,C", [(400, 2048), (301, 2056), (400, 4096), (333, 8192), (5, 1032)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_of_long_rows_and_backward_with_a_frozen_weight(rows, C, rms):
    x, w, dy = _rand((rows, C), 1.0, 1).requires_grad_(), _rand((C,), 1.0, 2), _rand((rows, C), 1.0, 3)
    b = None if rms else _rand((C,), 1.0, 4)
    y = ops.rms_norm(x, w, 1e-5) if rms else ops.layer_norm(x, w, b, 1e-5)
    y.backward(dy)
    xr = x.detach().double().requires_grad_()
    if rms:
        yr = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    else:
        yr = torch.nn.functional.layer_norm(xr, (C,), w.double(), b.double(), 1e-5)
    yr.backward(dy.double())
    # one bf16 rounding each (2^-9) and fp32 sums
    assert ((y.double() - yr).abs() <= 2.0 ** -8 * yr.abs() + 1e-4).all()
    assert ((x.grad.double() - xr.grad).abs() <= 2.0 ** -8 * xr.grad.abs() + 1e-4).all()


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 2040), (5, 2048), (5, 2056), (70, 14336)])
def test_gated_activation_at_the_edges_of_a_block(rows, H):
    from idrak_b200.ops.rowops import GATE_KINDS, _gate_ref
    gu, do = _rand((rows, 2 * H), 1.5, 3).requires_grad_(), _rand((rows, H), 1.0, 4)
    o = ops.gated_activation(gu, "silu")
    o.backward(do)
    gr = gu.detach().float().requires_grad_()
    ref = _gate_ref(gr[:, :H], GATE_KINDS["silu"]) * gr[:, H:]
    ref.backward(do.float())
    _close(o, ref)
    _close(gu.grad, gr.grad)


@pytest.mark.parametrize("rows,H", [(257, 8), (1000, 24), (31, 64), (4097, 136)])
def test_gated_activation_of_narrow_rows(rows, H):
    test_gated_activation_at_the_edges_of_a_block(rows, H)


@pytest.mark.parametrize("parts", [1, 24, 25, 32, 33, 57, 128])
def test_column_sums_over_any_number_of_partials(parts):
    """One block of rows per partial: fewer than the four a thread keeps in flight, a multiple, and remainders."""
    x = _rand((64 * parts - 3, 72), 1.0, 7)
    out = torch.ones(72, device="cuda")
    ops.colsum(x, out=out, accumulate=True)
    want = x.double().sum(0) + 1.0
    # fp32 sums of the rows in a fixed order: at most rows * 2^-24 of the sum of magnitudes
    assert ((out.double() - want).abs() <= x.shape[0] * 2.0 ** -24 * (x.double().abs().sum(0) + 1.0)).all()


@pytest.mark.parametrize("rms", [False, True])
def test_norm_parameter_gradients_from_one_launch(rms):
    x, dy = _rand((1000, 136), 1.0, 8).requires_grad_(), _rand((1000, 136), 1.0, 9)
    w, b = _rand((136,), 1.0, 10).requires_grad_(), _rand((136,), 1.0, 11).requires_grad_()
    (ops.rms_norm(x, w) if rms else ops.layer_norm(x, w, b)).backward(dy)
    xr = x.detach().double()
    xh = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5) if rms else torch.nn.functional.layer_norm(xr, (136,), eps=1e-5)
    want = (dy.double() * xh).sum(0)
    # one rounding to bf16 and fp32 sums of 1000 terms
    assert ((w.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-2).all()
    if not rms:
        want = dy.double().sum(0)
        assert ((b.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-2).all()


@pytest.mark.parametrize("C", [8, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 1032, 2048])
@pytest.mark.parametrize("rows", [1, 7, 300, 1001])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_backward_with_a_frozen_weight_of_any_width(C, rows, rms):
    """Rows held by 8, 16 or 32 lanes and by a block, the last block of rows not full, the residual's gradient added."""
    from idrak_b200.ops.rowops import norm_backward, norm_forward
    x, w, dy, dres = _rand((rows, C), 1.0, 1), _rand((C,), 1.0, 2), _rand((rows, C), 1.0, 3), _rand((rows, C), 1.0, 4)
    b = None if rms else _rand((C,), 1.0, 5)
    _, mean, rstd, _ = norm_forward(x, w, b, 1e-5, rms)
    xr = x.double().requires_grad_()
    if rms:
        yr = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    else:
        yr = torch.nn.functional.layer_norm(xr, (C,), w.double(), b.double(), 1e-5)
    yr.backward(dy.double())
    for extra in (None, dres):
        dx, dw, db = norm_backward(dy, x, w, mean, rstd, rms, not rms, extra, frozen=True)
        want = xr.grad if extra is None else xr.grad + extra.double()
        assert dw is None and db is None
        # fp32 sums of C terms and one rounding to bf16 (2^-9)
        assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
