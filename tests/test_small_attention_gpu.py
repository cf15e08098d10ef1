"""Attention of heads below 64 on the fp32 kernels, against the same statement in 64 bits and against torch's own operations."""
import math

import pytest
import torch

from idrak_b200.ops import attention_reference
from idrak_b200.ops.fused import _small_attention_grad, _split_qkv, qkv_attention

pytestmark = pytest.mark.gpu


def _case(B, S, H, Hkv, D, seed=0, sc=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = (torch.randn(B, S, (H + 2 * Hkv) * D, generator=g, device="cuda") * sc).to(torch.bfloat16)
    return qkv, torch.randn(B, S, H * D, generator=g, device="cuda").to(torch.bfloat16)


def _exact(qkv, do, H, Hkv, D, causal, scale=None):
    x = qkv.double().requires_grad_()
    q, k, v = _split_qkv(x, H, Hkv, D)
    B, S, _ = qkv.shape
    k, v = (t.repeat_interleave(H // Hkv, dim=2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * (scale or 1 / math.sqrt(D))
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v).reshape(B, S, H * D)
    return o.detach(), torch.autograd.grad(o, x, do.double())[0]


def _near(got, want):
    """fp32 sums (relative 1e-5 of the largest value) and one rounding to bf16 (half a unit in the last of 8 bits: 2^-8 of the value at most)."""
    return ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * want.abs().max()).all()


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H,Hkv,D", [(1, 1, 1, 1, 8), (8, 128, 4, 4, 32), (2, 31, 4, 2, 16), (3, 33, 2, 2, 24), (1, 200, 6, 2, 40), (40, 130, 4, 2, 32), (30, 100, 8, 8, 56), (70, 65, 4, 1, 16),
                                         (2, 97, 3, 1, 56), (1, 1000, 2, 1, 32)])
def test_forward_and_gradient(B, S, H, Hkv, D, causal):
    qkv, do = _case(B, S, H, Hkv, D)
    want, want_grad = _exact(qkv, do, H, Hkv, D, causal)
    x = qkv.clone().requires_grad_()
    out = qkv_attention(x, H, Hkv, D, causal)
    (grad,) = torch.autograd.grad(out, x, do)
    assert type(out.grad_fn).__name__.startswith("_SmallQkvAttention")
    assert _near(out, want) and _near(grad, want_grad)
    (again,) = torch.autograd.grad(qkv_attention(x, H, Hkv, D, causal), x, do)
    assert torch.equal(grad, again)


def test_scores_far_apart_and_a_scale():
    """Scores of several hundred: exponentials that vanish and rows led by one key."""
    qkv, do = _case(2, 70, 2, 1, 32, sc=8.0)
    want, want_grad = _exact(qkv, do, 2, 1, 32, True, 0.9)
    x = qkv.clone().requires_grad_()
    out = qkv_attention(x, 2, 1, 32, True, 0.9)
    (grad,) = torch.autograd.grad(out, x, do)
    # a score of 500 rounded to fp32 is off by 3e-5, and so is its probability
    assert ((out.double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-4 * want.abs().max()).all()
    assert ((grad.double() - want_grad).abs() <= 2.0 ** -7 * want_grad.abs() + 1e-3 * want_grad.abs().max()).all()


def test_what_torch_does_with_its_own_operations():
    """A gradient of the gradient, several upstream gradients at once, vmap over the call, a forward-mode derivative, saved-tensor hooks
    and an upstream gradient that is expanded: as before, through torch's operations where the kernels take no part."""
    H, Hkv, D = 2, 1, 16
    qkv, do = _case(2, 9, H, Hkv, D)
    ref = lambda t: attention_reference(*_split_qkv(t, H, Hkv, D)).reshape(*t.shape[:2], H * D)  # noqa: E731
    near = lambda a, b: (a.float() - b.float()).abs().max() <= 2.0 ** -7 * b.float().abs().max() + 1e-6  # noqa: E731
    x = qkv.clone().requires_grad_()
    grads = {}
    for name, f in (("kernel", lambda t: qkv_attention(t, H, Hkv, D)), ("ref", ref)):
        (g,) = torch.autograd.grad(f(x), x, do, create_graph=True)
        (g2,) = torch.autograd.grad(g.float().square().sum(), x)
        (many,) = torch.autograd.grad(f(x), x, torch.stack([do, 2 * do]), is_grads_batched=True)
        mapped = torch.func.vmap(lambda t: f(t[None])[0])(qkv)
        _, tangent = torch.func.jvp(f, (qkv,), (qkv,))
        (expanded,) = torch.autograd.grad(f(x), x, do[:1, :1].expand_as(do))
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
            y = f(x)
        (hooked,) = torch.autograd.grad(y, x, do)
        grads[name] = (g, g2, many, mapped, tangent, expanded, hooked)
    for a, b in zip(grads["kernel"], grads["ref"]):
        assert a.shape == b.shape and near(a.detach(), b.detach())
    assert near(_small_attention_grad(qkv, do, H, Hkv, D, True, 1 / math.sqrt(D)), torch.autograd.grad(ref(x), x, do)[0])


def test_strided_projection_and_rope():
    H, Hkv, D = 4, 2, 32
    qkv, do = _case(2, 40, H, Hkv, D)
    wide = torch.zeros(2, 40, qkv.shape[-1] + 8, dtype=torch.bfloat16, device="cuda")
    wide[..., 4:-4] = qkv
    assert torch.equal(qkv_attention(wide[..., 4:-4], H, Hkv, D), qkv_attention(qkv, H, Hkv, D))
    a = qkv_attention(qkv.clone(), H, Hkv, D, rope_theta=10000.0)
    from idrak_b200.ops.rowops import rope_reference
    q, k, v = _split_qkv(qkv, H, Hkv, D)
    pos = torch.arange(40, device="cuda").repeat(2)
    q, k = (rope_reference(t.reshape(80, -1, D), pos, 10000.0, None, 1.0).reshape(t.shape) for t in (q, k))
    want = attention_reference(q, k, v).reshape(2, 40, H * D)
    assert (a.float() - want.float()).abs().max() <= 2.0 ** -7 * want.float().abs().max()
