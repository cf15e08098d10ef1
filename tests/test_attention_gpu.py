"""tcgen05 flash attention forward/backward vs fp32 softmax(QK^T)V."""
import pytest
import torch

from idrak_b200 import ops

pytestmark = pytest.mark.gpu


def _rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)


def _close(a, b, tol):
    err = (a.float() - b.float()).abs().max().item()
    assert err <= tol, f"err {err}"


CASES = [  # B, Sq, Skv, H, Hkv, D, causal
    (1, 128, 128, 1, 1, 64, False),
    (1, 128, 128, 1, 1, 64, True),
    (2, 256, 256, 4, 4, 64, True),
    (2, 1024, 1024, 12, 12, 64, True),
    (1, 384, 384, 8, 2, 128, True),
    (1, 200, 200, 2, 2, 64, True),
    (1, 100, 333, 4, 1, 128, False),
    (1, 128, 512, 2, 2, 64, True),
]


@pytest.mark.parametrize("B,Sq,Skv,H,Hkv,D,causal", CASES)
def test_flash_forward(B, Sq, Skv, H, Hkv, D, causal):
    q, k, v = _rand((B, Sq, H, D), 1), _rand((B, Skv, Hkv, D), 2), _rand((B, Skv, Hkv, D), 3)
    out, lse = ops.flash_forward(q, k, v, causal)
    ref = ops.attention_reference(q.float(), k.float(), v.float(), causal)
    _close(out, ref, 2e-2)


def test_flash_forward_from_fused_qkv_buffer():
    B, S, H, D = 2, 256, 4, 64
    qkv = _rand((B, S, 3 * H * D), 5)
    q, k, v = (qkv[..., i * H * D:(i + 1) * H * D].unflatten(-1, (H, D)) for i in range(3))
    out, _ = ops.flash_forward(q, k, v, True)
    _close(out, ops.attention_reference(q.float(), k.float(), v.float(), True), 2e-2)


@pytest.mark.parametrize("B,Sq,Skv,H,Hkv,D,causal", CASES)
def test_flash_backward(B, Sq, Skv, H, Hkv, D, causal):
    q, k, v = (_rand((B, Sq, H, D), 1).requires_grad_(), _rand((B, Skv, Hkv, D), 2).requires_grad_(),
               _rand((B, Skv, Hkv, D), 3).requires_grad_())
    out = ops.attention(q, k, v, causal)
    do = _rand(out.shape, 4)
    out.backward(do)
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = ops.attention_reference(qr, kr, vr, causal)
    ref.backward(do.float())
    _close(q.grad, qr.grad, 5e-2)
    _close(k.grad, kr.grad, 5e-2)
    _close(v.grad, vr.grad, 5e-2)


@pytest.mark.parametrize("B,Sq,Skv,H,Hkv,D,causal", [
    (3, 130, 130, 64, 64, 128, True),      # many units per CTA, of one block and of two, the last two rows tall
    (2, 640, 640, 48, 16, 128, True),      # one to five blocks, three query heads on a key head
    (2, 640, 640, 48, 16, 64, True),
    (5, 128, 520, 40, 40, 128, False),     # one query block against five, the last eight keys wide
    (5, 520, 128, 40, 40, 64, False),
])
def test_flash_backward_walks_many_units(B, Sq, Skv, H, Hkv, D, causal):
    """Every CTA runs several units of different length one after the other: the next one's tiles, scores and sums come into
    the buffers of the one before."""
    q, k, v = _rand((B, Sq, H, D), 1), _rand((B, Skv, Hkv, D), 2), _rand((B, Skv, Hkv, D), 3)
    do = _rand((B, Sq, H, D), 4)
    out, lse = ops.flash_forward(q, k, v, causal)
    grads = ops.flash_backward(do, q, k, v, out, lse, causal)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ops.attention_reference(qr, kr, vr, causal).backward(do.float())
    for got, want in zip(grads, (qr.grad, kr.grad, vr.grad)):
        # out, P (or dS) and the gradient are rounded to 8 bits of mantissa, each 2^-9 of the value: 4 * 2^-9 with delta's share
        assert ((got.float() - want).norm() / want.norm()).item() < 2.0 ** -7
    for a, b in zip(grads, ops.flash_backward(do, q, k, v, out, lse, causal)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("B,Sq,Skv,H,Hkv,D,causal,window,parts", [
    (3, 515, 515, 16, 4, 64, True, None, 4),       # the last key block three keys tall
    (3, 515, 515, 16, 4, 128, True, None, 4),
    (1, 512, 512, 12, 4, 64, True, 100, 3),        # a group of three; key blocks that few query blocks see
    (2, 256, 700, 8, 4, 64, False, None, 2),
    (1, 130, 130, 4, 4, 64, True, None, 1),        # no group to deal out
    (1, 128, 128, 2, 1, 64, True, None, 1),        # too short to be worth it
    (8, 1024, 1024, 32, 8, 64, True, None, 1),     # units enough
])
def test_flash_backward_deals_the_heads_of_a_group(B, Sq, Skv, H, Hkv, D, causal, window, parts):
    """Key blocks whose query heads go to several units: parts in fp32, summed in their order, written through row strides."""
    from idrak_b200 import _native
    need = _native.lib().idrak_flash_bwd_workspace(B, H, Hkv, Sq, Skv, D, int(causal))
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert need == (2 * parts * B * Skv * Hkv * D if parts > 1 else 0)
    q, k, v = _rand((B, Sq, H, D), 1), _rand((B, Skv, Hkv, D), 2), _rand((B, Skv, Hkv, D), 3)
    do = _rand((B, Sq, H, D), 4)
    out, lse = ops.flash_forward(q, k, v, causal, window=window)
    both = torch.zeros((B, Skv, 2, Hkv, D), dtype=torch.bfloat16, device="cuda")
    dk, dv = both[:, :, 0], both[:, :, 1]
    grads = ops.flash_backward(do, q, k, v, out, lse, causal, grads=(torch.empty_like(q), dk, dv), window=window)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ops.attention_reference(qr, kr, vr, causal, window=window).backward(do.float())
    for got, want in zip(grads, (qr.grad, kr.grad, vr.grad)):
        assert ((got.float() - want).norm() / want.norm()).item() < 2.0 ** -7      # four roundings to bf16, as above
    again = ops.flash_backward(do, q, k, v, out, lse, causal, window=window)
    for x, y in zip(grads, again):
        assert torch.equal(x, y)


def _parts(B, Sq, Skv, H, Hkv, D, causal, window, packed):
    from idrak_b200 import _native
    need = _native.lib().idrak_flash_bwd_workspace_ex(B, H, Hkv, Sq, Skv, D, int(causal), window or 0, int(packed))
    assert need <= _native.lib().idrak_flash_bwd_workspace(B, H, Hkv, Sq, Skv, D, int(causal))
    return need // (2 * B * Skv * Hkv * D) or 1


@pytest.mark.parametrize("B,Sq,Skv,H,Hkv,D,causal,window,packed,parts", [
    (4, 256, 700, 8, 4, 128, False, None, False, 1),     # dealt 62 us, whole 44
    (8, 130, 130, 32, 8, 128, True, None, False, 1),
    (1, 2048, 2048, 32, 8, 128, True, 256, False, 1),    # units that a window has evened out
    (1, 2048, 2048, 16, 4, 128, True, 256, False, 2),
    (1, 2048, 2048, 16, 4, 128, True, None, False, 4),
    (1, 2048, 2048, 16, 4, 128, True, None, True, 1),    # lengths that only the device knows
    (1, 1024, 1024, 8, 1, 64, True, 200, False, 8),
    (1, 640, 640, 16, 1, 64, True, None, True, 16),
])
def test_flash_backward_deals_where_that_is_faster(B, Sq, Skv, H, Hkv, D, causal, window, packed, parts):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _parts(B, Sq, Skv, H, Hkv, D, causal, window, packed) == parts
    q, k, v = _rand((B, Sq, H, D), 1), _rand((B, Skv, Hkv, D), 2), _rand((B, Skv, Hkv, D), 3)
    do = _rand((B, Sq, H, D), 4)
    rs = ops.row_starts_from_spans([(0, 70), (70, 300), (300, Sq)], B, Sq, "cuda") if packed else None
    out, lse = ops.flash_forward(q, k, v, causal, window=window, row_start=rs)
    grads = ops.flash_backward(do, q, k, v, out, lse, causal, window=window, row_start=rs)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ops.attention_reference(qr, kr, vr, causal, window=window, row_start=rs).backward(do.float())
    for got, want in zip(grads, (qr.grad, kr.grad, vr.grad)):
        assert ((got.float() - want).norm() / want.norm()).item() < 2.0 ** -7      # four roundings to bf16, as above


MODES = [  # B, S, H, Hkv, D, window, spans, softcap
    (2, 512, 4, 4, 64, 128, None, None),
    (1, 640, 4, 2, 128, 200, None, None),
    (2, 512, 4, 4, 64, None, [(0, 100), (100, 384), (384, 400), (400, 512)], None),
    (1, 1000, 2, 1, 128, None, [(0, 7), (7, 530), (530, 1000)], None),
    (1, 384, 4, 4, 64, None, None, 30.0),
    (1, 384, 2, 2, 128, 96, [(0, 130), (130, 384)], 50.0),
]


@pytest.mark.parametrize("B,S,H,Hkv,D,window,spans,softcap", MODES)
def test_flash_window_packed_sequences_and_softcap(B, S, H, Hkv, D, window, spans, softcap):
    """Sliding window, sequences packed into one row (a lower key bound per position) and tanh soft-capping run inside
    the attention kernels, forward and backward; the oracle is the fp32 statement with explicit masks."""
    q, k, v = (_rand((B, S, H, D), 1).requires_grad_(), _rand((B, S, Hkv, D), 2).requires_grad_(),
               _rand((B, S, Hkv, D), 3).requires_grad_())
    row_start = ops.row_starts_from_spans(spans, B, S, "cuda") if spans else None
    out = ops.attention(q, k, v, True, None, window, row_start, softcap)
    do = _rand(out.shape, 4)
    out.backward(do)
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = ops.attention_reference(qr, kr, vr, True, None, window, row_start, softcap)
    ref.backward(do.float())
    _close(out, ref, 2e-2)
    _close(q.grad, qr.grad, 5e-2)
    _close(k.grad, kr.grad, 5e-2)
    _close(v.grad, vr.grad, 5e-2)


def test_packed_row_equals_the_sequences_run_one_by_one():
    """One launch over a packed row gives each sequence what a launch of its own gives (the same tiles of scores are
    masked instead of skipped, so the results agree to the rounding of the running maximum)."""
    B, S, H, D = 1, 768, 4, 64
    spans = [(0, 200), (200, 201), (201, 640), (640, 768)]
    q, k, v = _rand((B, S, H, D), 1), _rand((B, S, H, D), 2), _rand((B, S, H, D), 3)
    packed, _ = ops.flash_forward(q, k, v, True, None, None, ops.row_starts_from_spans(spans, B, S, "cuda"))
    for lo, hi in spans:
        alone, _ = ops.flash_forward(q[:, lo:hi].contiguous(), k[:, lo:hi].contiguous(), v[:, lo:hi].contiguous(), True)
        _close(packed[:, lo:hi], alone, 1e-2)


@pytest.mark.parametrize("B,H,Hkv,Sq,Skv,causal", [(5, 32, 8, 200, 200, True), (40, 4, 1, 257, 257, True), (5, 32, 8, 129, 500, True),
                                                   (1, 32, 4, 1281, 1281, True), (3, 64, 8, 128, 128, True), (3, 32, 8, 300, 300, False),
                                                   (3, 50, 10, 256, 640, False), (10, 16, 16, 385, 400, True)])
def test_two_query_tiles_have_the_bits_of_one(B, H, Hkv, Sq, Skv, causal):
    """Calls with a CTA of two query tiles for every SM against calls that one tile per CTA takes: the same arithmetic in the same
    order, at sizes where the second tile is empty, short or sees more keys. Rows of a warp move their maxima together on both."""
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(B, s, h, 128, generator=g, device="cuda").to(torch.bfloat16) for s, h in ((Sq, H), (Skv, Hkv), (Skv, Hkv)))
    o, lse = ops.flash_forward(q, k, v, causal)
    for b in range(B):                                                       # one sequence and few heads at a time: one tile per CTA
        for h in range(0, H, H // Hkv):
            part = slice(h, h + H // Hkv)
            ob, lb = ops.flash_forward(q[b:b + 1, :, part].contiguous(), k[b:b + 1, :, h * Hkv // H][:, :, None].contiguous(),
                                       v[b:b + 1, :, h * Hkv // H][:, :, None].contiguous(), causal)
            assert torch.equal(ob[0], o[b, :, part]) and torch.equal(lb[0], lse[b, part])
    if Sq <= Skv:
        ref = ops.attention_reference(q.float(), k.float(), v.float(), causal)
        # probabilities enter the product as bf16 (2^-9) and the result is rounded to bf16, values up to about 5
        assert (o.float() - ref).abs().max().item() <= 2.0 ** -8 * 5
