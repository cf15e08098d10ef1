"""Paged decode attention, paged KV writes and the device sampler vs plain PyTorch."""
import pytest
import torch

from idrak_b200.ops import decode as D

pytestmark = pytest.mark.gpu


def _rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("H,Hkv,Dh", [(4, 1, 128), (32, 8, 128), (12, 12, 64), (8, 2, 64)])
@pytest.mark.parametrize("splits", [1, 3, None])
def test_paged_decode_matches_reference(H, Hkv, Dh, splits):
    bs, nblocks, seqs = 16, 200, 5
    k_cache, v_cache = _rand((nblocks, bs, Hkv, Dh), 1), _rand((nblocks, bs, Hkv, Dh), 2)
    lens = torch.tensor([1, 17, 333, 64, 500], dtype=torch.int32, device="cuda")
    g = torch.Generator().manual_seed(3)
    table = torch.randperm(nblocks, generator=g)[: seqs * 32].reshape(seqs, 32).to(torch.int32).cuda()
    q = _rand((seqs, H, Dh), 4)
    out = D.paged_decode(q, k_cache, v_cache, table, lens, splits=splits)
    ref = D.paged_decode_reference(q, k_cache, v_cache, table, lens)
    assert (out.float() - ref.float()).abs().max().item() < 2e-2
    outw = D.paged_decode(q, k_cache, v_cache, table, lens, window=100, splits=splits)
    refw = D.paged_decode_reference(q, k_cache, v_cache, table, lens, window=100)
    assert (outw.float() - refw.float()).abs().max().item() < 2e-2


def test_kv_write_paged_from_fused_qkv():
    H, Hkv, Dh, T, bs = 8, 2, 64, 37, 16
    qkv = _rand((T, (H + 2 * Hkv) * Dh), 1)
    k = qkv[:, H * Dh:(H + Hkv) * Dh].unflatten(-1, (Hkv, Dh))
    v = qkv[:, (H + Hkv) * Dh:].unflatten(-1, (Hkv, Dh))
    kc = torch.zeros((10, bs, Hkv, Dh), dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    slots = (torch.randperm(160)[:T]).to(torch.int32).cuda()
    slots[5] = -1
    D.kv_write_paged(k, v, slots, kc, vc)
    flat_k, flat_v = kc.view(-1, Hkv, Dh), vc.view(-1, Hkv, Dh)
    for t in range(T):
        if t == 5:
            continue
        assert torch.equal(flat_k[slots[t]], k[t]) and torch.equal(flat_v[slots[t]], v[t])
    assert int((flat_k.abs().sum((1, 2)) > 0).sum()) == T - 1


def test_argmax_and_sampler():
    rows, V, ld = 7, 50257, 50304
    logits = _rand((rows, ld), 1) * 3
    ids = D.argmax_rows(logits, V)
    assert torch.equal(ids.cpu(), logits[:, :V].float().argmax(-1).to(torch.int32).cpu())
    dev = "cuda"
    t = torch.full((rows,), 0.8, device=dev)
    seeds = torch.arange(rows, dtype=torch.int64, device=dev) + 11
    # top_k = 1 is greedy whatever the seed
    one = D.sample_rows(logits, V, t, torch.ones(rows, dtype=torch.int32, device=dev), torch.ones(rows, device=dev),
                        torch.zeros(rows, device=dev), seeds, 0)
    assert torch.equal(one, ids)
    k = torch.full((rows,), 40, dtype=torch.int32, device=dev)
    p = torch.full((rows,), 0.9, device=dev)
    a = D.sample_rows(logits, V, t, k, p, torch.zeros(rows, device=dev), seeds, 3)
    b = D.sample_rows(logits, V, t, k, p, torch.zeros(rows, device=dev), seeds, 3)
    c = D.sample_rows(logits, V, t, k, p, torch.zeros(rows, device=dev), seeds, 4)
    assert torch.equal(a, b)                       # same (seed, step) -> same draw
    top40 = torch.topk(logits[:, :V].float(), 40, dim=-1).indices
    for r in range(rows):
        assert int(a[r]) in top40[r].tolist() and int(c[r]) in top40[r].tolist()
    # empirical frequencies follow the filtered distribution
    row = logits[:1].repeat(4000, 1).contiguous()
    n = row.shape[0]
    draws = D.sample_rows(row, V, torch.ones(n, device=dev), torch.full((n,), 4, dtype=torch.int32, device=dev),
                          torch.ones(n, device=dev), torch.zeros(n, device=dev),
                          torch.arange(n, dtype=torch.int64, device=dev), 0)
    vals, idx = torch.topk(logits[0, :V].float(), 4)
    want = torch.softmax(vals, 0)
    got = torch.stack([(draws == i).float().mean() for i in idx])
    assert (got - want).abs().max().item() < 0.04
    # a heavy repetition penalty moves the choice away from a token in the history
    hist = ids.reshape(rows, 1).contiguous()
    pen = D.sample_rows(logits, V, t, torch.ones(rows, dtype=torch.int32, device=dev), torch.ones(rows, device=dev),
                        torch.zeros(rows, device=dev), seeds, 0, history=hist,
                        repeat_penalty=torch.full((rows,), 50.0, device=dev))
    assert not torch.equal(pen, ids)


def test_sampler_ties_do_not_crowd_out_larger_logits():
    """All-equal logits with a few larger ones (a masked vocabulary looks like this): the larger ones must all be
    candidates, the tied places go to the lowest ids, and the draw repeats."""
    rows, V = 4, 4096
    dev = "cuda"
    logits = torch.zeros(rows, V, device=dev, dtype=torch.float32)
    big = [4000, 4010, 4095]
    for j, b in enumerate(big):
        logits[:, b] = 5.0 + j
    t = torch.ones(rows, device=dev)
    ones, zeros = torch.ones(rows, device=dev), torch.zeros(rows, device=dev)
    seeds = torch.arange(rows, dtype=torch.int64, device=dev)
    greedy = D.sample_rows(logits, V, t, torch.ones(rows, dtype=torch.int32, device=dev), ones, zeros, seeds, 0)
    assert greedy.tolist() == [4095] * rows
    k = torch.full((rows,), 8, dtype=torch.int32, device=dev)
    allowed = set(big) | {0, 1, 2, 3, 4}              # three larger logits, then five ties by ascending id
    seen = set()
    for step in range(200):
        a = D.sample_rows(logits, V, t, k, ones, zeros, seeds, step)
        b = D.sample_rows(logits, V, t, k, ones, zeros, seeds, step)
        assert torch.equal(a, b)
        seen |= set(a.tolist())
    assert seen <= allowed and set(big) <= seen, sorted(seen)


@pytest.mark.parametrize("H,Hkv,Dh,rot", [(8, 2, 64, 64), (32, 8, 128, 128), (4, 4, 128, 64), (6, 2, 256, 128)])
@pytest.mark.parametrize("qk_norm", [False, True])
def test_fused_norm_rope_kv_write_matches_the_separate_steps(H, Hkv, Dh, rot, qk_norm):
    """One launch = query / key RMS norm + RoPE (in place on the packed projection) + paged cache write; compared with
    the same steps composed on the CPU path of the op."""
    T, bs, nb = 45, 16, 12
    qkv = _rand((T, (H + 2 * Hkv) * Dh), 1)
    pos = torch.randint(0, 3000, (T,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(nb * bs)[:T].to(torch.int32).cuda()
    slots[7] = -1
    qn = (_rand((Dh,), 2).float() * 0.1 + 1).to(torch.bfloat16) if qk_norm else None
    kn = (_rand((Dh,), 3).float() * 0.1 + 1).to(torch.bfloat16) if qk_norm else None
    kc = torch.zeros((nb, bs, Hkv, Dh), dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    got = qkv.clone()
    D.norm_rope_kv(got, H, Hkv, Dh, pos, slots, kc, vc, None, None, qn, kn, 1e-6, 10000.0, rot)
    want = qkv.cpu().clone()
    kc2, vc2 = torch.zeros_like(kc).cpu(), torch.zeros_like(vc).cpu()
    D.norm_rope_kv(want, H, Hkv, Dh, pos.cpu(), slots.cpu(), kc2, vc2, None, None,
                   qn.cpu() if qn is not None else None, kn.cpu() if kn is not None else None, 1e-6, 10000.0, rot)
    assert (got.float().cpu() - want.float()).abs().max().item() < 3e-2
    assert (kc.float().cpu() - kc2.float()).abs().max().item() < 3e-2
    assert torch.equal(vc.cpu(), vc2)                       # values are copied, bit for bit
    # what the cache holds for keys is exactly what stayed in the projection buffer
    k_rows = got[:, H * Dh:(H + Hkv) * Dh].unflatten(-1, (Hkv, Dh))
    keep = slots >= 0
    assert torch.equal(kc.view(-1, Hkv, Dh)[slots[keep].long()], k_rows[keep])


@pytest.mark.parametrize("rot", [64, 192, 256])
@pytest.mark.parametrize("qk_norm", [False, True])
def test_every_rotary_width_of_a_head_of_256(rot, qk_norm):
    test_fused_norm_rope_kv_write_matches_the_separate_steps(6, 2, 256, rot, qk_norm)


@pytest.mark.parametrize("H,Hkv,Dh", [(32, 8, 128), (12, 12, 64), (4, 1, 128)])
@pytest.mark.parametrize("splits", [1, 4, None])
def test_int8_kv_cache_write_and_decode(H, Hkv, Dh, splits):
    """int8 codes + one scale per (slot, kv head): the fused write against the plain quantiser, and decode attention
    over the codes against the reference over the de-quantised cache."""
    bs, nblocks, seqs, T = 16, 120, 4, 600
    lens = [1, 50, 333, 216]
    table = torch.randperm(nblocks)[: seqs * 24].reshape(seqs, 24).to(torch.int32).cuda()
    kc = torch.zeros((nblocks, bs, Hkv, Dh), dtype=torch.int8, device="cuda")
    vc = torch.zeros_like(kc)
    ks = torch.zeros((nblocks, bs, Hkv), dtype=torch.float32, device="cuda")
    vs = torch.zeros_like(ks)
    qkv = _rand((T, (H + 2 * Hkv) * Dh), 5)
    slots, t = [], 0
    for s_, n in enumerate(lens):
        for p_ in range(n):
            slots.append(int(table[s_, p_ // bs]) * bs + p_ % bs)
    slots = torch.tensor(slots, dtype=torch.int32, device="cuda")
    D.norm_rope_kv(qkv, H, Hkv, Dh, None, slots, kc, vc, ks, vs)
    k_src = qkv[:, H * Dh:(H + Hkv) * Dh].unflatten(-1, (Hkv, Dh))
    q8, sc = D.quantize_kv_reference(k_src)
    got_codes = kc.view(-1, Hkv, Dh)[slots.long()].to(torch.int16)
    assert (got_codes - q8.to(torch.int16)).abs().max().item() <= 1          # division vs reciprocal at a tie
    assert torch.allclose(ks.view(-1, Hkv)[slots.long()], sc, rtol=1e-6)
    lens_t = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = _rand((seqs, H, Dh), 6)
    out = D.paged_decode(q, kc, vc, table, lens_t, splits=splits, k_scale=ks, v_scale=vs)
    ref = D.paged_decode_reference(q, kc, vc, table, lens_t, k_scale=ks, v_scale=vs)
    assert (out.float() - ref.float()).abs().max().item() < 2e-2
    # and close to attention over the unquantised keys / values (what the int8 cache costs)
    kb = torch.zeros((nblocks, bs, Hkv, Dh), dtype=torch.bfloat16, device="cuda")
    vb = torch.zeros_like(kb)
    D.norm_rope_kv(qkv, H, Hkv, Dh, None, slots, kb, vb)
    exact = D.paged_decode_reference(q, kb, vb, table, lens_t)
    assert (out.float() - exact.float()).abs().max().item() < 6e-2


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("hint,window", [(None, 0), (4096, 0), (4096, 300)])
def test_uneven_lengths_share_their_keys_by_the_built_in_rule(int8, Dh, hint, window):
    """Lengths at the edges of tiles (16) and shares (128 to 512), empty and long ones in one batch, with the split that the
    length bound gives. Probabilities enter the tensor core as bf16 (relative 2^-9) and the result is rounded to bf16:
    2^-8 of the largest value, which is at most about 4 here."""
    bs, Hkv, H = 16, 2, 8
    lens = [0, 1, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1025, 2000, 3000]
    width = 256
    need = [(n + bs - 1) // bs for n in lens]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist()
    table, at = torch.zeros(len(lens), width, dtype=torch.int32), 0
    for i, n in enumerate(need):
        table[i, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    table, lens_t = table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    kc, vc, q = _rand((sum(need), bs, Hkv, Dh), 1), _rand((sum(need), bs, Hkv, Dh), 2), _rand((len(lens), H, Dh), 3)
    scales = {}
    if int8:
        codes = [D.quantize_kv_reference(t.view(-1, Hkv, Dh)) for t in (kc, vc)]
        (kc, ks), (vc, vs) = ((c.view(-1, bs, Hkv, Dh), s.view(-1, bs, Hkv).contiguous()) for c, s in codes)
        scales = {"k_scale": ks, "v_scale": vs}
    out = D.paged_decode(q, kc, vc, table, lens_t, window=window, max_len_hint=hint, **scales)
    kd, vd = (kc.float() * ks[..., None], vc.float() * vs[..., None]) if int8 else (kc.float(), vc.float())
    ref = D.paged_decode_reference(q.float(), kd, vd, table, lens_t, window=window)
    assert (out.float() - ref).abs().max().item() <= 2.0 ** -8 * 4
    assert torch.equal(out, D.paged_decode(q, kc, vc, table, lens_t, window=window, max_len_hint=hint, **scales))


def test_decode_slots_refuses_what_indexing_refused():
    """A table on the host or with too few rows raises; a position outside its row of the table - also of a table that is a
    part of a wider one - gets no slot, shortens the sequence to its row and is reported."""
    from idrak_b200 import _native
    wide = torch.arange(100, 140, dtype=torch.int32, device="cuda").view(5, 8)
    table = wide[:, 2:5]
    pos = torch.tensor([0, 15, 47, 48, -1], dtype=torch.int32, device="cuda")
    slots, lens = D.decode_slots(pos[:3], table[:3], 16)
    want = [102 * 16, 110 * 16 + 15, 120 * 16 + 15]
    assert slots.tolist() == want and lens.tolist() == [1, 16, 48]
    _native.check_status("in range")
    slots, lens = D.decode_slots(pos, table, 16)
    assert slots.tolist() == want + [-1, -1] and lens.tolist() == [1, 16, 48, 48, 0]
    with pytest.raises(_native.NativeError, match="bad argument"):
        _native.check_status("slots")
    with pytest.raises(RuntimeError):
        D.decode_slots(pos[:3], table[:3].cpu(), 16)
    with pytest.raises(IndexError):
        D.decode_slots(pos, table[:4], 16)
    for other in (pos[:3].long(), pos[:3].repeat_interleave(2)[::2]):
        slots, lens = D.decode_slots(other, table, 16)
        assert slots.tolist() == want and lens.tolist() == [1, 16, 48]
    empty = D.decode_slots(pos[:0], table, 16)
    assert empty[0].numel() == 0 and empty[1].numel() == 0


@pytest.mark.parametrize("Dh", [64, 128])
@pytest.mark.parametrize("splits", [2, 8, 9, 64, 65, 125])
def test_any_number_of_shares_merges_in_order(Dh, splits):
    """Up to eight shares, one round of 64 and more than that, of sequences that fill them, some of them or one."""
    bs, Hkv, H, lens = 16, 2, 6, [4000, 2500, 33, 0]
    need = [(n + bs - 1) // bs for n in lens]
    table, at = torch.zeros(len(lens), max(need), dtype=torch.int32), 0
    for i, n in enumerate(need):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    kc, vc, q = _rand((at, bs, Hkv, Dh), 1), _rand((at, bs, Hkv, Dh), 2), _rand((len(lens), H, Dh), 3)
    table, lens_t = table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    out = D.paged_decode(q, kc, vc, table, lens_t, splits=splits)
    ref = D.paged_decode_reference(q.float(), kc.float(), vc.float(), table, lens_t)
    # probabilities enter the tensor core as bf16 (2^-9) and the result is rounded to bf16, values up to about 2
    assert (out.float() - ref).abs().max().item() <= 2.0 ** -8 * 2
    assert torch.equal(out, D.paged_decode(q, kc, vc, table, lens_t, splits=splits))


@pytest.mark.parametrize("H,Hkv,Dh,rot", [(12, 12, 256, 128), (12, 12, 128, 128), (12, 12, 128, 64), (9, 3, 64, 64)])
@pytest.mark.parametrize("T", [700, 3001])
@pytest.mark.parametrize("int8", [False, True])
def test_fused_norm_rope_kv_write_in_runs_of_heads(H, Hkv, Dh, rot, T, int8):
    """Enough tokens that a warp takes runs of heads, the last run of a token shorter: keys rotated once, values as they are."""
    bs = 16
    nb = (T + bs - 1) // bs
    qkv = _rand((T, (H + 2 * Hkv) * Dh), 1)
    pos = torch.randint(0, 3000, (T,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(nb * bs)[:T].to(torch.int32).cuda()
    kc, vc = (torch.zeros((nb, bs, Hkv, Dh), dtype=torch.int8 if int8 else torch.bfloat16, device="cuda") for _ in range(2))
    ks, vs = (torch.zeros((nb, bs, Hkv), device="cuda") if int8 else None for _ in range(2))
    got = qkv.clone()
    D.norm_rope_kv(got, H, Hkv, Dh, pos, slots, kc, vc, ks, vs, None, None, 1e-6, 10000.0, rot)
    heads = qkv.unflatten(-1, (H + 2 * Hkv, Dh))
    from idrak_b200.ops.rowops import rope_reference
    want = rope_reference(heads[:, :H + Hkv].contiguous(), pos, 10000.0, rot).float()
    mine = got.unflatten(-1, (H + 2 * Hkv, Dh))
    # both rounded to bf16 (they may fall on neighbours, 2^-7 apart), and fp32 angles of up to 3000 (2^-12 of a pair of up to 8)
    assert ((mine[:, :H + Hkv].float() - want).abs() <= 2.0 ** -7 * want.abs() + 4e-3).all()
    assert torch.equal(mine[:, H + Hkv:], heads[:, H + Hkv:])
    for cache, scale, part in ((kc, ks, mine[:, H:H + Hkv]), (vc, vs, heads[:, H + Hkv:])):
        held = cache.view(-1, Hkv, Dh)[slots.long()]
        if int8:
            codes, sc = D.quantize_kv_reference(part)
            assert (held.int() - codes.int()).abs().max() <= 1 and torch.allclose(scale.view(-1, Hkv)[slots.long()], sc, rtol=1e-6)
        else:
            assert torch.equal(held, part)


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("bs,H,Hkv,Dh", [(1, 4, 2, 64), (3, 8, 2, 128), (8, 9, 1, 128), (8, 8, 1, 64), (12, 16, 1, 64), (16, 2, 2, 128),
                                         (24, 16, 1, 128), (32, 10, 5, 64), (48, 8, 1, 128), (64, 6, 2, 128)])
@pytest.mark.parametrize("window", [0, 37])
def test_block_sizes_and_groups(int8, bs, H, Hkv, Dh, window):
    """Blocks that divide a tile of 16 keys, are divided by it, or neither; groups of 1 to 16 query heads, on either side of a column
    tile of 8; lengths at the edges of tiles and blocks. Slots past a sequence's end hold NaN (bf16) or scales of NaN (int8), which
    nothing may read into a result. The bound is that of the test of uneven lengths."""
    lens = [1, 7, 8, 15, 16, 17, 33, 64, 100, 257]
    need = [(n + bs - 1) // bs for n in lens]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(2)).tolist()
    table, at = torch.full((len(lens), max(need) + 1), -7, dtype=torch.int32), 0
    live = torch.zeros(sum(need), bs, dtype=torch.bool)
    for i, n in enumerate(need):
        blocks = order[at:at + n]
        table[i, :n] = torch.tensor(blocks, dtype=torch.int32)
        for j, b in enumerate(blocks):
            live[b, : min(bs, lens[i] - j * bs)] = True
        at += n
    table, lens_t, live = table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), live.cuda()
    kc, vc, q = _rand((sum(need), bs, Hkv, Dh), 1), _rand((sum(need), bs, Hkv, Dh), 2), _rand((len(lens), H, Dh), 3)
    scales = {}
    if int8:
        codes = [D.quantize_kv_reference(t.view(-1, Hkv, Dh)) for t in (kc, vc)]
        (kc, ks), (vc, vs) = ((c.view(-1, bs, Hkv, Dh), s.view(-1, bs, Hkv).contiguous()) for c, s in codes)
        kd, vd = kc.float() * ks[..., None], vc.float() * vs[..., None]
        ks[~live], vs[~live] = float("nan"), float("nan")
        scales = {"k_scale": ks, "v_scale": vs}
    else:
        kd, vd = kc.float(), vc.float()
        kc[~live], vc[~live] = float("nan"), float("nan")
    out = D.paged_decode(q, kc, vc, table, lens_t, window=window, **scales)
    ref = D.paged_decode_reference(q.float(), kd, vd, table, lens_t, window=window)
    assert (out.float() - ref).abs().max().item() <= 2.0 ** -8 * 4
