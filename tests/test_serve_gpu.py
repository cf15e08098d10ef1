"""Paged prefill / decode on the GPU against the training forward of the same bf16 model (teacher-forced), and an
end-to-end engine run with sampling on the device."""
import dataclasses

import pytest
import torch

from idrak_b200.models.decoder import build_decoder
from idrak_b200.models.spec import DecoderSpec
from idrak_b200.serve import GenerationOptions, LLMEngine
from idrak_b200.serve.runner import ModelRunner, PrefillItem

pytestmark = pytest.mark.gpu


def _spec(kind):
    if kind == "gpt2":
        return DecoderSpec.gpt2(layers=2, dim=256, heads=4, vocab=1000, max_positions=512)
    if kind == "llama128":
        return DecoderSpec.llama(layers=2, dim=256, heads=2, kv_heads=1, ff_dim=512, vocab=1000, max_positions=512)
    s = DecoderSpec.llama(layers=2, dim=256, heads=4, kv_heads=2, ff_dim=512, vocab=1000, max_positions=512)
    if kind == "windowed":
        s = dataclasses.replace(s, sliding_window=48)
    return s


@pytest.mark.parametrize("kind", ["llama", "llama128", "gpt2", "windowed"])
def test_paged_prefill_and_decode_match_forward(kind):
    dev = torch.device("cuda:0")
    spec = _spec(kind)
    model = build_decoder(spec, seed=5).to(dev, torch.bfloat16).eval()
    runner = ModelRunner(model, num_blocks=64, block_size=16)
    g = torch.Generator().manual_seed(1)
    lens = [37, 64, 5]
    steps = 70
    seqs = [torch.randint(0, spec.vocabulary, (n + steps,), generator=g).tolist() for n in lens]
    tables, nxt = [], 0
    for n in lens:
        need = (n + steps + 15) // 16
        tables.append(list(range(nxt, nxt + need)))
        nxt += need
    with torch.no_grad():
        full = [model(torch.tensor([s], dtype=torch.int32, device=dev))[0].float() for s in seqs]
    got = runner.prefill([PrefillItem(s[:n], 0, t) for s, n, t in zip(seqs, lens, tables)])
    for i, n in enumerate(lens):
        torch.testing.assert_close(got[i, : spec.vocabulary].float(), full[i][n - 1], rtol=3e-2, atol=3e-2)
    width = max(len(t) for t in tables)
    table = torch.tensor([t + [0] * (width - len(t)) for t in tables], dtype=torch.int32, device=dev)
    for k in range(steps):
        tok = torch.tensor([s[n + k] for s, n in zip(seqs, lens)], dtype=torch.int32, device=dev)
        pos = torch.tensor([n + k for n in lens], dtype=torch.int32, device=dev)
        lg = runner.decode(tok, pos, table)
        for i, n in enumerate(lens):
            torch.testing.assert_close(lg[i, : spec.vocabulary].float(), full[i][n + k], rtol=3e-2, atol=4e-2)
    # a shared prefix: the second half of a prompt computed against cached keys equals the whole prompt
    s, t = seqs[1], list(range(nxt, nxt + 5))
    runner.prefill([PrefillItem(s[:32], 0, t)])
    again = runner.prefill([PrefillItem(s[32:64], 32, t)])
    torch.testing.assert_close(again[0, : spec.vocabulary].float(), full[1][63], rtol=3e-2, atol=3e-2)


def test_engine_end_to_end_on_device():
    dev = torch.device("cuda:0")
    spec = _spec("llama")
    model = build_decoder(spec, seed=5).to(dev, torch.bfloat16).eval()
    for p in model.parameters():
        p.data.mul_(2.0)
    eng = LLMEngine(model, num_blocks=256, max_batch=16)
    g = torch.Generator().manual_seed(2)
    prompts = [torch.randint(0, 1000, (int(n),), generator=g).tolist() for n in torch.randint(4, 90, (24,), generator=g)]
    greedy = eng.generate(prompts, GenerationOptions.greedy_options(32))
    assert all(len(r.output) == 32 for r in greedy)
    # greedy tokens are the arg-max of the training forward wherever its top-2 margin is clear
    checked = 0
    for p, r in list(zip(prompts, greedy))[:6]:
        ids = p + r.output
        with torch.no_grad():
            lg = model(torch.tensor([ids], dtype=torch.int32, device=dev))[0].float()
        top = lg.topk(2, -1)
        for k, tok in enumerate(r.output):
            row = len(p) - 1 + k
            if float(top.values[row, 0] - top.values[row, 1]) > 0.25:
                assert int(top.indices[row, 0]) == tok
                checked += 1
    assert checked > 50
    o = GenerationOptions(temperature=0.8, top_k=40, top_p=0.9, repeat_penalty=1.1, seed=3, max_tokens=24,
                          return_logprobs=True)
    a = eng.generate(prompts[:8], o)
    b = eng.generate(prompts[:8], o)
    assert [r.output for r in a] == [r.output for r in b]            # seeded sampling repeats
    assert all(len(r.logprobs) == 24 and max(r.logprobs) <= 0 for r in a)
    st = eng.stats()
    assert st["free_blocks"] == 256 and st["running"] == 0


@pytest.mark.parametrize("quant", ["", "int8", "int4"])
@pytest.mark.parametrize("rows", [1, 9, 40])
def test_few_row_decode_agrees_with_the_layer_by_layer_path(quant, rows):
    """The fused decode path (bf16 or packed projections) against the modules' own forwards over the same cache. Both round
    activations to bf16 at every layer (relative 2^-9, ten roundings over two layers), the fused one at fewer places."""
    from idrak_b200.models import DecoderSpec, build_decoder
    from idrak_b200.quant import quantize_model
    from idrak_b200.serve import ModelRunner
    torch.manual_seed(0)
    spec = DecoderSpec.llama(layers=2, dim=256, heads=4, kv_heads=2, ff_dim=512, vocab=500, max_positions=256, head_dim=64)
    model = build_decoder(spec, seed=1).to("cuda", torch.bfloat16)
    if quant:
        quantize_model(model, quant)
    runner = ModelRunner(model, rows * 4, 16)
    for c in runner.k_cache + runner.v_cache:
        c.copy_(torch.randn(c.shape, device="cuda"))
    table = torch.randperm(rows * 4, device="cuda").to(torch.int32).view(rows, 4)
    positions = torch.randint(0, 64, (rows,), device="cuda", dtype=torch.int32)
    tokens = torch.randint(0, 500, (rows,), device="cuda", dtype=torch.int32)
    assert runner._few_row_path()
    fused = runner.decode(tokens, positions, table).float()
    runner._few_rows_ok = False
    plain = runner.decode(tokens, positions, table).float()
    rms = plain.pow(2).mean().sqrt()
    assert ((fused - plain).pow(2).mean().sqrt() <= 10 * 2.0 ** -9 * rms) and fused.isfinite().all()


@pytest.mark.parametrize("quant", ["", "int8", "int4"])
@pytest.mark.parametrize("lengths,shared", [((5,), 0), ((64,), 0), ((9, 300, 9), 0), ((16, 16), 0), ((20, 11), 16)])
def test_prefill_calls_the_same_kernels_as_the_modules(quant, lengths, shared):
    """Prefill through the kernels directly (fresh prompts, of equal length, behind a shared prefix) against the modules' own
    forwards: the same kernels in the same order, so logits and caches agree bit for bit."""
    from idrak_b200.models import DecoderSpec, build_decoder
    from idrak_b200.quant import quantize_model
    from idrak_b200.serve import ModelRunner, PrefillItem
    spec = DecoderSpec.llama(layers=2, dim=256, heads=4, kv_heads=2, ff_dim=512, vocab=500, max_positions=512, head_dim=64)
    model = build_decoder(spec, seed=1).to("cuda", torch.bfloat16)
    if quant:
        quantize_model(model, quant)
    runner = ModelRunner(model, 40, 16)
    g = torch.Generator().manual_seed(0)
    items, block = [], 0
    for n in lengths:
        need = (shared + n + 15) // 16
        items.append(PrefillItem(torch.randint(0, 500, (n,), generator=g).tolist(), shared, list(range(block, block + need))))
        block += need
    if shared:
        for c in runner.k_cache + runner.v_cache:
            c.copy_(torch.randn(c.shape, device="cuda"))
    results = []
    for few in (True, False):
        runner._few_rows_ok = few
        logits = runner.prefill(items).float()
        results.append((logits, runner.prefill(items, all_logits=True).float(), [c.float().clone() for c in runner.k_cache + runner.v_cache]))
    (a, a_all, a_cache), (b, b_all, b_cache) = results
    for x, y in [(a, b), (a_all, b_all)] + list(zip(a_cache, b_cache)):
        assert torch.equal(x, y) and x.isfinite().all()


def _small(seed=1):
    spec = DecoderSpec.llama(layers=2, dim=256, heads=4, kv_heads=2, ff_dim=512, vocab=500, max_positions=256, head_dim=64)
    return build_decoder(spec, seed=seed).to("cuda", torch.bfloat16)


def _step(model_or_runner, graphed=False):
    """Logits of a prefill of two prompts (every token) and of the decode step after it, on a given or a fresh runner."""
    runner = model_or_runner if isinstance(model_or_runner, ModelRunner) else ModelRunner(model_or_runner, 8, 16)
    items = [PrefillItem(list(range(7, 27)), 0, [0, 1]), PrefillItem(list(range(40, 45)), 0, [2])]
    every = runner.prefill(items, all_logits=True).clone()
    last = runner.prefill(items).clone()
    tok, pos = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in ([3, 4], [20, 5]))
    table = torch.tensor([[0, 1], [2, 3]], dtype=torch.int32, device="cuda")
    step = (runner.decode_graphed(tok, pos, table, 21) if graphed else runner.decode(tok, pos, table)).clone()
    return every, last, step


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("quant", ["", "int8"])
def test_runner_follows_adapters_that_come_and_go(quant):
    """Adapters attached after a runner's first calls, taken off for a while, and put back: prefill, decode and recorded
    decode steps give what a runner made at that moment gives, bit for bit."""
    from idrak_b200.adapters.lora import add_adapters
    from idrak_b200.quant import quantize_model
    from idrak_b200.text.finetuning import adapters_disabled
    model = _small()
    if quant:
        quantize_model(model, quant)
    plain, graphed = ModelRunner(model, 8, 16), ModelRunner(model, 8, 16)
    bare, bare_graphed = _step(plain), _step(graphed, True)
    torch.manual_seed(0)
    for p in add_adapters(model, rank=8):
        p.data.normal_(0, 0.05)
    adapted = _step(model)
    assert not torch.equal(adapted[0], bare[0]) and not torch.equal(adapted[2], bare[2])
    assert _same(_step(plain), adapted) and _same(_step(graphed, True), _step(ModelRunner(model, 8, 16), True))
    with adapters_disabled(model):
        assert _same(_step(plain), bare) and _same(_step(graphed, True), bare_graphed)
        inside = ModelRunner(model, 8, 16)                  # its first call finds no adapters
        assert _same(_step(inside), bare)
    for r in (plain, inside):
        assert _same(_step(r), adapted)


@pytest.mark.parametrize("kind", ["int8", "int4", "fp8"])
def test_runner_follows_weights_packed_after_its_first_call(kind):
    from idrak_b200.quant import quantize_model
    model = _small()
    plain, graphed = ModelRunner(model, 8, 16), ModelRunner(model, 8, 16)
    _step(plain), _step(graphed, True)
    quantize_model(model, kind)
    assert _same(_step(plain), _step(model)) and _same(_step(graphed, True), _step(ModelRunner(model, 8, 16), True))


def test_prefill_runs_hooks_and_replaced_modules():
    """Hooks on norms and feed-forwards, a feed-forward that is not the library's, a runner with its own block."""
    model = _small()
    want, _, _ = _step(model)
    seen = []
    blk = model.blocks[1]
    for m in (blk.attn_norm, blk.mlp_norm, blk.mlp, model.norm):
        handle = m.register_forward_hook(lambda mod, args, out: seen.append(mod))
        assert torch.equal(_step(model)[0], want)
        assert m in seen
        handle.remove()

    class Doubled(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, x, residual=None):
            y = self.inner(x) * 2
            return y if residual is None else y + residual

    class OwnBlock(ModelRunner):
        calls = 0

        def _block(self, blk, x, attend):
            OwnBlock.calls += 1
            return super()._block(blk, x, attend)

    assert torch.equal(_step(OwnBlock(model, 8, 16))[0], want) and OwnBlock.calls >= 2 * len(model.blocks)
    blk.mlp = Doubled(blk.mlp)
    assert not torch.equal(ModelRunner(model, 8, 16).prefill([PrefillItem([5, 6, 7], 0, [0])], all_logits=True), want[:3])


@pytest.mark.parametrize("kind", ["int8", "int4"])
def test_packed_projections_of_a_model_with_folded_norms(kind):
    """Norms folded into the projections, the projections packed afterwards: the few-row decode step still normalises."""
    from idrak_b200.quant import quantize_model
    from idrak_b200.serve.runner import fold_norms_into_projections
    model = _small()
    for blk in model.blocks:
        blk.attn_norm.weight.data.uniform_(0.5, 2.0)
    assert fold_norms_into_projections(model)
    quantize_model(model, kind)
    runner = ModelRunner(model, 8, 16)
    fused = _step(runner)[2].float()
    assert runner._few_row_path()
    runner._few_rows_ok = False
    plain = _step(runner)[2].float()
    # both round activations to bf16 (2^-9) at each of the ten steps of two layers
    assert (fused - plain).pow(2).mean().sqrt() <= 10 * 2.0 ** -9 * plain.pow(2).mean().sqrt()


@pytest.mark.parametrize("dim,heads,kv_heads,head_dim", [(256, 4, 2, 64), (512, 4, 1, 128)])
@pytest.mark.parametrize("extra", [{}, {"qk_norm": True}, {"qkv_bias": True}, {"norm_offset": 1.0, "activation": "gelu"}, {"int8": True}])
def test_native_prefill_launches_what_the_runner_would(dim, heads, kv_heads, head_dim, extra, monkeypatch):
    """The blocks as one native call against the runner's own launches: the same kernels on the same operands, so logits and caches
    agree bit for bit - one token, prompts of one length side by side, odd lengths, on both sides of 64 rows."""
    import dataclasses
    from idrak_b200.models import DecoderSpec, build_decoder
    from idrak_b200.serve import ModelRunner, PrefillItem, native_prefill
    extra = dict(extra)
    int8 = extra.pop("int8", False)
    spec = dataclasses.replace(DecoderSpec.llama(layers=2, dim=dim, heads=heads, kv_heads=kv_heads, ff_dim=1152, vocab=300, max_positions=512,
                                                 head_dim=head_dim), **extra)
    model = build_decoder(spec, seed=2).to("cuda", torch.bfloat16)
    ran = []
    inner = native_prefill.run
    monkeypatch.setattr(native_prefill, "run", lambda *a: ran.append(inner(*a)) or ran[-1])
    g = torch.Generator().manual_seed(1)
    for lengths in ((1,), (45,), (16, 16, 7), (8, 8), (300, 33)):
        out = []
        for native in (True, False):
            runner = ModelRunner(model, 80, 16, cache_dtype=torch.int8 if int8 else None)
            if not native:
                runner._native_blocks = lambda *a: None
            items, block = [], 0
            g.manual_seed(sum(lengths))
            for n in lengths:
                items.append(PrefillItem(torch.randint(0, 300, (n,), generator=g).tolist(), 0, list(range(block, block + (n + 15) // 16))))
                block += (n + 15) // 16
            caches = runner.k_cache + runner.v_cache + (runner.k_scale + runner.v_scale if int8 else [])
            out.append([runner.prefill(items).clone(), runner.prefill(items, all_logits=True).clone()] + [c[:-1].clone() for c in caches])
        assert all(torch.equal(x, y) and x.float().isfinite().all() for x, y in zip(*out))
    assert len(ran) == 10 and all(r is not None for r in ran)


def test_native_prefill_refuses_what_it_does_not_cover():
    from idrak_b200.models import DecoderSpec, build_decoder
    from idrak_b200.serve import ModelRunner, PrefillItem
    model = _small()
    runner = ModelRunner(model, 20, 16)
    items = [PrefillItem([1, 2, 3], 0, [0]), PrefillItem([4] * 20, 0, [1, 2])]
    want = runner.prefill(items).clone()
    w = model.blocks[0].attn.o_weight
    model.blocks[0].attn.o_weight = torch.nn.Parameter(torch.cat([w.data, w.data], 1)[:, : w.shape[1]])      # rows not side by side
    assert torch.equal(runner.prefill(items), want)
    assert torch.equal(runner.prefill([PrefillItem([4] * 4, 16, [1, 2])])[0], want[1])                       # behind a cached prefix
