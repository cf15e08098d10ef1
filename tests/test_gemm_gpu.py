"""tcgen05 GEMM against a plain PyTorch fp32 statement of the same contract."""
import math

import pytest
import torch

from idrak_b200.ops import gemm, gemm_reference, linear

pytestmark = pytest.mark.gpu


def _rand(shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _check(out, ref, tol=2e-2):
    out, ref = out.float(), ref.float()
    err = (out - ref).abs().max().item()
    denom = ref.abs().max().item() + 1e-6
    assert err / denom < tol, f"max err {err} vs scale {denom}"


SHAPES = [(128, 256, 64), (256, 512, 128), (384, 768, 768), (1024, 2304, 768), (200, 136, 72), (64, 64, 64),
          (130, 100, 1000), (4096, 768, 3072), (128, 50304, 768)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_majors(M, N, K, a_mn, b_mn):
    if (a_mn and M % 8) or (b_mn and N % 8) or K % 8:
        pytest.skip("leading dimension must be a multiple of 8")
    a = _rand((K, M) if a_mn else (M, K), 1.0, 1)
    b = _rand((K, N) if b_mn else (N, K), 1.0, 2)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, splits=1)
    ref = gemm_reference(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    _check(out, ref)


@pytest.mark.parametrize("splits", [2, 3, 8])
def test_gemm_splitk_matches_and_is_deterministic(splits):
    M, N, K = 768, 768, 4096
    a, b = _rand((K, M), 1.0, 3), _rand((K, N), 1.0, 4)
    ref = gemm_reference(a, b, a_mn=True, b_mn=True, out_dtype=torch.float32)
    o1 = gemm(a, b, a_mn=True, b_mn=True, splits=splits, out_dtype=torch.float32)
    o2 = gemm(a, b, a_mn=True, b_mn=True, splits=splits, out_dtype=torch.float32)
    _check(o1, ref, 5e-3)
    assert torch.equal(o1, o2)


@pytest.mark.parametrize("M", [1, 7, 16, 32, 33, 48, 64])
@pytest.mark.parametrize("N,K,splits", [(512, 256, 1), (6144, 4096, None), (4096, 1024, 4), (1000, 520, 1)])
def test_gemm_few_rows(M, N, K, splits):
    """Decode-sized products take the few-row layout (part of the A tile per stage, more stages): every epilogue the
    serving path uses, with and without split-K, and N / K that are not tile multiples."""
    a, b = _rand((M, K), 1.0, 11), _rand((N, K), 0.05, 12)
    bias, res = _rand((N,), 1.0, 13), _rand((M, N), 1.0, 14)
    _check(gemm(a, b, splits=splits), gemm_reference(a, b, out_dtype=torch.float32))
    _check(gemm(a, b, bias=bias, residual=res, splits=splits),
           gemm_reference(a, b, bias=bias, residual=res, out_dtype=torch.float32))
    out, pre = gemm(a, b, bias=bias, act="gelu", splits=splits)
    ref, ref_pre = gemm_reference(a, b, bias=bias, act="gelu", out_dtype=torch.float32)
    _check(pre, ref_pre)
    _check(out, ref)
    o32 = gemm(a, b, splits=splits, out_dtype=torch.float32)
    assert torch.equal(o32, gemm(a, b, splits=splits, out_dtype=torch.float32))
    _check(o32, gemm_reference(a, b, out_dtype=torch.float32), 5e-3)


def test_gemm_epilogues():
    M, N, K = 512, 1024, 256
    a, b = _rand((M, K), 1.0, 5), _rand((N, K), 0.1, 6)
    bias, res = _rand((N,), 1.0, 7), _rand((M, N), 1.0, 8)
    out = gemm(a, b, bias=bias, residual=res)
    _check(out, gemm_reference(a, b, bias=bias, residual=res, out_dtype=torch.float32))
    out, pre = gemm(a, b, bias=bias, act="gelu")
    ref, ref_pre = gemm_reference(a, b, bias=bias, act="gelu", out_dtype=torch.float32)
    _check(pre, ref_pre)
    _check(out, ref)
    g = gemm(a, b, act="gelu_grad", aux=pre)
    _check(g, gemm_reference(a, b, act="gelu_grad", aux=pre, out_dtype=torch.float32))
    # the training pair: activation and derivative out of the forward epilogue, one multiply in the backward one
    out_d, dact = gemm(a, b, bias=bias, act="gelu_d")
    ref_d, ref_dact = gemm_reference(a, b, bias=bias, act="gelu_d", out_dtype=torch.float32)
    _check(out_d, ref_d)
    _check(dact, ref_dact)
    _check(gemm(a, b, act="mul_aux", aux=dact), gemm_reference(a, b, act="mul_aux", aux=dact, out_dtype=torch.float32))
    acc = torch.ones((M, N), dtype=torch.float32, device="cuda")
    gemm(a, b, out=acc, beta=True, alpha=0.5)
    _check(acc, gemm_reference(a, b, alpha=0.5, out_dtype=torch.float32) + 1.0)


def test_linear_autograd_matches_torch():
    x = _rand((4, 96, 256), 1.0, 9).requires_grad_()
    w = _rand((384, 256), 0.05, 10).requires_grad_()
    b = _rand((384,), 0.1, 11).requires_grad_()
    y = linear(x, w, b)
    dy = _rand(y.shape, 1.0, 12)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(dy.float())
    _check(y, yr)
    _check(x.grad, xr.grad)
    _check(w.grad, wr.grad)
    _check(b.grad, br.grad)


def test_autotune_measures_once_and_keeps_results_equal(tmp_path):
    from idrak_b200 import config
    from idrak_b200.runtime import reset_tuner, tuner
    config.settings.set("IDRAK_AUTOTUNE", True)
    config.settings.set("IDRAK_TUNING_CACHE", str(tmp_path / "tuning.json"))
    reset_tuner()
    try:
        a, b = _rand((48, 2048), 1.0, 21), _rand((1536, 2048), 0.05, 22)
        first = gemm(a, b)
        t = tuner()
        assert t.measured == 1 and any(k.startswith("gemm.splits:64x1536x2048") for k in t.entries())
        second = gemm(a, b)
        assert t.measured == 1
        ref = gemm_reference(a, b, out_dtype=torch.float32)
        _check(first, ref)
        _check(second, ref)
    finally:
        config.settings._overrides.pop("IDRAK_AUTOTUNE", None)
        config.settings._overrides.pop("IDRAK_TUNING_CACHE", None)
        reset_tuner()


def _pair_case(M, N, K, a_mn, b_mn):
    a = _rand((K, M) if a_mn else (M, K), 1.0, 31)
    b = _rand((K, N) if b_mn else (N, K), 0.05, 32)
    ref = gemm_reference(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    out = gemm(a, b, a_mn=a_mn, b_mn=b_mn, splits=1)
    _check(out, ref)
    assert torch.equal(out, gemm(a, b, a_mn=a_mn, b_mn=b_mn, splits=1))
    if not a_mn and not b_mn:
        bias, res = _rand((N,), 1.0, 33), _rand((M, N), 1.0, 34)
        _check(gemm(a, b, bias=bias, residual=res, splits=1), gemm_reference(a, b, bias=bias, residual=res, out_dtype=torch.float32))
        o, pre = gemm(a, b, bias=bias, act="gelu", splits=1)
        r, r_pre = gemm_reference(a, b, bias=bias, act="gelu", out_dtype=torch.float32)
        _check(pre, r_pre)
        _check(o, r)
        _check(gemm(a, b, act="gelu_grad", aux=pre, splits=1), gemm_reference(a, b, act="gelu_grad", aux=pre, out_dtype=torch.float32))
        o, dact = gemm(a, b, bias=bias, act="gelu_d", splits=1)
        r, r_dact = gemm_reference(a, b, bias=bias, act="gelu_d", out_dtype=torch.float32)
        _check(dact, r_dact)
        _check(o, r)
        _check(gemm(a, b, act="mul_aux", aux=dact, splits=1), gemm_reference(a, b, act="mul_aux", aux=dact, out_dtype=torch.float32))
        acc = torch.ones((M, N), dtype=torch.float32, device="cuda")
        gemm(a, b, out=acc, beta=True, alpha=0.5, splits=1)
        _check(acc, gemm_reference(a, b, alpha=0.5, out_dtype=torch.float32) + 1.0)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(2048, 2304, 768), (4096, 768, 3072), (1504, 1000, 520), (16384, 768, 768)])
def test_gemm_large_products(M, N, K, a_mn, b_mn):
    """Products large enough for the CTA-pair kernel (256 x 256 tiles on two SMs; IDRAK_GEMM_PAIR=2 sends every such
    product there, the default only the shapes where it measured faster, 0 none): all operand layouts, sizes that are
    not tile multiples, every epilogue."""
    _pair_case(M, N, K, a_mn, b_mn)
    from idrak_b200 import _native
    _native.check_status("large products")


@pytest.mark.parametrize("N", [264, 392, 512])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_narrow_tiles_of_a_small_product_give_the_same_bits(N, a_mn, b_mn):
    """The most row tiles that still get 128 columns per tile, and one more, which gets 256: an element's sum over K has one
    order, so the rows that both calls share agree to the bit."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, K = sms // 4 * 128, 136
    a, b = _rand((rows + 128, K), 1.0, 1), _rand((N, K), 1.0, 2)
    bias, res = _rand((N,), 1.0, 3), _rand((rows + 128, N), 1.0, 4)
    def run(m):
        x = a[:m].t().contiguous() if a_mn else a[:m]
        w = b.t().contiguous() if b_mn else b
        return gemm(x, w, a_mn=a_mn, b_mn=b_mn, bias=bias, residual=res[:m], splits=1)
    narrow = run(rows)
    assert torch.equal(narrow, run(rows + 128)[:rows])
    # fp32 accumulation, one rounding to bf16 (half an ulp is 2^-9) and the fp32 reference's own
    ref = gemm_reference(a[:rows], b, out_dtype=torch.float32) + bias.float() + res[:rows].float()
    assert ((narrow.float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 63, 64, 65])
@pytest.mark.parametrize("N,K", [(8, 1024), (136, 72), (768, 768), (4096, 1032), (18944, 1024), (19200, 1024), (100, 2048), (128, 8)])
def test_products_of_few_rows_keep_the_contract(M, N, K):
    """Calls on either side of the rule that sends them to the few-row kernel: rows and widths at its edges, rows that it cannot read
    (strides between 16 bytes), an output, bias and residual given. One fp32 sum over K and one rounding to bf16 either way: half an
    ulp (2^-9 relative) each for kernel and reference, and sums of K products of magnitude about 1 in another order."""
    a, b = _rand((M, K), 1.0, 41), _rand((N, K), 0.2, 42)
    bias, res, out = _rand((N,), 1.0, 43), _rand((M, N), 1.0, 44), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ref = gemm_reference(a, b, out_dtype=torch.float32)
    full = ref + bias.float() + res.float()
    for got, want in ((gemm(a, b), ref), (gemm(a, b, bias=bias, residual=res, out=out), full), (gemm(a, b, splits=1), ref)):
        assert ((got.float() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5).all()
    assert gemm(a, b, bias=bias, residual=res, out=out) is out
    if K < 1024 or N > 18944:                                     # the dense kernel does not cut K: the same bits for any number of rows
        assert torch.equal(gemm(a, b), gemm(a, b, splits=1))
        assert torch.equal(gemm(a, b), gemm(torch.cat([a, a[:1].expand(200, K)]), b, splits=1)[:M])
    wide = torch.zeros(M, K + 3, dtype=torch.bfloat16, device="cuda")
    if M > 1:
        wide[:, :K] = a
        with pytest.raises(Exception):
            gemm(wide[:, :K], b)
    assert gemm(a, b, out_dtype=torch.float32).dtype == torch.float32
    from idrak_b200 import _native
    _native.check_status("few rows")


@pytest.mark.parametrize("M", [65, 80, 127, 128, 129, 160, 192, 193, 255, 256])
@pytest.mark.parametrize("N,K", [(8, 1024), (264, 1032), (768, 3072), (4096, 1024), (300, 136)])
def test_products_of_some_more_rows(M, N, K):
    """The kernel for 65 to 256 rows on either side of the rule that sends products to it, and called by itself at sizes that the rule
    does not give it: one pass of 128 rows, two, a ragged last tile of features, an uncut K with the dense kernel's bits."""
    from idrak_b200.ops.skinny import wide_linear
    a, b = _rand((M, K), 1.0, 51), _rand((N, K), 0.2, 52)
    bias, res, out = _rand((N,), 1.0, 53), _rand((M, N), 1.0, 54), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    ref = gemm_reference(a, b, out_dtype=torch.float32)
    full = ref + bias.float() + res.float()
    for got, want in ((gemm(a, b), ref), (gemm(a, b, bias=bias, residual=res, out=out), full), (wide_linear(a, b), ref),
                      (wide_linear(a, b, bias, res, torch.empty_like(out)), full)):
        # fp32 sums in another order and one rounding to bf16, as in the test of few rows
        assert ((got.float() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5).all()
    assert torch.equal(wide_linear(a, b, one_pass=True), gemm(a, b, splits=1)) and torch.equal(wide_linear(a, b), wide_linear(a, b))
    from idrak_b200 import _native
    _native.check_status("wide")


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(8, 8, 8), (72, 64, 64), (264, 128, 512), (64, 192, 1032), (520, 392, 200), (296, 72, 1000), (64, 64, 8192),
                                   (1024, 520, 128), (3072, 576, 64), (1024, 64, 1024), (1032, 256, 1024)])
def test_small_products(M, N, K, a_mn, b_mn):
    """The kernel of products of a few tiles on either side of the rules that send them to it, ragged in each direction, in each
    operand order, over views whose rows lie further apart than they are long; every form of the epilogue."""
    def operand(rows, cols, sd, seed):
        return _rand((rows, cols + 24), sd, seed)[:, 8 : 8 + cols]
    a = operand(K, M, 1.0, 61) if a_mn else operand(M, K, 1.0, 61)
    b = operand(K, N, 0.2, 62) if b_mn else operand(N, K, 0.2, 62)
    bias, res, aux = _rand((N,), 1.0, 63), operand(M, N, 1.0, 64), _rand((M, N), 1.0, 65)
    order = dict(a_mn=a_mn, b_mn=b_mn)
    # sums of K products of standard deviation 0.2 in fp32 in another order, and one rounding to bf16 (half an ulp: 2^-8)
    tol = lambda want: 2.0 ** -8 * want.abs() + 1e-5 * K ** 0.5
    for kw in (dict(), dict(bias=bias, residual=res, alpha=0.5), dict(act="mul_aux", aux=aux), dict(act="gelu_d", bias=bias)):
        got, want = gemm(a, b, **order, **kw), gemm_reference(a, b, **order, **kw, out_dtype=torch.float32)
        pairs = zip(got, want) if isinstance(got, tuple) else ((got, want),)
        for g, w in pairs:                  # the derivative that the oracle returns is itself rounded: one ulp
            assert ((g.float() - w.float()).abs() <= tol(w.float()) * (2 if isinstance(got, tuple) else 1)).all()
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.ones(M, N + 3, device="cuda", dtype=dtype)[:, 1 : N + 1]          # rows that start anywhere
        want = gemm_reference(a, b, **order, out_dtype=torch.float32) + 1
        got = gemm(a, b, **order, out=out, beta=True)
        assert ((got.float() - want).abs() <= tol(want)).all()
    assert torch.equal(gemm(a, b, **order, splits=0), gemm(a, b, **order, splits=0))
    if not (a_mn or b_mn) and K <= 960:      # up to 15 blocks K is not cut: in one pass, with the bits of the kernel for larger products
        assert torch.equal(gemm(a, b, bias=bias, residual=res, splits=0), gemm(a, b, bias=bias, residual=res, splits=1))
    from idrak_b200 import _native
    _native.check_status("small")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("tokens,M,N", [(8, 8, 8), (65, 72, 136), (1000, 384, 128), (1024, 512, 128), (1500, 200, 64), (8192, 64, 64), (4096, 2304, 768)])
def test_weight_and_bias_gradient(tokens, M, N, accumulate, dtype):
    """One launch for both where the weight gradient is small (all sizes but the last): the weight gradient has the bits it has alone, and
    the column sums are as close to the 64-bit ones as a tree of fp32 sums has to be."""
    from idrak_b200.ops import _grad
    from idrak_b200.ops.gemm import bias_grad, weight_bias_grad, weight_grad
    dy, x = _rand((tokens, M + 8), 1.0, 71)[:, :M], _rand((tokens, N), 1.0, 72)
    times, grads = 2 if accumulate else 1, []
    for fused in (True, False):
        w, b = (torch.nn.Parameter(torch.zeros(s, device="cuda", dtype=dtype)) for s in ((M, N), (M,)))
        w.grad, b.grad = torch.ones_like(w), torch.ones_like(b)
        _grad.enable((w, b))
        for _ in range(times):
            if fused:
                assert weight_bias_grad(dy, x, w, b, dy) == (None, None)
            else:
                weight_grad(dy, x, w), bias_grad(dy, b, dy)
        grads.append((w.grad, b.grad))
        _grad.next_step()
    assert torch.equal(grads[0][0], grads[1][0])
    want = dy.double().sum(0)
    # every fp32 addition is off by 2^-24 of its partial sum, and a value passes fewer than log2(tokens) + 16 of them; a bf16 store by 2^-8
    bound = dy.double().abs().sum(0) * 2.0 ** -24 * (math.log2(tokens) + 16) * times
    if dtype == torch.bfloat16:
        bound = bound + want.abs() * 2.0 ** -8 * (3 if accumulate else 1)      # the first store of 1 x, the second of 2 x
    assert ((grads[0][1].double() - times * want).abs() <= bound).all()
    new = weight_bias_grad(dy, x, None, None)
    assert torch.equal(new[0], gemm(dy, x, a_mn=True, b_mn=True)) and new[1].dtype == torch.bfloat16
    from idrak_b200 import _native
    _native.check_status("weight and bias gradient")


@pytest.mark.parametrize("M,N,K", [(257, 4096, 4096), (384, 4096, 1032), (300, 28672, 256), (1030, 4096, 200), (520, 28672, 192), (2100, 28672, 128)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_products_of_an_odd_number_of_row_tiles(M, N, K, b_mn):
    """Sizes on either side of the rule that keeps a product on single CTAs: a tile fewer than pairs, a wave fewer, all tiles cut."""
    a, b, res = _rand((M, K), 1.0, 81), _rand((K, N) if b_mn else (N, K), 0.2, 82), _rand((M, N), 1.0, 83)
    ref = gemm_reference(a, b, b_mn=b_mn, residual=res, out_dtype=torch.float32)
    # fp32 sums in another order and one rounding to bf16, as in the test of few rows
    assert ((gemm(a, b, b_mn=b_mn, residual=res).float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * K ** 0.5).all()
    from idrak_b200 import _native
    _native.check_status("row tiles")
