"""Each CUDA kernel alone against its plain PyTorch statement (tests/kernel_refs.py), at sizes
other than the engine's: odd widths, head sizes in steps of 16, any grouping, windows, page edges."""


import pytest
import torch

import kernel_refs as ref

pytestmark = pytest.mark.gpu

DEV = "cuda"


def ops():
    from lily_b200.csrc import ops as o
    return o


def tol(dtype):
    return dict(atol=2e-5, rtol=2e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


DTYPES = [torch.float32, torch.bfloat16]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden,vocab", [(64, 256), (136, 331), (4096, 1009)])
def test_embed(dtype, hidden, vocab):
    g = torch.Generator(device=DEV).manual_seed(0)
    table = torch.randn(vocab, hidden, device=DEV, generator=g).to(dtype)
    ids = torch.randint(0, vocab, (37,), device=DEV, generator=g, dtype=torch.int32)
    assert torch.equal(ops().embed(table, ids), ref.embed(table, ids))
    # ids below zero name request slots whose token the sampler left on the device
    future = torch.randint(0, vocab, (9,), device=DEV, generator=g, dtype=torch.int32)
    mixed = ids.clone()
    mixed[::3] = -(torch.arange(0, 13, device=DEV, dtype=torch.int32) % 9 + 1)
    assert torch.equal(ops().embed(table, mixed, future=future), ref.embed(table, mixed, future=future))
    assert torch.equal(ops().embed(table, mixed, future=future)[0], table[future[0].long()].float())


def test_scatter_tokens():
    g = torch.Generator(device=DEV).manual_seed(17)
    tokens = torch.randint(0, 1000, (5,), device=DEV, generator=g, dtype=torch.int32)
    logit_rows = torch.tensor([0, 1, 2, 9, 30], device=DEV, dtype=torch.int32)        # three decode tokens, two portions' ends
    token_req = torch.tensor([0, 1, 2] + [3] * 7 + [4] * 21, device=DEV, dtype=torch.int32)
    slots = torch.tensor([4, 1, 7, 2, 5], device=DEV, dtype=torch.int32)
    a = torch.full((9,), -5, device=DEV, dtype=torch.int32)
    b = a.clone()
    ops().scatter_tokens(tokens, logit_rows, token_req, slots, a)
    ref.scatter_tokens(tokens, logit_rows, token_req, slots, b)
    assert torch.equal(a, b) and a[4] == tokens[0] and a[5] == tokens[4] and a[0] == -5


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("wdtype", DTYPES)
@pytest.mark.parametrize("hidden", [64, 136, 1000, 4096, 12288])
def test_add_rmsnorm(dtype, wdtype, hidden):
    if dtype == torch.float32 and wdtype == torch.bfloat16:
        pytest.skip("float32 activations keep float32 gains")
    g = torch.Generator(device=DEV).manual_seed(1)
    n = 19
    resid = torch.randn(n, hidden, device=DEV, generator=g) * 3
    delta = torch.randn(n, hidden, device=DEV, generator=g).to(dtype)
    w = (1 + 0.1 * torch.randn(hidden, device=DEV, generator=g)).to(wdtype)
    for d in (delta, None):
        r1, r2 = resid.clone(), resid.clone()
        got = ops().add_rmsnorm(r1, d, w, 1e-5, dtype)
        want = ref.add_rmsnorm(r2, d, w, 1e-5, dtype)
        torch.testing.assert_close(r1, r2, atol=0, rtol=0)
        torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    rows = torch.tensor([18, 0, 7, 7], device=DEV, dtype=torch.int32)
    r1 = resid.clone()
    got = ops().add_rmsnorm(r1, delta, w, 1e-6, dtype, rows=rows)
    want = ref.add_rmsnorm(resid.clone(), delta, w, 1e-6, dtype, rows=rows)
    assert torch.equal(r1, resid)                       # gathered rows leave the residual alone
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("inter", [128, 200, 352, 12288])
def test_silu_mul(dtype, inter):
    g = torch.Generator(device=DEV).manual_seed(2)
    gu = (torch.randn(23, 2 * inter, device=DEV, generator=g) * 2).to(dtype)
    torch.testing.assert_close(ops().silu_mul(gu).float(), ref.silu_mul(gu).float(), **tol(dtype))


@pytest.mark.parametrize("m,n,k", [(1, 64, 64), (7, 331, 136), (65, 129, 200), (33, 1009, 4096), (300, 24, 17)])
def test_gemm_fp32_is_true_fp32(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.randn(m, k, device=DEV, generator=g)
    w = torch.randn(n, k, device=DEV, generator=g)
    b = torch.randn(n, device=DEV, generator=g)
    want = (x.double() @ w.double().t() + b.double()).float()
    got = ops().linear(x, w, b)
    # float32 accumulation error grows like sqrt(k) * 2^-24 * |x||w|; TF32 would be ~1e-3 relative
    assert float((got - want).abs().max()) < 4e-6 * (k ** 0.5) * 4
    # a row's result does not depend on the other rows in the batch
    assert torch.equal(ops().linear(x[:1].contiguous(), w, b), got[:1])


def test_linear_bf16_and_fp32_logits():
    g = torch.Generator(device=DEV).manual_seed(4)
    x = torch.randn(9, 136, device=DEV, generator=g).bfloat16()
    w = torch.randn(331, 136, device=DEV, generator=g).bfloat16()
    b = torch.randn(331, device=DEV, generator=g).bfloat16()
    want = x.float() @ w.float().t()
    torch.testing.assert_close(ops().linear(x, w).float(), want, atol=0.1, rtol=2e-2)
    out = ops().linear(x, w, out_dtype=torch.float32)
    assert out.dtype == torch.float32
    torch.testing.assert_close(out, want, atol=1e-3, rtol=1e-4)       # logits keep the accumulator's precision
    # the product may be rounded to bfloat16 before the bias is added: half an ulp at its magnitude (~64)
    torch.testing.assert_close(ops().linear(x, w, b).float(), want + b.float(), atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (8, 6144, 4096), (8, 4096, 12288), (5, 331, 128), (16, 1000, 256),
                                   (17, 136, 64), (33, 2000, 1024), (64, 4096, 1024), (3, 24576, 4096), (64, 24, 64),
                                   (8, 5120, 25600), (16, 4096, 12288),                                     # a long slice of x
                                   (1, 5120, 25600), (2, 5120, 25600), (3, 10240, 8192), (3, 300, 16384)])   # x read from global memory
def test_skinny_gemm_partial_sums(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(11)
    x = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    w = torch.randn(n, k, device=DEV, generator=g).bfloat16()
    parts = ops().linear_split(x, w, splits=max(1, min(5, k // 512)))
    assert parts is not None and parts.dtype == torch.float32 and parts.shape[1:] == (m, n)
    auto = ops().linear_split(x, w)                     # the kernel's own rule may leave the shape to the library
    if auto is not None:
        torch.testing.assert_close(auto.sum(0), parts.sum(0), atol=2e-5 * (k ** 0.5) * 4, rtol=1e-4)       # other slices, other rounding
    want = x.double() @ w.double().t()
    got = parts.double().sum(0)
    assert float((got - want).abs().max()) < 2e-5 * (k ** 0.5) * 4      # float32 accumulation of exact products
    # a token's result does not depend on the other tokens in the batch
    alone = ops().linear_split(x[:1].contiguous(), w, splits=parts.shape[0])
    assert torch.equal(alone[:, 0], parts[:, 0])
    # shapes the kernel does not take are left to the library product
    assert ops().linear_split(torch.zeros(65, k, device=DEV).bfloat16(), w) is None
    assert ops().linear_split(torch.zeros(2, 72, device=DEV).bfloat16(), torch.zeros(8, 72, device=DEV).bfloat16()) is None
    assert ops().linear_split(x.float(), w.float()) is None


SWIGLU_SHAPES = [(8, 12288, 4096, 128), (1, 12288, 4096, 128), (5, 1408, 512, 128), (8, 200, 64, None),
                 (3, 264, 1088, 8), (7, 25600, 5120, 128), (8, 352, 128, None), (2, 128, 12288, 64)]


@pytest.mark.parametrize("m,inter,k,run", SWIGLU_SHAPES)
def test_skinny_swiglu(m, inter, k, run):
    """The gate/up product with SiLU*mul in one weight-streaming kernel against the plain statement: tall and low
    matrices, deep k, both layouts of the fused matrix, 1 to 8 tokens; scratch and counters left as they are, and a
    token's result does not depend on its neighbours."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(12)
    x = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * inter, k, device=DEV, generator=g) * k ** -0.5).bfloat16()
    need = o.swiglu_skinny_need(m, inter, k, torch.bfloat16, run, whenever_possible=True)
    assert need is not None
    scratch = torch.full((need[0],), float("nan"), device=DEV)
    counters = torch.zeros(need[1], device=DEV, dtype=torch.int32)
    got = o.swiglu_skinny(x, w, run, scratch, counters)
    gu = x.double() @ w.double().t()
    want = ref.silu_mul(gu.float(), torch.float32, block=run)
    torch.testing.assert_close(got.float(), want, atol=2e-2, rtol=2e-2)
    assert float((got.float() - want).abs().mean()) < 2e-3
    assert int(counters.abs().sum()) == 0
    again = o.swiglu_skinny(x, w, run, scratch, counters)
    assert torch.equal(again, got) and int(counters.abs().sum()) == 0
    alone = o.swiglu_skinny(x[:1].contiguous(), w, run, scratch, counters)
    assert torch.equal(alone[0], got[0])
    assert o.swiglu_skinny_need(9, inter, k, torch.bfloat16, run) is None
    assert o.swiglu_skinny_need(m, inter, k, torch.bfloat16, run) is not None
    assert torch.equal(o.swiglu_skinny(x, w, run), got)
    assert o.swiglu_skinny_need(m, inter, k, torch.float32, run) is None
    assert o.swiglu_skinny_need(m, inter, k + 8, torch.bfloat16, run) is None


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (2048, 6144, 4096), (300, 1000, 136), (65, 331, 200), (1, 24, 8),
                                   (777, 512, 4096), (129, 257, 72), (1100, 5000, 520), (2048, 4096, 12288), (4100, 2500, 72)])
def test_gemm_tcgen05(m, n, k):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(13)
    x = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    w = torch.randn(n, k, device=DEV, generator=g).bfloat16()
    b = torch.randn(n, device=DEV, generator=g).bfloat16()
    want = x.float() @ w.float().t()
    got = o.gemm_tc(x, w)
    assert o.gemm_tc_status() == 0
    # exact bfloat16 products summed in float32, rounded once to bfloat16
    torch.testing.assert_close(got.float(), want, atol=2e-2 * (k ** 0.5), rtol=1e-2)
    assert float((got.float() - want).abs().max()) <= float(want.abs().max()) * 2 ** -7
    torch.testing.assert_close(o.gemm_tc(x, w, b).float(), want + b.float(), atol=2e-2 * (k ** 0.5) + 0.1, rtol=1e-2)
    assert o.gemm_tc_status() == 0
    assert torch.equal(o.gemm_tc(x, w), got) and o.gemm_tc_status() == 0          # again: the same bits


@pytest.mark.parametrize("activation", ["relu2", "silu", "gelu_tanh"])
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (2048, 3072, 2048), (300, 1000, 136), (65, 331, 200), (777, 520, 4096)])
def test_gemm_tcgen05_activation_epilogue(activation, m, n, k):
    """The plain product with an activation on the float32 sums before they are rounded, and the feed-forward's
    ``linear_activation`` that takes this kernel for 65 tokens and more."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(15)
    x = (torch.randn(m, k, device=DEV, generator=g) * 0.5).bfloat16()
    w = (torch.randn(n, k, device=DEV, generator=g) * (k ** -0.5) * 2).bfloat16()
    z = x.float() @ w.float().t()
    want = {"relu2": torch.clamp(z, min=0) ** 2, "silu": torch.nn.functional.silu(z),
            "gelu_tanh": torch.nn.functional.gelu(z, approximate="tanh")}[activation]
    got = o.gemm_tc(x, w, plain_activation=activation)
    assert o.gemm_tc_status() == 0 and got.shape == (m, n)
    torch.testing.assert_close(got.float(), want, atol=2e-2, rtol=2e-2)
    via = o.linear_activation(x, w, activation)
    torch.testing.assert_close(via.float(), want, atol=2e-2, rtol=2e-2)
    unfused = o.activation(o.linear(x, w, out_dtype=torch.float32), torch.bfloat16, activation)
    torch.testing.assert_close(unfused.float(), want, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("m,inter,k", [(128, 128, 64), (2048, 12288, 4096), (300, 384, 136), (70, 256, 4096)])
def test_gemm_tcgen05_silu_mul_epilogue(m, inter, k):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(14)
    x = (torch.randn(m, k, device=DEV, generator=g) * 0.5).bfloat16()
    gate = (torch.randn(inter, k, device=DEV, generator=g) * (k ** -0.5)).bfloat16()
    up = (torch.randn(inter, k, device=DEV, generator=g) * (k ** -0.5)).bfloat16()
    mixed = torch.stack((gate.view(inter // 128, 128, k), up.view(inter // 128, 128, k)), dim=1).reshape(2 * inter, k).contiguous()
    gt, ut = x.float() @ gate.float().t(), x.float() @ up.float().t()
    want = torch.nn.functional.silu(gt) * ut
    got = o.gemm_tc(x, mixed, silu_mul_block=True)
    assert o.gemm_tc_status() == 0 and got.shape == (m, inter)
    torch.testing.assert_close(got.float(), want, atol=2e-2, rtol=2e-2)
    # the same interleaved product through the unfused path: library product, then SiLU*mul in runs of 128
    two = o.linear(x, mixed)
    torch.testing.assert_close(o.silu_mul(two, block=128).float(), want, atol=3e-2, rtol=3e-2)
    torch.testing.assert_close(o.silu_mul(two, block=128).float(), ref.silu_mul(two, block=128).float(), atol=2e-2, rtol=2e-2)


def test_kernels_add_up_partial_sums():
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(12)
    m, h, nq, nkv, d, page = 7, 136, 4, 2, 16, 16
    parts = torch.randn(3, m, h, device=DEV, generator=g)
    whole = (parts[0] + parts[1]) + parts[2]
    w = (1 + 0.1 * torch.randn(h, device=DEV, generator=g)).bfloat16()
    r1, r2 = torch.randn(m, h, device=DEV, generator=g), None
    r2 = r1.clone()
    a = o.add_rmsnorm(r1, parts, w, 1e-6, torch.bfloat16)
    b = o.add_rmsnorm(r2, whole, w, 1e-6, torch.bfloat16)
    assert torch.equal(a, b) and torch.equal(r1, r2)
    gu = torch.randn(3, m, 2 * 200, device=DEV, generator=g)
    assert torch.equal(o.silu_mul(gu, torch.bfloat16), o.silu_mul((gu[0] + gu[1]) + gu[2], torch.bfloat16))
    torch.testing.assert_close(o.silu_mul(gu, torch.bfloat16).float(),
                               ref.silu_mul(gu.sum(0)).float(), atol=2e-2, rtol=2e-2)
    qkv = torch.randn(3, m, (nq + 2 * nkv) * d, device=DEV, generator=g)
    pos = torch.arange(m, device=DEV, dtype=torch.int32) + 5
    req = torch.zeros(m, device=DEV, dtype=torch.int32)
    table = torch.tensor([[2, 1]], device=DEV, dtype=torch.int32)
    cos, sin = torch.rand(32, d // 2, device=DEV, generator=g), torch.rand(32, d // 2, device=DEV, generator=g)
    gain = torch.ones(d, device=DEV).bfloat16()
    c1 = torch.zeros(3, 2, nkv, page, d, device=DEV).bfloat16()
    c2 = c1.clone()
    q1 = o.qk_norm_rope_write(qkv, gain, gain, 1e-6, cos, sin, pos, req, table, c1, nq, nkv, d, d, page)
    q2 = o.qk_norm_rope_write((qkv[0] + qkv[1]) + qkv[2], gain, gain, 1e-6, cos, sin, pos, req, table, c2, nq, nkv, d, d, page)
    assert q1.dtype == torch.bfloat16 and torch.equal(q1, q2) and torch.equal(c1, c2) and float(c1.abs().max()) > 0


def _cache(pages, nkv, page_size, d, dtype, g):
    return (torch.randn(pages + 1, 2, nkv, page_size, d, device=DEV, generator=g)).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,rd,norm", [(4, 2, 16, 16, True), (8, 2, 32, 32, False), (6, 2, 48, 24, True),
                                               (5, 1, 80, 80, False), (32, 8, 128, 128, True), (3, 3, 256, 64, True),
                                               (7, 7, 64, 64, True), (2, 1, 256, 256, True), (9, 3, 128, 128, False)])
def test_qk_norm_rope_write(dtype, nq, nkv, d, rd, norm):
    g = torch.Generator(device=DEV).manual_seed(5)
    page, n, reqs = 16, 50, 3
    qkv = torch.randn(n, (nq + 2 * nkv) * d, device=DEV, generator=g).to(dtype)
    token_req = torch.tensor([i % reqs for i in range(n)], device=DEV, dtype=torch.int32)
    # distinct (request, position) pairs so that no two tokens write the same place
    positions = torch.arange(n, device=DEV, dtype=torch.int32) + 3
    table = (torch.randperm(reqs * 6, device=DEV, generator=g) + 1).view(reqs, 6).to(torch.int32)
    cos = torch.rand(128, rd // 2, device=DEV, generator=g)
    sin = torch.rand(128, rd // 2, device=DEV, generator=g)
    qg = (1 + 0.1 * torch.randn(d, device=DEV, generator=g)).to(dtype) if norm else None
    kg = (1 + 0.1 * torch.randn(d, device=DEV, generator=g)).to(dtype) if norm else None
    c1 = _cache(18, nkv, page, d, dtype, g)
    c0, c2 = c1.clone(), c1.clone()
    got = ops().qk_norm_rope_write(qkv, qg, kg, 1e-6, cos, sin, positions, token_req, table, c1, nq, nkv, d, rd, page)
    want = ref.qk_norm_rope_write(qkv, qg, kg, 1e-6, cos, sin, positions, token_req, table, c2, nq, nkv, d, rd, page)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    torch.testing.assert_close(c1.float(), c2.float(), **tol(dtype))
    assert not torch.equal(c1, c0)
    # without rotation tables and without the cache write
    c3 = c1.clone()
    got = ops().qk_norm_rope_write(qkv, qg, kg, 1e-6, None, None, positions, token_req, table, c3, nq, nkv, d, 0, page,
                                   write_kv=False)
    want = ref.qk_norm_rope_write(qkv, qg, kg, 1e-6, None, None, positions, token_req, table, c2.clone(), nq, nkv, d,
                                  0, page, write_kv=False)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    assert torch.equal(c3, c1)


def _attention_case(dtype, nq, nkv, d, page, prefixes, news, window, seed=6, spike=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    reqs = len(prefixes)
    width = max(-(-(p + n) // page) for p, n in zip(prefixes, news))
    pages = reqs * width
    cache = _cache(pages, nkv, page, d, dtype, g)
    table = (torch.randperm(pages, device=DEV, generator=g) + 1).view(reqs, width).to(torch.int32)
    total = sum(news)
    q = torch.randn(total, nq * d, device=DEV, generator=g).to(dtype)
    if spike:
        # one far key per request dominates: its key is a scaled copy of the first query of that request
        at = 0
        for r, (p, n) in enumerate(zip(prefixes, news)):
            far = 1 if p + n > 2 else 0
            pg, off = int(table[r, far // page]), far % page
            for h in range(nkv):
                cache[pg, 0, h, off] = (q[at].view(nq, d)[h * (nq // nkv)].float() * 4).to(dtype)
            at += n
    cu = torch.tensor([0] + list(torch.tensor(news).cumsum(0)), device=DEV, dtype=torch.int32)
    pre = torch.tensor(prefixes, device=DEV, dtype=torch.int32)
    return cache, table, q, cu, pre


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,page,window", [
    (4, 2, 16, 16, None), (8, 2, 32, 16, None), (6, 2, 48, 8, 40), (5, 1, 80, 32, None), (32, 8, 128, 64, None),
    (2, 2, 256, 16, 100), (16, 2, 64, 16, 33), (40, 1, 32, 16, None), (40, 2, 64, 16, None), (6, 2, 192, 32, 500),
    (8, 8, 128, 8, 64)])
def test_attention_prefill(dtype, nq, nkv, d, page, window):
    prefixes, news = [0, 17, 130, 5, 300, 64], [1, 70, 33, 200, 129, 2]      # lengths of the reference's own test
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, prefixes, news, window, spike=True)
    rows = ops().prefill_tile_rows(dtype, d)
    treq = [r for r, n in enumerate(news) for _ in range(0, n, rows)]
    tstart = [s for r, n in enumerate(news) for s in range(0, n, rows)]
    treq_t = torch.tensor(treq, device=DEV, dtype=torch.int32)
    tstart_t = torch.tensor(tstart, device=DEV, dtype=torch.int32)
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    ops().attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, got, nq, nkv, d, page, d ** -0.5, window)
    ref.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, want, nq, nkv, d, page, d ** -0.5, window)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))


def _tiles_of(news, rows):
    treq = [r for r, n in enumerate(news) for _ in range(0, n, rows)]
    tstart = [s for r, n in enumerate(news) for s in range(0, n, rows)]
    return (torch.tensor(treq, device=DEV, dtype=torch.int32), torch.tensor(tstart, device=DEV, dtype=torch.int32))


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("nq,nkv,page,window", [(8, 2, 64, None), (4, 4, 128, None), (6, 1, 256, None), (4, 2, 64, 200),
                                                 (2, 1, 64, 100), (4, 2, 128, 129), (6, 2, 64, None), (3, 3, 64, 70)])
def test_attention_prefill_tcgen05(nq, nkv, page, window, d):
    """The tcgen05 kernel (tiles of 128 rows; head sizes 128 and 64) against the plain statement: cached prefixes
    that end inside a page and inside a key tile, portions shorter and longer than a tile, one token."""
    o, dtype = ops(), torch.bfloat16
    rows = o.prefill_tile_rows(dtype, d, page, 10 ** 6)
    assert rows == 128 and o.uses_tcgen05_attention(dtype, d, page, 4096) and not o.uses_tcgen05_attention(dtype, d, 16, 4096)
    prefixes, news = [0, 17, 130, 5, 700, 64, 1000], [1, 70, 333, 200, 129, 2, 640]
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, prefixes, news, window, spike=True)
    treq_t, tstart_t = _tiles_of(news, rows)
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    o.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, got, nq, nkv, d, page, d ** -0.5, window, tile_rows=rows,
                        heads_per_block=1)
    assert o.attention_tc_status() == 0
    ref.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, want, nq, nkv, d, page, d ** -0.5, window)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    if (nq // nkv) % 2 == 0:
        # the form with two heads of a kv head a block
        both = torch.zeros_like(q)
        o.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, both, nq, nkv, d, page, d ** -0.5, window, tile_rows=rows,
                            heads_per_block=2)
        assert o.attention_tc_status() == 0
        torch.testing.assert_close(both.float(), want.float(), **tol(dtype))
    else:
        with pytest.raises(o.KernelError, match="heads a block"):
            o.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, torch.zeros_like(q), nq, nkv, d, page, d ** -0.5,
                                window, tile_rows=rows, heads_per_block=2)
    # the mma.sync kernel on the same case, cut into its own tiles, agrees too
    base = o.prefill_tile_rows(dtype, d)
    breq, bstart = _tiles_of(news, base)
    other = torch.zeros_like(q)
    o.attention_prefill(q, cache, table, cu, pre, breq, bstart, other, nq, nkv, d, page, d ** -0.5, window)
    torch.testing.assert_close(got.float(), other.float(), **tol(dtype))


@pytest.mark.parametrize("d", [128, 64])
def test_attention_prefill_tcgen05_rising_scores(d):
    """Scores that grow by far more than 2^8 from one key tile to the next, for every row: the kernel
    must rescale the output in tensor memory each time (the path that ordinary data rarely takes)."""
    o, dtype, nq, nkv, page = ops(), torch.bfloat16, 4, 2, 64
    g = torch.Generator(device=DEV).manual_seed(21)
    prefixes, news = [300, 0], [520, 700]
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, prefixes, news, None, seed=22)
    u = torch.randn(d, device=DEV, generator=g)
    q = (0.5 * q.float().view(-1, nq, d) + u).view(q.shape).to(dtype)
    for r, (p, n) in enumerate(zip(prefixes, news)):
        for pos, c in ((40, 0.25), (190, 0.5), (330, 1.0), (470, 1.5), (p + n - 90, 2.5), (p + n - 3, 4.0)):
            pg, off = int(table[r, pos // page]), pos % page
            cache[pg, 0, :, off] = (c * u).to(dtype)
            cache[pg, 1, :, off] = c
    rows = o.prefill_tile_rows(dtype, d, page, 10 ** 6)
    treq_t, tstart_t = _tiles_of(news, rows)
    want = torch.zeros_like(q)
    ref.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, want, nq, nkv, d, page, d ** -0.5, None)
    for heads in (1, 2):
        got = torch.zeros_like(q)
        o.attention_prefill(q, cache, table, cu, pre, treq_t, tstart_t, got, nq, nkv, d, page, d ** -0.5, None, tile_rows=rows,
                            heads_per_block=heads)
        assert o.attention_tc_status() == 0
        torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    assert float(want.float()[-1].view(nq, d)[0].mean()) > 3.5          # the last row sees the strongest key


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("splits", [1, 3, 6, 7, 8, 12, 40, 300])         # 300: past what the combine kernel stages in shared memory
@pytest.mark.parametrize("nq,nkv,d,page,window", [
    (4, 2, 16, 16, None), (8, 2, 32, 16, None), (6, 2, 48, 8, 40), (5, 1, 80, 32, None), (32, 8, 128, 64, None),
    (2, 2, 256, 16, 100), (40, 1, 32, 16, None), (16, 16, 64, 16, 7), (40, 2, 64, 16, None), (6, 2, 192, 32, 500),
    (8, 8, 128, 8, 64)])
def test_attention_decode(dtype, splits, nq, nkv, d, page, window):
    seqs = [1, 8, 65, 500, 1000, 3, 257]                                     # prefixes up to 999, as the reference tests
    prefixes, news = [s - 1 for s in seqs], [1] * len(seqs)
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, prefixes, news, window, seed=7, spike=True)
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    need = ops().decode_scratch_floats(len(seqs), nq, d, splits)
    scratch = torch.full((max(need, 1),), float("nan"), device=DEV)
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    ops().attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, window)
    ref.attention_decode(q, cache, table, seq_t, want, None, splits, nq, nkv, d, page, d ** -0.5, window)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))


@pytest.mark.parametrize("from_projection", [False, True])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("nq,nkv,d,page,window", [(32, 8, 128, 64, None), (8, 2, 64, 16, None), (40, 2, 64, 16, 70), (5, 1, 128, 8, 300)])
def test_attention_decode_with_three_stages(from_projection, splits, nq, nkv, d, page, window):
    """The tensor-core kernel with three key/value tiles a block (the plan's form for many rows of about one length):
    rows of one tile, of two, of exactly the three that are asked for ahead, and longer; a spike in every row; from
    finished queries and from the projection, where the block with the new position writes its key and value first."""
    o = ops()
    dtype = torch.bfloat16
    seqs = [1, 64, 65, 128, 129, 192, 193, 500, 1000, 3, 257]
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, [n - 1 for n in seqs], [1] * len(seqs), window, seed=17, spike=True)
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    scratch = torch.full((max(o.decode_scratch_floats(len(seqs), nq, d, splits), 1),), float("nan"), device=DEV)
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    if not from_projection:
        o.attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, window, stages=3)
        ref.attention_decode(q, cache, table, seq_t, want, None, splits, nq, nkv, d, page, d ** -0.5, window)
    else:
        g = torch.Generator(device=DEV).manual_seed(171)
        qkv = torch.cat([q, torch.randn(len(seqs), 2 * nkv * d, device=DEV, generator=g).to(dtype)], 1)
        gain = (1 + 0.1 * torch.randn(d, device=DEV, generator=g)).to(dtype)
        cos, sin = torch.rand(1100, d // 2, device=DEV, generator=g), torch.rand(1100, d // 2, device=DEV, generator=g)
        one, two = cache.clone(), cache.clone()
        o.attention_decode_fused(qkv, gain, gain, 1e-6, cos, sin, one, table, seq_t, got, scratch, splits, nq, nkv, d, d, page,
                                 d ** -0.5, window, stages=3)
        o.attention_decode_fused(qkv, gain, gain, 1e-6, cos, sin, two, table, seq_t, want, scratch, splits, nq, nkv, d, d, page,
                                 d ** -0.5, window)
        ref_out = torch.zeros_like(q)
        ref.attention_decode_fused(qkv, gain, gain, 1e-6, cos, sin, cache.clone(), table, seq_t, ref_out, None, splits, nq, nkv, d,
                                   d, page, d ** -0.5, window)
        assert torch.equal(one, two)                                   # the same key and value written
        torch.testing.assert_close(want.float(), ref_out.float(), **tol(dtype))
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    with pytest.raises(Exception, match="stages"):
        o.attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, window, stages=4)


@pytest.mark.parametrize("rows,splits,stages", [(11, 1, 0), (11, 3, 0), (11, 2, 3), (64, 1, 0), (64, 2, 0), (129, 1, 0)])
@pytest.mark.parametrize("nq,nkv,d,page,window,keep", [
    (32, 8, 128, 64, None, 0), (32, 8, 128, 128, 100, 0), (16, 8, 64, 64, None, 0), (16, 8, 64, 128, 70, 65), (40, 2, 128, 64, 64, 3)])
def test_attention_decode_by_whole_tiles(nq, nkv, d, page, window, keep, rows, splits, stages):
    """Pages of whole tiles come by TMA: against the same cache in pages of 16, which are fetched piece by piece, and the reference.  Rows of one key up to several
    tiles in an order of their own (64 rows over 8 kv heads are taken longest first, 129 are not), and infinities and NaN where no key is.
    Without a window both add up the same ranges; with one they start at different keys."""
    o, dtype = ops(), torch.bfloat16
    lens = [1, 64, 65, 128, 129, 192, 193, 500, 1000, 3, 257]
    seqs = [lens[(7 * i) % 11] + (i // 11) for i in range(rows)]
    cache, table, q, cu, pre = _attention_case(dtype, nq, nkv, d, page, [n - 1 for n in seqs], [1] * rows, window, seed=19, spike=True)
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    for r, n in enumerate(seqs):
        if n % page:
            cache[int(table[r, n // page]), 0, :, n % page:] = float("nan")
            cache[int(table[r, n // page]), 1, :, n % page:] = float("inf")
    k = page // 16
    pieces = cache.view(cache.shape[0], 2, nkv, k, 16, d).permute(0, 3, 1, 2, 4, 5).reshape(-1, 2, nkv, 16, d).contiguous()
    small = (table[:, :, None] * k + torch.arange(k, device=DEV, dtype=torch.int32)).reshape(rows, -1).contiguous()
    scratch = torch.full((max(o.decode_scratch_floats(rows, nq, d, splits), 1),), float("nan"), device=DEV)
    got, other, want = torch.zeros_like(q), torch.zeros_like(q), torch.zeros_like(q)
    args = dict(window=window, stages=stages, keep_first=keep)
    o.attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, **args)
    o.attention_decode(q, pieces, small, seq_t, other, scratch, splits, nq, nkv, d, 16, d ** -0.5, **args)
    ref.attention_decode(q, cache, table, seq_t, want, None, splits, nq, nkv, d, page, d ** -0.5, window, keep_first=keep)
    assert o.attention_tc_status() == 0
    if window is None:
        assert torch.equal(got, other)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    if keep:
        return
    # from the projection: the block with the new position puts its key and value into the tile
    g = torch.Generator(device=DEV).manual_seed(23)
    qkv = torch.randn(2, rows, (nq + 2 * nkv) * d, device=DEV, generator=g)
    cos, sin = torch.rand(1100, d // 2, device=DEV, generator=g), torch.rand(1100, d // 2, device=DEV, generator=g)
    for r, n in enumerate(seqs):
        cache[int(table[r, (n - 1) // page]), :, :, (n - 1) % page] = float("nan")
    written = cache.clone()
    o.attention_decode_fused(qkv, None, None, 1e-6, cos, sin, written, table, seq_t, got, scratch, splits, nq, nkv, d, d, page, d ** -0.5,
                             window, stages=stages)
    ref.attention_decode_fused(qkv, None, None, 1e-6, cos, sin, cache, table, seq_t, want, None, splits, nq, nkv, d, d, page, d ** -0.5, window)
    assert o.attention_tc_status() == 0
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    for r, n in enumerate(seqs):
        at = int(table[r, (n - 1) // page])
        torch.testing.assert_close(written[at, :, :, (n - 1) % page].float(), cache[at, :, :, (n - 1) % page].float(), **tol(dtype))


@pytest.mark.parametrize("splits,stages", [(1, 0), (3, 0), (40, 0), (1, 3)])
@pytest.mark.parametrize("from_projection", [False, True])
def test_a_wait_for_a_tile_that_runs_out_is_reported(monkeypatch, from_projection, splits, stages):
    """With no poll allowed every block gives its wait up while its copies are on their way: it waits for them, says so and leaves NaN, the
    next call is as if nothing had been."""
    o, nq, nkv, d, page = ops(), 16, 4, 128, 64
    seqs = [1, 64, 129, 700, 2000]
    cache, table, q, _, _ = _attention_case(torch.bfloat16, nq, nkv, d, page, [n - 1 for n in seqs], [1] * len(seqs), None, seed=3)
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    qkv = torch.randn(1, len(seqs), (nq + 2 * nkv) * d, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4))
    scratch = torch.empty(max(o.decode_scratch_floats(len(seqs), nq, d, splits), 1), device=DEV)

    def run():
        out = torch.zeros_like(q)
        if from_projection:
            o.attention_decode_fused(qkv, None, None, 1e-6, None, None, cache, table, seq_t, out, scratch, splits, nq, nkv, d, 0, page, d ** -0.5,
                                     stages=stages)
        else:
            o.attention_decode(q, cache, table, seq_t, out, scratch, splits, nq, nkv, d, page, d ** -0.5, stages=stages)
        torch.cuda.synchronize()
        return out
    want = run()
    assert o.attention_decode_lost() == 0 and torch.isfinite(want).all()
    monkeypatch.setattr(o, "DECODE_POLLS", 0)
    assert torch.isnan(run()).all()
    assert 1 <= o.attention_decode_lost() <= len(seqs) and o.attention_decode_lost() == 0
    monkeypatch.undo()
    assert torch.equal(run(), want) and o.attention_tc_status() == 0


def test_three_stages_are_refused_where_they_do_not_fit():
    o = ops()
    nq, nkv, d, page = 2, 2, 256, 16
    cache, table, q, cu, pre = _attention_case(torch.bfloat16, nq, nkv, d, page, [99], [1], None, seed=3)
    seq_t = torch.tensor([100], device=DEV, dtype=torch.int32)
    with pytest.raises(Exception, match="stages"):
        o.attention_decode(q, cache, table, seq_t, torch.zeros_like(q), None, 1, nq, nkv, d, page, d ** -0.5, stages=3)
    cache, table, q, cu, pre = _attention_case(torch.float32, 4, 2, 16, 16, [99], [1], None, seed=3)
    with pytest.raises(Exception, match="stages"):
        o.attention_decode(q, cache, table, seq_t, torch.zeros_like(q), None, 1, 4, 2, 16, 16, 0.25, stages=3)


@pytest.mark.parametrize("requests,longest", [(1, 40000), (2, 30000), (4, 20000)])
def test_attention_decode_of_a_few_long_rows(requests, longest):
    """A few rows of tens of thousands of keys: the plan leaves the clusters (16 blocks a row at most) for one full
    wave of ranges through scratch and the combine kernel, from the qkv product as the engine would run it; one far
    key among them carries the row (its key is the query scaled up)."""
    o = ops()
    dtype, nq, nkv, d, page = torch.bfloat16, 32, 8, 128, 64
    plan = o.plan_decode_attention(dtype, requests, nq, nkv, d, longest)
    assert plan.arm == "wave" and plan.splits > 16 // requests + 8 and plan.fused and plan.scratch_floats > 0
    seqs = [longest - 1777 * i for i in range(requests)]
    cache, table, _, cu, pre = _attention_case(dtype, nq, nkv, d, page, [n - 1 for n in seqs], [1] * requests, None, seed=10)
    g = torch.Generator(device=DEV).manual_seed(92)
    qkv = torch.randn(3, requests, (nq + 2 * nkv) * d, device=DEV, generator=g) * 0.6
    far = 12345                                                     # a position in the middle of some range
    q_sum = qkv.sum(0)
    for r in range(requests):
        pg, off = int(table[r, far // page]), far % page
        for h in range(nkv):
            cache[pg, 0, h, off] = (q_sum[r].view(nq + 2 * nkv, d)[h * (nq // nkv)] * 3).to(dtype)
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    scratch = torch.full((plan.scratch_floats,), float("nan"), device=DEV)
    got, want = (torch.zeros(requests, nq * d, device=DEV, dtype=dtype) for _ in range(2))
    one, two = cache.clone(), cache.clone()
    o.attention_decode_fused(qkv, None, None, 1e-6, None, None, one, table, seq_t, got, scratch, plan.splits, nq, nkv, d, 0,
                             page, d ** -0.5)
    ref.attention_decode_fused(qkv, None, None, 1e-6, None, None, two, table, seq_t, want, None, plan.splits, nq, nkv, d, 0,
                                page, d ** -0.5)
    torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
    torch.testing.assert_close(one.float(), two.float(), atol=2 ** -7, rtol=2 ** -7)
    # the far key matters: without it the heads that look at it give another result
    cache2 = cache.clone()
    for r in range(requests):
        cache2[int(table[r, far // page]), 0, :, far % page] = 0
    other = torch.zeros_like(got)
    o.attention_decode_fused(qkv, None, None, 1e-6, None, None, cache2, table, seq_t, other, scratch, plan.splits, nq, nkv, d, 0,
                             page, d ** -0.5)
    assert float((other.float() - got.float()).abs().max()) > 0.05


@pytest.mark.parametrize("planes", [1, 3])
@pytest.mark.parametrize("splits", [1, 4, 6, 12])
@pytest.mark.parametrize("nq,nkv,d,page,window,rd,gains", [
    (32, 8, 128, 64, None, 128, True), (8, 2, 64, 16, None, 64, False), (40, 2, 64, 16, 70, 32, True),
    (6, 2, 192, 32, None, 0, True), (2, 2, 256, 16, 100, 256, False), (5, 1, 128, 8, None, 128, True)])
def test_attention_decode_from_the_projection(planes, splits, nq, nkv, d, page, window, rd, gains):
    """One kernel from the qkv product to the attention output (bfloat16, tensor-core head sizes) against the two
    kernels it replaces: the same output and the same cache afterwards, with per-head gains or without, full,
    partial or no rotation, a window, the product as bfloat16 or as float32 partial sums, and sequence lengths whose
    new position opens a page, ends one, or is the only one.  (Up to a last bit of bfloat16: the two sum a head's
    squares in different orders.)"""
    o = ops()
    dtype = torch.bfloat16
    seqs = [1, 8, 65, 500, 1000, 3, 257, 64, 129]
    prefixes, news = [n - 1 for n in seqs], [1] * len(seqs)
    cache, table, _, cu, pre = _attention_case(dtype, nq, nkv, d, page, prefixes, news, window, seed=8)
    g = torch.Generator(device=DEV).manual_seed(81)
    n, width = len(seqs), (nq + 2 * nkv) * d
    qkv = torch.randn(planes, n, width, device=DEV, generator=g) * 0.7 if planes > 1 else \
        torch.randn(n, width, device=DEV, generator=g).to(dtype)
    qg = (1 + 0.1 * torch.randn(d, device=DEV, generator=g)).to(dtype) if gains else None
    kg = (1 + 0.1 * torch.randn(d, device=DEV, generator=g)).to(dtype) if gains else None
    cos = torch.rand(1100, rd // 2, device=DEV, generator=g) if rd else None
    sin = torch.rand(1100, rd // 2, device=DEV, generator=g) if rd else None
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    pos = seq_t - 1
    req = torch.arange(n, device=DEV, dtype=torch.int32)
    scratch = torch.full((max(o.decode_scratch_floats(n, nq, d, splits), 1),), float("nan"), device=DEV)
    two, one = cache.clone(), cache.clone()
    q = o.qk_norm_rope_write(qkv, qg, kg, 1e-6, cos, sin, pos, req, table, two, nq, nkv, d, rd, page)
    want = torch.zeros(n, nq * d, device=DEV, dtype=dtype)
    o.attention_decode(q, two, table, seq_t, want, scratch, splits, nq, nkv, d, page, d ** -0.5, window)
    got = torch.zeros_like(want)
    o.attention_decode_fused(qkv, qg, kg, 1e-6, cos, sin, one, table, seq_t, got, scratch, splits, nq, nkv, d, rd, page,
                             d ** -0.5, window)
    last_bit = dict(atol=2 ** -7, rtol=2 ** -7)
    torch.testing.assert_close(one.float(), two.float(), **last_bit, msg="the cache after the step")
    assert float((one.float() - two.float()).abs().gt(0).float().mean()) < 1e-3        # and nearly everywhere the same bits
    torch.testing.assert_close(got.float(), want.float(), **last_bit)
    # and against the plain statement of the fused step itself (float32 inside, rounded once)
    plain_cache, plain_out = cache.clone(), torch.zeros_like(want)
    ref.attention_decode_fused(qkv, qg, kg, 1e-6, cos, sin, plain_cache, table, seq_t, plain_out, None, splits, nq, nkv, d, rd,
                                page, d ** -0.5, window)
    torch.testing.assert_close(one.float(), plain_cache.float(), **last_bit, msg="the cache against the plain statement")
    torch.testing.assert_close(got.float(), plain_out.float(), atol=2e-2, rtol=2e-2)
    # a layer that reads another layer's cache: nothing is written
    kept = two.clone()
    o.attention_decode_fused(qkv * 0.5 if planes > 1 else qkv, qg, kg, 1e-6, cos, sin, kept, table, seq_t, got, scratch, splits,
                             nq, nkv, d, rd, page, d ** -0.5, window, write_kv=False)
    assert torch.equal(kept, two)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,page", [(4, 2, 16, 16), (8, 2, 128, 64), (6, 2, 48, 8)])
def test_attention_window_edge_and_page_edge(dtype, nq, nkv, d, page):
    """A key that dominates every score, placed first just inside and then just outside the window
    of the last query (and on the last slot of a page): inside it owns the output, outside it must
    not be seen at all.  Prefill and decode kernels, same cache."""
    o = ops()
    window, seq = 2 * page + 3, 5 * page + 2
    g = torch.Generator(device=DEV).manual_seed(15)
    width = -(-seq // page)
    table = (torch.randperm(width, device=DEV, generator=g) + 1).view(1, width).to(torch.int32)
    q = torch.randn(1, nq * d, device=DEV, generator=g).to(dtype)
    qpos = seq - 1
    for key_pos, inside in ((qpos - window + 1, True), (qpos - window, False), (3 * page - 1, True)):
        cache = (torch.randn(width + 1, 2, nkv, page, d, device=DEV, generator=g) * 0.1).to(dtype)
        pg, off = int(table[0, key_pos // page]), key_pos % page
        for h in range(nkv):
            cache[pg, 0, h, off] = (q.view(nq, d)[h * (nq // nkv)].float() * 8).to(dtype)
            cache[pg, 1, h, off] = 7.0
        for decode in (True, False):
            got, want = torch.zeros_like(q), torch.zeros_like(q)
            seq_t = torch.tensor([seq], device=DEV, dtype=torch.int32)
            if decode:
                scratch = torch.empty(max(1, o.decode_scratch_floats(1, nq, d, 2)), device=DEV)
                o.attention_decode(q, cache, table, seq_t, got, scratch, 2, nq, nkv, d, page, d ** -0.5, window)
                ref.attention_decode(q, cache, table, seq_t, want, None, 2, nq, nkv, d, page, d ** -0.5, window)
            else:
                cu = torch.tensor([0, 1], device=DEV, dtype=torch.int32)
                pre = torch.tensor([seq - 1], device=DEV, dtype=torch.int32)
                z = torch.zeros(1, device=DEV, dtype=torch.int32)
                o.attention_prefill(q, cache, table, cu, pre, z, z, got, nq, nkv, d, page, d ** -0.5, window)
                ref.attention_prefill(q, cache, table, cu, pre, z, z, want, nq, nkv, d, page, d ** -0.5, window)
            torch.testing.assert_close(got.float(), want.float(), **tol(dtype))
            first_head = got.view(nq, d)[0].float()
            if inside:
                assert float((first_head - 7.0).abs().max()) < 0.5, (key_pos, decode)
            else:
                assert float(first_head.abs().max()) < 1.0, (key_pos, decode)


def test_attention_refuses_what_it_cannot_do():
    o = ops()
    q = torch.zeros(1, 2 * 704, device=DEV)                     # the CUDA-core kernel takes head sizes up to 640
    cache = torch.zeros(2, 2, 2, 16, 704, device=DEV)
    table = torch.ones(1, 1, device=DEV, dtype=torch.int32)
    seq = torch.ones(1, device=DEV, dtype=torch.int32)
    with pytest.raises(o.KernelError, match="head_dim"):
        o.attention_decode(q, cache, table, seq, torch.zeros_like(q), None, 1, 2, 2, 704, 16, 1.0)
    with pytest.raises(o.KernelError, match="CUDA"):
        o.silu_mul(torch.zeros(2, 4))


@pytest.mark.parametrize("vocab", [256, 331, 1009, 151936])
def test_argmax_and_penalties(vocab):
    g = torch.Generator(device=DEV).manual_seed(8)
    logits = torch.randn(5, vocab, device=DEV, generator=g)
    logits[2, vocab - 1] = 50.0
    logits[3, 7] = logits[3, 100] = 40.0                         # a tie goes to the lower index
    got = ops().argmax(logits)
    assert got.tolist() == torch.argmax(logits, -1).tolist() and got[3] == 7 and got[2] == vocab - 1
    rows = torch.tensor([0, 0, 1, 4], device=DEV, dtype=torch.int32)
    toks = torch.tensor([3, 9, 3, vocab - 1], device=DEV, dtype=torch.int32)
    cnt = torch.tensor([2, 0, 1, 5], device=DEV, dtype=torch.int32)
    bias = torch.tensor([0.0, 1.5, -2.0, 0.0], device=DEV)
    rep = torch.tensor([1.3, 1.0, 1.0, 1.0, 2.0], device=DEV)
    freq = torch.tensor([0.1, 0.2, 0.0, 0.0, 0.05], device=DEV)
    pres = torch.tensor([0.5, 0.0, 0.0, 0.0, 0.25], device=DEV)
    a, b = logits.clone(), logits.clone()
    ops().apply_penalties(a, rows, toks, cnt, bias, rep, freq, pres)
    ref.apply_penalties(b, rows, toks, cnt, bias, rep, freq, pres)
    torch.testing.assert_close(a, b, atol=1e-6, rtol=1e-6)


@pytest.mark.parametrize("vocab", [256, 1009, 151936])
def test_top_logprobs(vocab):
    g = torch.Generator(device=DEV).manual_seed(23)
    logits = torch.randn(5, vocab, device=DEV, generator=g) * 3
    logits[1, 7] = logits[1, 11] = float(logits[1].max()) + 1.0          # a tie at the top
    ks = [0, 2, 5, 20, 64]
    tokens, lps, counts = ops().top_logprobs(logits, torch.tensor(ks, device=DEV, dtype=torch.int32))
    want = torch.log_softmax(logits.double(), -1)
    for r, k in enumerate(ks):
        n = int(counts[r])
        if k == 0:
            assert n == 0
            continue
        assert k <= n <= ops().top_logprobs_cap()
        got = sorted(zip(tokens[r, :n].tolist(), lps[r, :n].tolist()), key=lambda tv: (-tv[1], tv[0]))[:k]
        top = torch.topk(want[r], k)
        assert sorted(t for t, _ in got) == sorted(top.indices.tolist())
        for t, v in got:
            assert abs(v - float(want[r, t])) < 1e-4
    rt, rl, rc = ref.top_logprobs(logits, torch.tensor(ks, device=DEV, dtype=torch.int32))
    assert rc.tolist() == counts.tolist()


@pytest.mark.parametrize("vocab,copies", [(256, 1), (1009, 1), (151936, 1), (151936, 4)])
def test_sample_matches_filtered_distribution(vocab, copies):
    """(Four copies of the cases at the large vocabulary: more blocks than the device holds at once, which the
    launcher gives half the threads each.)"""
    import plain_impl

    g = torch.Generator(device=DEV).manual_seed(9)
    cases = [(0.7, -1, 1.0, 0.0), (1.0, 5, 1.0, 0.0), (1.3, -1, 0.6, 0.0), (0.9, 50, 0.8, 0.05), (1.0, -1, 1.0, 0.2),
             (0.0, -1, 1.0, 0.0), (1.0, 1, 1.0, 0.0), (2.0, -1, 0.05, 0.0)] * copies
    rows = len(cases)
    logits = torch.randn(rows, vocab, device=DEV, generator=g) * 3
    t = torch.tensor([c[0] for c in cases], device=DEV)
    k = torch.tensor([c[1] for c in cases], device=DEV, dtype=torch.int32)
    p = torch.tensor([c[2] for c in cases], device=DEV)
    mp = torch.tensor([c[3] for c in cases], device=DEV)
    for u_val in (0.0, 0.123, 0.5, 0.77, 0.999999):
        u = torch.full((rows,), u_val, device=DEV)
        toks, lps = ops().sample(logits, t, k, p, mp, u, want_logprob=True)
        for r, (temp, kk, pp, mm) in enumerate(cases):
            tok = int(toks[r])
            if temp == 0 or kk == 1:
                assert tok == int(torch.argmax(logits[r]))
                assert abs(float(lps[r]) - float(torch.log_softmax(logits[r], -1)[tok])) < 1e-4
                continue
            probs = plain_impl.filtered_probs(logits[r].cpu(), temp, kk, pp, mm).double()
            assert probs[tok] > 0, (r, tok)
            cum = torch.cumsum(probs, 0)
            lo, hi = float(cum[tok] - probs[tok]), float(cum[tok])
            assert lo - 1e-5 <= u_val < hi + 1e-5, (r, u_val, lo, hi)      # the drawn token's interval holds u
            assert abs(float(lps[r]) - float(torch.log(probs[tok]))) < 1e-3


def test_sample_frequencies():
    # chi-square of many draws against the softmax, as the reference tests its sampler
    # (tests/test_engine.py:157-184 there): 12 tokens, temperature 1, 40000 draws.
    g = torch.Generator(device=DEV).manual_seed(10)
    vocab, draws = 12, 40000
    row = torch.randn(vocab, device=DEV, generator=g)
    logits = row.repeat(draws, 1).contiguous()
    u = torch.rand(draws, device=DEV, generator=g)
    ones = torch.ones(draws, device=DEV)
    toks, _ = ops().sample(logits, ones, torch.full((draws,), -1, device=DEV, dtype=torch.int32), ones,
                           torch.zeros(draws, device=DEV), u)
    counts = torch.bincount(toks.long(), minlength=vocab).double().cpu()
    expect = torch.softmax(row.double().cpu(), 0) * draws
    chi2 = float(((counts - expect) ** 2 / expect).sum())
    assert chi2 < 31.26                                         # df = 11, p = 0.001


@pytest.mark.parametrize("n,k", [(16, 2048), (17, 2052), (2400, 4100), (5, 260), (4750, 516), (130, 32), (70, 64), (513, 132), (2048, 2304)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 8, 9, 200, 257])
def test_gemm_fp32_rows_and_tiles_give_the_same_bits(m, n, k):
    """Both kernels of the float32 product sum in the same order: a row is the same bits alone, in a few rows and in
    many, with a last tile, run or stage that is not whole; one that is not on 16 bytes goes element by element."""
    g = torch.Generator(device=DEV).manual_seed(m * 31 + n + k)
    x, w = torch.randn(m, k, device=DEV, generator=g), torch.randn(n, k, device=DEV, generator=g)
    got = ops().linear(x, w)
    want = x.double() @ w.double().t()
    # sqrt(k) * 2^-24 of products near one, and as much for the largest of m * n
    assert float((got - want).abs().max()) < 4e-6 * (k ** 0.5) * 4
    assert torch.equal(ops().linear(x[-1:].contiguous(), w), got[-1:])
    many = torch.cat([x, torch.zeros(1500, k, device=DEV)])
    assert torch.equal(ops().linear(many, w)[:m], got)
    off = torch.empty(n * k + 1, device=DEV)[1:].view(n, k).copy_(w)
    assert torch.equal(ops().linear(x, off), got)


@pytest.mark.parametrize("nq,nkv,d,dv,page,window,in_keys", [
    (8, 2, 30, 30, 16, None, False), (12, 2, 64, 36, 16, 40, False), (4, 1, 640, 512, 16, None, True), (5, 1, 320, 320, 8, None, False),
    (18, 2, 20, 22, 16, 300, False)])
def test_attention_fp32_wide_and_element_by_element(nq, nkv, d, dv, page, window, in_keys):
    """float32 attention where the tiles come in pieces of 16 bytes (two buffers, or one where two do not fit) and where
    a head size is no multiple of four; more and fewer query heads a kv head than a block has warps."""
    seqs, prefixes, news = [1, 31, 32, 33, 257], [0, 30, 5, 0, 200], [1, 2, 33, 65, 31]
    g = torch.Generator(device=DEV).manual_seed(d + dv)
    width = max(-(-s // page) for s in seqs + [p + n for p, n in zip(prefixes, news)])
    row = nkv * (d if in_keys else d + dv)
    cache = torch.randn(len(seqs) * width + 1, page * row, device=DEV, generator=g)
    table = (torch.randperm(len(seqs) * width, device=DEV, generator=g) + 1).view(len(seqs), width).to(torch.int32)
    opts = dict(dv=dv, values_in_keys=in_keys)
    for decode in (True, False):
        n = len(seqs) if decode else sum(news)
        q = torch.randn(n, nq * d, device=DEV, generator=g)
        got, want = torch.zeros(n, nq * dv, device=DEV), torch.zeros(n, nq * dv, device=DEV)
        if decode:
            seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
            ref.attention_decode(q, cache, table, seq_t, want, None, 1, nq, nkv, d, page, d ** -0.5, window, **opts)
            for splits in (1, 3):
                scratch = torch.full((max(ops().decode_scratch_floats(n, nq, dv, splits), 1),), float("nan"), device=DEV)
                ops().attention_decode(q, cache, table, seq_t, got.zero_(), scratch, splits, nq, nkv, d, page, d ** -0.5, window, **opts)
                torch.testing.assert_close(got, want, **tol(torch.float32))
        else:
            cu = torch.tensor([0] + list(torch.tensor(news).cumsum(0)), device=DEV, dtype=torch.int32)
            pre = torch.tensor(prefixes, device=DEV, dtype=torch.int32)
            tiles = _tiles_of(news, ops().prefill_tile_rows(torch.float32, d))
            ref.attention_prefill(q, cache, table, cu, pre, *tiles, want, nq, nkv, d, page, d ** -0.5, window, **opts)
            ops().attention_prefill(q, cache, table, cu, pre, *tiles, got, nq, nkv, d, page, d ** -0.5, window, **opts)
            torch.testing.assert_close(got, want, **tol(torch.float32))


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("window,keep,cap,sinks", [(None, 0, None, False), (70, 0, 30.0, False), (70, 9, None, False), (None, 0, None, True)])
@pytest.mark.parametrize("nq,nkv,d,dv,page", [(2, 2, 4, 8, 16), (4, 2, 132, 128, 16), (9, 3, 128, 64, 64), (14, 2, 128, 128, 8), (16, 2, 256, 252, 16),
                                              (7, 1, 100, 100, 1)])
def test_attention_decode_fp32_keys_over_warps(nq, nkv, d, dv, page, window, keep, cap, sinks, splits):
    """float32 decode rows whose keys are cut over warps: fewer query heads than the kernel's one, two, four or eight, one piece of
    128 columns and two, rows that end inside a warp's four keys and inside a round of all warps, ranges without keys, the
    window's and the kept positions, a sink a head, a row so far ahead that its weight is all there is."""
    seqs = [1, 2, 5, 31, 33, 64, 65, 257]
    g = torch.Generator(device=DEV).manual_seed(d + dv + splits)
    width = max(-(-s // page) for s in seqs)
    cache = torch.randn(len(seqs) * width + 1, page * nkv * (d + dv), device=DEV, generator=g)
    cache[0] = float("nan")                                    # a page that no row owns
    table = (torch.randperm(len(seqs) * width, device=DEV, generator=g) + 1).view(len(seqs), width).to(torch.int32)
    q = torch.randn(len(seqs), nq * d, device=DEV, generator=g)
    q[3] *= 40.0
    opts = dict(dv=dv, keep_first=keep, softcap=cap)
    if sinks:
        opts["sinks"] = torch.randn(nq, device=DEV, generator=g) * 3.0
    seq_t = torch.tensor(seqs, device=DEV, dtype=torch.int32)
    got, want = (torch.zeros(len(seqs), nq * dv, device=DEV) for _ in range(2))
    scratch = torch.full((max(ops().decode_scratch_floats(len(seqs), nq, dv, splits), 1),), float("nan"), device=DEV)
    ref.attention_decode(q, cache, table, seq_t, want, None, 1, nq, nkv, d, page, d ** -0.5, window, **opts)
    ops().attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, window, **opts)
    torch.testing.assert_close(got, want, **tol(torch.float32))


def _nan_keys_case(dtype, nq, nkv, d, page, seqs_places):
    """A row for each (length, place of a key that is NaN in one column for the first kv head; None: no such key)."""
    g = torch.Generator(device=DEV).manual_seed(d + len(seqs_places))
    rows = len(seqs_places)
    width = max(-(-n // page) for n, _ in seqs_places)
    cache = torch.randn(rows * width + 1, 2, nkv, page, d, device=DEV, generator=g).to(dtype)
    table = (torch.randperm(rows * width, device=DEV, generator=g) + 1).view(rows, width).to(torch.int32)
    for r, (_, place) in enumerate(seqs_places):
        if place is not None:
            cache[int(table[r, place // page]), 0, 0, place % page, 3] = float("nan")
    q = torch.randn(rows, nq * d, device=DEV, generator=g).to(dtype)
    return cache, table, q, torch.tensor([n for n, _ in seqs_places], device=DEV, dtype=torch.int32)


def _nan_keys_reach_their_rows(dtype, nq, nkv, d, page, splits, seqs, **opts):
    cases = [(n, p) for n in seqs for p in sorted({None, 0, 4, 64, n - 1}, key=str) if p is None or p < n]
    cache, table, q, seq_t = _nan_keys_case(dtype, nq, nkv, d, page, cases)
    got, want = torch.zeros_like(q), torch.zeros_like(q)
    scratch = torch.full((max(ops().decode_scratch_floats(len(cases), nq, d, splits), 1),), float("nan"), device=DEV)
    ref.attention_decode(q, cache, table, seq_t, want, None, 1, nq, nkv, d, page, d ** -0.5, **opts)
    ops().attention_decode(q, cache, table, seq_t, got, scratch, splits, nq, nkv, d, page, d ** -0.5, **opts)
    first = nq // nkv * d                                      # the columns of the first kv head's query heads
    for r, (n, place) in enumerate(cases):
        assert bool(torch.isnan(got[r, :first]).all()) == (place is not None) and torch.isfinite(got[r, first:]).all(), (n, place)
    torch.testing.assert_close(got.float(), want.float(), equal_nan=True, **tol(dtype))


@pytest.mark.parametrize("splits", [1, 3, 9, 40])
@pytest.mark.parametrize("nq,nkv,d,cap", [(2, 2, 128, None), (6, 2, 64, None), (8, 2, 128, 30.0), (16, 2, 128, None), (4, 2, 256, None)])
def test_attention_decode_fp32_a_nan_key_reaches_its_row(nq, nkv, d, cap, splits):
    """A key that is seen and whose score is a NaN makes the row one, wherever it lies: alone among its warp's four keys, in the first round of a
    warp and in later ones, alone in its range; ranges merged by the combine kernel's plain loops and its staged ones."""
    _nan_keys_reach_their_rows(torch.float32, nq, nkv, d, 16, splits, [1, 2, 5, 13, 65, 129, 257], softcap=cap)


@pytest.mark.parametrize("splits,stages", [(1, 0), (3, 0), (9, 0), (40, 0), (1, 3), (2, 3)])
@pytest.mark.parametrize("nq,nkv,d,page", [(16, 4, 128, 16), (16, 4, 128, 64), (16, 8, 64, 128), (40, 2, 128, 64)])
def test_attention_decode_bf16_a_nan_key_reaches_its_row(nq, nkv, d, page, splits, stages):
    """The same on tensor cores, where a warp has 16 keys of every tile: ranges that end with one key, merged in the block, in clusters and by the
    combine kernel; tiles piece by piece and by TMA."""
    _nan_keys_reach_their_rows(torch.bfloat16, nq, nkv, d, page, splits, [1, 2, 65, 129, 193, 385], stages=stages)


@pytest.mark.parametrize("tokens", [1, 2, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("width,ff,experts,identity,top,activation,on_input,shared", [
    (64, 64, 3, 0, 2, "silu", False, False), (192, 320, 16, 2, 4, "swish_clamped", False, False),
    (2048, 2048, 16, 0, 3, "relu2", False, True), (128, 192, 40, 0, 8, "silu", True, True), (256, 64, 2, 6, 7, "swish_clamped", False, True),
    (64, 128, 256, 0, 8, "relu2", True, False), (1216, 512, 64, 0, 8, "silu", False, False), (1856, 2048, 12, 0, 8, "silu", False, False)])
def test_experts_of_a_few_tokens(tokens, width, ff, experts, identity, top, activation, on_input, shared):
    """The kernels that stream the chosen experts' weights (up to 16 tokens and 128 pairs; beyond, the grouped products): odd
    numbers of tokens, experts nobody chose, steps of identity choices alone, fewer tiles of k than warps."""
    g = torch.Generator(device=DEV).manual_seed(tokens * 7 + width)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    bf = torch.bfloat16
    h = rand(tokens, width).to(bf)
    router = rand(experts + identity + (1 if shared else 0), width) * 0.5
    gu = (rand(experts, (1 if activation == "relu2" else 2) * ff, width) / width ** 0.5).to(bf)
    dn = (rand(experts, width, ff) / ff ** 0.5).to(bf)
    sh = rand(2, tokens, width) if shared else None
    r = ops().moe_route(h, router, None, top, experts, shared_gate=shared, outputs=experts + identity)
    got = ops().moe_experts(h, r, gu, dn, 7.0, 1.702, activation=activation, weight_on_input=on_input, shared=sh)
    plain = ref.ExpertRouting(r.chosen, r.weights, top, r.gate)
    want = ref.moe_experts(h, plain, gu, dn, 7.0, 1.702, activation=activation, weight_on_input=on_input, shared=sh)
    # the activations are rounded to 8 bits once here, 2^-9 of each of ff terms; the grouped products round their outputs too
    scale = float(want.abs().max())
    assert float((got - want).abs().max()) < 1.6e-2 * scale
    # a token's sum does not depend on its neighbours, bit for bit, while both take the same kernels
    few = lambda n: bool(ops().library().lily_moe_few_takes(n, top, experts, width, ff) and ops().library().lily_moe_few_pays(n, top, experts, width, ff))
    if few(tokens) and few(1):
        keep = slice(tokens - 1, tokens)
        alone = ops().moe_route(h[keep], router, None, top, experts, shared_gate=shared, outputs=experts + identity)
        assert torch.equal(alone.chosen, r.chosen[keep])
        one = ops().moe_experts(h[keep].contiguous(), alone, gu, dn, 7.0, 1.702, activation=activation, weight_on_input=on_input,
                                shared=sh[:, keep].contiguous() if shared else None)
        assert torch.equal(one, got[keep])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("requests,heads,groups,pd,n_state", [
    (1, 2, 1, 64, 128), (9, 64, 8, 64, 128), (3, 6, 3, 24, 64), (2, 4, 2, 7, 20), (5, 8, 1, 33, 256), (2, 2, 2, 16, 300), (300, 2, 1, 80, 512),
    (4, 3, 1, 5, 17), (3, 2, 1, 9, 64), (3, 2, 1, 9, 68), (300, 4, 2, 70, 132), (2, 3, 1, 40, 260),
    (64, 2, 1, 64, 44), (65, 2, 1, 64, 44), (256, 4, 1, 64, 260), (257, 4, 1, 64, 260)])
def test_ssd_scan_of_one_token_a_request(dtype, requests, heads, groups, pd, n_state):
    """A decode step's scan: rows of a head that no warp fills, states of one to four pieces a lane, many and few requests; a state
    that is no multiple of four takes the general kernel."""
    g = torch.Generator(device=DEV).manual_seed(requests + pd)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    inner = heads * pd
    xbc, proj = rand(requests, inner + 2 * groups * n_state).to(dtype), rand(requests, 5 + heads).to(dtype)
    vec = [rand(heads) for _ in range(3)]
    state = rand(requests + 2, inner * n_state + 4 * (requests % 2))
    cu = torch.arange(requests + 1, device=DEV, dtype=torch.int32)
    slots = (torch.randperm(requests + 1, device=DEV, generator=g) + 1)[:requests].to(torch.int32)
    mine, theirs = state.clone(), state.clone()
    got = ops().ssd_scan(xbc, proj, 5, *vec, mine, cu, slots, requests, heads, pd, n_state, groups)
    want = ref.ssd_scan(xbc, proj, 5, *vec, theirs, cu, slots, requests, heads, pd, n_state, groups)
    # float32 throughout: n_state products a sum, 2^-24 each
    torch.testing.assert_close(got, want, rtol=2e-5, atol=2e-5 * n_state ** 0.5)
    torch.testing.assert_close(mine, theirs, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("requests,heads,d", [(1, 32, 64), (7, 3, 32), (40, 2, 128), (2, 5, 256), (3, 4, 48), (64, 8, 32), (65, 8, 32)])
def test_wkv_scan_of_one_token_a_request(dtype, requests, heads, d):
    g = torch.Generator(device=DEV).manual_seed(requests + d)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    r, k, v = (rand(requests, heads * d).to(dtype) for _ in range(3))
    lw, u = -torch.exp(rand(requests, heads * d)), rand(heads, d)
    state = rand(requests + 2, heads * d * d + 8)
    cu = torch.arange(requests + 1, device=DEV, dtype=torch.int32)
    slots = (torch.randperm(requests + 1, device=DEV, generator=g) + 1)[:requests].to(torch.int32)
    mine, theirs = state.clone(), state.clone()
    got = ops().wkv_scan(r, k, v, lw, u, mine, cu, slots, requests, heads, d)
    want = ref.wkv_scan(r, k, v, lw, u, theirs, cu, slots, requests, heads, d)
    torch.testing.assert_close(got, want, rtol=2e-5, atol=2e-5 * d ** 0.5)
    torch.testing.assert_close(mine, theirs, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rows,hidden", [(1, 1024), (3, 1056), (64, 2048), (65, 2048), (70, 516), (5, 1028), (66, 4100), (3, 8192), (9, 9000), (2, 1027)])
@pytest.mark.parametrize("planes,gains,bias,write", [((1, 17), 2, True, True), ((9, 0), 1, False, True), ((0, 0), 2, True, False), ((8, None), 0, False, True)])
def test_add_rmsnorm_multi_in_pieces(rows, hidden, planes, gains, bias, write):
    """Rows over a cluster, in a block's registers (whole and with a last piece that few threads have) and a number at a time; sums of one to
    seventeen planes (0: bfloat16, None: no such sum), outputs and stream as the plain statement."""
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    deltas = [None if n is None else (rand(n, rows, hidden) if n else rand(rows, hidden).bfloat16()) for n in planes]
    vectors, b = [rand(hidden) for _ in range(gains)], rand(hidden) if bias else None
    mine, theirs = rand(rows, hidden), None
    theirs, kept = mine.clone(), mine.clone()
    got = ops().add_rmsnorm_multi(mine, deltas, vectors, 1e-6, torch.bfloat16, b, write)
    want = ref.add_rmsnorm_multi(theirs, deltas, vectors, 1e-6, torch.bfloat16, b, write)
    assert len(got) == gains
    for x, y in zip(got, want):
        torch.testing.assert_close(x.float(), y.float(), rtol=1e-2, atol=1e-2)             # one rounding to bfloat16 apart
    torch.testing.assert_close(mine, theirs, rtol=1e-5, atol=1e-5)
    if not write:
        assert torch.equal(mine, kept)


@pytest.mark.parametrize("hidden", [1024, 1056, 1536, 2560, 3584, 3616])
@pytest.mark.parametrize("rows", [1, 9, 64])
def test_norms_of_a_few_rows_over_clusters(rows, hidden):
    """Rows over the eight blocks of a cluster whose shares end inside a warp, or do not: each sum is over the row's columns and nothing else, so a
    column too much or too few (1.4e-4 of every result at 3,616 columns) is beyond what is allowed for three roundings of 2^-24."""
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    unit = lambda x: x * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-6)
    resid, delta, gain = rand(rows, hidden), rand(3, rows, hidden), rand(hidden)
    mine = resid.clone()
    got = ops().add_rmsnorm(mine, delta, gain, 1e-6, torch.float32)
    total = resid.double() + delta.double().sum(0)
    torch.testing.assert_close(got.double(), unit(total) * gain, rtol=5e-5, atol=1e-5)
    torch.testing.assert_close(mine.double(), total, rtol=1e-5, atol=1e-5)
    a, b, f = rand(2, rows, hidden), rand(1, rows, hidden), rand(1, rows, hidden)
    got = ops().normed_mean([a, b], [gain, resid[0].contiguous()], 1e-6, add=f)
    want = (unit(a.double().sum(0)) * gain + unit(b[0].double()) * resid[0]) / 2 + f[0]
    torch.testing.assert_close(got.double().view(rows, hidden), want, rtol=5e-5, atol=1e-5)
    mine, bias = resid.clone(), rand(hidden)
    both = ops().add_rmsnorm_multi(mine, [delta, b], [gain, resid[0].contiguous()], 1e-6, torch.float32, bias, True)
    total = resid.double() + delta.double().sum(0) + b[0].double() + bias
    for got, vector in zip(both, (gain, resid[0])):
        torch.testing.assert_close(got.double(), unit(total) * vector, rtol=5e-5, atol=1e-5)
    torch.testing.assert_close(mine.double(), total, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("tokens,rank,cols", [(1, 1, 5), (2, 64, 2048), (8, 31, 130), (9, 33, 257), (21, 200, 128), (2364, 33, 128), (2371, 33, 130), (3, 130, 384),
                                              (4, 64, 64), (5, 65, 100), (1193, 64, 516), (2380, 5, 132)])
def test_wkv_decay_by_rows_asked_for_ahead(tokens, rank, cols):
    g = torch.Generator(device=DEV).manual_seed(rank)
    a, w2t, w0 = (torch.randn(*s, device=DEV, generator=g) for s in ((tokens, rank), (rank, cols), (cols,)))
    w2t = w2t / rank ** 0.5
    torch.testing.assert_close(ops().wkv_decay(a, w2t, w0), ref.wkv_decay(a, w2t, w0), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n,k", [(1, 64), (15, 128), (64, 448), (331, 512), (2048, 2048), (5000, 576), (10304, 192)])
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16])
def test_linear_of_a_few_rows(m, n, k):
    """bfloat16 products of up to 16 rows: tiles of rows and eighths of k that are not whole, fewer tiles of k than warps, several
    tiles a block; with and without a bias, both result types."""
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((m, k), (n, k)))
    b = torch.randn(n, device=DEV, generator=g)
    want = x.double() @ w.double().t()
    got = ops().linear(x, w, out_dtype=torch.float32)
    # float32 sums of exact products: 2^-24 of sqrt(k) terms near one, and the largest of m * n
    assert float((got - want).abs().max()) < 4e-6 * (k ** 0.5) * 4
    assert float((ops().linear(x, w, b, out_dtype=torch.float32) - (want + b)).abs().max()) < 4e-6 * (k ** 0.5) * 4
    assert torch.equal(ops().linear(x, w), got.bfloat16())
    low = ops().linear(x, w, b.bfloat16())
    assert float((low - (want + b.bfloat16())).abs().max()) < 2 ** -8 * float(want.abs().max() + 4)
    assert torch.equal(ops().linear(x[-1:].contiguous(), w), ops().linear(x, w)[-1:])


@pytest.mark.parametrize("m,n,k,here", [
    (8, 32, 25600, True), (8, 32, 25664, False), (8, 512, 25664, True), (8, 5120, 8192, True), (8, 5120, 8256, False), (9, 1024, 18944, True),
    (9, 1024, 19008, False), (9, 3072, 19008, True), (16, 5120, 4096, True), (16, 5120, 4160, False), (16, 40000, 1024, True), (16, 40000, 960, False),
    (16, 18944, 4160, False), (16, 18960, 4160, True), (16, 8192, 12288, True), (16, 8192, 12352, False), (16, 80000, 1984, False)])
def test_linear_of_a_few_rows_on_both_sides_of_its_line(m, n, k, here):
    """Where the kernel for few rows hands over to the library (with 148 SMs): the same numbers either way."""
    g = torch.Generator(device=DEV).manual_seed(n + k)
    x, w = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((m, k), (n, k)))
    assert ops().few_rows_take(x, w) == here or ops().sm_count() != 148
    want = x.double() @ w.double().t()
    # the tensor cores cut off what they add to an accumulator: k / 16 additions of 2^-23 of at most the largest sum
    assert float((ops().linear(x, w, out_dtype=torch.float32) - want).abs().max()) < k / 16 * 2 ** -23 * float(want.abs().max())
    assert float((ops().linear(x, w) - want).abs().max()) < 2 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.float16, torch.float64])
@pytest.mark.parametrize("m", [1, 9, 16, 17])
def test_linear_takes_a_bias_of_any_float_type(m, dtype):
    """Few rows and many: a bias that no kernel reads as it is gets converted first."""
    g = torch.Generator(device=DEV).manual_seed(m)
    x, w = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((m, 192), (40, 192)))
    b = torch.randn(40, device=DEV, generator=g).to(dtype)
    want = x.double() @ w.double().t() + b.double()
    assert float((ops().linear(x, w, b, out_dtype=torch.float32) - want).abs().max()) < 4e-6 * (192 ** 0.5) * 4
    low = ops().linear(x, w, b)                       # sum and bias are rounded to 8 bits, 2^-9 each
    assert low.dtype == torch.bfloat16 and float((low - want).abs().max()) < 2 ** -8 * float(want.abs().max() + 4)


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh", "swish_clamped"])
@pytest.mark.parametrize("m,inter,k,run", [(1, 8, 64, 8), (5, 72, 192, 24), (8, 3000, 576, 8), (3, 2432, 512, 128)])
def test_gate_up_of_a_few_rows(activation, m, inter, k, run):
    """Every activation in the product's epilogue, runs of all lengths, several tiles a block and fewer outputs than a tile's rows."""
    g = torch.Generator(device=DEV).manual_seed(m + k)
    x = torch.randn(m, k, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * inter, k, device=DEV, generator=g) * 2 * k ** -0.5).bfloat16()
    how = dict(limit=1.5, alpha=1.702) if activation == "swish_clamped" else {}
    need = ops().swiglu_skinny_need(m, inter, k, torch.bfloat16, run, whenever_possible=True)
    got = ops().swiglu_skinny(x, w, run, torch.zeros(need[0], device=DEV), torch.zeros(need[1], device=DEV, dtype=torch.int32),
                              activation=activation, **how)
    want = ref.silu_mul((x.double() @ w.double().t()).float(), torch.float32, block=run, activation=activation, **how)
    assert float((got.float() - want).abs().max()) < 2 ** -8 * float(want.abs().max())      # rounded once, to 8 bits


def test_linear_split_in_one_plane():
    """Where finished rows are the faster way the product comes as one float32 plane, the same numbers as its slices added up; at the
    edges of that rule (1.25 tiles a SM and two, K 4,096) it comes in slices on the other side."""
    g = torch.Generator(device=DEV).manual_seed(0)
    o, sms = ops(), ops().sm_count()
    for n, k, whole in ((20 * sms, 4160, True), (20 * sms - 16, 4160, False), (20 * sms - 16, 4096, True), (32 * sms, 512, True), (32 * sms + 1, 512, False)):
        assert o.few_rows_whole_pays(2, n, k) == whole
        x, w = torch.randn(2, k, device=DEV, generator=g).bfloat16(), torch.randn(n, k, device=DEV, generator=g).bfloat16()
        parts = o.linear_split(x, w)
        assert (parts is not None and parts.shape[0] == 1) == whole or o.library().lily_skinny_gemm_splits(2, n, k) <= 1
        if parts is not None:
            assert float((parts.sum(0) - x.double() @ w.double().t()).abs().max()) < 4e-6 * (k ** 0.5) * 4
    for m, n, k in ((2, 2048, 2048), (16, 4096, 12288), (8, 24, 64)):
        x, w = torch.randn(m, k, device=DEV, generator=g).bfloat16(), torch.randn(n, k, device=DEV, generator=g).bfloat16()
        one = ops().linear_split(x, w)
        assert tuple(one.shape) == (1, m, n) and one.dtype == torch.float32
        assert float((one[0] - x.double() @ w.double().t()).abs().max()) < 4e-6 * (k ** 0.5) * 4


@pytest.mark.parametrize("heads_per_block", [1, 2])
@pytest.mark.parametrize("nq,nkv,d,window,sink,planes", [(16, 4, 128, None, True, True), (4, 2, 64, None, False, True), (6, 3, 64, 100, True, True),
                                                         (8, 4, 128, None, True, False)])
def test_attention_prefill_tcgen05_sink_and_planes(nq, nkv, d, window, sink, planes, heads_per_block):
    """The sink's unit and the planes of values of every kv head on the tcgen05 kernel: one-row tiles, cached prefixes, rows whose
    scores all lie far below the sink's and rows with a key far above it."""
    o, page = ops(), 64
    prefixes, news = [0, 17, 130, 300], [1, 200, 129, 64]
    cache, table, q, cu, pre = _attention_case(torch.bfloat16, nq, nkv, d, page, prefixes, news, window, spike=True)
    q[5:40] = (q[5:40].float() * 6).bfloat16()
    rows = int(o.library().lily_attention_prefill_tc_rows())
    tiles = _tiles_of(news, rows)
    shape = (nkv, len(q), nq * d) if planes else (len(q), nq * d)
    got = torch.zeros(shape, device=DEV, dtype=torch.bfloat16)
    o.attention_prefill(q, cache, table, cu, pre, *tiles, got, nq, nkv, d, page, d ** -0.5, window, tile_rows=rows, sink=sink,
                        all_values=planes, heads_per_block=heads_per_block)
    assert o.attention_tc_status() == 0
    if planes:
        wide = torch.zeros(len(q), nq * nkv * d, device=DEV)
        ref.attention_prefill(q, cache, table, cu, pre, *tiles, wide, nq, nkv, d, page, d ** -0.5, window, sink=sink, all_values=True)
        wide = wide.view(len(q), nq, nkv, d)
        own = torch.arange(nq, device=DEV) // (nq // nkv)
        want = torch.stack([wide[:, torch.arange(nq, device=DEV), (own + z) % nkv] for z in range(nkv)]).reshape(shape)
    else:
        want = torch.zeros(shape, device=DEV)
        ref.attention_prefill(q, cache, table, cu, pre, *tiles, want, nq, nkv, d, page, d ** -0.5, window, sink=sink)
    torch.testing.assert_close(got.float(), want.float(), **tol(torch.bfloat16))


@pytest.mark.parametrize("nq,nkv,d,window,keep,cap,planes", [
    (4, 4, 128, None, 0, None, True), (3, 3, 64, None, 0, 20.0, False), (8, 2, 128, 90, 70, None, False), (4, 2, 64, 64, 3, 15.0, True),
    (6, 6, 128, 100, 130, 30.0, True)])
def test_sink_prompts_with_caps_kept_positions_and_single_heads(nq, nkv, d, window, keep, cap, planes):
    """A sink with a soft cap, with kept first positions beside a window, and one query head a kv head: the same from the tcgen05 and the
    mma.sync kernels' tiles, and as the plain statement."""
    o, page = ops(), 64
    prefixes, news = [0, 30, 200], [40, 129, 200]
    cache, table, q, cu, pre = _attention_case(torch.bfloat16, nq, nkv, d, page, prefixes, news, window, spike=True)
    shape = (nkv, len(q), nq * d) if planes else (len(q), nq * d)
    how = dict(sink=True, all_values=planes, softcap=cap, keep_first=keep)
    if planes:
        wide = torch.zeros(len(q), nq * nkv * d, device=DEV)
        ref.attention_prefill(q, cache, table, cu, pre, *_tiles_of(news, 32), wide, nq, nkv, d, page, d ** -0.5, window, **how)
        wide, heads = wide.view(len(q), nq, nkv, d), torch.arange(nq, device=DEV)
        want = torch.stack([wide[:, heads, (heads // (nq // nkv) + z) % nkv] for z in range(nkv)]).reshape(shape)
    else:
        want = torch.zeros(shape, device=DEV)
        ref.attention_prefill(q, cache, table, cu, pre, *_tiles_of(news, 32), want, nq, nkv, d, page, d ** -0.5, window, **how)
    for rows in (int(o.library().lily_attention_prefill_tc_rows()), int(o.library().lily_attention_prefill_mma_rows())):
        got = torch.zeros(shape, device=DEV, dtype=torch.bfloat16)
        o.attention_prefill(q, cache, table, cu, pre, *_tiles_of(news, rows), got, nq, nkv, d, page, d ** -0.5, window, tile_rows=rows, **how)
        assert o.attention_tc_status() == 0
        torch.testing.assert_close(got.float(), want.float(), **tol(torch.bfloat16))


def test_sink_prompts_take_the_tiles_they_fill():
    o = ops()
    rows = lambda d, news, heads, planes: o.prefill_tile_rows(torch.bfloat16, d, 64, sum(news), sink=True, all_values=planes, heads=heads, new_lens=news)
    for d, news, heads, planes, want in ((128, [128], 16, False, 128), (128, [127], 16, False, 64), (128, [16] * 16, 32, False, 64), (128, [16] * 16, 32, True, 64),
                                         (128, [64] * 2, 16, True, 128), (128, [300, 45, 211, 127, 512], 16, True, 128), (64, [300], 16, False, 64),
                                         (64, [400], 16, False, 128), (64, [16] * 8, 16, True, 64), (64, [256] * 4, 16, True, 128),
                                         (64, [300], 32, True, 128), (64, [300, 20], 32, True, 64)):
        assert rows(d, news, heads, planes) == want, (d, news, heads, planes)
    assert o.prefill_tile_rows(torch.bfloat16, 128, 64, 500, sink=True) == 128


@pytest.mark.parametrize("lens", [[17], [64, 5, 130], [128, 1, 257, 40], [16, 300]])
@pytest.mark.parametrize("heads,groups,pd,n_state", [(4, 2, 64, 128), (3, 1, 16, 16), (2, 1, 80, 48), (8, 4, 128, 64)])
def test_ssd_scan_in_chunks_on_the_tensor_cores(lens, heads, groups, pd, n_state):
    """bfloat16 portions as chunks of matrix products: chunks and tiles that are not whole, short portions beside long ones, heads of
    less and more than 64 columns, slow and fast decays (e^-30 a token) in one chunk; no further from 64 bits than token by token."""
    from lily_b200.csrc import ops as o
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + pd)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    n, inner = sum(lens), heads * pd
    xbc, proj = rand(n, inner + 2 * groups * n_state).bfloat16(), rand(n, 8 + heads).bfloat16()
    dt_bias, a_log, d_skip = rand(heads), torch.linspace(-5.0, 3.0, heads, device=DEV), rand(heads)
    state = rand(len(lens) + 1, inner * n_state)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=DEV, dtype=torch.int32)
    slots = torch.arange(len(lens), 0, -1, device=DEV, dtype=torch.int32)
    plan = o.scan_plan(lens, DEV, inner * n_state)
    assert plan.fine is not None and plan.fine.num_chunks
    errs = []
    x64, p64, s64 = xbc.double(), proj.double(), state.double()
    want = torch.empty(n, inner, device=DEV, dtype=torch.float64)
    per = heads // groups
    for r in range(len(lens)):
        s = s64[int(slots[r])].view(heads, pd, n_state)
        for t in range(int(cu[r]), int(cu[r + 1])):
            x = x64[t, :inner].view(heads, pd)
            b, c = (x64[t, inner + k * groups * n_state:inner + (k + 1) * groups * n_state].view(groups, n_state).repeat_interleave(per, 0) for k in (0, 1))
            dt = torch.nn.functional.softplus(p64[t, 4:4 + heads] + dt_bias.double())
            s.copy_(torch.exp(-torch.exp(a_log.double()) * dt)[:, None, None] * s + (dt[:, None] * x)[:, :, None] * b[:, None, :])
            want[t] = (torch.einsum("hpn,hn->hp", s, c) + d_skip.double()[:, None] * x).reshape(inner)
    for chunks in (False, True):
        o._SSD_CHUNKS = chunks
        try:
            mine = state.clone()
            got = o.ssd_scan(xbc, proj, 4, dt_bias, a_log, d_skip, mine, cu, slots, len(lens), heads, pd, n_state, groups, plan=plan)
        finally:
            o._SSD_CHUNKS = True
        errs.append((float((got.double() - want).norm() / want.norm()), float((mine.double() - s64)[1:].norm() / s64[1:].norm())))
        assert torch.equal(mine[0], state[0])
    # float32 sums either way: 2^-24 a product and term
    assert errs[1][0] < 2e-6 and errs[1][1] < 2e-6, errs
    assert errs[1][0] < errs[0][0] + 2e-8 and errs[1][1] < errs[0][1] + 2e-8, errs


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where,at", [("x", 3), ("x", 78), ("x", 150), ("B", 20), ("C", 21), ("dt", 37), ("state", 0)])
def test_ssd_chunks_keep_non_finite_numbers_where_they_are(bad, where, at):
    """A number that is not finite spoils its own column (value, state) and its own head from its token on, as it does token by
    token: bit for bit nothing in earlier tokens, other columns, other heads or the other request."""
    from lily_b200.csrc import ops as o
    lens, heads, pd, n_state = [170, 40], 3, 80, 32
    g = torch.Generator(device=DEV).manual_seed(at)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    n, inner = sum(lens), heads * pd
    xbc, proj, state = rand(n, inner + 2 * n_state).bfloat16(), rand(n, heads).bfloat16(), rand(3, inner * n_state)
    vec = [rand(heads), torch.tensor([-5.0, -2.0, -3.0], device=DEV), rand(heads)]
    cu, slots = torch.tensor([0, 170, 210], device=DEV, dtype=torch.int32), torch.tensor([2, 1], device=DEV, dtype=torch.int32)
    plan = o.scan_plan(lens, DEV, inner * n_state)

    def run(xbc, proj, state):
        state = state.clone()
        return o.ssd_scan(xbc, proj, 0, *vec, state, cu, slots, 2, heads, pd, n_state, 1, plan=plan).view(n, heads, pd), state[1:].view(2, heads, pd, n_state)

    y0, s0 = run(xbc, proj, state)
    assert bool(y0.isfinite().all()) and bool(s0.isfinite().all())
    xbc, proj, state = xbc.clone(), proj.clone(), state.clone()
    same, held = torch.ones(n, heads, pd, dtype=torch.bool, device=DEV), torch.ones_like(s0, dtype=torch.bool)
    if where == "x":
        xbc[at, pd + 70] = bad                            # head 1, value column 70
        same[at:170, 1, 70] = held[1, 1, 70] = False
    elif where == "B":
        xbc[at, inner + 5] = bad                          # state column 5 of every head
        same[at:170], held[1, :, :, 5] = False, False
    elif where == "C":
        xbc[at, inner + n_state + 5] = bad
        same[at] = False
    elif where == "dt":
        proj[at, 2] = bad
        if bad == float("-inf"):                          # a step of size zero
            assert bool(run(xbc, proj, state)[0].isfinite().all())
            return
        same[at:170, 2], held[1, 2] = False, False
    else:
        state[2].view(heads, pd, n_state)[0, 33, 7] = bad
        same[:170, 0, 33] = held[1, 0, 33, 7] = False
    y1, s1 = run(xbc, proj, state)
    assert torch.equal(y1[same], y0[same]) and torch.equal(s1[held], s0[held])
    if where != "dt":                                     # (behind an infinite step nothing of the state is left to be spoiled by)
        assert not bool(y1[~same].isfinite().any()) and not bool(s1[~held].isfinite().any())
    else:
        assert not bool(y1[at, 2].isfinite().any())


def test_ssd_chunks_where_a_decay_is_beyond_float32():
    """exp(a_log) dt past the largest float32: the state is forgotten at every token, and what the token brings is all there is."""
    from lily_b200.csrc import ops as o
    n, heads, pd, n_state = 140, 2, 64, 64
    g = torch.Generator(device=DEV).manual_seed(1)
    rand = lambda *s: torch.randn(*s, device=DEV, generator=g)
    xbc, proj, state = rand(n, heads * pd + 2 * n_state).bfloat16(), rand(n, heads).abs().bfloat16() + 8, rand(2, heads * pd * n_state)
    vec = [torch.zeros(heads, device=DEV), torch.tensor([88.0, 90.0], device=DEV), rand(heads)]
    cu, slots = torch.tensor([0, n], device=DEV, dtype=torch.int32), torch.ones(1, device=DEV, dtype=torch.int32)
    plan = o.scan_plan([n], DEV, heads * pd * n_state)
    got = o.ssd_scan(xbc, proj, 0, *vec, state, cu, slots, 1, heads, pd, n_state, 1, plan=plan).double()
    x, b, c = xbc.double().split([heads * pd, n_state, n_state], 1)
    dt = torch.nn.functional.softplus(proj.double())
    want = ((b * c).sum(1)[:, None] * dt + vec[2].double())[:, :, None] * x.view(n, heads, pd)
    assert float((got.view_as(want) - want).norm() / want.norm()) < 2e-6


def test_scan_plan_cuts_only_for_who_runs_it():
    """No tensor-core cut, lists on the device or workspace for a scan that will not use them: float32, sizes the kernels refuse, the selective
    scan, portions that are faster in one piece."""
    o = ops()
    floats, bf = 64 * 64 * 128, (torch.bfloat16, 64, 64, 128, 64 * 64 + 16 * 128)
    for chunks in (False, (torch.float32,) + bf[1:], (torch.bfloat16, 64, 64, 136, 64 * 64 + 16 * 136)):
        plan = o.scan_plan([190] * 64, DEV, floats, chunks=chunks)
        assert plan.fine is None and plan.direct is None and o.scan_workspace_floats(plan, 64, 64, 128) == 0
        plan = o.scan_plan([300] + [100] * 40, DEV, floats, chunks=chunks)
        assert plan.fine is None and plan.num_chunks == 3 and o.scan_workspace_floats(plan, 64, 64, 128) == 3 * (floats + 64)
    for lens, want in (([17], 0), ([24], 1), ([17] * 8, 0), ([32] * 8, 0), ([64] * 8, 8), ([1] * 16 + [17], 0), ([1] * 16 + [40], 1), ([33, 391], 5)):
        plan = o.scan_plan(lens, DEV, floats, chunks=bf)
        assert (plan.fine.num_chunks if plan.fine else 0) == want, lens
        assert o.scan_workspace_floats(plan, 64, 64, 128) == want * (floats + 64)
    # more chunks than a grid of the tensor-core kernels has room for
    assert o.scan_plan([150] * 16383, DEV, 256).fine.num_chunks == 32766 and o.scan_plan([150] * 16384, DEV, 256).fine is None
