"""Each CUDA kernel alone against its plain torch reference (tests/torch_kernels.py), at other sizes
than the engine's tiny models: widths that are no power of two, head sizes in steps of 16,
odd group sizes, pages of odd length."""

from __future__ import annotations

import random

import pytest
import torch

import torch_kernels as ref

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def _tol(dtype):
    return dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=2 ** -7, atol=2 ** -7)


def _randn(*shape, dtype, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [64, 100, 2048, 3000])
def test_embedding(dtype, width):
    from liteinfer_b200 import ops

    table = _randn(777, width, dtype=dtype)
    ids = torch.tensor([0, 776, 5, 5, 123, 1000, -1], dtype=torch.int32, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.embedding(ids, table, torch.empty(7, width, dtype=dtype, device="cuda"), flag)
    assert torch.equal(out[:5], table[ids[:5].long()])
    assert torch.equal(out[5:], torch.zeros_like(out[5:])) and int(flag) == 1


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [64, 100, 2048, 5000])
def test_rmsnorm_variants(dtype, width):
    from liteinfer_b200 import ops

    x = _randn(37, width, dtype=dtype, seed=1, scale=3.0)
    delta = _randn(37, width, dtype=dtype, seed=2)
    w = (1 + 0.1 * _randn(width, dtype=torch.float32, seed=3)).to(dtype)
    rows = torch.tensor([36, 0, 5, 5], dtype=torch.int32, device="cuda")
    for kwargs in ({}, {"delta": delta, "write_residual": True}, {"delta": delta, "rows": rows}, {"rows": rows}):
        xa, xb = x.clone(), x.clone()
        n = 4 if "rows" in kwargs else 37
        got = ops.rmsnorm(xa, w, 1e-5, torch.empty(n, width, dtype=dtype, device="cuda"), **kwargs)
        want = ref.rmsnorm(xb, w, 1e-5, torch.empty(n, width, dtype=dtype, device="cuda"), **kwargs)
        torch.testing.assert_close(got.float(), want.float(), **_tol(dtype))
        torch.testing.assert_close(xa.float(), xb.float(), **_tol(dtype))   # the residual stream moved on (or not)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_pytorch_tanh", "relu"])
@pytest.mark.parametrize("width", [176, 100, 8192])
def test_act_mul(dtype, act, width):
    from liteinfer_b200 import ops

    gu = _randn(19, 2 * width, dtype=dtype, scale=2.0)
    got = ops.act_mul(gu, torch.empty(19, width, dtype=dtype, device="cuda"), act)
    want = ref.act_mul(gu, torch.empty(19, width, dtype=dtype, device="cuda"), act)
    torch.testing.assert_close(got.float(), want.float(), **_tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_add_and_bias(dtype):
    from liteinfer_b200 import ops

    x, d, b = _randn(9, 100, dtype=dtype), _randn(9, 100, dtype=dtype, seed=5), _randn(100, dtype=dtype, seed=6)
    torch.testing.assert_close(ops.add_(x.clone(), d).float(), (x.float() + d.float()).to(dtype).float())
    torch.testing.assert_close(ops.add_bias_(x.clone(), b).float(), (x.float() + b.float()).to(dtype).float())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (7, 1000, 96), (130, 100, 50), (64, 128256 // 64, 2048), (3, 5, 7)])
def test_gemm_simt(dtype, M, N, K):
    from liteinfer_b200 import ops

    x, w, b = _randn(M, K, dtype=dtype), _randn(N, K, dtype=dtype, seed=1, scale=0.05), _randn(N, dtype=dtype, seed=2)
    got = ops.gemm_simt(x, w, torch.empty(M, N, dtype=dtype, device="cuda"), b)
    want = (x.double() @ w.double().t() + b.double())
    tol = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=2 ** -7, atol=2 ** -7)
    torch.testing.assert_close(got.double(), want, **tol)


def test_gemm_simt_rows_do_not_depend_on_the_batch():
    from liteinfer_b200 import ops

    x, w = _randn(70, 320, dtype=torch.float32), _randn(1000, 320, dtype=torch.float32, seed=1)
    full = ops.gemm_simt(x, w, torch.empty(70, 1000, device="cuda"))
    one = ops.gemm_simt(x[33:34].contiguous(), w, torch.empty(1, 1000, device="cuda"))
    assert torch.equal(full[33:34], one)


# One chunk of k and part of one; several in a cluster of odd size; four a block and the first k beyond that; eight; a k that is
# not a multiple of four.
@pytest.mark.parametrize("N,K", [(33, 40), (100, 128), (1000, 772), (64, 1024), (96, 2052), (65, 4096), (40, 4100), (65, 8196), (70, 301)])
def test_gemm_simt_widths_agree_bit_for_bit(N, K):
    from liteinfer_b200 import ops

    x, w = _randn(200, K, dtype=torch.float32), _randn(N, K, dtype=torch.float32, seed=1)
    b = _randn(N, dtype=torch.float32, seed=2)
    full = ops.gemm_simt(x, w, torch.empty(200, N, device="cuda"), b)
    # Chains of at most 128 products and then at most 34 sums, each rounding by 2^-24 of what it has.
    bound = (x.double().abs() @ w.double().abs().t() + b.double().abs()) * (128 + 34) * 2.0 ** -24
    assert bool(((full.double() - (x.double() @ w.double().t() + b.double())).abs() <= bound).all())
    for M in (1, 2, 4, 5, 8, 9, 16, 17, 63, 64, 65, 129):
        part = ops.gemm_simt(x[3:3 + M].contiguous(), w, torch.empty(M, N, device="cuda"), b)
        assert torch.equal(part, full[3:3 + M]), M
    if K % 4 == 0:
        wide = torch.randn(2, 17, K + 8, device="cuda")
        batched = ops.batched_linear(wide[:, :, 4:K + 4], torch.stack([w, 2 * w]), torch.empty(2, 17, N, device="cuda"))
        for i in range(2):
            one = ops.gemm_simt(wide[i, :, 4:K + 4].contiguous(), (i + 1) * w, torch.empty(17, N, device="cuda"))
            assert torch.equal(batched[i], one)


# More rows than a grid has tiles of 64 for: the first launch's last rows and the second's.
@pytest.mark.parametrize("dtype", DTYPES)
def test_gemm_simt_of_more_rows_than_a_grid_takes(dtype):
    from liteinfer_b200 import ops

    M, N, K = 65535 * 64 + 70, 3, 8
    x, w, b = _randn(M, K, dtype=dtype), _randn(N, K, dtype=dtype, seed=1), _randn(N, dtype=dtype, seed=2)
    got = ops.gemm_simt(x, w, torch.full((M, N), float("nan"), dtype=dtype, device="cuda"), b)
    # Eight products, their sum and the bias, each rounding by 2^-24 of what it has, and the result's own rounding.
    want, size = x.double() @ w.double().t() + b.double(), x.double().abs() @ w.double().abs().t() + b.double().abs()
    assert bool(((got.double() - want).abs() <= size * (9 * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0))).all())


# As many rows as the narrow kernel takes at once and one more, at a k that is the last of twelve chunks a block, the first of
# thirteen, between, the narrow kernel's last and the first beyond it.
@pytest.mark.parametrize("K", [12288, 12292, 14336, 16384, 16388])
def test_gemm_simt_of_a_deep_k(K):
    from liteinfer_b200 import ops

    N = 130
    x, w = _randn(256, K, dtype=torch.float32), _randn(N, K, dtype=torch.float32, seed=1)
    full = ops.gemm_simt(x, w, torch.empty(256, N, device="cuda"))
    # Chains of at most 128 products and then the chunks' sums, each rounding by 2^-24 of what it has.
    bound = (x.double().abs() @ w.double().abs().t()) * (128 + -(-K // 128)) * 2.0 ** -24
    assert bool(((full.double() - x.double() @ w.double().t()).abs() <= bound).all())
    for M in (1, 4, 8, 12, 13, 16, 17, 48, 255):
        part = ops.gemm_simt(x[1:1 + M].contiguous(), w, torch.empty(M, N, device="cuda"))
        assert torch.equal(part, full[1:1 + M]), M


@pytest.mark.parametrize("N,K", [(512, 256), (4096, 1024), (1000, 4096)])
def test_a_second_operand_that_the_kernel_just_ahead_writes(N, K):
    """The activation ahead lets the next kernel start while it still runs; what it writes is read behind it all the same."""
    from liteinfer_b200 import ops

    x, pairs = _randn(12, K, dtype=torch.float32), [_randn(N, 2 * K, dtype=torch.float32, seed=1 + i) for i in range(2)]
    want = []
    for pair in pairs:
        y = ops.act_mul(pair, torch.empty(N, K, device="cuda"), "silu")
        torch.cuda.synchronize()
        want.append(ops.gemm_simt(x, y, torch.empty(12, N, device="cuda")))
    torch.cuda.synchronize()
    products = (ops.gemm_simt, ops.linear,
                lambda a, b, out: ops.batched_linear(a[None], b[None], out[None])[0])
    y, got = torch.empty(N, K, device="cuda"), []
    for i in range(12):                 # y holds the other weights until the kernel ahead has written it
        ops.act_mul(pairs[i % 2], y, "silu")
        got.append(products[i % 3](x, y, torch.empty(12, N, device="cuda")))
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2]), i


@pytest.mark.parametrize("M,N,K", [(1, 3072, 2048), (8, 2048, 8192), (64, 1000, 96), (300, 512, 64), (2048, 256, 2048)])
def test_linear_bfloat16(M, N, K):
    from liteinfer_b200 import ops

    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    got = ops.linear(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"))
    want = x.double() @ w.double().t()
    torch.testing.assert_close(got.double(), want, rtol=2 ** -7, atol=2 ** -7)


def _paged_case(dtype, heads, kv_heads, head_dim, page_size, q_lens, ctx_lens, seed=0, poison=True):
    """Random pool, shuffled pages, sequences with given new-query and context lengths."""
    g = torch.Generator().manual_seed(seed)
    B = len(q_lens)
    pages_per = [-(-c // page_size) for c in ctx_lens]
    num_pages = sum(pages_per) + 3
    perm = torch.randperm(num_pages, generator=g).tolist()
    width = max(pages_per) + 2
    table = torch.full((B, width), -1, dtype=torch.int32)
    at = 0
    for s, n in enumerate(pages_per):
        table[s, :n] = torch.tensor(perm[at:at + n], dtype=torch.int32)
        at += n
    T = sum(q_lens)
    row = (heads + 2 * kv_heads) * head_dim
    qkv = _randn(T, row, dtype=dtype, seed=seed + 1)
    fill = float("nan") if poison else 0.0
    k_pool = torch.full((num_pages, kv_heads, page_size, head_dim), fill, dtype=dtype, device="cuda")
    v_pool = torch.full_like(k_pool, fill)
    # Earlier tokens of every context: random keys and values written straight into the pages.
    for s in range(B):
        old = ctx_lens[s] - q_lens[s]
        kk = _randn(old, kv_heads, head_dim, dtype=dtype, seed=seed + 10 + s)
        vv = _randn(old, kv_heads, head_dim, dtype=dtype, seed=seed + 50 + s)
        for p in range(old):
            page = int(table[s, p // page_size])
            k_pool[page, :, p % page_size] = kk[p]
            v_pool[page, :, p % page_size] = vv[p]
    qsl = torch.tensor([0] + torch.tensor(q_lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    ctx = torch.tensor(ctx_lens, dtype=torch.int32, device="cuda")
    positions = torch.cat([torch.arange(c - q, c) for q, c in zip(q_lens, ctx_lens)]).to(torch.int32).cuda()
    seq_of = torch.cat([torch.full((q,), s) for s, q in enumerate(q_lens)]).to(torch.int32).cuda()
    return dict(qkv=qkv, k_pool=k_pool, v_pool=v_pool, table=table.cuda(), qsl=qsl, ctx=ctx, positions=positions,
                seq_of=seq_of, B=B, T=T)


ATTENTION_SHAPES = [  # heads, kv_heads, head_dim, page_size
    (4, 2, 16, 16), (6, 3, 48, 8), (10, 2, 80, 5), (8, 8, 64, 16), (32, 8, 128, 16), (3, 1, 32, 64), (2, 1, 256, 16),
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", ATTENTION_SHAPES)
@pytest.mark.parametrize("window", [0, 7])
def test_rope_write_then_attention(dtype, heads, kv_heads, head_dim, page_size, window):
    """Portions, whole prompts and single tokens in one launch, over shuffled pages with NaN in every unwritten slot."""
    from liteinfer_b200 import ops

    q_lens, ctx_lens = [1, 40, 1, 7, 33, 2], [90, 60, 3, 7, 33, 65]
    case = _paged_case(dtype, heads, kv_heads, head_dim, page_size, q_lens, ctx_lens)
    inv_freq = (1.0 / (10000.0 ** (torch.arange(0, head_dim, 2).float() / head_dim))).cuda()
    outs = []
    for impl in (ops, ref):
        qkv, k_pool, v_pool = case["qkv"].clone(), case["k_pool"].clone(), case["v_pool"].clone()
        impl.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, inv_freq, heads,
                           kv_heads, head_dim, head_dim)
        out = torch.empty(case["T"], heads * head_dim, dtype=dtype, device="cuda")
        impl.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"],
                             case["B"], max(q_lens), heads, kv_heads, head_dim, head_dim ** -0.5, window)
        outs.append((qkv, k_pool, v_pool, out))
    for got, want in zip(outs[0], outs[1]):
        written = ~torch.isnan(want.float())
        assert torch.equal(torch.isnan(got.float()), ~written)      # nothing written outside the requests' slots
        torch.testing.assert_close(got.float()[written], want.float()[written], **_tol(dtype))
    assert torch.isfinite(outs[0][3].float()).all()


# Launches of few blocks, whose keys two blocks share from eight tiles of 64 on (one tile short of it, just there, an odd
# number of tiles, keys hidden by a window, a sequence too short to share beside one that is not).
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 64), (3, 1, 128), (8, 8, 128), (32, 1, 64)])
@pytest.mark.parametrize("q_lens,ctx_lens,window", [([40], [448], 0), ([40], [449], 0), ([130, 2], [1111, 70], 0), ([70, 33], [700, 1000], 600),
                                                    ([3], [2000], 513)])
def test_prompt_attention_with_shared_keys(heads, kv_heads, head_dim, q_lens, ctx_lens, window):
    from liteinfer_b200 import ops

    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, q_lens, ctx_lens)
    qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads, head_dim, 0)
    common = (case["table"], case["qsl"], case["ctx"])
    out = torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device="cuda")
    ops.paged_attention_tcgen05(qkv, qkv.stride(0), out, k_pool, v_pool, *common, torch.arange(len(q_lens), dtype=torch.int32, device="cuda"),
                                len(q_lens), max(q_lens), heads, kv_heads, head_dim, head_dim ** -0.5, window)
    want = torch.empty_like(out)
    ref.paged_attention(qkv, qkv.shape[1], want, k_pool, v_pool, *common, len(q_lens), max(q_lens), heads, kv_heads, head_dim,
                        head_dim ** -0.5, window)
    torch.testing.assert_close(out.float(), want.float(), **_tol(torch.bfloat16))
    assert ops.gemm_error_flag("cuda:0") == 0


# Grids on both sides of the numbers of blocks up to which a launch goes out in pairs (74 and 148 at head size 64, 74 at 128),
# contexts that are known, unknown and those of a padded shape, whose grid has blocks without queries.
@pytest.mark.parametrize("head_dim,n,q_len", [(64, 1, 444), (64, 1, 570), (64, 1, 580), (64, 1, 1184), (64, 1, 1200), (64, 2, 1184), (64, 4, 592), (64, 3, 790),
                                                (128, 2, 1184), (128, 2, 1200)])
@pytest.mark.parametrize("extra", [0, 5, 300])
def test_prompt_attention_in_pairs_where_the_grid_has_room(head_dim, n, q_len, extra):
    from liteinfer_b200 import ops

    heads, kv_heads = 8, 1                                  # 16 queries a tile of rows
    q_lens, ctx_lens = [q_len] + [q_len // 2] * (n - 1), [q_len + extra] + [q_len // 2 + extra] * (n - 1)
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, q_lens, ctx_lens)
    qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads, head_dim, 0)
    common = (case["table"], case["qsl"], case["ctx"])
    want = torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device="cuda")
    ref.paged_attention(qkv, qkv.shape[1], want, k_pool, v_pool, *common, n, q_len, heads, kv_heads, head_dim, head_dim ** -0.5, 0)
    places = torch.tensor([*range(n), -1], dtype=torch.int32, device="cuda")
    for places_n, longest, context in ((n, q_len, max(ctx_lens)), (n, q_len, 0), (n + 1, q_len * 5 // 4, 4096)):
        out = torch.empty_like(want)
        ops.paged_attention_tcgen05(qkv, qkv.stride(0), out, k_pool, v_pool, *common, places, places_n, longest, heads, kv_heads,
                                    head_dim, head_dim ** -0.5, max_context_len=context)
        torch.testing.assert_close(out.float(), want.float(), **_tol(torch.bfloat16))
    assert ops.gemm_error_flag("cuda:0") == 0


# Prompts, portions and single tokens of 32-bit numbers in one launch: tiles of one query and of eight, groups of 1 to 8 heads, units of
# keys that only some of a tile's queries see, pages that are not there (NaN wherever no request owns a slot).
@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(4, 4, 64, 16), (4, 2, 20, 5), (12, 4, 64, 16), (8, 2, 128, 8), (16, 2, 100, 16),
                                                               (9, 1, 64, 16)])
@pytest.mark.parametrize("window,keep_first,softcap,sink", [(0, 0, 0.0, False), (70, 0, 0.0, True), (100, 68, 20.0, False),
                                                            (-96, 0, 0.0, False)])
def test_prompts_in_32_bit_share_their_keys(heads, kv_heads, head_dim, page_size, window, keep_first, softcap, sink):
    from liteinfer_b200 import ops

    q_lens, ctx_lens = [9, 1, 33, 2, 8, 1, 150, 7], [9, 200, 33, 130, 264, 1, 301, 64]
    case = _paged_case(torch.float32, heads, kv_heads, head_dim, page_size, q_lens, ctx_lens)
    sinks = _randn(heads, dtype=torch.float32, seed=9) if sink else None
    ops.rope_kv_write(case["qkv"], case["positions"], case["seq_of"], case["table"], case["k_pool"], case["v_pool"], None,
                      heads, kv_heads, head_dim, 0)
    args = (case["qkv"], case["qkv"].shape[1])
    rest = (case["k_pool"], case["v_pool"], case["table"], case["qsl"], case["ctx"], case["B"], max(q_lens), heads, kv_heads,
            head_dim, head_dim ** -0.5)
    options = dict(window=max(window, 0), chunk=max(-window, 0), keep_first=keep_first, softcap=softcap, sink=sinks)
    out = lambda: torch.full((case["T"], heads * head_dim), float("nan"), device="cuda")
    want = ref.paged_attention(*args, out(), *rest, **options)
    for plan in (None, _plan_for(q_lens, ctx_lens)):
        got = ops.paged_attention(*args, out(), *rest, plan=plan, **options)
        torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5)


# Portions of few queries on either side of the line between the two kernels, whose sums are the same: as many queries as teams take and
# one more, each portion also as the end of one of eight queries, which never is theirs.
@pytest.mark.parametrize("heads,kv_heads,head_dim,few", [(4, 4, 64, 5), (8, 4, 64, 3), (12, 4, 64, 2), (4, 4, 128, 3), (4, 4, 100, 6), (8, 4, 128, 3),
                                                         (16, 4, 128, 2), (16, 2, 128, 1)])
@pytest.mark.parametrize("context", [20, 333])
def test_portions_of_few_queries_in_32_bit(heads, kv_heads, head_dim, few, context):
    from liteinfer_b200 import ops

    scale = head_dim ** -0.5
    for queries in (2, few, few + 1):
        if queries < 2:
            continue
        lens = [8, 1, 8]
        case = _paged_case(torch.float32, heads, kv_heads, head_dim, 16, lens, [context] * 3, poison=False)
        out = lambda n: torch.full((n, heads * head_dim), float("nan"), device="cuda")
        ops.rope_kv_write(case["qkv"], case["positions"], case["seq_of"], case["table"], case["k_pool"], case["v_pool"], None,
                          heads, kv_heads, head_dim, 0)
        tail = (case["k_pool"], case["v_pool"], case["table"])
        whole = ops.paged_attention(case["qkv"], case["qkv"].shape[1], out(17), *tail, case["qsl"], case["ctx"], 3, 8, heads, kv_heads,
                                    head_dim, scale, plan=_plan_for(lens, [context] * 3))
        short = torch.cat([case["qkv"][8 - queries:9], case["qkv"][17 - queries:]])
        lens = [queries, 1, queries]
        qsl = torch.tensor([0, queries, queries + 1, 2 * queries + 1], dtype=torch.int32, device="cuda")
        for plan in (None, _plan_for(lens, [context] * 3)):
            got = ops.paged_attention(short, short.shape[1], out(len(short)), *tail, qsl, case["ctx"], 3, queries, heads, kv_heads, head_dim,
                                      scale, plan=plan)
            assert torch.equal(got, torch.cat([whole[8 - queries:9], whole[17 - queries:]]))


# Rows walked by one warp and by teams, one unit of keys and several rounds of them, every width of values.
@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(3, 1, 64, 16), (9, 1, 20, 16), (2, 2, 128, 16), (6, 3, 256, 8),
                                                               (2, 1, 320, 16), (34, 2, 33, 5)])
@pytest.mark.parametrize("window,keep_first,softcap,sink", [(0, 0, 0.0, False), (70, 0, 0.0, True), (100, 68, 20.0, False),
                                                            (-96, 0, 0.0, False)])
def test_generic_attention_cuts_agree_bit_for_bit(heads, kv_heads, head_dim, page_size, window, keep_first, softcap, sink):
    from liteinfer_b200 import ops

    ctx = 1100
    case = _paged_case(torch.float32, heads, kv_heads, head_dim, page_size, [ctx], [ctx])
    sinks = _randn(heads, dtype=torch.float32, seed=9) if sink else None
    ops.rope_kv_write(case["qkv"], case["positions"], case["seq_of"], case["table"], case["k_pool"], case["v_pool"], None,
                      heads, kv_heads, head_dim, 0)

    def attend(start, count):
        qkv = case["qkv"][start:start + count]
        out = torch.empty(count, heads * head_dim, device="cuda")
        ops.paged_attention_generic(qkv, qkv.stride(0), out, case["k_pool"], case["v_pool"], case["table"],
                                    torch.tensor([0, count], dtype=torch.int32, device="cuda"),
                                    torch.tensor([start + count], dtype=torch.int32, device="cuda"), 1, count, heads, kv_heads,
                                    head_dim, head_dim ** -0.5, window, keep_first, softcap, sinks)
        return out

    whole = attend(0, ctx)
    q, k, v = (t.double().unflatten(1, (-1, head_dim)) for t in case["qkv"].split(
        [heads * head_dim, kv_heads * head_dim, kv_heads * head_dim], dim=1))
    k, v = (t.repeat_interleave(heads // kv_heads, dim=1) for t in (k, v))
    score = torch.einsum("thd,shd->hts", q, k) * head_dim ** -0.5
    score = softcap * torch.tanh(score / softcap) if softcap else score
    i, j = torch.arange(ctx, device="cuda")[:, None], torch.arange(ctx, device="cuda")[None]
    seen = j <= i
    if window > 0:
        seen &= (i - j < window) | (j < keep_first)
    elif window < 0:
        seen &= i // -window == j // -window
    score = score.masked_fill(~seen, -torch.inf)
    if sink:
        score = torch.cat([score, sinks.double()[:, None, None].expand(-1, ctx, 1)], -1)
    want = torch.einsum("hts,shd->thd", torch.softmax(score, -1)[..., :ctx], v).flatten(1)
    torch.testing.assert_close(whole.double(), want, rtol=1e-5, atol=1e-5)
    for start, count in ((0, 1), (62, 2), (64, 1), (127, 3), (130, 1), (500, 9), (1099, 1)):
        assert torch.equal(attend(start, count), whole[start:start + count]), (start, count)


# As many sequences as give a block sixteen warps, eight, four and two, at rows of less than a unit of keys and of many.
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(16, 16, 64), (12, 4, 128), (8, 8, 300)])
def test_generic_attention_of_any_number_of_sequences(heads, kv_heads, head_dim):
    from liteinfer_b200 import ops

    lengths = [1, 31, 33, 400]
    case = _paged_case(torch.float32, heads, kv_heads, head_dim, 16, [1] * 4, lengths)
    case["k_pool"].copy_(_randn(*case["k_pool"].shape, dtype=torch.float32, seed=5))
    case["v_pool"].copy_(_randn(*case["v_pool"].shape, dtype=torch.float32, seed=6))

    def attend(n):
        qkv = case["qkv"][:4].repeat(n // 4, 1)
        out = torch.empty(n, heads * head_dim, device="cuda")
        return ops.paged_attention_generic(qkv, qkv.stride(0), out, case["k_pool"], case["v_pool"], case["table"].repeat(n // 4, 1),
                                           torch.arange(n + 1, dtype=torch.int32, device="cuda"), case["ctx"].repeat(n // 4), n, 1,
                                           heads, kv_heads, head_dim, head_dim ** -0.5)

    few = attend(4)
    want = torch.empty_like(few)
    ref.paged_attention(case["qkv"], case["qkv"].shape[1], want, case["k_pool"], case["v_pool"], case["table"], case["qsl"], case["ctx"],
                        4, 1, heads, kv_heads, head_dim, head_dim ** -0.5, 0)
    torch.testing.assert_close(few, want, **_tol(torch.float32))
    for n in (8, 12, 20, 36, 40, 80, 152):
        assert torch.equal(attend(n), few.repeat(n // 4, 1)), n


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_finds_one_far_key(dtype):
    """One key among hundreds is made to dominate: the output must be that key's value, wherever its page lies."""
    from liteinfer_b200 import ops

    heads, kv_heads, d, page = 4, 2, 64, 16
    ctx = 700
    for far in (0, 15, 16, 333, 698):
        case = _paged_case(dtype, heads, kv_heads, d, page, [1], [ctx], seed=far, poison=True)
        qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
        # the new token's own key/value must be in the pool too (position ctx-1)
        ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads,
                          kv_heads, d, 0)
        q = qkv[:, :heads * d].view(1, heads, d)
        pg, off = int(case["table"][0, far // page]), far % page
        for h in range(kv_heads):
            k_pool[pg, h, off] = (q[0, h * 2].float() * 8).to(dtype)    # aligned with the first head of the group
        out = torch.empty(1, heads * d, dtype=dtype, device="cuda")
        ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 1,
                            heads, kv_heads, d, 1.0)
        for h in range(kv_heads):
            torch.testing.assert_close(out.view(heads, d)[h * 2].float(), v_pool[pg, h, off].float(),
                                       rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("dtype", DTYPES)
def test_window_edge(dtype):
    """With a window of w the key at distance w-1 is seen and the key at distance w is not."""
    from liteinfer_b200 import ops

    heads, kv_heads, d, page, w, ctx = 2, 1, 32, 8, 11, 50
    for distance, seen in ((w - 1, True), (w, False)):
        case = _paged_case(dtype, heads, kv_heads, d, page, [1], [ctx], seed=3, poison=False)
        qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
        ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads,
                          kv_heads, d, 0)
        far = ctx - 1 - distance
        pg, off = int(case["table"][0, far // page]), far % page
        k_pool[pg, 0, off] = (qkv[0, :d].float() * 10).to(dtype)
        v_pool[pg, 0, off] = 100.0
        out = torch.empty(1, heads * d, dtype=dtype, device="cuda")
        ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 1,
                            heads, kv_heads, d, 1.0, w)
        assert (out[0, :d].float().mean() > 50) == seen


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab", [512, 1000, 128256])
def test_argmax(dtype, vocab):
    from liteinfer_b200 import ops

    logits = _randn(5, vocab, dtype=dtype)
    logits[2, vocab - 1] = 50.0
    logits[3, 7] = logits[3, 300] = 60.0     # equal values: the lower index wins
    got = ops.argmax(logits, torch.empty(5, dtype=torch.int32, device="cuda"))
    want = ref.argmax(logits.cpu(), torch.empty(5, dtype=torch.int32))
    assert got.cpu().tolist() == want.tolist() and got[2] == vocab - 1 and got[3] == 7


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab", [50, 1000])
def test_sample_matches_the_rule(dtype, vocab):
    """Temperature, top-k and top-p, with ties at the boundaries, against the row-by-row rule."""
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(0)
    rows = 24
    logits = (torch.randn(rows, vocab, generator=g) * 2).to(dtype)
    logits[1, 3] = logits[1, 17] = logits[1, 30] = logits[1].float().max() + 1     # ties at the top
    logits[2] = logits[2].float().round().to(dtype)                               # many ties everywhere
    temps = torch.tensor([0.0, 1.0, 0.7, 2.5] * 6)
    top_k = torch.tensor([0, 1, 2, 5, 0, 40, 3, 0, vocab, vocab + 5, 7, 0] * 2, dtype=torch.int32)
    top_p = torch.tensor([1.0, 0.9, 0.5, 1.0, 0.1, 0.95] * 4)
    for trial in range(4):
        u = torch.rand(rows, generator=g)
        got = ops.sample(logits.cuda(), temps.cuda(), top_k.cuda(), top_p.cuda(), u.cuda(),
                         torch.empty(rows, dtype=torch.int32, device="cuda")).cpu()
        for r in range(rows):
            want = ref.sample_row(logits[r], float(temps[r]), int(top_k[r]), float(top_p[r]), float(u[r]))
            if int(got[r]) != want:
                # A draw that lands within rounding of a boundary of the running sum may fall either side of it.
                lo = ref.sample_row(logits[r], float(temps[r]), int(top_k[r]), float(top_p[r]), max(0.0, float(u[r]) - 1e-5))
                hi = ref.sample_row(logits[r], float(temps[r]), int(top_k[r]), float(top_p[r]), min(0.999999, float(u[r]) + 1e-5))
                assert int(got[r]) in (lo, hi), f"row {r}: got {int(got[r])}, rule gives {want}"


def _sample_rule(x, k, p, u):
    """The sampling rule for one row x (already divided by its temperature), sums in 64 bits, by a stable sort: the column
    drawn, and the columns that could be."""
    n = x.numel()
    order = torch.sort(x, descending=True, stable=True).indices
    w = torch.exp(x - x.max()).double()
    keep = order[:k] if 0 < k < n else order
    if 0.0 < p < 1.0:
        before = torch.cumsum(w[keep], 0) - w[keep]
        keep = keep[before <= p * float(w[keep].sum())]
    keep = keep.sort().values
    run = torch.cumsum(w[keep], 0)
    return int(keep[min(int((run <= u * float(run[-1])).sum()), len(keep) - 1)]), keep


# One block a row, two, four, eight; rows that start anywhere; rows too long for the blocks' shared memory, and for 16-bit
# column numbers; as many rows as make bfloat16 be staged undivided.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab,rows", [(1, 12), (31, 12), (8192, 12), (8193, 12), (20011, 12), (32766, 84), (50257, 12), (128256, 48),
                                        (400003, 12), (600001, 12)])
def test_sample_splits_a_row_over_blocks(dtype, vocab, rows):
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(vocab)
    logits = (torch.randn(rows, vocab, generator=g) * 2.5).to(dtype)
    logits[1] = 3.25                                        # all equal: only the index decides
    logits[2] = logits[2].float().round().to(dtype)         # a few values, thousands of ties
    logits[3, :-1] = -torch.inf                             # one column left
    logits[4, : vocab // 2] = torch.finfo(dtype).min        # masked with the type's lowest value
    logits[5] = logits[5] * 40                              # most probabilities vanish
    temps = torch.tensor([0.7, 1.0, 1.3, 1.0, 0.0, 1.0] * (rows // 6))
    top_k = torch.tensor([50, 1000, 0, 7, 3, 200, 0, 0, 4097, 0, vocab // 2, 1] * (rows // 12), dtype=torch.int32)
    top_p = torch.tensor([1.0, 0.5, 0.9, 0.95, 0.9, 0.99, 0.9, 0.3, 0.999, 1.0, 0.05, 0.5] * (rows // 12))
    for trial in range(2):
        u = torch.rand(rows, generator=g)
        got = ops.sample(logits.cuda(), temps.cuda(), top_k.cuda(), top_p.cuda(), u.cuda(),
                         torch.empty(rows, dtype=torch.int32, device="cuda")).cpu()
        for r in range(rows):
            if float(temps[r]) == 0.0 or int(top_k[r]) == 1:
                assert int(got[r]) == int(torch.argmax(logits[r].float())), r
                continue
            x = logits[r].float() / temps[r]
            # The kernel's weights are 32-bit exponentials (2^-22 of their own) cut to multiples of 2^-32 of the largest, so
            # its running sums are within `off` of the whole, and the draw and the cut of top-p move by no more.
            off = 2.0 ** -22 + vocab * 2.0 ** -32
            k, p, v = int(top_k[r]), float(top_p[r]), float(u[r])
            rules = [_sample_rule(x, k, p + dp, min(max(v + du, 0.0), 0.9999999)) for du in (-2 * off, 0.0, 2 * off)
                     for dp in ((-2 * off, 0.0, 2 * off) if p < 1 else (0.0,))]
            low, high = min(at for at, _ in rules), max(at for at, _ in rules)
            assert low <= int(got[r]) <= high, f"row {r}: got {int(got[r])}, the rule gives {low} to {high}"
            assert any(bool((keep == int(got[r])).any()) for _, keep in rules), f"row {r}: {int(got[r])} is not in what is kept"


# What is told apart by sorting: a top-k at and around the 1,024 candidates that are sorted at most; boundary bins of a handful and of
# thousands of columns (scale 0.02: the whole row lies in a few bins); one block a row and eight.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab", [2048, 8192, 50257])
@pytest.mark.parametrize("scale", [0.02, 0.5, 3.0])
def test_sample_among_few_and_many_candidates(dtype, vocab, scale):
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(vocab + int(100 * scale))
    ks, ps, rows = [2, 32, 33, 512, 513, 1023, 1024, 1025, 0, 0, 0, 0], [1.0, 0.3, 0.999], 36
    logits = (torch.randn(rows, vocab, generator=g) * scale).to(dtype)
    temps = torch.tensor([1.0, 0.6, 1.7] * (rows // 3))
    top_k, top_p = torch.tensor([k for k in ks for _ in ps], dtype=torch.int32), torch.tensor(ps * len(ks))
    u = torch.rand(rows, generator=g)
    got = ops.sample(logits.cuda(), temps.cuda(), top_k.cuda(), top_p.cuda(), u.cuda(),
                     torch.empty(rows, dtype=torch.int32, device="cuda")).cpu()
    off = 2.0 ** -22 + vocab * 2.0 ** -32          # as in the test above
    for r in range(rows):
        x = logits[r].float() / temps[r]
        k, p, v = int(top_k[r]), float(top_p[r]), float(u[r])
        rules = [_sample_rule(x, k, p + dp, min(max(v + du, 0.0), 0.9999999)) for du in (-2 * off, 0.0, 2 * off)
                 for dp in ((-2 * off, 0.0, 2 * off) if p < 1 else (0.0,))]
        low, high = min(at for at, _ in rules), max(at for at, _ in rules)
        assert low <= int(got[r]) <= high, f"row {r}: got {int(got[r])}, the rule gives {low} to {high}"
        assert any(bool((keep == int(got[r])).any()) for _, keep in rules), f"row {r}: {int(got[r])} is not in what is kept"


# Rows whose k-th value lies far below their maximum: low temperatures, a few large values over many small ones, one value far above all; as
# many columns as can be chosen and one more than are sorted.  One block a row, a cluster, and a cluster of the most a block's memory holds.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vocab", [1000, 8192, 32000, 151936])
def test_sample_far_below_the_maximum(dtype, vocab):
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(vocab)
    ks, ps = [2, 50, 127, 129, 511, 513], [1.0, 0.9, 0.999999]
    kinds = [(0.05, "wide"), (0.2, "wide"), (1.0, "peaked"), (0.02, "peaked"), (1.0, "alone")]
    cases = [(k, p, t, kind) for k in ks for p in ps for t, kind in kinds]
    def row(kind):
        x = torch.randn(vocab, generator=g) * 2.5
        if kind == "peaked":
            x = x * 0.6 + 3 * torch.empty(vocab).exponential_(1.0, generator=g)
        if kind == "alone":
            x[int(torch.randint(vocab, (1,), generator=g))] = 400.0 + float(torch.rand(1, generator=g))
        return x
    logits = torch.stack([row(kind) for *_, kind in cases]).to(dtype)
    u = torch.rand(len(cases), generator=g)
    got = ops.sample(logits.cuda(), torch.tensor([t for _, _, t, _ in cases]).cuda(), torch.tensor([k for k, *_ in cases], dtype=torch.int32).cuda(),
                     torch.tensor([p for _, p, *_ in cases]).cuda(), u.cuda(), torch.empty(len(cases), dtype=torch.int32, device="cuda")).cpu()
    off = 2.0 ** -22 + vocab * 2.0 ** -32          # as in the tests above
    for r, (k, p, t, _) in enumerate(cases):
        x, v = logits[r].float() / t, float(u[r])
        rules = [_sample_rule(x, k, p + dp, min(max(v + du, 0.0), 0.9999999)) for du in (-2 * off, 0.0, 2 * off)
                 for dp in ((-2 * off, 0.0, 2 * off) if p < 1 else (0.0,))]
        low, high = min(at for at, _ in rules), max(at for at, _ in rules)
        assert low <= int(got[r]) <= high, f"{cases[r]}: got {int(got[r])}, the rule gives {low} to {high}"
        assert any(bool((keep == int(got[r])).any()) for _, keep in rules), f"{cases[r]}: {int(got[r])} is not in what is kept"


# Parameters that travel with the launch, up to as many rows as it takes, and one row more through the pinned copy.
@pytest.mark.parametrize("rows", [1, 3, 128, 129])
def test_sampler_brings_its_parameters_along(rows):
    from liteinfer_b200 import SamplingParams, ops
    from liteinfer_b200.sampling.sampler import Sampler

    g = torch.Generator().manual_seed(rows)
    logits = (torch.randn(rows, 3000, generator=g) * 2.5).cuda()
    kinds = [dict(temperature=0.8, top_k=40), dict(temperature=0.0), dict(temperature=1.3, top_p=0.8), dict(temperature=1.0)]
    params = [SamplingParams(seed=i, **kinds[i % 4]) for i in range(rows)]
    got = Sampler(0)(logits, params)
    uniform = torch.tensor([0.0 if p.greedy else random.Random(p.seed).random() for p in params]).cuda()
    want = ops.sample(logits, torch.tensor([p.temperature for p in params]).cuda(),
                      torch.tensor([max(p.top_k, 0) for p in params], dtype=torch.int32).cuda(),
                      torch.tensor([p.top_p for p in params]).cuda(), uniform, torch.empty(rows, dtype=torch.int32, device="cuda"))
    assert torch.equal(got, want)


def test_sample_distribution():
    """Many draws of one row follow softmax(logits / T) restricted to the top-k."""
    from liteinfer_b200 import ops

    vocab, n = 40, 20000
    g = torch.Generator().manual_seed(1)
    row = torch.randn(vocab, generator=g)
    logits = row.repeat(n, 1).cuda()
    u = torch.rand(n, generator=g).cuda()
    got = ops.sample(logits, torch.full((n,), 0.8).cuda(), torch.full((n,), 10, dtype=torch.int32).cuda(),
                     torch.ones(n).cuda(), u, torch.empty(n, dtype=torch.int32, device="cuda")).cpu()
    keep = torch.topk(row, 10).indices
    p = torch.zeros(vocab)
    p[keep] = torch.softmax(row[keep] / 0.8, -1)
    freq = torch.bincount(got.long(), minlength=vocab).float() / n
    assert float((freq - p).abs().max()) < 0.015
    assert set(got.tolist()) <= set(keep.tolist())


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(3072, 2048), (2048, 8192), (1000, 96), (17, 40), (128256 // 8, 2048), (48, 16384)])
def test_gemm_skinny(M, N, K):
    from liteinfer_b200 import ops

    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    b = _randn(N, dtype=torch.bfloat16, seed=2)
    got = ops.gemm_skinny(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), b)
    want = x.double() @ w.double().t() + b.double()
    torch.testing.assert_close(got.double(), want, rtol=2 ** -7, atol=2 ** -7)


def test_gemm_skinny_rows_do_not_depend_on_the_batch():
    from liteinfer_b200 import ops

    x, w = _randn(64, 2048, dtype=torch.bfloat16), _randn(555, 2048, dtype=torch.bfloat16, seed=1, scale=0.05)
    full = ops.gemm_skinny(x, w, torch.empty(64, 555, dtype=torch.bfloat16, device="cuda"))
    for rows in (1, 8, 20):
        part = ops.gemm_skinny(x[:rows].contiguous(), w, torch.empty(rows, 555, dtype=torch.bfloat16, device="cuda"))
        assert torch.equal(part, full[:rows])


def test_linear_hands_narrow_batches_to_the_streaming_kernel():
    """Up to 8 rows of x always, up to 16 for weights of few rows: `linear` then gives what the kernel gives."""
    from liteinfer_b200 import ops

    for M, N, streams in ((8, 8192, True), (12, 2048, True), (16, 4096, True), (17, 2048, False), (12, 8192, False)):
        x, w = _randn(M, 512, dtype=torch.bfloat16), _randn(N, 512, dtype=torch.bfloat16, seed=1, scale=0.05)
        before = ops.kernels.launch_count
        out = ops.linear(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"))
        assert (ops.kernels.launch_count > before) == streams     # library products are not counted
        torch.testing.assert_close(out.double(), x.double() @ w.double().t(), rtol=2 ** -7, atol=2 ** -7)
        if streams:
            assert torch.equal(out, ops.gemm_stream(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda")))


def test_gemm_skinny_refuses_what_it_cannot_do():
    from liteinfer_b200 import ops
    from liteinfer_b200.ops import KernelLibraryError

    x, w = _randn(65, 64, dtype=torch.bfloat16), _randn(16, 64, dtype=torch.bfloat16)
    with pytest.raises(KernelLibraryError, match="refuses"):
        ops.gemm_skinny(x, w, torch.empty(65, 16, dtype=torch.bfloat16, device="cuda"))
    x, w = _randn(2, 100, dtype=torch.bfloat16), _randn(16, 100, dtype=torch.bfloat16)
    with pytest.raises(KernelLibraryError, match="refuses"):
        ops.gemm_skinny(x, w, torch.empty(2, 16, dtype=torch.bfloat16, device="cuda"))
    # ...while `linear` takes any shape, by handing what the kernel refuses to the library product.
    out = ops.linear(x, w, torch.empty(2, 16, dtype=torch.bfloat16, device="cuda"))
    torch.testing.assert_close(out.double(), x.double() @ w.double().t(), rtol=2 ** -7, atol=2 ** -7)


def _plan_for(q_lens, ctx_lens):
    from liteinfer_b200.parts.context import AttentionPlan

    dec = [i for i, q in enumerate(q_lens) if q == 1]
    pre = [i for i, q in enumerate(q_lens) if q > 1]
    starts = [0]
    for q in q_lens:
        starts.append(starts[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    return AttentionPlan(num_decode=len(dec), decode_seqs=i32(dec), decode_tokens=i32([starts[i] for i in dec]),
                         num_prefill=len(pre), prefill_seqs=i32(pre),
                         max_prefill_query_len=max([q_lens[i] for i in pre], default=0),
                         max_decode_context_len=max([ctx_lens[i] for i in dec], default=0))


def _splits(splits, monkeypatch):
    """`"11 as a cluster"`: 11 splits with the streaming kernel's merge through a cluster switched on."""
    if isinstance(splits, str):
        monkeypatch.setenv("LITEINFER_ATTN_CLUSTER_MERGE", "1")
        return int(splits.split()[0])
    return splits


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(4, 2, 64, 16), (8, 8, 64, 8), (32, 8, 128, 16),
                                                               (6, 2, 128, 5), (64, 1, 64, 32), (5, 1, 64, 16)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("splits", [None, 1, 3, 32, "2 as a cluster", "11 as a cluster", "16 as a cluster"])
def test_tensor_core_attention_against_the_plain_kernel(heads, kv_heads, head_dim, page_size, window, splits,
                                                        monkeypatch):
    """Portions and single tokens, planned (split decode rows beside unsplit portions) or not, over
    contexts that straddle the 64-key tiles, with NaN in every slot no request owns."""
    from liteinfer_b200 import ops

    splits = _splits(splits, monkeypatch)
    q_lens = [1, 130, 1, 7, 64, 1, 1, 2]
    ctx_lens = [700, 190, 1, 7, 64, 63, 65, 129]
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, page_size, q_lens, ctx_lens)
    qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads,
                      head_dim, 0)
    args = (qkv, qkv.shape[1])
    rest = (k_pool, v_pool, case["table"], case["qsl"], case["ctx"], case["B"], max(q_lens), heads, kv_heads,
            head_dim, head_dim ** -0.5, window)
    want = ref.paged_attention(*args, torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device="cuda"), *rest)
    out = torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    plan = None if splits is None else _plan_for(q_lens, ctx_lens)
    got = ops.paged_attention(*args, out, *rest, plan=plan, decode_splits=splits if splits and splits > 1 else None)
    assert torch.isfinite(got.float()).all()
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)


# Contexts at the edges of one block's tiles, of sixteen blocks' and of one tile a block, together in a launch; many sequences, whose
# blocks at head size 128 are more than two an SM (320 of them) and as many again behind a second split.
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("ctx_lens,splits", [([1, 64, 256, 257, 320, 1024, 1025, 6144, 6145], 32), ([1, 256, 257, 448, 704, 6145], 7),
                                             ([70 + 5 * i for i in range(40)], None), ([300 + 9 * i for i in range(40)], 2)])
@pytest.mark.parametrize("window,softcap,sink", [(0, 0.0, False), (300, 0.0, True), (0, 20.0, False)])
def test_decode_splits_follow_the_context(head_dim, ctx_lens, splits, window, softcap, sink):
    from liteinfer_b200 import ops

    heads, kv_heads, q_lens = 16, 8, [1] * len(ctx_lens)
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, q_lens, ctx_lens)
    qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads,
                      head_dim, 0)
    args = (qkv, qkv.shape[1])
    rest = (k_pool, v_pool, case["table"], case["qsl"], case["ctx"], case["B"], 1, heads, kv_heads, head_dim, head_dim ** -0.5, window)
    extra = dict(softcap=softcap, sink=_randn(heads, dtype=torch.float32, seed=9) if sink else None)
    want = ref.paged_attention(*args, torch.empty(case["T"], heads * head_dim, dtype=torch.bfloat16, device="cuda"), *rest, **extra)
    got = ops.paged_attention(*args, torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda"),
                              *rest, plan=_plan_for(q_lens, ctx_lens), decode_splits=splits, **extra)
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)
    assert ops.gemm_error_flag("cuda:0") == 0


# Blocks of head size 128 (148 SMs): two an SM, three, between one wave of three and two of two, and beyond.
def test_three_blocks_an_sm_where_they_save_a_wave():
    from liteinfer_b200.ops import kernels

    narrow, wide = kernels.decode_capacity(128, True), kernels.decode_wide_capacity()
    assert 2 * wide == 3 * narrow
    form = lambda blocks: bool(kernels._fn("li_paged_attention_stream_wide")(128, blocks))
    assert [form(b) for b in (1, narrow, narrow + 1, wide, wide + 1, 2 * narrow, 2 * narrow + 1, 4 * narrow)] == [
        False, False, True, True, False, False, True, True]
    assert not kernels._fn("li_paged_attention_stream_wide")(64, wide)


# Launches of one wave and of more in every form, contexts of every length, as they come and longest first, some of the places empty.
@pytest.mark.parametrize("head_dim,n", [(64, 20), (64, 100), (128, 30), (128, 50), (128, 64), (128, 76)])
def test_decode_longest_first(head_dim, n, monkeypatch):
    from liteinfer_b200 import ops
    from liteinfer_b200.ops import kernels

    heads, kv_heads = 16, 8
    ctx_lens = [1 + (37 * i * i) % 700 for i in range(n)]
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, [1] * n, ctx_lens, poison=False)
    rest = (case["k_pool"], case["v_pool"], case["table"], case["qsl"], case["ctx"], case["B"], 1, heads, kv_heads, head_dim,
            head_dim ** -0.5)
    out = lambda: torch.full((n, heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    plan, launched = _plan_for([1] * n, ctx_lens), []
    plain = ops.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest, plan=plan)
    order = sorted(range(n), key=lambda i: -ctx_lens[i])
    plan.decode_longest_first = torch.tensor(order + [-1] * 3, dtype=torch.int32, device="cuda")
    plan.decode_seqs = torch.cat([plan.decode_seqs, plan.decode_longest_first[n:]])
    plan.num_decode += 3
    kernel = kernels.paged_attention_mma
    monkeypatch.setattr(kernels, "paged_attention_mma", lambda *args, **options: launched.append(args[8]) or kernel(*args, **options))
    got = ops.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest, plan=plan)
    assert torch.equal(got, plain) or (n <= 30 and torch.allclose(got.float(), plain.float(), rtol=2 ** -6, atol=2 ** -6))
    more = (n + 3) * kv_heads > kernels.decode_capacity(head_dim, True)
    assert launched[0] is (plan.decode_longest_first if more else plan.decode_seqs)
    want = ref.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest)
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)


# A count that is asked for is every sequence's, also of one with fewer tiles than blocks or as few as one block would take.
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("splits", [1, 2, 5, 8, 32, None])
def test_splits_that_are_asked_for_are_taken(head_dim, splits, monkeypatch):
    from liteinfer_b200 import ops
    from liteinfer_b200.ops import kernels

    heads, kv_heads, ctx_lens = 8, 2, [1, 100, 256, 300, 449, 1000, 3000]
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, [1] * len(ctx_lens), ctx_lens, poison=False)
    rest = (case["k_pool"], case["v_pool"], case["table"], case["qsl"], case["ctx"], case["B"], 1, heads, kv_heads, head_dim,
            head_dim ** -0.5)
    out = lambda: torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest, plan=_plan_for([1], [64]))        # (what is kept is made)
    partials = []       # the log-sum-exps of the launch: a split that the kernel wrote holds a number or minus infinity
    empty = torch.empty

    def marked(*shape, **options):
        made = empty(*shape, **options)
        if options.get("dtype") == torch.float32 and made.dim() == 1:
            made.fill_(float("nan"))
            partials.append(made)
        return made

    monkeypatch.setattr(kernels.torch, "empty", marked)
    got = ops.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest, plan=_plan_for([1] * len(ctx_lens), ctx_lens),
                              decode_splits=splits)
    monkeypatch.undo()
    want = ref.paged_attention(case["qkv"], case["qkv"].shape[1], out(), *rest)
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)
    written = [not bool(torch.isnan(p).any()) for p in partials]
    assert written == ([] if splits == 1 else [splits is not None])      # None: the short ones have one block, and no partial result


# Launches that know the longest context only, one sequence at every edge of what the kernel gives its own keys: the last that one block
# takes and the next, a tile a block, sixteen blocks, the last with sixteen and the first with more, beside others; from 32 blocks down to 2.
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("kv_heads,ctx_lens", [(2, [1, 64, 256, 257, 320, 321, 1024, 1025, 3072, 3073, 6145]), (8, [256, 257, 320, 321, 448, 449, 700, 6145]),
                                               (8, [60 + 61 * i for i in range(24)])])
@pytest.mark.parametrize("window,softcap,sink", [(0, 0.0, False), (300, 0.0, True), (0, 20.0, False)])
def test_decode_takes_the_splits_its_keys_pay_for(head_dim, kv_heads, ctx_lens, window, softcap, sink):
    from liteinfer_b200 import ops

    heads, q_lens = 16, [1] * len(ctx_lens)
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, 16, q_lens, ctx_lens, poison=False)
    args = (case["qkv"], case["qkv"].shape[1])
    rest = (case["k_pool"], case["v_pool"], case["table"], case["qsl"], case["ctx"], case["B"], 1, heads, kv_heads, head_dim,
            head_dim ** -0.5, window)
    extra = dict(softcap=softcap, sink=_randn(heads, dtype=torch.float32, seed=9) if sink else None)
    out = lambda: torch.full((case["T"], heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    want = ref.paged_attention(*args, out(), *rest, **extra)
    got = ops.paged_attention(*args, out(), *rest, plan=_plan_for(q_lens, ctx_lens), **extra)
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)
    assert ops.gemm_error_flag("cuda:0") == 0


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [(32, 8, 64, 16), (8, 8, 64, 8), (16, 1, 128, 16),
                                                               (6, 2, 128, 5), (5, 1, 64, 32)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("splits", [1, 3, 32, "11 as a cluster", "16 as a cluster"])
def test_decode_attention_with_rotary_and_cache_write_fused(heads, kv_heads, head_dim, page_size, window, splits,
                                                            monkeypatch):
    """One launch that rotates q and the newest key, stores key and value and attends, against the two
    launches it replaces: the same output and the same pages, to the bit; contexts end at, just before and
    just after the edges of pages and of 64-key tiles."""
    from liteinfer_b200 import ops

    splits = _splits(splits, monkeypatch)
    ctx_lens = [700, 1, 64, 65, 63, 129, 320, 16, 17]
    q_lens = [1] * len(ctx_lens)
    case = _paged_case(torch.bfloat16, heads, kv_heads, head_dim, page_size, q_lens, ctx_lens, seed=3)
    inv_freq = (1.0 / (500000.0 ** (torch.arange(0, head_dim, 2).float() / head_dim))).cuda()
    plan = _plan_for(q_lens, ctx_lens)
    rest = (case["table"], case["qsl"], case["ctx"], case["B"], 1, heads, kv_heads, head_dim, head_dim ** -0.5, window)
    q_width, kv_width = heads * head_dim, kv_heads * head_dim

    qkv, k_two, v_two = case["qkv"].clone(), case["k_pool"].clone(), case["v_pool"].clone()
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_two, v_two, inv_freq, heads, kv_heads,
                      head_dim, head_dim)
    want = ops.paged_attention(qkv, qkv.shape[1], torch.empty(case["T"], q_width, dtype=torch.bfloat16, device="cuda"),
                               k_two, v_two, *rest, plan=plan, decode_splits=splits)

    qkv, k_one, v_one = case["qkv"].clone(), case["k_pool"].clone(), case["v_pool"].clone()
    assert ops.fused_decode_supports(torch.bfloat16, heads, kv_heads, head_dim, head_dim, plan)
    newest = ops.NewestToken(inv_freq, qkv[:, q_width:], qkv[:, q_width + kv_width:])
    got = ops.paged_attention(qkv, qkv.shape[1], torch.empty(case["T"], q_width, dtype=torch.bfloat16, device="cuda"),
                              k_one, v_one, *rest, plan=plan, decode_splits=splits, newest=newest)
    assert torch.equal(got, want)
    for one, two in ((k_one, k_two), (v_one, v_two)):
        assert torch.equal(torch.isnan(one.float()), torch.isnan(two.float()))
        assert torch.equal(torch.nan_to_num(one.float()), torch.nan_to_num(two.float()))

    # A layer that reads another layer's pages: the newest token is there already and nothing is written.
    frozen_k, frozen_v = k_two.clone(), v_two.clone()
    newest = ops.NewestToken(inv_freq, qkv[:, q_width:], qkv[:, q_width + kv_width:], store=False)
    again = ops.paged_attention(qkv, qkv.shape[1], torch.empty_like(got), frozen_k, frozen_v, *rest, plan=plan,
                                decode_splits=splits, newest=newest)
    assert torch.equal(again, want)
    assert torch.equal(torch.nan_to_num(frozen_k.float()), torch.nan_to_num(k_two.float()))


def test_tensor_core_attention_finds_one_far_key_under_splits():
    from liteinfer_b200 import ops

    heads, kv_heads, d, page, ctx = 8, 2, 128, 16, 3000
    for far in (0, 63, 64, 1500, 2998):
        case = _paged_case(torch.bfloat16, heads, kv_heads, d, page, [1], [ctx], seed=far)
        qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
        ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads,
                          kv_heads, d, 0)
        q = qkv[:, :heads * d].view(1, heads, d)
        pg, off = int(case["table"][0, far // page]), far % page
        for h in range(kv_heads):
            k_pool[pg, h, off] = (q[0, h * 4].float() * 4).to(torch.bfloat16)
        out = torch.empty(1, heads * d, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 1,
                            heads, kv_heads, d, 1.0, 0, plan=_plan_for([1], [ctx]))
        for h in range(kv_heads):
            torch.testing.assert_close(out.view(heads, d)[h * 4].float(), v_pool[pg, h, off].float(),
                                       rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("words,n_late", [(40, 0), (2105, 8), (16384, 64), (16385, 3)])
def test_stage_batch_equals_copy_and_scatter(words, n_late):
    """The kernel that reads a pinned batch in place and places the late tokens gives what the copy followed by the
    scatter gives; a batch beyond its limit is refused (the caller copies)."""
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(words)
    tok_len, n = (16 if words < 16384 else 3000), max(n_late, 1)    # layout: tokens first, dst 4 words behind, src after it
    host = torch.randint(0, 1000, (words,), generator=g, dtype=torch.int32)
    dst = torch.full((n,), -1, dtype=torch.int32)
    places = torch.randperm(tok_len, generator=g).to(torch.int32)
    for i in range(0, min(n_late, 2 * tok_len), 2):      # every second entry names a place, each place once
        dst[i] = places[i // 2]
    at = tok_len + 4
    host[at:at + n] = dst
    host[at + n:at + 2 * n] = torch.randint(0, 32, (n,), generator=g, dtype=torch.int32)
    host = host.pin_memory()
    source = torch.randint(0, 50000, (32,), generator=g, dtype=torch.int32).cuda()
    views = lambda t: (t[:tok_len], t[at:at + n], t[at + n:at + 2 * n])
    want = host.cuda()
    if n_late:
        ops.scatter_tokens(*views(want), source)
    device = torch.full((words,), -7, dtype=torch.int32, device="cuda")
    done = ops.stage_batch(device, host, *views(device), source if n_late else None)
    assert done == (words <= ops.kernels.STAGE_KERNEL_MAX_WORDS)
    if done:
        torch.cuda.synchronize()
        assert torch.equal(device, want)


@pytest.mark.parametrize("apart", [(), ("tokens",), ("dst",), ("src",), ("tokens", "dst", "src")])
@pytest.mark.parametrize("words,off", [(3000, 0), (3001, 1), (1025, 3)])
def test_stage_batch_with_tensors_of_their_own(apart, words, off):
    """Tokens and the lists of places may be tensors outside the batch, and the batch may start anywhere."""
    from liteinfer_b200 import ops

    g = torch.Generator().manual_seed(words)
    n = 40
    host = torch.randint(0, 1000, (words + off,), generator=g, dtype=torch.int32)
    host[off + 400:off + 400 + n] = torch.randperm(300, generator=g)[:n].to(torch.int32)
    host[off + 400:off + 400 + n:3] = -1
    host[off + 500:off + 500 + n] = torch.randint(0, 32, (n,), generator=g, dtype=torch.int32)
    host = host.pin_memory()[off:]
    source = torch.randint(0, 50000, (32,), generator=g, dtype=torch.int32).cuda()
    device = torch.full((words + off,), -7, dtype=torch.int32, device="cuda")[off:]
    at = {"tokens": slice(0, 300), "dst": slice(400, 400 + n), "src": slice(500, 500 + n)}
    parts = {name: host[place].cuda() if name in apart else device[place] for name, place in at.items()}
    assert ops.stage_batch(device, host, parts["tokens"], parts["dst"], parts["src"], source)
    tokens = host[:300].clone()
    for d, s in zip(host[400:400 + n].tolist(), host[500:500 + n].tolist()):
        if d >= 0:
            tokens[d] = int(source[s])
    want = host.clone()
    if "tokens" not in apart:
        want[:300] = tokens
    assert torch.equal(parts["tokens"].cpu(), tokens) and torch.equal(device.cpu(), want)


@pytest.mark.parametrize("shapes", [[(3, 5)], [(16, 128, 128), (7,), (4, 1000)], [(1,)] * 40])
def test_zeroed_slots(shapes):
    """The slots named, and no others, are zero in every state tensor, whatever a slot's size and alignment."""
    from liteinfer_b200 import ops

    slots = 70
    tensors = [torch.full((slots, *shape), 3.0, dtype=DTYPES[i % 2], device="cuda") for i, shape in enumerate(shapes)]
    states = ops.SlotStates(tensors)
    states.zero([4])
    assert all(bool((t[4] == 0).all()) and int((t == 0).sum()) == t[4].numel() for t in tensors)
    named = [0, *range(5, slots)]
    states.zero(named)
    for t in tensors:
        assert bool((t[0] == 0).all() and (t[4:] == 0).all() and (t[1:4] == 3).all())


# Sequences of less than a chunk of eight tokens, whole chunks, and a rest, together and each alone, at every head size the
# staged kernel has; the plain recurrence checks the first.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,vdim", [(16, 128, 128), (4, 128, 32), (20, 64, 64), (40, 32, 96), (3, 256, 16)])
def test_delta_rule_chunks(dtype, heads, dim, vdim):
    from liteinfer_b200 import ops

    lengths = [21, 1, 8, 9, 40, 2]
    n, count = sum(lengths), len(lengths)
    qkv = _randn(n, 2 * heads * dim + heads * vdim, dtype=dtype)
    ab = _randn(n, 2 * heads, dtype=dtype, seed=1)
    a_log, dt_bias = _randn(heads, dtype=torch.float32, seed=2), _randn(heads, dtype=torch.float32, seed=3)
    before = _randn(count, heads, vdim, dim, dtype=torch.float32, seed=4)

    def run(first, last):
        rows = slice(sum(lengths[:first]), sum(lengths[:last]))
        state, out = before[first:last].clone(), torch.empty(rows.stop - rows.start, heads * vdim, device="cuda")
        starts = torch.tensor([0] + torch.tensor(lengths[first:last]).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        slots = torch.arange(last - first, dtype=torch.int32, device="cuda")
        ops.gated_delta_rule(qkv[rows], ab[rows], a_log, dt_bias, state, starts, slots, last - first, heads, heads, dim, vdim, out,
                             max(2, max(lengths[first:last])))
        return out, state

    out, state = run(0, count)
    at = 0
    for i, length in enumerate(lengths[:5]):
        alone, kept = run(i, i + 1)
        assert torch.equal(alone, out[at:at + length]) and torch.equal(kept[0], state[i]), i
        at += length
    q, k, v = (t.double().unflatten(1, (heads, -1)) for t in qkv[:21].split([heads * dim, heads * dim, heads * vdim], dim=1))
    q, k = (t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    beta, raw = torch.sigmoid(ab[:21, :heads].double()), ab[:21, heads:].double() + dt_bias.double()
    decay = torch.exp(-a_log.double().exp() * torch.nn.functional.softplus(raw))
    S = before[0].double()                                  # [heads, vdim, dim]
    for t in range(21):
        S = decay[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
        S = S + u[:, :, None] * k[t][:, None, :]
        want = torch.einsum("hvd,hd->hv", S, q[t]) * dim ** -0.5
        torch.testing.assert_close(out[t].double(), want.flatten(), rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(state[0].double(), S, rtol=1e-4, atol=1e-4)


def test_split_policy():
    from liteinfer_b200.ops import decode_splits_for

    assert decode_splits_for(1, 8, 100) == 1            # fewer than four key tiles: nothing to split
    assert decode_splits_for(1, 8, 4096) == 32
    assert 2 <= decode_splits_for(8, 8, 4096) <= 16
    assert decode_splits_for(64, 8, 4096) == 1


def test_split_policy_with_the_cluster_merge(monkeypatch):
    """With the switch on, the streaming kernel gets a count whose splits can be one cluster each, all of them
    resident at once."""
    from liteinfer_b200.ops import decode_splits_for, kernels

    monkeypatch.setenv("LITEINFER_ATTN_CLUSTER_MERGE", "1")
    for batch in (1, 4, 8, 16):
        chosen = decode_splits_for(batch, 8, 4096, 64, True)
        assert 2 <= chosen <= 16 and kernels.cluster_capacity(64, chosen) >= batch * 8, (batch, chosen)


def _interleave(gate, up):
    rest = gate.shape[1:]
    return torch.stack([gate.reshape(-1, 8, *rest), up.reshape(-1, 8, *rest)], dim=1).reshape(2 * gate.shape[0], *rest).contiguous()


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("inter,K,act", [(8192, 2048, "silu"), (112, 120, "gelu_pytorch_tanh"), (176, 64, "relu")])
@pytest.mark.parametrize("with_bias", [False, True])
def test_gated_linear_is_product_activation_and_multiply_in_one(M, inter, K, act, with_bias):
    from liteinfer_b200 import ops

    dt = torch.bfloat16
    x = _randn(M, K, dtype=dt)
    gate, up = _randn(inter, K, dtype=dt, seed=1, scale=0.05), _randn(inter, K, dtype=dt, seed=2, scale=0.05)
    bg, bu = _randn(inter, dtype=dt, seed=3), _randn(inter, dtype=dt, seed=4)
    w = _interleave(gate, up)
    b = _interleave(bg, bu) if with_bias else None
    got = ops.gated_linear(x, w, torch.empty(M, inter, dtype=dt, device="cuda"), act, b)
    # the same thing in two kernels, through the same layout: bit for bit
    gu = ops.linear(x, w, torch.empty(M, 2 * inter, dtype=dt, device="cuda"), b)
    two = ops.act_mul_interleaved(gu, torch.empty(M, inter, dtype=dt, device="cuda"), act)
    assert torch.equal(got, two)
    # and the plain formula on the plain layout
    gu_plain = torch.cat([x.double() @ gate.double().t() + (bg.double() if with_bias else 0),
                          x.double() @ up.double().t() + (bu.double() if with_bias else 0)], dim=1).to(dt)
    want = ref.act_mul(gu_plain, torch.empty(M, inter, dtype=dt, device="cuda"), act)
    torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)


@pytest.mark.parametrize("dtype", DTYPES)
def test_act_mul_interleaved(dtype):
    from liteinfer_b200 import ops

    gu = _randn(5, 2 * 176, dtype=dtype, scale=2.0)
    got = ops.act_mul_interleaved(gu, torch.empty(5, 176, dtype=dtype, device="cuda"), "silu")
    want = ref.act_mul_interleaved(gu, torch.empty(5, 176, dtype=dtype, device="cuda"), "silu")
    torch.testing.assert_close(got.float(), want.float(), **_tol(dtype))


def test_skinny_slices_leave_their_counters_at_zero():
    from liteinfer_b200 import ops
    from liteinfer_b200.ops.kernels import scratch_for

    # Few rows of w: wide blocks; very few and a long k: slices of k as well.
    assert ops.gemm_skinny_plan(16384, 2048) == (2, 1) and ops.gemm_skinny_plan(3072, 2048) == (8, 1)
    assert ops.gemm_skinny_plan(8192, 2048) == (8, 1) and ops.gemm_skinny_plan(9600, 64) == (4, 1)
    assert ops.gemm_skinny_plan(2048, 8192) == (16, 1) and ops.gemm_skinny_plan(64, 32768) == (16, 4)
    x, w = _randn(8, 32768, dtype=torch.bfloat16), _randn(64, 32768, dtype=torch.bfloat16, seed=1, scale=0.02)
    outs = [ops.gemm_skinny(x, w, torch.empty(8, 64, dtype=torch.bfloat16, device="cuda")) for _ in range(3)]
    torch.testing.assert_close(outs[0].double(), x.double() @ w.double().t(), rtol=2 ** -7, atol=2 ** -6)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    torch.cuda.synchronize()
    assert int(scratch_for(x.device).gemm_counters.abs().sum()) == 0
    assert int(scratch_for(x.device).attention_counters.abs().sum()) == 0


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (2048, 2048, 2048), (300, 1000, 96), (77, 136, 40), (129, 3072, 2048),
                                   (1024, 16384, 512), (256, 2048, 8192)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_gemm_tcgen05(M, N, K, with_bias):
    """The tcgen05 / TMA / tensor-memory product against a float64 product, at sizes that leave ragged tiles in
    every direction, for the kernel of single CTAs (fewer than 256 rows or columns) and the one of CTA pairs; no
    wait inside the kernel may have given up."""
    from liteinfer_b200 import ops

    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    b = _randn(N, dtype=torch.bfloat16, seed=2) if with_bias else None
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05(x, w, out, b)
    want = x.double() @ w.double().t() + (b.double() if with_bias else 0)
    assert ops.gemm_error_flag("cuda:0") == 0
    torch.testing.assert_close(out.double(), want, rtol=2 ** -7, atol=2 ** -6)


@pytest.mark.parametrize("M,inter,K,act", [(2048, 8192, 2048, "silu"), (130, 176, 64, "gelu_pytorch_tanh"),
                                           (500, 112, 120, "relu"), (300, 504, 96, "silu"), (257, 128, 4096, "gelu")])
def test_gemm_tcgen05_gated_epilogue(M, inter, K, act):
    """act(gate) * up in the product's epilogue equals the library product followed by the activation kernel,
    bit for bit without a bias (the same sums rounded at the same places)."""
    from liteinfer_b200 import ops

    dt = torch.bfloat16
    x = _randn(M, K, dtype=dt)
    w = _interleave(_randn(inter, K, dtype=dt, seed=1, scale=0.05), _randn(inter, K, dtype=dt, seed=2, scale=0.05))
    got = ops.gemm_tcgen05(x, w, torch.empty(M, inter, dtype=dt, device="cuda"), None, act)
    gu = ops.linear(x, w, torch.empty(M, 2 * inter, dtype=dt, device="cuda"))
    two = ops.act_mul_interleaved(gu, torch.empty(M, inter, dtype=dt, device="cuda"), act)
    assert ops.gemm_error_flag("cuda:0") == 0
    # the library may add its products in another order: a rounding of the bfloat16 product apart at most
    torch.testing.assert_close(got.float(), two.float(), rtol=2 ** -6, atol=2 ** -6)


@pytest.mark.parametrize("heads,kv_heads,page_size", [(4, 1, 16), (32, 8, 16), (8, 8, 32), (16, 2, 64), (128, 1, 16),
                                                      (24, 8, 16), (5, 1, 32), (7, 7, 16)])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("d", [64, 128])
def test_tcgen05_attention_against_the_plain_kernel(heads, kv_heads, page_size, window, d, monkeypatch):
    """The tcgen05 / TMA / tensor-memory attention kernel: portions, whole prompts and single tokens over shuffled
    pages, NaN in every slot no request owns, contexts that straddle the 64-key tiles; no wait may give up."""
    from liteinfer_b200 import ops

    q_lens, ctx_lens = [1, 130, 1, 7, 64, 2, 257], [700, 190, 1, 7, 64, 129, 300]
    case = _paged_case(torch.bfloat16, heads, kv_heads, d, page_size, q_lens, ctx_lens)
    qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
    ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads, d, 0)
    rest = (k_pool, v_pool, case["table"], case["qsl"], case["ctx"])
    tail = (case["B"], max(q_lens), heads, kv_heads, d, d ** -0.5, window)
    want = ref.paged_attention(qkv, qkv.shape[1], torch.empty(case["T"], heads * d, dtype=torch.bfloat16, device="cuda"),
                               *rest, *tail)
    out = torch.full((case["T"], heads * d), float("nan"), dtype=torch.bfloat16, device="cuda")
    assert ops.tcgen05_attention_supports(torch.bfloat16, heads, kv_heads, d, page_size)
    ops.paged_attention_tcgen05(qkv, qkv.shape[1], out, *rest, None, *tail)
    assert ops.gemm_error_flag("cuda:0") == 0
    assert torch.isfinite(out.float()).all()
    torch.testing.assert_close(out.float(), want.float(), rtol=2 ** -6, atol=2 ** -6)


def test_tcgen05_attention_refuses_what_it_cannot_do():
    from liteinfer_b200 import ops

    assert not ops.tcgen05_attention_supports(torch.bfloat16, 129, 1, 64, 16)    # a group larger than a block's rows
    assert not ops.tcgen05_attention_supports(torch.bfloat16, 4, 2, 96, 16)      # head size 96: the plain kernel
    assert not ops.tcgen05_attention_supports(torch.bfloat16, 4, 2, 64, 8)       # pages of 8
    assert not ops.tcgen05_attention_supports(torch.float32, 4, 2, 64, 16)


@pytest.mark.parametrize("M", [1, 5, 8, 13])
@pytest.mark.parametrize("N,K", [(3072, 2048), (2048, 8192), (1000, 96), (64, 32768)])
def test_streaming_product_adds_into_the_residual_stream(M, N, K, monkeypatch):
    """With `residual` the weight-streaming kernel adds its result into the stream itself (the same bits as the
    product followed by the 32-bit sum rounded once) and leaves the new rows' sums of squares in parts."""
    from liteinfer_b200 import ops

    monkeypatch.setattr(ops.kernels, "FUSED_NORM", True)       # the fusion is a switch (off by default)
    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    b = _randn(N, dtype=torch.bfloat16, seed=2)
    stream = _randn(M, N, dtype=torch.bfloat16, seed=3, scale=2.0)
    product = ops.linear(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), b)
    want = (stream.float() + product.float()).to(torch.bfloat16)
    got = stream.clone()
    stats = ops.linear(x, w, None, b, residual=got)
    assert isinstance(stats, ops.RowStats) and stats.sumsq.shape == (-(-N // 16), M)
    assert torch.equal(got, want)
    torch.testing.assert_close(stats.sumsq.sum(0), want.float().pow(2).sum(-1), rtol=1e-5, atol=1e-5)
    again = stream.clone()
    assert torch.equal(ops.linear(x, w, None, b, residual=again).sumsq, stats.sumsq) and torch.equal(again, got)


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K,gated", [(3072, 2048, False), (16384, 2048, True), (1000, 96, False), (352, 64, True),
                                       (128256 // 4, 2048, False)])
def test_streaming_product_folds_the_norm_in(M, N, K, gated):
    """A pending norm as the product's input: weight * x / rms(x) with the statistics from the parts that the
    product before left, for all rows or for rows picked by index; against the norm kernel followed by the
    product, within bfloat16 rounding (the fused form rounds once less), and against float64."""
    from liteinfer_b200 import ops

    rows_total = M + 3
    hidden = _randn(rows_total, K, dtype=torch.bfloat16, seed=4, scale=3.0)
    wn = (1 + 0.1 * _randn(K, dtype=torch.float32, seed=5)).to(torch.bfloat16)
    w = _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.02)          # results of magnitude one
    # the statistics as a product of 7 column tiles would have left them
    parts = torch.stack([c.float().pow(2).sum(-1) for c in hidden.chunk(7, dim=1)])
    for rows in (None, torch.tensor(list(range(rows_total - 1, rows_total - 1 - M, -1)), dtype=torch.int32, device="cuda")):
        if rows is None:
            source, stats = hidden[:M].contiguous(), ops.RowStats(parts[:, :M].contiguous())
        else:
            source, stats = hidden, ops.RowStats(parts.contiguous())
        pending = ops.PendingNorm(source, wn, 1e-5, stats, rows)
        normed = pending.materialise()
        picked = source if rows is None else source[rows.long()]
        exact = (picked.double() / torch.sqrt(picked.double().pow(2).mean(-1, keepdim=True) + 1e-5)) * wn.double()
        if gated:
            got = ops.gated_linear(pending, w, torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda"), "silu")
            two = ops.gated_linear(normed, w, torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda"), "silu")
        else:
            got = ops.linear(pending, w, None)
            two = ops.linear(normed, w, None)
            torch.testing.assert_close(got.double(), exact @ w.double().t(), rtol=2 ** -6, atol=2 ** -6)
        # (the two-kernel form rounds the normalised row once more than the fused one: each is within a rounding of
        # the exact product, so they are within two of each other)
        torch.testing.assert_close(got.float(), two.float(), rtol=2 ** -5, atol=2 ** -5)


def test_fused_decode_layer_chain_matches_the_unfused_one(monkeypatch):
    """Norm -> product -> residual -> norm -> gated product -> product -> residual, as a decode step of five
    tokens runs it (two fused products per half layer), against the same chain kernel by kernel."""
    from liteinfer_b200.parts.block import apply_norm, run_part
    from liteinfer_b200.parts.feed_forward import GatedMLP
    from liteinfer_b200.parts.norm import RMSNorm
    from liteinfer_b200 import ops

    dev, dt, h, inter = torch.device("cuda:0"), torch.bfloat16, 256, 512
    norm = RMSNorm(h, 1e-5, dt, dev)
    hidden = _randn(5, h, dtype=dt, seed=2)
    norm.bind({"weight": (1 + 0.1 * _randn(h, dtype=torch.float32, seed=1)).to(dt)})
    mlp = GatedMLP(h, inter, "silu", dt, dev)
    mlp.bind({n: _randn(*s.shape, dtype=dt, seed=10 + i, scale=0.05) for i, (n, s) in enumerate(mlp.tensor_specs().items())})
    # unfused: materialised norms, deltas added by the next norm
    a = hidden.clone()
    d1 = mlp.forward(norm.forward(a, None), None)
    d2 = mlp.forward(norm.forward(a, d1), None)
    want = (a.float() + d2.float())
    # fused: the parts add into the stream and hand on statistics
    monkeypatch.setattr(ops.kernels, "FUSED_NORM", True)
    b = hidden.clone()
    s1 = run_part(mlp, apply_norm(norm, b, None, mlp), b, None)
    assert isinstance(s1, ops.RowStats)
    pending = apply_norm(norm, b, s1, mlp)
    assert isinstance(pending, ops.PendingNorm)
    s2 = run_part(mlp, pending, b, None)
    assert isinstance(s2, ops.RowStats)
    torch.testing.assert_close(b.float(), want, rtol=2 ** -6, atol=2 ** -6)
    torch.testing.assert_close(s2.sumsq.sum(0), b.float().pow(2).sum(-1), rtol=1e-5, atol=1e-5)


# More tiles than two for every SM with rows of 19 to 24 chunks of 128 k, of 25 to 32 and of more; and very many tiles; short rows
# in rounds of tiles that one block of eight warps and two of six take alike, and that they do not.
@pytest.mark.parametrize("M", [1, 8, 9])
@pytest.mark.parametrize("N,K", [(4752, 2312), (6144, 3072), (5001, 3080), (9000, 4096), (4752, 4104), (57000, 2440),
                                 (8000, 2312), (14208, 2560), (17600, 2440), (8000, 2816)])
def test_gemm_stream_of_long_rows(M, N, K):
    from liteinfer_b200 import ops

    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    b = _randn(N, dtype=torch.bfloat16, seed=2)
    got = ops.gemm_stream(x, w, torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), b)
    torch.testing.assert_close(got.double(), x.double() @ w.double().t() + b.double(), rtol=2 ** -7, atol=2 ** -7)
    if N % 16 == 0:
        pairs = (x.double() @ w.double().t()).view(M, -1, 2, 8).bfloat16().double()
        want = (pairs[:, :, 0] * torch.sigmoid(pairs[:, :, 0])).bfloat16().double() * pairs[:, :, 1]
        got = ops.gemm_stream(x, w, torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda"), None, "silu")
        # Both factors are rounded to 2^-8 of themselves, the gate's through an activation of slope up to 1.1, and their product.
        torch.testing.assert_close(got.double(), want.flatten(1), rtol=2 ** -5, atol=2 ** -6)
    assert ops.gemm_error_flag("cuda:0") == 0


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(3072, 2048), (2048, 8192), (1000, 96), (17, 40), (128256 // 8, 2048), (48, 16384),
                                 (16384, 2048), (5000, 200)])
def test_gemm_stream(M, N, K):
    """The persistent product with per-warp TMA rings against a float64 product: tiles past N, chunks past K (a k
    that is no multiple of 128, of 64, or smaller than one chunk), more tiles than blocks and fewer."""
    from liteinfer_b200 import ops

    x, w = _randn(M, K, dtype=torch.bfloat16), _randn(N, K, dtype=torch.bfloat16, seed=1, scale=0.05)
    b = _randn(N, dtype=torch.bfloat16, seed=2)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    got = ops.gemm_stream(x, w, out, b)
    want = x.double() @ w.double().t() + b.double()
    assert ops.gemm_error_flag("cuda:0") == 0
    torch.testing.assert_close(got.double(), want, rtol=2 ** -7, atol=2 ** -6 if K > 4096 else 2 ** -7)
    again = ops.gemm_stream(x, w, torch.empty_like(out), b)
    assert torch.equal(got, again)


def test_gemm_stream_rows_do_not_depend_on_the_batch():
    from liteinfer_b200 import ops

    x, w = _randn(16, 2048, dtype=torch.bfloat16), _randn(555, 2048, dtype=torch.bfloat16, seed=1, scale=0.05)
    full = ops.gemm_stream(x, w, torch.empty(16, 555, dtype=torch.bfloat16, device="cuda"))
    for rows in (1, 5, 8, 12):
        part = ops.gemm_stream(x[:rows].contiguous(), w, torch.empty(rows, 555, dtype=torch.bfloat16, device="cuda"))
        assert torch.equal(part, full[:rows])


@pytest.mark.parametrize("M", [1, 8, 13])
@pytest.mark.parametrize("inter,K,act", [(8192, 2048, "silu"), (112, 120, "gelu_pytorch_tanh"), (176, 64, "relu")])
def test_gemm_stream_epilogues(M, inter, K, act):
    """act(gate) * up in the epilogue equals the product followed by the activation kernel; the residual sum equals
    the product followed by a 32-bit sum rounded once, and leaves the sums of squares of the new rows."""
    from liteinfer_b200 import ops

    dt = torch.bfloat16
    x = _randn(M, K, dtype=dt)
    w = _interleave(_randn(inter, K, dtype=dt, seed=1, scale=0.05), _randn(inter, K, dtype=dt, seed=2, scale=0.05))
    b = _interleave(_randn(inter, dtype=dt, seed=3), _randn(inter, dtype=dt, seed=4))
    gu = ops.gemm_stream(x, w, torch.empty(M, 2 * inter, dtype=dt, device="cuda"), b)
    two = ops.act_mul_interleaved(gu, torch.empty(M, inter, dtype=dt, device="cuda"), act)
    got = ops.gemm_stream(x, w, torch.empty(M, inter, dtype=dt, device="cuda"), b, act)
    assert torch.equal(got, two)
    stream = _randn(M, 2 * inter, dtype=dt, seed=9, scale=2.0)
    want = (stream.float() + gu.float()).to(dt)
    stats = ops.gemm_stream(x, w, None, b, residual=stream)
    assert torch.equal(stream, want)
    torch.testing.assert_close(stats.sumsq.sum(0), want.float().pow(2).sum(-1), rtol=1e-5, atol=1e-5)
    assert ops.gemm_error_flag("cuda:0") == 0


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("w,ctx", [(11, 50), (64, 129), (65, 129), (16, 81), (100, 700)])
def test_window_edge_on_the_tensor_core_paths(d, w, ctx, monkeypatch):
    """With a window of w the key at distance w - 1 is seen and the key at distance w is not, on every path that
    bfloat16 heads of 64 and 128 take: single tokens with their keys unsplit and split, through the kernel with
    TMA rings and the one with shared-memory tiles, with the rotary encoding and the cache write fused in, and a
    portion of three tokens through the tcgen05 kernel.  The edge falls inside a tile of 64 keys, on its first key,
    on its last, and on a page's edge."""
    from liteinfer_b200 import ops

    heads, kv_heads, page, dt = 8, 2, 16, torch.bfloat16
    inv_freq = (1.0 / (500000.0 ** (torch.arange(0, d, 2).float() / d))).cuda()

    def planted(q_len, distance, rotate):
        case = _paged_case(dt, heads, kv_heads, d, page, [q_len], [ctx], seed=w + distance, poison=False)
        qkv, k_pool, v_pool = case["qkv"], case["k_pool"], case["v_pool"]
        rotated = qkv.clone()          # what the queries look like once they are rotated (or not)
        ref.rope_kv_write(rotated, case["positions"], case["seq_of"], case["table"], k_pool.clone(), v_pool.clone(),
                          inv_freq if rotate else None, heads, kv_heads, d, d if rotate else 0, store=False)
        far = ctx - 1 - distance
        pg, off = int(case["table"][0, far // page]), far % page
        last = rotated[q_len - 1, :heads * d].view(heads, d)
        for h in range(kv_heads):
            k_pool[pg, h, off] = (last[h * (heads // kv_heads)].float() * 10).to(dt)
            v_pool[pg, h, off] = 100.0
        return case, qkv, k_pool, v_pool

    def sees(out, q_len):
        return float(out[q_len - 1].view(heads, d)[0].float().mean()) > 50

    for distance, seen in ((w - 1, True), (w, False)):
        # single tokens, keys and values already in their pages
        for stream in ("1", "0"):
            monkeypatch.setenv("LITEINFER_DECODE_STREAM", stream)
            for splits in (1, 3):
                case, qkv, k_pool, v_pool = planted(1, distance, False)
                ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads,
                                  kv_heads, d, 0)
                out = torch.empty(1, heads * d, dtype=dt, device="cuda")
                ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 1,
                                    heads, kv_heads, d, 1.0, w, plan=_plan_for([1], [ctx]), decode_splits=splits)
                assert sees(out, 1) == seen, (stream, splits, distance)
        monkeypatch.setenv("LITEINFER_DECODE_STREAM", "1")
        # the rotary encoding and the cache write inside the attention launch
        for splits in (1, 3):
            case, qkv, k_pool, v_pool = planted(1, distance, True)
            q_width, kv_width = heads * d, kv_heads * d
            newest = ops.NewestToken(inv_freq, qkv[:, q_width:], qkv[:, q_width + kv_width:])
            out = torch.empty(1, heads * d, dtype=dt, device="cuda")
            ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 1,
                                heads, kv_heads, d, 1.0, w, plan=_plan_for([1], [ctx]), decode_splits=splits, newest=newest)
            assert sees(out, 1) == seen, ("fused", splits, distance)
        # a portion of three tokens: the tcgen05 kernel
        case, qkv, k_pool, v_pool = planted(3, distance, False)
        ops.rope_kv_write(qkv, case["positions"], case["seq_of"], case["table"], k_pool, v_pool, None, heads, kv_heads, d, 0)
        assert ctx - 1 - distance < ctx - 3      # the planted key lies before the portion's own keys
        out = torch.empty(3, heads * d, dtype=dt, device="cuda")
        assert ops.tcgen05_attention_supports(dt, heads, kv_heads, d, page)
        ops.paged_attention(qkv, qkv.shape[1], out, k_pool, v_pool, case["table"], case["qsl"], case["ctx"], 1, 3,
                            heads, kv_heads, d, 1.0, w, plan=_plan_for([3], [ctx]))
        assert sees(out, 3) == seen, ("portion", distance)
    assert ops.gemm_error_flag("cuda:0") == 0
