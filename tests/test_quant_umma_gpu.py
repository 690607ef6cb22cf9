"""Raw GGUF blocks through the tensor cores (`csrc/kernels/quant_umma.cu`) against the dequantised weights in 64 bits: edges of the
row and column tiles, one and many blocks, parts of K, ragged and empty groups."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _raw(name, rows, K, seed):
    from pocketllm_b200.formats import gguf_quants as gq
    w = (np.random.default_rng(seed).standard_normal((rows, K)) * 0.02).astype(np.float32)
    blocks = gq.quantize(w, name)
    return torch.from_numpy(blocks).cuda().view(-1), torch.from_numpy(gq.dequantize(blocks, name).reshape(rows, K)).cuda().double()


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


# products are exact and sums fp32 (a few hundred terms to a block, a few blocks): 2^-24 * sqrt(K) / 2 at most, 1e-6 at K = 3072
TOL = 1e-6


@pytest.mark.parametrize("name", ["iq2_xxs", "q4_k", "q5_k"])
@pytest.mark.parametrize("M,N,K", [(1, 128, 256), (1, 300, 3072), (5, 64, 768), (16, 129, 1536), (17, 256, 512), (33, 130, 1280), (64, 2, 2304), (65, 384, 1024), (128, 200, 256), (256, 130, 512)])
def test_linear(name, M, N, K):
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw(name, N, K, M + N)
    g = torch.Generator("cuda").manual_seed(K)
    x = torch.randn(M, K, device="cuda", generator=g) * torch.logspace(-4, 4, M, device="cuda")[:, None]
    x = x.to(torch.bfloat16)
    assert _rel(go.gguf_linear(x, raw, name, N, epi=2), x.double() @ w.T) < TOL
    gamma = 1 + 0.1 * torch.randn(K, device="cuda", generator=g)
    n = (x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6) * gamma).to(torch.bfloat16).double()
    # a norm that rounds to the other side of a bf16 tie: a part of the values by 2^-8 at most
    assert _rel(go.gguf_linear(x, raw, name, N, gamma=gamma, epi=2), n @ w.T) < 2e-4
    assert _rel(go.gguf_linear(x, raw, name, N), x.double() @ w.T) < 2 ** -8
    if N % 2 == 0:
        z = x[:, :].double() / x.double().norm(dim=1, keepdim=True) * 30
        xs = z.to(torch.bfloat16)
        a, b = (xs.double() @ w.T).chunk(2, -1)
        assert _rel(go.gguf_linear(xs, raw, name, N, epi=1), torch.nn.functional.silu(a) * b) < 2 ** -8


@pytest.mark.parametrize("name", ["iq2_xxs", "q4_k", "q5_k"])
@pytest.mark.parametrize("M,N,K", [(1, 128, 256), (1, 300, 3072), (5, 64, 768), (8, 2, 2304)])
def test_few_rows_of_small_weights_on_the_tensor_cores(name, M, N, K):
    """Sizes that `gguf_linear` decodes in registers, in the kernel all the same; zeros and infinities too."""
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw(name, N, K, M + N)
    g = torch.Generator("cuda").manual_seed(K)
    x = (torch.randn(M, K, device="cuda", generator=g) * torch.logspace(-4, 4, M, device="cuda")[:, None]).to(torch.bfloat16)
    gamma = 1 + 0.1 * torch.randn(K, device="cuda", generator=g)
    run = lambda x, gamma=None, epi=2: go._umma_linear(x, raw, name, N, gamma, 1e-6, epi, None)
    n = (x.float() * torch.rsqrt((x.float() ** 2).mean(-1, keepdim=True) + 1e-6) * gamma).to(torch.bfloat16).double()
    assert _rel(run(x), x.double() @ w.T) < TOL and _rel(run(x, gamma), n @ w.T) < 2e-4 and _rel(run(x, epi=0), x.double() @ w.T) < 2 ** -8
    x[0] = 0
    x[-1, 3] = float("inf") if M > 1 else 0.0
    y = run(x)
    assert (y[0] == 0).all() and (M == 1 or (not torch.isfinite(y[-1]).any() and _rel(y[1:-1], x[1:-1].double() @ w.T) < TOL))


@pytest.mark.parametrize("name", ["iq2_xxs", "q4_k", "q5_k"])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 8, 9])
def test_linear_on_both_sides_of_the_rule(name, M):
    """Weights of the last size that few rows decode in registers, and one block row more."""
    from pocketllm_b200.ops import gguf_ops as go
    K, N = 8192, (1 << 24 if name != "iq2_xxs" or M > 2 else 1 << 25) // (1 << (M - 1).bit_length()) // 8192
    raw, w = _raw(name, 32, K, M)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    for n in (N, N + 32):
        assert go._registers_faster(name, M, n * K) == (n == N and M <= 8)
        y = go.gguf_linear(x, raw.repeat(n // 32), name, n, epi=2).view(M, n // 32, 32)
        want = x.double() @ w.T
        assert _rel(y[:, 0], want) < TOL and torch.equal(y[:, :1].expand_as(y), y)


@pytest.mark.parametrize("name", ["iq2_xxs", "q4_k", "q5_k"])
@pytest.mark.parametrize("M,N", [(256, 2048), (257, 2048), (384, 2080), (385, 2080)])
def test_linear_on_both_sides_of_the_row_limits(name, M, N):
    """Up to 2^24 weights 256 rows are the most, above 384; beyond that the weight is rounded to bf16, whose 2^-9 a sum takes over."""
    from pocketllm_b200.ops import gguf_ops as go
    K = 8192
    raw, w = _raw(name, 32, K, M)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    y = go.gguf_linear(x, raw.repeat(N // 32), name, N, epi=2).view(M, N // 32, 32)
    inside = M < (go.UMMA_MAX_ROWS if N * K <= 1 << 24 else go.UMMA_MAX_ROWS_LARGE)
    assert inside == (M in (256, 384))
    want = (x.double() @ w.T)[:, None].expand(-1, N // 32, -1)
    assert _rel(y, want) < (TOL if inside else 2 ** -8)


def test_linear_rows_of_zeros_and_infinities():
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw("q5_k", 256, 512, 0)
    x = torch.randn(4, 512, device="cuda").to(torch.bfloat16)
    x[1] = 0
    x[2, 7] = float("inf")
    x[3] *= 2.0 ** 100
    y = go.gguf_linear(x, raw, "q5_k", 256, epi=2)
    assert (y[1] == 0).all() and not torch.isfinite(y[2]).any()
    assert _rel(y[0], x[0].double() @ w.T) < TOL and _rel(y[3], x[3].double() @ w.T) < TOL


def test_one_row_of_any_stride():
    """A single row is contiguous whatever its row stride says."""
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw("q5_k", 520, 512, 3)
    x = torch.randn(512, 1, device="cuda").to(torch.bfloat16).t()
    assert x.stride(0) == 1 and x.is_contiguous()
    assert _rel(go.gguf_linear(x, raw, "q5_k", 520, epi=2), x.double() @ w.T) < TOL
    assert _rel(go._umma_linear(x, raw, "q5_k", 520, None, 0.0, 2, None), x.double() @ w.T) < TOL


@pytest.mark.parametrize("M", [1, 20])
def test_first_rows_of_a_longer_buffer(M):
    """An odd number of IQ2 blocks is no whole number of words, the buffer behind it is."""
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw("iq2_xxs", 130, 256, 4)
    x = torch.randn(M, 256, device="cuda").to(torch.bfloat16)
    assert raw.numel() % 4 == 0
    assert _rel(go.gguf_linear(x, raw, "iq2_xxs", 129, epi=2), x.double() @ w[:129].T) < TOL


@pytest.mark.parametrize("t13,t2", [("iq2_xxs", "iq2_xxs"), ("q4_k", "iq2_xxs"), ("iq2_xxs", "q5_k")])
@pytest.mark.parametrize("T,E,topk,limit", [(1, 16, 4, 0.0), (9, 40, 3, 0.0), (17, 40, 4, 0.0), (33, 40, 3, 0.0), (90, 8, 2, 0.5), (300, 5, 2, 0.0)])
def test_experts(t13, t2, T, E, topk, limit):
    from pocketllm_b200.ops import gguf_ops as go
    H, I = 512, 256 + 512 * (T % 2)
    raw13, w13 = _raw(t13, E * 2 * I, H, 1)
    raw2, w2 = _raw(t2, E * H, I, 2)
    w13, w2 = w13.view(E, 2 * I, H), w2.view(E, H, I)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    # the last expert gets nothing, the first one more than the others
    ids = torch.stack([torch.randperm(E - 1, generator=g)[:topk] for _ in range(T)]).int()
    ids[::2, 0] = torch.where((ids[::2, 1:] == 0).any(-1), ids[::2, 0], torch.zeros_like(ids[::2, 0]))
    weight = torch.rand(T, topk, generator=g)
    ids, weight = ids.cuda(), weight.cuda()
    routes = go.group_routes(ids, weight, E)

    def exact(lo, hi):
        y = torch.zeros(T, H, device="cuda", dtype=torch.float64)
        for e in range(lo, hi):
            t, j = (ids == e).nonzero(as_tuple=True)
            a, b = (x[t].double() @ w13[e].T).chunk(2, -1)
            if limit:
                a, b = a.clamp(max=limit), b.clamp(-limit, limit)
            y.index_add_(0, t, weight[t, j, None].double() * ((torch.nn.functional.silu(a) * b) @ w2[e].T))
        return y

    run = lambda **k: go.gguf_moe_forward(x, k.pop("a", raw13), k.pop("b", raw2), t13, t2, E, I, *routes, limit=limit, routes=routes, **k)
    # fp32 sums and the exponential of a SiLU; hidden values in two fp16 terms (2^-22)
    want = exact(0, E)
    assert _rel(run(), want) < 2e-6
    half = E // 2
    n13, n2 = raw13.numel() // E * half, raw2.numel() // E * half
    assert _rel(run(a=raw13[:n13], b=raw2[:n2], local_experts=half), exact(0, half)) < 2e-6
    assert _rel(run(a=raw13[n13:].clone(), b=raw2[n2:].clone(), expert_offset=half, local_experts=E - half), exact(half, E)) < 2e-6
    if not limit:       # hidden values in one fp16 term
        assert _rel(go.gguf_moe_forward_grouped(x, raw13, raw2, t13, t2, E, I, routes), want) < 5e-4


@pytest.mark.parametrize("t13,t2,E,topk,H,I", [("iq2_xxs", "iq2_xxs", 64, 8, 1536, 768), ("q4_k", "q5_k", 16, 2, 2048, 1280), ("iq2_xxs", "q4_k", 40, 3, 3072, 512)])
def test_a_token_gives_the_same_bits_in_any_company(t13, t2, E, topk, H, I):
    """One token alone (K in parts over CTAs) and the same token among others (all parts in one CTA), up to the four routes per expert
    from which prompts take the grouped form."""
    from pocketllm_b200.ops import gguf_ops as go
    def raw(name, rows, K, seed):        # any payload, scale fields 2^-11
        n = {"iq2_xxs": 66, "q4_k": 144, "q5_k": 176}[name]
        b = torch.randint(0, 256, (rows * K // 256, n), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        b[:, :2 if name == "iq2_xxs" else 4] = torch.tensor([0, 0x10] * (1 if name == "iq2_xxs" else 2), dtype=torch.uint8)
        return b.view(-1)

    raw13, raw2 = raw(t13, E * 2 * I, H, 1), raw(t2, E * H, I, 2)
    g = torch.Generator().manual_seed(0)
    T = 4 * E // topk
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(E, generator=g)[:topk] for _ in range(T)]).int().cuda()
    weight = torch.rand(T, topk, generator=g).cuda()
    assert go._umma_splits(topk * (2 * I // 128), H, go._umma_slots(t13, 16)) > 1

    def run(n, **k):
        routes = go.group_routes(ids[:n].contiguous(), weight[:n].contiguous(), E)
        return go.gguf_moe_forward(x[:n].contiguous(), k.pop("a", raw13), k.pop("b", raw2), t13, t2, E, I, *routes, routes=routes, **k)

    half, n13, n2 = E // 2, raw13.numel() // 2, raw2.numel() // 2
    for kw in ({}, dict(a=raw13[n13:].clone(), b=raw2[n2:].clone(), expert_offset=half, local_experts=half)):
        alone = run(1, **kw)
        for n in (2, 3, 5, 8, 17, T):
            assert torch.equal(run(n, **kw)[:1], alone), n


@pytest.mark.parametrize("t13,t2,E,topk,H,I,cut", [("iq2_xxs", "iq2_xxs", 64, 8, 1536, 768, (False, False)), ("iq2_xxs", "iq2_xxs", 64, 2, 4096, 1024, (True, False)),
                                                   ("iq2_xxs", "iq2_xxs", 64, 2, 1024, 3072, (False, True)),
                                                   ("q4_k", "q5_k", 16, 2, 2048, 1280, (True, False)), ("iq2_xxs", "q4_k", 40, 3, 3072, 512, (True, False))])
def test_a_token_in_any_company_and_the_parts_of_its_products(t13, t2, E, topk, H, I, cut, monkeypatch):
    """One token alone (K in parts over CTAs) and the same token among others (all parts in one CTA), up to the four routes per expert
    from which prompts take the grouped form."""
    from pocketllm_b200.ops import gguf_ops as go
    def raw(name, rows, K, seed):        # any payload, scale fields 2^-11
        n = {"iq2_xxs": 66, "q4_k": 144, "q5_k": 176}[name]
        b = torch.randint(0, 256, (rows * K // 256, n), dtype=torch.uint8, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        b[:, :2 if name == "iq2_xxs" else 4] = torch.tensor([0, 0x10] * (1 if name == "iq2_xxs" else 2), dtype=torch.uint8)
        return b.view(-1)

    raw13, raw2 = raw(t13, E * 2 * I, H, 1), raw(t2, E * H, I, 2)
    g = torch.Generator().manual_seed(0)
    T = 4 * E // topk
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(E, generator=g)[:topk] for _ in range(T)]).int().cuda()
    weight = torch.rand(T, topk, generator=g).cuda()
    calls, product = [], go._umma
    monkeypatch.setattr(go, "_umma", lambda *a: (calls.append(a[10:13]), product(*a)))      # columns, parts, splits

    def run(n, **k):
        routes = go.group_routes(ids[:n].contiguous(), weight[:n].contiguous(), E)
        return go.gguf_moe_forward(x[:n].contiguous(), k.pop("a", raw13), k.pop("b", raw2), t13, t2, E, I, *routes, routes=routes, **k)

    half, n13, n2 = E // 2, raw13.numel() // 2, raw2.numel() // 2
    for kw in ({}, dict(a=raw13[n13:].clone(), b=raw2[n2:].clone(), expert_offset=half, local_experts=half)):
        calls.clear()
        alone = run(1, **kw)
        assert [(c, p > 1, s == p) for c, p, s in calls] == [(16, b, True) for b in cut]      # which products are cut, into CTAs of their own
        for n in (2, 3, 5, 8, 17, T):
            calls.clear()
            assert torch.equal(run(n, **kw)[:1], alone), n
        assert [(c, p > 1, s) for c, p, s in calls] == [(16, b, 1) for b in cut]                # and with all tokens all parts are one CTA's


def _e4m3(x, w, scale, epi, resid, columns, splits, failed=0):
    from ctypes import c_float, c_int, c_void_p
    from pocketllm_b200 import ops
    M, K = x.shape
    N = w.shape[0]
    lib, null = ops._lib.kernels(), c_void_p(0)
    staged, factor = torch.empty(M, K, device="cuda", dtype=torch.float16), torch.empty(M, device="cuda")
    cols = N // 2 if epi == 1 else N
    y = torch.full((M, cols), float("nan"), device="cuda", dtype=torch.float32 if epi == 2 else torch.bfloat16)
    tiles = -(-N // 128) if epi != 1 else -(-(N // 2) // 64)
    ws, counters = torch.empty(max(1, tiles * splits * columns * 128), device="cuda"), torch.zeros(tiles, device="cuda", dtype=torch.int32)
    status = torch.full((1,), failed, device="cuda", dtype=torch.int32)
    ops._check(lib.pk_quant_stage_rows(ops._ptr(x), c_int(0), c_int(K), c_int(K), null, c_int(M), null, c_float(0), c_int(0), null, null, null, c_int(20), c_int(1),
                                       ops._ptr(staged), ops._ptr(factor), null, c_int(0), ops._stream()), "stage")
    if splits == 0:         # the kernel of up to 16 rows
        ops._check(lib.pk_rows_fp8(ops._ptr(w), ops._ptr(scale), c_int(K // 128), c_int(M), c_int(N), c_int(K), ops._ptr(staged), ops._ptr(factor), c_int(epi),
                                   ops._ptr(y), c_int(cols), ops._ptr(resid), c_int(ops._sm_count()), ops._stream()), "rows")
        return y
    for _ in range(2):      # the counters are zero again after a launch
        ops._check(lib.pk_quant_rows(ops._ptr(w), c_int(20), c_int(N), c_int(K), null, c_int(1), c_int(M), ops._ptr(staged), ops._ptr(factor), c_int(1), c_int(epi),
                                     ops._ptr(y), c_int(cols), ops._ptr(resid), c_float(0), c_int(columns), c_int(splits), c_int(splits), ops._ptr(ws), ops._ptr(counters),
                                     ops._ptr(status), ops._ptr(scale), c_int(K // 128), c_int(ops._sm_count()), ops._stream()), "rows")
    assert int(status) == failed and not counters.any()
    return y


@pytest.mark.parametrize("M,N,K,splits", [(3, 128, 128, 1), (16, 130, 640, 5), (17, 384, 1280, 3), (33, 40, 512, 2), (64, 512, 2176, 4), (5, 38400, 256, 1),
                                          (1, 16, 128, 0), (8, 130, 640, 0), (9, 40, 1280, 0), (16, 4112, 5120, 0), (5, 66, 17408, 0)])
def test_e4m3_blocks(M, N, K, splits):
    g = torch.Generator("cuda").manual_seed(M)
    w = (torch.randn(N, K, device="cuda", generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    scale = torch.rand(-(-N // 128), K // 128, device="cuda", generator=g) * 1e-3 + 1e-4
    wd = w.double() * scale.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    x = (torch.randn(M, K, device="cuda", generator=g) * torch.logspace(-2, 2, M, device="cuda")[:, None]).to(torch.bfloat16)
    resid = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16)
    columns = 32 if M <= 32 else 64
    want = x.double() @ wd.T
    assert _rel(_e4m3(x, w, scale, 2, None, columns, splits), want) < TOL
    assert _rel(_e4m3(x, w, scale, 0, None, columns, splits), want) < 2 ** -8
    assert _rel(_e4m3(x, w, scale, 4, resid, columns, splits), want + resid.double()) < 2 ** -8
    a, b = want.chunk(2, -1)
    assert _rel(_e4m3(x, w, scale, 1, None, columns, splits), torch.nn.functional.silu(a) * b) < 2 ** -8


@pytest.mark.parametrize("splits", [1, 3])
def test_after_a_wait_that_ran_out(splits):
    """A product that finds the error word set gives NaN in every place and leaves the counters of its parts at zero."""
    w = torch.randn(300, 768, device="cuda").to(torch.float8_e4m3fn)
    x, scale = torch.randn(20, 768, device="cuda").to(torch.bfloat16), torch.ones(3, 6, device="cuda")
    assert torch.isnan(_e4m3(x, w, scale, 2, None, 32, splits, failed=31)).all()
    assert torch.isnan(_e4m3(x, w, scale, 1, None, 32, splits, failed=31)).all()
    assert _rel(_e4m3(x, w, scale, 2, None, 32, splits), x.double() @ w.double().T) < TOL


@pytest.mark.parametrize("M", [1, 15, 17, 100])
@pytest.mark.parametrize("N,K", [(1, 64), (64, 576), (65, 5120), (128, 192)])
def test_narrow_linear(M, N, K):
    from ctypes import c_int
    from pocketllm_b200 import ops
    g = torch.Generator("cuda").manual_seed(M + N)
    x, w = (torch.randn(r, K, device="cuda", generator=g).to(torch.bfloat16) for r in (M, N))
    y = torch.full((M, N + 3), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops._check(ops._lib.kernels().pk_linear_narrow(ops._ptr(x), c_int(K), ops._ptr(w), c_int(M), c_int(N), c_int(K), ops._ptr(y), c_int(N + 3), ops._stream()), "narrow")
    assert _rel(y[:, :N], x.double() @ w.double().T) < 2 ** -8 and torch.isnan(y[:, N:]).all()


@pytest.mark.parametrize("T,topk,E", [(1, 8, 256), (3, 2, 5), (700, 8, 256), (129, 6, 2000), (40, 1, 11000), (1, 6, 2000), (2, 3, 65), (1, 4, 11999)])
def test_grouped_routes(T, topk, E):
    from pocketllm_b200.ops import gguf_ops as go
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, E, (T, topk), generator=g, dtype=torch.int32)
    ids[::3] = ids[0, 0]
    weight = torch.rand(T, topk, generator=g)
    routes = go.group_routes(ids.cuda(), weight.cuda(), E)
    order = torch.sort(ids.view(-1), stable=True).indices
    seg, tok, w = (t.cpu() for t in routes)
    assert torch.equal(seg[1:].long(), torch.bincount(ids.view(-1), minlength=E).cumsum(0)) and int(seg[0]) == 0
    assert torch.equal(routes.src.cpu().long(), order) and torch.equal(tok.long(), order // topk) and torch.equal(w, weight.view(-1)[order])


@pytest.mark.parametrize("T,E,H", [(1, 256, 3072), (3, 33, 1002), (9, 40, 1000), (127, 64, 256), (128, 60, 96), (130, 65, 3072), (300, 256, 1000), (281, 256, 96), (282, 256, 96), (1130, 64, 132), (2000, 40, 64)])
def test_router_logits(T, E, H):
    from pocketllm_b200.ops import gguf_ops as go
    g = torch.Generator("cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(E, H, device="cuda", generator=g) * H ** -0.5
    ids, weight = go.router_topk(x, w, 4, score_func="sigmoid", norm_topk=False)
    p = torch.sigmoid(x.double() @ w.double().T)
    top = p.topk(5, -1).values
    clear = ((top[:, :-1] - top[:, 1:]) > 1e-5).all(-1)          # a choice that fp32 sums decide as well
    assert clear.float().mean() > 0.9 and torch.equal(ids[clear].long(), p.topk(4, -1).indices[clear])
    assert (weight.double() - p.gather(1, ids.long())).abs().max() < 2e-6


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("N,K,split", [(8, 64, 0), (40, 128, 16), (130, 960, 0), (66, 4096, 32), (4112, 192, 0), (40, 512, 16), (24, 6144, 0), (300, 3072, 0), (16, 12544, 0)])
def test_bf16_rows(M, N, K, split):
    """Rows of whole steps of 64: fewer steps than the ring holds and more, K cut over warps, ragged groups, two inputs."""
    from pocketllm_b200.ops import mixer_ops as mo
    g = torch.Generator("cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    x, x2, w, st = r(M, K), r(M, K), r(N, K) * K ** -0.5, torch.zeros(1, device="cuda", dtype=torch.int32)
    want = x.double() @ w.double().T
    y = lambda n, dt: torch.full((M, n), float("nan"), device="cuda", dtype=dt)
    assert _rel(mo.linear(x, w, y(N, torch.float32), st), want) < TOL
    assert _rel(mo.linear(x, w, y(N, torch.bfloat16), st), want) < 2 ** -8
    a, b = want.chunk(2, -1)
    assert _rel(mo.linear(x, w, y(N // 2, torch.bfloat16), st, swiglu=True), torch.nn.functional.silu(a) * b) < 2 ** -8
    if split:
        want[:, split:] = x2.double() @ w[split:].double().T
        assert _rel(mo.linear2(x, x2, split, w, y(N, torch.float32), st), want) < TOL


@pytest.mark.parametrize("K", [4096, 14336])
def test_bf16_rows_round_their_sums(K):
    """Tensor cores cut sums off; a running sum of K values would be off by 2^-24 per 16 of them (5e-7 and 2e-6 here). Sums of 16 that
    are added with rounding stay within a few 2^-24."""
    from pocketllm_b200.ops import mixer_ops as mo
    g = torch.Generator("cuda").manual_seed(K)
    for x in (torch.randn(3, K, device="cuda", generator=g), torch.rand(3, K, device="cuda", generator=g)):
        x, w = x.to(torch.bfloat16), (torch.randn(256, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
        y = mo.linear(x, w, torch.empty(3, 256, device="cuda"), torch.zeros(1, device="cuda", dtype=torch.int32))
        assert _rel(y, x.double() @ w.double().T) < 4 * 2 ** -24


@pytest.mark.parametrize("M,K", [(1, 8), (300, 256), (3, 1016), (3, 1024), (2, 1028), (7, 3072), (2, 12296)])
@pytest.mark.parametrize("mode", [1, 2])
def test_rmsnorm_by_width(M, K, mode):
    """On both sides of the 16-byte form's rule, with a residual sum and without."""
    from pocketllm_b200 import ops
    g = torch.Generator("cuda").manual_seed(M + K)
    x, gamma, y = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16), torch.randn(K, device="cuda", generator=g), torch.randn(1, M, K, device="cuda", generator=g)
    h = torch.empty_like(x)
    scale = gamma.double() + (1 if mode == 1 else 0)
    norm = lambda v: v.double() * torch.rsqrt((v.double() ** 2).mean(-1, keepdim=True) + 1e-6) * scale
    assert _rel(ops.rmsnorm(x, gamma, mode=mode), norm(x)) < 2 ** -8
    out = ops.rmsnorm(x, gamma, mode=mode, parts=y, hidden_out=h)
    assert torch.equal(h, (x + y[0]).to(torch.bfloat16)) and _rel(out, norm(h)) < 2 ** -8


@pytest.mark.parametrize("name,N,K,rows,E", [("iq2_xxs", 130, 256, 40, 7), ("iq2_xxs", 2, 768, 25, 5), ("q4_k", 130, 512, 40, 7), ("iq2_xxs", 6, 256, 16500, 1), ("q5_k", 4, 256, 16500, 3)])
@pytest.mark.parametrize("columns", [16, 64])
def test_groups_at_any_place(name, N, K, rows, E, columns):
    """Groups that begin on any four bytes, and more token tiles than are looked up."""
    from ctypes import c_float, c_int, c_void_p
    from pocketllm_b200 import ops
    from pocketllm_b200.ops import gguf_ops as go
    raw, w = _raw(name, E * N, K, rows)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, K, generator=g).to(torch.bfloat16).cuda()
    cut = torch.sort(torch.randint(0, rows + 1, (E - 1,), generator=g)).values
    seg = torch.cat([torch.zeros(1, dtype=torch.long), cut, torch.tensor([rows])])
    st = go._Staged(x, name, rows, 1)
    for epi in (2, 3):
        y = torch.full((rows, N if epi == 2 else N // 2), float("nan"), device="cuda")
        go._umma(st, raw, name, N, K, seg.int().cuda(), E, epi, y, 0.0, columns, 1, 1, None)
        for e in range(E):
            a, b = int(seg[e]), int(seg[e + 1])
            want = x[a:b].double() @ w[e * N:(e + 1) * N].T
            if epi == 3:
                u, v = want.chunk(2, -1)
                want = torch.nn.functional.silu(u) * v
            assert a == b or _rel(y[a:b], want) < TOL * (1 if epi == 2 else 4)      # the exponential of a SiLU and its product


@pytest.mark.parametrize("name,M,N,K", [("q8_0", 64, 32768, 3072), ("q5_k", 400, 6400, 3072)])
def test_product_behind_the_decode_of_its_weight(name, M, N, K):
    """The decode to the scratch is the launch directly before the product (no norm, status given): a weight tile read before it is
    written has the NaN that the scratch is filled with, or the other weight. Weights are rounded to bf16: 2^-9 of each, 2^-8 of a sum."""
    from pocketllm_b200.ops import gguf_ops as go
    sides = []
    for seed in (M, M + 1):
        raw, w = _raw(name, 32, K, seed)
        x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
        sides.append((raw.repeat(N // 32), x, (x.double() @ w.T)[:, None].expand(-1, N // 32, -1)))
    status = torch.zeros(1, device="cuda", dtype=torch.int32)
    go.gguf_linear(sides[0][1], sides[0][0], name, N, epi=2, status=status)
    (scratch,) = (b for k, b in go._scratch.items() if k[1] == torch.cuda.current_stream().cuda_stream)
    for i in range(20):
        raw, x, want = sides[i % 2]
        if i % 4 < 2:
            scratch.fill_(float("nan"))
        y = go.gguf_linear(x, raw, name, N, epi=2, status=status)
        assert _rel(y.view(want.shape), want) < 2 ** -8
    assert status.item() == 0


def test_mixer_linear_behind_the_launch_that_makes_its_weight():
    """More than eight rows times a weight that the launch directly before writes over NaN."""
    from pocketllm_b200.ops import gguf_ops as go, mixer_ops as mo
    M, N, K = 20, 32768, 3072
    raw, w = _raw("q8_0", 32, K, 5)
    raw = raw.repeat(N // 32)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    want = (x.double() @ w.T)[:, None].expand(-1, N // 32, -1)
    y, status = torch.empty(M, N, device="cuda"), torch.zeros(1, device="cuda", dtype=torch.int32)
    scratch = go._dequant_scratch(raw, "q8_0", N, K)
    for _ in range(10):
        scratch.fill_(float("nan"))
        y.zero_()
        assert go._dequant_scratch(raw, "q8_0", N, K).data_ptr() == scratch.data_ptr()
        mo.linear(x, scratch, y, status)
        assert _rel(y.view(want.shape), want) < 2 ** -8
    assert status.item() == 0
