"""The float32 kernels of the 32-bit mode (the streaming product, attention of single tokens and of portions) against
float64 statements of the same operation, at the sizes where their tiles end."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24                         # unit roundoff of float32


def ops():
    from litellmengine_b200.csrc import ops as o
    return o


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (1, 5, 132), (2, 33, 128), (3, 100, 520), (4, 31, 1024), (5, 17, 8), (8, 4096, 4096),
                                   (7, 1000, 1540), (9, 64, 256), (13, 331, 2052), (16, 6144, 1024), (16, 3, 12288), (1, 70000, 16)])
def test_streaming_product(M, N, K):
    torch.manual_seed(M * 1000 + N)
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    ref = x.double() @ w.double().T
    got = ops().linear(x, w)
    assert got.dtype == torch.float32
    # a lane adds at most ceil(K / 128) * 4 products one by one, then at most 5 + 3 levels of a tree
    bound = (4 * -(-K // 128) + 9) * U * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - ref).abs() <= bound).all())
    assert torch.equal(ops().linear(x, w), got)
    if K > 4:
        w[N // 2, K - 1] = float("inf")                       # what a lane past the row's end must not multiply by zero
        bad = ops().linear(x, w)
        assert bool(torch.isinf(bad[:, N // 2]).all()) and bool(torch.isfinite(bad).sum() == M * (N - 1))


@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (17, 130, 72), (32, 128, 128), (33, 1000, 136), (64, 257, 520), (65, 300, 1000),
                                   (128, 4096, 512), (129, 31, 4096), (500, 1024, 2048), (2050, 160, 64)])
def test_tensor_core_product(M, N, K):
    """Tiles of 32, 64 and 128 tokens and 128 weight rows, blocks of 64 along K, whole and in parts."""
    torch.manual_seed(M * 1000 + N)
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    x[0, :8] *= 1e18                                          # a wide range of exponents in one sum
    w[0, :8] *= 1e-18
    ref = x.double() @ w.double().T
    got = ops().linear_f32_tcgen05(x, w)
    # what is left out of a product is at most 2^-24 of it, a block's 24 additions are cut at the last place, the blocks' sums rounded
    bound = (1.01 * U + 24 * 2 * U + -(-K // 64) * U) * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - ref).abs() <= bound).all())
    assert float((got - ref).norm() / ref.norm()) < 4e-7
    assert ops().stream_status(DEV).tolist() == [0, 0]
    if K >= 128 and M > 1 and N > 3:                           # infinities and NaN as plain multiply-adds give them
        x[1, 5], w[2, 70], w[3, 9] = float("inf"), float("-inf"), float("nan")
        x[0] = w[1] = 1e30
        lib, got = torch.mm(x, w.t()), ops().linear_f32_tcgen05(x, w)
        assert torch.equal(torch.isnan(got), torch.isnan(lib)) and torch.equal(torch.isinf(got), torch.isinf(lib))
        assert torch.equal(got[torch.isinf(got)], lib[torch.isinf(lib)])
        assert ops().stream_status(DEV).tolist() == [0, 0]


@pytest.mark.parametrize("M,N,K", [(17, 512, 64), (32, 130, 4096), (33, 257, 1024), (64, 300, 12288), (65, 512, 4096), (128, 512, 12288),
                                   (300, 9472, 512), (500, 1024, 4096)])
@pytest.mark.parametrize("kind", ["signed", "same", "cut"])
def test_tensor_core_product_is_as_near_as_float32_sums(M, N, K, kind):
    """Every row against 64 bits, for values of either sign, of one sign, and for values whose pieces, if they were cut instead of
    rounded, would leave out 2^-21 of every product.  A block's last additions are cut at the place of their sum, its smaller
    terms matter little, and the blocks' sums are rounded: 1 to 3 units of 2^-24 together.  A product without the third pieces is 2^-17 off."""
    g = torch.Generator(device=DEV).manual_seed(M * 1000 + K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    if kind == "same":
        x, w = x.abs(), w.abs()
    elif kind == "cut":
        x, w = torch.full_like(x, 1 + 2.0 ** -7 - 2.0 ** -23), torch.full_like(w, 1 + 2.0 ** -7 - 2.0 ** -23)
    ref = x.double() @ w.double().T
    error = lambda got: float(((got - ref).norm(dim=1) / ref.norm(dim=1)).max())
    assert error(ops().linear_f32_tcgen05(x, w)) < 5 * U
    # the largest numbers round to an infinity of bfloat16: those sums are made again, without the split
    x[1, 0], w[:, 0] = 3.4028234e38, 2.0 ** -120
    ref = x.double() @ w.double().T
    got = ops().linear_f32_tcgen05(x, w)
    assert float(((got[1] - ref[1]).abs() / ref[1].abs()).max()) < K * U and bool(torch.isfinite(got).all())
    others = [m for m in range(M) if m != 1]
    assert float(((got - ref)[others].norm(dim=1) / ref[others].norm(dim=1)).max()) < 5 * U
    assert ops().stream_status(DEV).tolist() == [0, 0]


def test_the_product_of_each_size_takes_its_path():
    o = ops()
    w = torch.randn(4096, 512, device=DEV)
    for rows, k in ((16, 512), (17, 512), (300, 512), (17, 508), (40, 256)):
        x, ww = torch.randn(rows, k, device=DEV), w[:, :k].contiguous()
        before = o.launch_count
        y = o.linear(x, ww)
        own = o.launch_count - before
        assert (own > 0) == (rows <= 16 or (k % 8 == 0 and ww.numel() >= o.F32_TENSOR_MIN_WEIGHTS)), (rows, k, own)
        ref = x.double() @ ww.double().t()
        assert float((y - ref).norm() / ref.norm()) < 2e-6


def pages_of(lens, nkv, d, page, g):
    width = max(-(-n // page) for n in lens)
    perm = torch.randperm(len(lens) * width + 2, generator=g)
    cache = torch.full((len(perm), 2, nkv, page, d), 33.0)
    table = torch.stack([perm[b * width:(b + 1) * width] for b in range(len(lens))]).to(torch.int32)
    ks, vs = [], []
    for b, n in enumerate(lens):
        k, v = torch.randn(n, nkv, d, generator=g), torch.randn(n, nkv, d, generator=g)
        j = torch.arange(n)
        cache[table[b, j // page].long(), 0, :, j % page] = k
        cache[table[b, j // page].long(), 1, :, j % page] = v
        ks.append(k), vs.append(v)
    return cache.to(DEV), table.to(DEV), ks, vs


def plain(q, k, v, pos, span, scale):
    """q [H, d] at `pos` over k, v [S, G, d] in float64; span as the kernels take it."""
    lo = max(0, pos - span + 1) if span and span > 0 else pos - pos % -span if span else 0
    rep = q.shape[0] // k.shape[1]
    kk, vv = (t[lo:pos + 1].double().repeat_interleave(rep, dim=1) for t in (k, v))
    p = torch.softmax(torch.einsum("hd,shd->hs", q.double(), kk) * scale, -1)
    return torch.einsum("hs,shd->hd", p, vv)


def tolerance(d, keys, scale_of_scores):
    """Rounding of a score (d products, then its exponential's argument) and of the sums over the keys."""
    return U * (8 * d ** 0.5 + 4 * scale_of_scores + 4 * math.sqrt(keys)) * 4


@pytest.mark.parametrize("nq,nkv,d,page", [(4, 4, 64, 16), (4, 2, 128, 16), (8, 2, 128, 5), (8, 1, 128, 16), (16, 2, 64, 64), (2, 2, 128, 1)])
@pytest.mark.parametrize("span", [None, 1, 37, -50])
@pytest.mark.parametrize("splits", [1, 3])
def test_single_tokens(nq, nkv, d, page, span, splits):
    g = torch.Generator().manual_seed(nq * 100 + d + page)
    lens = [1, 7, 8, 9, 63, 64, 65, 200, 313]
    cache, table, ks, vs = pages_of(lens, nkv, d, page, g)
    B, i32 = len(lens), lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q = torch.randn(B + 1, nq * d, generator=g).to(DEV)
    out, status = torch.zeros_like(q), i32([0, 0])
    # the rows in another order, with padding; one row belongs to nobody
    order = [r for r in range(B)][::-1]
    rows = i32([-1] + [r + 1 for r in order] + [-1])
    ops().attention_f32_decode(q, out, cache, rows, B + 2, i32([0] + [n - 1 for n in lens]), i32([0] + list(range(B))), i32(list(range(B))),
                               table, nq, nkv, d, page, span, d ** -0.5, splits, status)
    for b, n in enumerate(lens):
        ref = plain(q[b + 1].view(nq, d).cpu(), ks[b], vs[b], n - 1, span, d ** -0.5)
        err = float((out[b + 1].view(nq, d).double().cpu() - ref).abs().max())
        assert err <= tolerance(d, n, 6.0) * float(vs[b].abs().max()), (n, err)
    assert status.tolist() == [0, 0] and float(out[0].abs().max()) == 0.0


@pytest.mark.parametrize("nq,nkv,d,page", [(4, 4, 64, 16), (8, 2, 128, 16), (3, 1, 128, 5), (4, 2, 64, 1)])
@pytest.mark.parametrize("span", [None, 1, 70, -100])
def test_portions(nq, nkv, d, page, span):
    """(keys cached after the step, query rows at their end), around the edges of 64 and 128 rows and of 64 keys."""
    g = torch.Generator().manual_seed(nq * 100 + d + page)
    reqs = [(2, 2), (64, 64), (65, 65), (130, 129), (200, 3), (300, 127), (257, 257)]
    cache, table, ks, vs = pages_of([n for n, _ in reqs], nkv, d, page, g)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    T = sum(t for _, t in reqs)
    q = torch.randn(T, nq * d, generator=g).to(DEV)
    out, status, R = torch.zeros_like(q), i32([0, 0]), ops().PREFILL_TILE_ROWS
    starts = [sum(t for _, t in reqs[:i]) for i in range(len(reqs))]
    tiles = [(e, r) for e, (_, t) in enumerate(reqs) for r in range(0, t, R)][::-1] + [(-1, -1)]
    ops().attention_f32_prefill(q, out, cache, i32(tiles), len(tiles), i32(list(range(len(reqs)))), i32(starts), i32([t for _, t in reqs]),
                                i32([n for n, _ in reqs]), table, nq, nkv, d, page, span, d ** -0.5, status)
    for e, (n, t) in enumerate(reqs):
        for r in {0, 1, t // 2, min(63, t - 1), min(64, t - 1), t - 1}:
            ref = plain(q[starts[e] + r].view(nq, d).cpu(), ks[e], vs[e], n - t + r, span, d ** -0.5)
            err = float((out[starts[e] + r].view(nq, d).double().cpu() - ref).abs().max())
            assert err <= tolerance(d, n, 6.0) * float(vs[e].abs().max()), (n, t, r, err)
    assert status.tolist() == [0, 0]


@pytest.mark.parametrize("span", [None, 70, -100])
def test_a_value_that_is_not_finite_reaches_only_who_sees_it(span):
    """Infinities and NaN among the values of a portion: rows before them, or with their window behind them, stay finite."""
    g = torch.Generator().manual_seed(5)
    nq, nkv, d, page, n, t = 4, 2, 128, 16, 300, 250
    cache, table, ks, vs = pages_of([n], nkv, d, page, g)
    bad = {60: float("nan"), 200: float("inf"), 281: float("-inf")}
    for j, x in bad.items():
        cache[table[0, j // page].long(), 1, :, j % page] = x
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    q = torch.randn(t, nq * d, generator=g).to(DEV)
    out, status, R = torch.zeros_like(q), i32([0, 0]), ops().PREFILL_TILE_ROWS
    tiles = [(0, r) for r in range(0, t, R)][::-1]
    ops().attention_f32_prefill(q, out, cache, i32(tiles), len(tiles), i32([0]), i32([0]), i32([t]), i32([n]), table, nq, nkv, d, page, span,
                                d ** -0.5, status)
    for r in range(t):
        pos = n - t + r
        lo = max(0, pos - span + 1) if span and span > 0 else pos - pos % -span if span else 0
        seen = any(lo <= j <= pos for j in bad)
        assert bool(torch.isfinite(out[r]).all()) != seen, pos
        if not seen:
            ref = plain(q[r].view(nq, d).cpu(), ks[0], vs[0], pos, span, d ** -0.5)
            assert float((out[r].view(nq, d).double().cpu() - ref).abs().max()) <= tolerance(d, n, 6.0) * float(vs[0].abs().max()), pos


@pytest.mark.parametrize("splits", [1, 2])
def test_single_tokens_with_scores_of_minus_infinity(splits):
    """Keys whose product with the query overflows downwards weigh nothing, also where a warp meets nothing else at first."""
    g = torch.Generator().manual_seed(6)
    nq, nkv, d, page, n = 8, 2, 128, 16, 200
    cache, table, ks, vs = pages_of([n], nkv, d, page, g)
    far = [j for j in range(n) if j % 64 < 16 or j >= 184]
    for j in far:
        ks[0][j] = 0.0
        ks[0][j, :, 0] = -1e30
        cache[table[0, j // page].long(), 0, :, j % page] = ks[0][j].to(DEV)
    q = torch.randn(1, nq * d, generator=g)
    q.view(nq, d)[:, 0] = 1e10
    for j in set(range(n)) - set(far):
        ks[0][j, :, 0] = 0.0
        cache[table[0, j // page].long(), 0, :, j % page] = ks[0][j].to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    out, status = torch.zeros(1, nq * d, device=DEV), i32([0, 0])
    ops().attention_f32_decode(q.to(DEV), out, cache, None, 1, i32([n - 1]), i32([0]), i32([0]), table, nq, nkv, d, page, None, d ** -0.5,
                               splits, status)
    ref = plain(q[0].view(nq, d), ks[0], vs[0], n - 1, None, d ** -0.5)
    assert float((out.view(nq, d).double().cpu() - ref).abs().max()) <= tolerance(d, n, 6.0) * float(vs[0].abs().max())
