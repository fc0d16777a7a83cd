"""The one-pass tcgen05 prompt kernels where the running maximum moves late: in the first or second half of a tile of keys, in
many rows or in one, by little or by more than exp2 holds; portions of every remainder of 128 rows, whole and windowed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
D, PAGE, NQ, NKV = 128, 16, 4, 2


@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("loud,times", [([], 1.0), ([130, 200, 255, 383], 12.0), ([64, 129, 450], 60.0), (list(range(0, 600, 37)), 400.0)])
def test_maxima_that_move_and_rows_behind_the_last(loud, times, window):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(5 + len(loud))
    reqs = [(2, 2), (65, 65), (127, 127), (128, 128), (257, 129), (600, 255), (640, 1 + 128), (513, 513)]      # (cached and new, new)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    width = max(-(-n // PAGE) for n, _ in reqs)
    table = torch.randperm(len(reqs) * width, generator=g, device=DEV).to(torch.int32).view(len(reqs), width).contiguous()
    cache = torch.zeros(len(reqs) * width, 2, NKV, PAGE, D, device=DEV, dtype=torch.bfloat16)
    kv = []
    for b, (n, _) in enumerate(reqs):
        x = torch.randn(2, n, NKV, D, generator=g, device=DEV)
        for k in loud:                          # keys whose scores leave those before them far behind, for queries of either sign
            if k < n:
                x[0, k] *= times
        x = x.to(torch.bfloat16)
        j = torch.arange(n, device=DEV)
        for s in (0, 1):
            cache[table[b, j // PAGE].long(), s, :, j % PAGE] = x[s]
        kv.append(x)
    T = sum(t for _, t in reqs)
    starts = [sum(t for _, t in reqs[:b]) for b in range(len(reqs))]
    q = torch.randn(T, NQ * D, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((T, NQ * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    tiles = [(b, r) for b, (_, t) in enumerate(reqs) for r in range(0, t, 128)] + [(-1, -1)]
    status = i32([0, 0])
    ops.paged_attention_prefill_tcgen05(q, out, cache, i32(tiles), len(tiles), i32(list(range(len(reqs)))), i32(starts), i32([t for _, t in reqs]),
                                        i32([n for n, _ in reqs]), table, NQ, NKV, D, PAGE, window, D ** -0.5, status)
    assert status.tolist() == [0, 0]
    for b, (n, t) in enumerate(reqs):
        k, v = (x.to(F64).repeat_interleave(NQ // NKV, 1) for x in kv[b])
        s = torch.einsum("thd,shd->hts", q[starts[b]:starts[b] + t].view(t, NQ, D).to(F64), k) * D ** -0.5
        i, j = torch.arange(n - t, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
        see = (j <= i) & ((i - j < window) if window else torch.ones_like(i - j, dtype=torch.bool))
        p = torch.softmax(s.masked_fill(~see, float("-inf")), -1)
        want = torch.einsum("hts,shd->thd", p, v).reshape(t, -1)
        # weights are rounded to bfloat16, of 8 bits (2^-8 of a weight at most), so is the result; a score's float32 sum of 128 products, of
        # up to 2^-23 * |q . k| each as the tensor cores cut them, moves a weight by that much in relation to itself
        carried = torch.einsum("hts,shd->thd", p, v.abs()).reshape(t, -1)
        cut = float(s.abs().max()) * 128 * 2.0 ** -23
        bound = 2.0 ** -8 * (carried + want.abs()) * 1.02 + 2 * cut * carried + 1e-6
        got = out[starts[b]:starts[b] + t].to(F64)
        assert bool(((got - want).abs() <= bound).all()), (n, t, float(((got - want).abs() / bound).max()))


@pytest.mark.parametrize("loud,times", [([47, 48, 95], 12.0), ([96, 143, 144, 300], 60.0), (list(range(0, 500, 29)), 400.0)])
@pytest.mark.parametrize("window", [None, 60])
def test_latent_maxima_that_move(loud, times, window):
    """The same of the latent kernel's tiles of 96 keys, in halves of 48, and pairs of tiles of 128 query rows."""
    from litellmengine_b200.csrc import ops as o
    g = torch.Generator(device=DEV).manual_seed(len(loud))
    H, R, K = 2, 64, o.LATENT_TILE_KEYS
    reqs = [(2, 2), (97, 97), (130, 129), (400, 257), (500, 3), (511, 511)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    first = [max(0, n - t - window + 1) if window else 0 for n, t in reqs]
    count = [-(-(n - f) // K) * K for (n, _), f in zip(reqs, first)]
    at = [sum(count[:b]) for b in range(len(reqs))]
    gathered, kv = (torch.zeros(sum(count), w, device=DEV, dtype=torch.bfloat16) for w in (R + 64, H * 256))
    for (n, _), f, a in zip(reqs, first, at):
        k = torch.randn(n - f, H * 256, generator=g, device=DEV)
        for j in loud:
            if j < n - f:
                k.view(-1, H, 256)[j, :, :128] *= times
        kv[a:a + n - f] = k.to(torch.bfloat16)
        gathered[a:a + n - f] = torch.randn(n - f, R + 64, generator=g, device=DEV).to(torch.bfloat16)
    T, starts = sum(t for _, t in reqs), [sum(t for _, t in reqs[:b]) for b in range(len(reqs))]
    q = torch.randn(T, H * 192, generator=g, device=DEV).to(torch.bfloat16)
    tiles, status = [(b, r) for b, (_, t) in enumerate(reqs) for r in range(0, t, o.LATENT_TILE_ROWS)], i32([0, 0])
    segs = i32([list(x) for x in zip(range(len(reqs)), first, at, count)])
    out = torch.full((T, H * 128), float("nan"), device=DEV, dtype=torch.bfloat16)
    o.latent_prefill(q, kv, gathered, out, i32(tiles), len(tiles), segs, i32(starts), i32([t for _, t in reqs]), i32([n for n, _ in reqs]), H, R,
                     window, 192 ** -0.5, status)
    assert status.tolist() == [0, 0]
    for b, (n, t) in enumerate(reqs):
        a, f = at[b], first[b]
        kh = kv[a:a + n - f].view(n - f, H, 256).to(F64)
        k = torch.cat([kh[..., :128], gathered[a:a + n - f, None, R:].to(F64).expand(n - f, H, 64)], -1)
        s = torch.einsum("thd,shd->hts", q[starts[b]:starts[b] + t].view(t, H, 192).to(F64), k) * 192 ** -0.5
        i, j = torch.arange(n - t, n, device=DEV)[:, None], torch.arange(f, n, device=DEV)[None, :]
        see = (j <= i) & ((i - j < window) if window else torch.ones_like(i - j, dtype=torch.bool))
        p = torch.softmax(s.masked_fill(~see, float("-inf")), -1)
        want, carried = (torch.einsum("hts,shd->thd", p, v).reshape(t, -1) for v in (kh[..., 128:], kh[..., 128:].abs()))
        cut = float(s.abs().max()) * 192 * 2.0 ** -23                      # the bound of the test above
        bound = 2.0 ** -8 * (carried + want.abs()) * 1.02 + 2 * cut * carried + 1e-6
        got = out[starts[b]:starts[b] + t].to(F64)
        assert bool(((got - want).abs() <= bound).all()), (n, t, float(((got - want).abs() / bound).max()))


@pytest.mark.parametrize("loud,times", [([], 1.0), ([127, 128, 200, 383], 12.0), ([64, 129, 450], 60.0), (list(range(0, 600, 37)), 400.0)])
@pytest.mark.parametrize("window", [None, 70])
def test_biased_maxima_that_move(loud, times, window):
    """The same with a temperature per head and a logarithmic bias of the distance, whose two tables take turns tile by tile."""
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(15 + len(loud))
    reqs = [(2, 2), (65, 65), (128, 128), (257, 129), (600, 255), (640, 1 + 128), (513, 513)]      # (cached and new, new)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    width = max(-(-n // PAGE) for n, _ in reqs)
    table = torch.randperm(len(reqs) * width, generator=g, device=DEV).to(torch.int32).view(len(reqs), width).contiguous()
    cache = torch.zeros(len(reqs) * width, 2, NKV, PAGE, D, device=DEV, dtype=torch.bfloat16)
    kv = []
    for b, (n, _) in enumerate(reqs):
        x = torch.randn(2, n, NKV, D, generator=g, device=DEV)
        for k in loud:
            if k < n:
                x[0, k] *= times
        x = x.to(torch.bfloat16)
        j = torch.arange(n, device=DEV)
        for s in (0, 1):
            cache[table[b, j // PAGE].long(), s, :, j % PAGE] = x[s]
        kv.append(x)
    T, starts = sum(t for _, t in reqs), [sum(t for _, t in reqs[:b]) for b in range(len(reqs))]
    q = torch.randn(T, NQ * D, generator=g, device=DEV).to(torch.bfloat16)
    three = torch.tensor([[1.0, 0.0, 0.0], [0.7, 1.5, 0.3], [1.3, 0.4, 5.0], [0.2, 3.0, 1.0]], device=DEV)      # temperature, r1, r2
    out = torch.full((T, NQ * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    tiles = [(b, r) for b, (_, t) in enumerate(reqs) for r in range(0, t, 128)] + [(-1, -1)]
    status = i32([0, 0])
    ops.paged_attention_prefill_tcgen05_biased(q, out, cache, i32(tiles), len(tiles), i32(list(range(len(reqs)))), i32(starts),
                                               i32([t for _, t in reqs]), i32([n for n, _ in reqs]), table, NQ, NKV, D, PAGE, window, D ** -0.5,
                                               status, three)
    assert status.tolist() == [0, 0]
    temp, r1, r2 = (c.to(F64)[:, None, None] for c in three.unbind(1))
    for b, (n, t) in enumerate(reqs):
        k, v = (x.to(F64).repeat_interleave(NQ // NKV, 1) for x in kv[b])
        i, j = torch.arange(n - t, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
        off = r1 * torch.log1p(r2 * (i - j).clamp(min=0))
        s = torch.einsum("thd,shd->hts", q[starts[b]:starts[b] + t].view(t, NQ, D).to(F64), k) * D ** -0.5 * temp
        see = (j <= i) & ((i - j < window) if window else torch.ones_like(i - j, dtype=torch.bool))
        p = torch.softmax((s - off).masked_fill(~see, float("-inf")), -1)
        want, carried = (torch.einsum("hts,shd->thd", p, x).reshape(t, -1) for x in (v, v.abs()))
        # the bound of the first test; the bias is a float32 product of r1 and a logarithm that is within 2^-21 of its size or of 1
        cut = float(s.abs().max()) * 128 * 2.0 ** -23 + (1 + float(off.max())) * 4 * 2.0 ** -21
        bound = 2.0 ** -8 * (carried + want.abs()) * 1.02 + 2 * cut * carried + 1e-6
        got = out[starts[b]:starts[b] + t].to(F64)
        assert bool(((got - want).abs() <= bound).all()), (n, t, float(((got - want).abs() / bound).max()))
