"""The one-pass tcgen05 prompt kernel where the running maximum moves late: in the first or second half of a tile of 128 keys, in
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
