"""The tcgen05 prompt kernel with kept first keys, sinks, a gate per head and a result that is a column range, against
float64 and against the mma.sync kernel, at the edges of its tiles of 128 rows and 128 keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("window,keep", [(None, 0), (1, 0), (1, 1), (100, 5), (128, 128), (129, 127), (64, 130), (257, 300), (-200, 0)])
@pytest.mark.parametrize("nq,nkv,page", [(4, 2, 16), (8, 1, 64)])
def test_kept_keys_sinks_gates_and_columns(nq, nkv, page, window, keep):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(nq + keep)
    d, scale = 128, 128 ** -0.5
    reqs = [(2, 2), (128, 128), (129, 129), (300, 127), (700, 257), (1000, 30), (520, 520)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    width = max(-(-n // page) for n, _ in reqs)
    order = torch.randperm(len(reqs) * width, generator=g, device=DEV).to(torch.int32)
    table = order.view(len(reqs), width).contiguous()
    cache = torch.zeros(len(order), 2, nkv, page, d, device=DEV, dtype=torch.bfloat16)
    ks = [torch.randn(2, n, nkv, d, generator=g, device=DEV).to(torch.bfloat16) for n, _ in reqs]
    for b, kv in enumerate(ks):
        j = torch.arange(kv.shape[1], device=DEV)
        for x in (0, 1):
            cache[table[b, j // page].long(), x, :, j % page] = kv[x]
    span = abs(window) if window else 0
    for b, (n, t) in enumerate(reqs):          # pages that no query of the step sees are somebody else's by now
        lo = n - t - span + 1 if window and window > 0 else (n - t) // span * span if window else 0
        for page_at in range(-(-keep // page), max(0, lo) // page):
            cache[table[b, page_at].long()] = float("nan")
            if page_at % 2:
                table[b, page_at] = -1
    T = sum(t for _, t in reqs)
    starts = [sum(t for _, t in reqs[:b]) for b in range(len(reqs))]
    q = torch.randn(T, nq * d, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(T, nq + 3, generator=g, device=DEV)
    sinks = torch.randn(nq, generator=g, device=DEV) * 3
    tiles = [(b, r) for b, (_, t) in enumerate(reqs) for r in range(0, t, 128)] + [(-1, -1)]
    status = i32([0, 0])
    args = lambda out, off: (q, out, off, cache, i32(tiles), len(tiles), i32(list(range(len(reqs)))), i32(starts), i32([t for _, t in reqs]),
                             i32([n for n, _ in reqs]), table, nq, nkv, d, page, window, scale, status)
    wide = torch.full((T, nq * d + 24), 7.0, device=DEV, dtype=torch.bfloat16)
    assert ops.prefill_tcgen05_biased_supported(d, page, nq // nkv)
    ops.paged_attention_prefill_tcgen05_ext(*args(wide, 16), head_gate=gate, gate_off=2, out_scale=0.5, keep_first=keep, sink=sinks)
    assert status.tolist() == [0, 0]
    assert float((wide[:, :16].float() - 7).abs().max()) == 0 and float((wide[:, 16 + nq * d:].float() - 7).abs().max()) == 0
    share = 0.5 * torch.sigmoid(gate[:, 2:2 + nq].to(F64))
    for b, (n, t) in enumerate(reqs):
        k, v = (x.to(F64).repeat_interleave(nq // nkv, 1) for x in ks[b])
        s = torch.einsum("thd,shd->hts", q[starts[b]:starts[b] + t].view(t, nq, d).to(F64), k) * scale
        i, j = torch.arange(n - t, n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
        near = (i - j < window) if window and window > 0 else (j >= i - i % span) if window else torch.ones_like(i - j, dtype=torch.bool)
        see = (j <= i) & (near | (j < keep))
        s = torch.cat([s.masked_fill(~see, float("-inf")), sinks.to(F64)[:, None, None].expand(nq, t, 1)], -1)
        p = torch.softmax(s, -1)[..., :n]
        ref = torch.einsum("hts,shd->thd", p, v)
        bound = share[starts[b]:starts[b] + t, :, None] * (2 ** -8 * (ref.abs() + torch.einsum("hts,shd->thd", p, v.abs())) + 1e-3)
        got = wide[starts[b]:starts[b] + t, 16:16 + nq * d].view(t, nq, d).to(F64)
        ref = ref * share[starts[b]:starts[b] + t, :, None]
        assert bool(((got - ref).abs() <= bound).all()), (n, t, float(((got - ref).abs() / bound).max()))
