"""Long prompt steps of latent attention: the path that maps the cached rows to per-head keys and values against the
path over the rows themselves, and its kernels against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


def ops():
    from litellmengine_b200.csrc import ops as o
    return o


@pytest.mark.parametrize("H,R,window", [(1, 64, None), (3, 128, None), (2, 512, 100), (2, 512, 1), (3, 256, 300)])
def test_kernels(H, R, window):
    """(cached after the step, queries at the end) around the edges of 96 keys and of 128 and 256 query rows."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(H * 100 + R)
    reqs = [(2, 2), (96, 96), (97, 97), (130, 129), (256, 256), (400, 257), (500, 3), (900, 300)]
    page, DK, K = 16, R + 64, o.LATENT_TILE_KEYS
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    width = max(-(-n // page) for n, _ in reqs)
    order = torch.randperm(len(reqs) * width, generator=g, device=DEV).to(torch.int32)
    table = order.view(len(reqs), width).contiguous()
    cache = torch.full((len(reqs) * width, 1, page, DK), float("nan"), device=DEV, dtype=torch.bfloat16)
    rows = [torch.randn(n, DK, generator=g, device=DEV).to(torch.bfloat16) for n, _ in reqs]
    for b, r in enumerate(rows):
        j = torch.arange(len(r), device=DEV)
        cache[table[b, j // page].long(), 0, j % page] = r
    T = sum(t for _, t in reqs)
    starts = [sum(t for _, t in reqs[:b]) for b in range(len(reqs))]
    first = [max(0, n - t - window + 1) if window else 0 for n, t in reqs]
    count = [-(-(n - f) // K) * K for (n, _), f in zip(reqs, first)]
    at = [sum(count[:b]) for b in range(len(reqs))]
    segs, status = i32([list(x) for x in zip(range(len(reqs)), first, at, count)]), i32([0, 0])
    slots, q_len, kv_len = i32(list(range(len(reqs)))), i32([t for _, t in reqs]), i32([n for n, _ in reqs])
    gathered = o.latent_gather(cache, segs, len(reqs), sum(count), max(count), slots, kv_len, table, page, status)
    want = torch.zeros(sum(count), DK, device=DEV, dtype=torch.bfloat16)
    for (n, _), f, a, r in zip(reqs, first, at, rows):
        want[a:a + n - f] = r[f:]
    assert torch.equal(gathered, want)
    w = (torch.randn(H * 256, R, generator=g, device=DEV) * R ** -0.5).to(torch.bfloat16)
    kv = torch.mm(gathered[:, :R], w.t())
    q32 = torch.randn(T, H * 192, generator=g, device=DEV)
    pos = i32([p for n, t in reqs for p in range(n - t, n)])
    inv = torch.rand(32, generator=g, device=DEV)
    for pairs in (False, True):
        qp = o.latent_q_pack(q32, pos, inv, H, 128, 64, 64, rot_pairs=pairs, rot_mag=1.25)
        qn, packed = o.latent_q_split(q32, pos, inv, H, 128, 64, R, 64, torch.bfloat16, rot_pairs=pairs, rot_mag=1.25)
        assert torch.equal(qp.view(T, H, 192)[..., :128].permute(1, 0, 2), qn)
        assert torch.allclose(qp.view(T, H, 192)[..., 128:].float(), packed.view(T, H, DK)[..., R:].float(), rtol=2 ** -7, atol=1e-6)
    R2 = o.LATENT_TILE_ROWS
    tiles = i32([(b, r) for b, (_, t) in enumerate(reqs) for r in range(0, t, R2)])
    out = torch.full((T, H * 128), 7.0, device=DEV, dtype=torch.bfloat16)
    scale = 192 ** -0.5
    gate = torch.randn(T, H + 5, generator=g, device=DEV) if R == 512 else None
    o.latent_prefill(qp, kv, gathered, out, tiles, len(tiles), segs, i32(starts), q_len, kv_len, H, R, window, scale, status,
                     gate=gate, gate_off=3)
    assert status.tolist() == [0, 0]
    share = torch.sigmoid(gate[:, 3:3 + H].to(F64)) if gate is not None else torch.ones(T, H, device=DEV, dtype=F64)
    for b, (n, t) in enumerate(reqs):
        a, f = at[b], first[b]
        kh = kv[a:a + n - f].view(n - f, H, 256).to(F64)
        k = torch.cat([kh[..., :128], gathered[a:a + n - f, None, R:].to(F64).expand(n - f, H, 64)], -1)
        qq = qp[starts[b]:starts[b] + t].view(t, H, 192).to(F64)
        s = torch.einsum("thd,shd->hts", qq, k) * scale
        i, j = torch.arange(n - t, n, device=DEV)[:, None], torch.arange(f, n, device=DEV)[None, :]
        see = (j <= i) & ((i - j < window) if window else True)
        p = torch.softmax(s.masked_fill(~see, float("-inf")), -1)
        ref = torch.einsum("hts,shd->thd", p, kh[..., 128:])
        share_b = share[starts[b]:starts[b] + t, :, None]
        ref = ref * share_b
        got = out[starts[b]:starts[b] + t].view(t, H, 128).to(F64)
        # weights and result rounded to bfloat16 (2^-9 each), the weights' errors weighted by the values they meet
        bound = 2 ** -8 * (ref.abs() + share_b * torch.einsum("hts,shd->thd", p, kh[..., 128:].abs())) + 1e-3
        assert bool(((got - ref).abs() <= bound).all()), (n, t, float(((got - ref).abs() / bound).max()))



@pytest.mark.parametrize("H,D,P,dims", [(50, 128, 64, 64), (41, 128, 64, 20), (3, 128, 64, 36), (2, 64, 32, 0), (90, 8, 8, 6), (1, 2048, 64, 64), (2, 8184, 8, 8),
                                        (3, 8192, 64, 48), (1, 24640, 64, 64)])
@pytest.mark.parametrize("pairs", [False, True])
def test_queries_are_packed_whatever_the_heads(H, D, P, dims, pairs):
    """More heads than a block takes at once, angles that cover parts of a group of eight, heads wider than a block."""
    o, T = ops(), 5
    g = torch.Generator(device=DEV).manual_seed(H + D)
    q = torch.randn(T, H * (D + P), generator=g, device=DEV)
    pos = torch.tensor([0, 1, 7, 500, 40000], dtype=torch.int32, device=DEV)
    inv = torch.rand(max(1, dims // 2), generator=g, device=DEV)
    got = o.latent_q_pack(q, pos, inv, H, D, P, dims, rot_pairs=pairs, rot_mag=1.25).view(T, H, D + P)
    x = q.view(T, H, D + P).to(F64).clone()
    angle = (pos.float()[:, None] * inv[:dims // 2]).to(F64)          # the product is a 32-bit one
    c, s = 1.25 * torch.cos(angle)[:, None], 1.25 * torch.sin(angle)[:, None]
    part = x[..., D:D + dims]
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    a, b = part[..., u].clone(), part[..., v].clone()
    part[..., u], part[..., v] = a * c - b * s, b * c + a * s
    assert torch.equal(got[..., :D], q.view(T, H, D + P)[..., :D].to(torch.bfloat16))
    assert torch.equal(got[..., D + dims:], q.view(T, H, D + P)[..., D + dims:].to(torch.bfloat16))
    # one rounding to bfloat16 of a number that is a few 2^-24 off
    assert bool(((got.to(F64) - x).abs() <= 2.0 ** -8 * x.abs() + 1e-5).all())


@pytest.mark.parametrize("window", [None, 200])
def test_long_step_of_every_kind_of_entry(window):
    """Portions with and without earlier tokens beside single tokens, in one step, over both paths."""
    from litellmengine_b200.config import config_from_dict
    from litellmengine_b200.engine import ModelRunner, StepEntry
    m = {"heads": 3, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 96, "kv_rank": 128, "scale": 192 ** -0.5,
         "rot": {"base": 10000.0, "dims": 64}}
    if window:
        m["mask"] = {"size": window}
    cfg = {"architecture": "Vugedra", "vocab": 64, "width": 256, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    runner = ModelRunner.from_config(config_from_dict(cfg), seed=3, device=DEV, max_total_tokens=8192, max_requests=8, max_tokens_per_step=2048)
    mixer = runner.model.blocks[0].mixer
    past, new = [0, 130, 500, 77, 400, 0], [700, 1, 260, 129, 1, 2]
    g = torch.Generator(device=DEV).manual_seed(1)
    slots = [runner.admit() for _ in past]
    x = lambda n: torch.randn(n, 256, generator=g, device=DEV).to(torch.bfloat16)
    for s, p in zip(slots, past):
        if p:
            b = runner.prepare([StepEntry(s, [0] * p)])
            mixer.forward(x(p), runner.model.stage_context(0, b, runner.cache))
            runner.finish(b)
    b = runner.prepare([StepEntry(s, [0] * n) for s, n in zip(slots, new)])
    ctx, xs = runner.model.stage_context(0, b, runner.cache), x(sum(new))
    assert sum(new) >= 1025 and mixer._expand is not None
    before = ops().launch_count
    got = mixer.forward(xs, ctx)
    launched = ops().launch_count - before
    held, mixer._expand = mixer._expand, None
    ref = mixer.forward(xs, ctx)
    mixer._expand = held
    # both paths round queries, keys (or folded queries) and sums to bfloat16 a handful of times, 2^-9 each
    err = (got - ref).double().norm(dim=1) / ref.double().norm(dim=1)
    assert float(err.max()) < 6 * 2 ** -8, float(err.max())
    assert launched > 5
    runner.check_status()
    limit, mixer.EXPANDED_BYTES = mixer.EXPANDED_BYTES, 1000          # more rows than may be expanded at once: the other path
    assert torch.equal(mixer.forward(xs, ctx), ref)
    mixer.EXPANDED_BYTES = limit


def long_step(window=None, seed=3):
    """A mixer, a step of 1,100 tokens (a prompt, short and long portions, a single token) and its inputs."""
    from litellmengine_b200.config import config_from_dict
    from litellmengine_b200.engine import ModelRunner, StepEntry
    m = {"heads": 3, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 96, "kv_rank": 128, "scale": 192 ** -0.5,
         "rot": {"base": 10000.0, "dims": 64}}
    cfg = {"architecture": "Vugedra", "vocab": 64, "width": 256, "norm": {"eps": 1e-5},
           "layers": [{"type": "latent_attention", "mixer": m, "mlp": None}]}
    runner = ModelRunner.from_config(config_from_dict(cfg), seed=seed, device=DEV, max_total_tokens=4096, max_requests=8, max_tokens_per_step=2048)
    mixer, g = runner.model.blocks[0].mixer, torch.Generator(device=DEV).manual_seed(1)
    x = lambda n: torch.randn(n, 256, generator=g, device=DEV).to(torch.bfloat16)
    past, new = [0, 130, 500, 77], [800, 1, 296, 3]
    slots = [runner.admit() for _ in past]
    for s, p in zip(slots, past):
        if p:
            b = runner.prepare([StepEntry(s, [0] * p)])
            mixer.forward(x(p), runner.model.stage_context(0, b, runner.cache))
            runner.finish(b)
    b = runner.prepare([StepEntry(s, [0] * n) for s, n in zip(slots, new)])
    ctx, xs = runner.model.stage_context(0, b, runner.cache), x(sum(new))
    held, mixer._expand = mixer._expand, None
    rows = mixer.forward(xs, ctx)                              # the path over the cached rows
    mixer._expand = held
    return runner, mixer, ctx, xs, rows


def test_a_step_that_is_being_captured_keeps_to_the_cached_rows():
    """A graph that serves any division of its tokens must not hold one step's segments, however many tokens it has."""
    _, mixer, ctx, xs, rows = long_step()
    assert not torch.equal(mixer.forward(xs, ctx), rows)       # by itself the step is expanded
    ctx.batch.any_division = True
    assert torch.equal(mixer.forward(xs, ctx), rows)


def test_tile_sizes_are_the_kernels(monkeypatch):
    _, mixer, ctx, xs, _ = long_step()
    for name, other in (("LATENT_TILE_ROWS", 128), ("LATENT_TILE_KEYS", 48)):      # the lists were made with the right ones
        with monkeypatch.context() as m:
            m.setattr(ops(), name, other)
            with pytest.raises(ops().KernelError):
                mixer.forward(xs, ctx)


def test_out_of_memory_in_the_expanded_path_takes_the_other(monkeypatch):
    _, mixer, ctx, xs, rows = long_step()
    def full(*a, **k):
        raise torch.cuda.OutOfMemoryError("no room for keys and values")
    monkeypatch.setattr(ops(), "latent_q_pack", full)
    assert torch.equal(mixer.forward(xs, ctx), rows)


@pytest.mark.parametrize("window,gated", [(None, False), (100, True)])
def test_a_row_that_is_not_finite_reaches_only_who_sees_it(window, gated):
    """Cached rows with infinities and NaN in a portion: the queries before them, and those that have them behind their window, stay
    as they would be without."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(7)
    H, R, n, t, past = 2, 128, 700, 600, 100
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    first = max(0, past - window + 1) if window else 0
    count, K = -(-(n - first) // o.LATENT_TILE_KEYS) * o.LATENT_TILE_KEYS, o.LATENT_TILE_ROWS
    rows = torch.zeros(count, R + 64, device=DEV, dtype=torch.bfloat16)
    rows[:n - first] = torch.randn(n - first, R + 64, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(H * 256, R, generator=g, device=DEV) * R ** -0.5).to(torch.bfloat16)
    kv = torch.mm(rows[:, :R], w.t())
    bad = {190: float("nan"), 420: float("inf"), 640: float("nan")}
    for p, x in bad.items():
        kv.view(count, H, 256)[p - first, :, 128:] = x                     # values only: the scores stay finite
    kv.view(count, H, 256)[640 - first] = float("nan")
    q = torch.randn(t, H * 192, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(t, H, generator=g, device=DEV) if gated else None
    out, status, scale = torch.zeros(t, H * 128, device=DEV, dtype=torch.bfloat16), i32([0, 0]), 192 ** -0.5
    tiles = i32([(0, r) for r in range(0, t, K)])
    o.latent_prefill(q, kv, rows, out, tiles, len(tiles), i32([[0, first, 0, count]]), i32([0]), i32([t]), i32([n]), H, R, window, scale, status,
                     gate=gate)
    assert status.tolist() == [0, 0]
    j = torch.arange(first, n, device=DEV)
    i = torch.arange(past, n, device=DEV)[:, None]
    see = (j <= i) & ((i - j < window) if window else True)
    spoiled = torch.stack([see[:, p - first] for p in bad], 1).any(1)
    kh = kv[:n - first].view(-1, H, 256).to(F64)
    k = torch.cat([kh[..., :128], rows[:n - first, None, R:].to(F64).expand(-1, H, 64)], -1).nan_to_num(0.0)
    s = torch.einsum("thd,shd->hts", q.view(t, H, 192).to(F64), k) * scale
    p = torch.softmax(s.masked_fill(~see, float("-inf")), -1)
    v = kh[..., 128:].nan_to_num(0.0, 0.0, 0.0)
    ref, bound = torch.einsum("hts,shd->thd", p, v), 2 ** -8 * torch.einsum("hts,shd->thd", p, v.abs())
    if gated:
        ref, bound = (x * torch.sigmoid(gate.to(F64))[:, :, None] for x in (ref, bound))
    got = out.view(t, H, 128).to(F64)
    assert not bool(torch.isfinite(got[spoiled]).any())
    assert bool(((got - ref).abs() <= bound + 2 ** -8 * ref.abs() + 1e-3)[~spoiled].all()) and int((~spoiled).sum()) > 60
