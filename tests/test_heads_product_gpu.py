"""The paired q/k/v product with norms, rotation and the cache write in its epilogue, against the plain paired product and the kernels
that do these behind it: bit for bit what is only rounded, to one rounding what is normed (the sum of squares is added in another
order) or turned (which of its two products is rounded first is the compiler's)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nq,nkv,K,page", [(4, 2, 72, 16), (3, 1, 200, 64), (16, 8, 128, 8), (9, 3, 64, 32)])
@pytest.mark.parametrize("norm,pairs", [(True, 64), (False, 64), (False, 32), (True, 32), (False, 0)])
def test_like_the_kernels_behind_the_product(nq, nkv, K, page, norm, pairs):
    from litellmengine_b200.csrc import ops
    d = 128
    g = torch.Generator(device=DEV).manual_seed(nq + K + pairs)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    w = (torch.randn((nq + 2 * nkv) * d, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    qw, kw = (torch.randn(d, generator=g, device=DEV) for _ in range(2)) if norm else (None, None)
    inv = (10000.0 ** (-torch.arange(pairs, device=DEV) / max(1, pairs))).contiguous() if pairs else None
    for T in (1, 127, 129, 257, 640, 700):
        x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
        ends = [T // 3, T]                                       # two requests, each behind tokens of its own
        entry = i32([0] * ends[0] + [1] * (T - ends[0]))
        pos = i32(list(range(5, 5 + ends[0])) + list(range(70, 70 + T - ends[0])))
        width = -(-(75 + T) // page)
        table = torch.randperm(2 * width + 1, generator=g, device=DEV).to(torch.int32)[:2 * width].view(2, width).contiguous()
        slots, status = i32([1, 0]), i32([0, 0])
        caches = [torch.full((2 * width + 1, 2, nkv, page, d), 3.0, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
        angles = ops.rope_angles(pos, inv) if pairs else None
        proj = ops.linear_pair(x, w, torch.float32)
        if pairs == 32:
            c = caches[0]
            q = ops.attention_prepare(proj, 0, nq * d, (nq + nkv) * d, None, qw, kw, "head" if norm else None, 1e-6, None, c[:, 0], c[:, 1], pos, entry,
                                      slots, table, nq, nkv, d, d, page, status, torch.bfloat16, rotation=(inv, 64, 1.0, False))
        else:
            q = ops.qk_norm_rope_kv_write(proj, caches[0], pos, entry, slots, table, qw, kw, 1e-6, inv, 2 * pairs, nq, nkv, d, page, True, status,
                                          q_dtype=torch.bfloat16, angles=angles)
        got = ops.linear_pair_heads(x, w, caches[1], pos, entry, slots, table, qw, kw, 1e-6, angles, nq, nkv, page, status)
        assert status.tolist() == [0, 0] and ops.stream_status(torch.device(DEV)).tolist() == [0, 0]
        for a, b in ((q, got), (caches[0], caches[1])):
            if not norm and not pairs:
                assert torch.equal(a, b), T
            else:                                                # one bfloat16 rounding of a value that may be a few 2^-24 off
                # (a turned entry is the difference of two products: what is off is a part of the head's largest entries)
                off = 2.0 ** -21 * float(a.abs().max())
                assert bool(((a.float() - b.float()).abs() <= 2.0 ** -7 * a.float().abs() + off).all()), T
                assert float((a != b).float().mean()) < 0.01


def test_a_page_outside_the_cache_is_told_and_left_out():
    from litellmengine_b200.csrc import ops
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    x, w = torch.ones(130, 64, device=DEV, dtype=torch.bfloat16), torch.ones(384, 64, device=DEV, dtype=torch.bfloat16)
    cache, status = torch.zeros(3, 2, 1, 64, 128, device=DEV, dtype=torch.bfloat16), i32([0, 0])
    z = torch.zeros(130, dtype=torch.int32, device=DEV)
    q = ops.linear_pair_heads(x, w, cache, torch.arange(130, dtype=torch.int32, device=DEV), z, i32([0]), i32([[0, 7, 2]]), None, None, 0.0, None, 1, 1, 64, status)
    assert status[0] == 3 and 64 <= int(status[1]) < 128
    assert bool((q == 64).all()) and bool((cache[0] == 64).all()) and bool((cache[1] == 0).all()) and bool((cache[2, :, :, :2] == 64).all())
    assert bool((cache[2, :, :, 2:] == 0).all())


def test_which_products_come_here():
    from litellmengine_b200.csrc import ops
    bf = lambda *s: torch.zeros(*s, device=DEV, dtype=torch.bfloat16)
    w, cache = bf(6144, 4096), bf(1, 2, 8, 16, 128)
    takes = lambda T, **k: ops.heads_product(bf(T, 4096), k.get("w", w), k.get("cache", cache), k.get("d", 128))
    assert takes(640) and takes(2900) and not takes(500) and not takes(128) and not takes(599)
    assert not takes(2900, d=64) and not takes(2900, cache=cache.float()) and not takes(2900, w=w.float()) and not takes(2900, cache=None)


@pytest.mark.parametrize("H,K", [(1, 64), (3, 200), (8, 136), (11, 64)])
@pytest.mark.parametrize("turned", [False, True])
def test_latent_queries_like_the_kernel_behind_the_product(H, K, turned):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(H + K)
    w = (torch.randn(H * 192, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    inv = 10000.0 ** (-torch.arange(32, device=DEV) / 32.0)
    for T in (1, 128, 129, 255, 257, 700):
        x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
        pos = torch.randint(0, 40000, (T,), generator=g, device=DEV, dtype=torch.int32)
        angles = ops.rope_angles(pos, inv) if turned else None
        want = ops.latent_q_pack(ops.linear_pair(x, w, torch.float32), pos, inv, H, 128, 64, 64 if turned else 0, rot_pairs=True)
        got = ops.linear_pair_latent_q(x, w, angles, H)
        if not turned:
            assert torch.equal(got, want), T
        else:                                                    # as above: which product of a turned entry is rounded first
            off = 2.0 ** -21 * float(want.abs().max())
            assert bool(((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + off).all()), T
            assert float((got != want).float().mean()) < 0.01
            assert torch.equal(got.view(T, H, 192)[..., :128], want.view(T, H, 192)[..., :128])
    assert ops.stream_status(torch.device(DEV)).tolist() == [0, 0]
