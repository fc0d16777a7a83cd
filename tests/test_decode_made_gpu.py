"""The decode attention kernel that makes its queries, keys and values itself, against the two kernels it stands for: the same
results and the same pages, bit for bit, at the edges of its pages, tiles of 64 keys and splits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("d,nq,nkv,page", [(128, 16, 8, 16), (128, 8, 1, 64), (128, 4, 4, 8), (64, 6, 2, 32), (64, 16, 1, 16)])
@pytest.mark.parametrize("splits", [1, 2, 5])
@pytest.mark.parametrize("norm,rotation,parts", [(True, "angles", 1), (True, "frequencies", 3), (False, None, 2), (False, "angles", 1)])
def test_like_the_two_kernels(d, nq, nkv, page, splits, norm, rotation, parts):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(d + nq + splits)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    past = [0, 1, 7, 15, 16, 31, 62, 63, 64, 65, 127, 128, 190, 255, 256, 500, 701]
    T, width = len(past), -(-702 // page)
    order = torch.randperm(T * width + 3, generator=g, device=DEV).to(torch.int32)
    table = order[:T * width].view(T, width).contiguous()
    cache = torch.randn(T * width + 3, 2, nkv, page, d, generator=g, device=DEV).to(torch.bfloat16)
    qkv = torch.randn(parts, T, (nq + 2 * nkv) * d, generator=g, device=DEV)
    qkv = ops.PartialSum(qkv) if parts > 1 else qkv[0]
    perm = torch.randperm(T, generator=g, device=DEV).to(torch.int32)        # which entry a token belongs to, and which slot that has
    slots = torch.randperm(T, generator=g, device=DEV).to(torch.int32)
    pos = i32(past)
    qw, kw = (torch.randn(d, generator=g, device=DEV) for _ in range(2)) if norm else (None, None)
    inv = (10000.0 ** (-torch.arange(d // 2, device=DEV) * 2.0 / d)).contiguous() if rotation else None
    angles = ops.rope_angles(pos, inv) if rotation == "angles" else None
    other, status = cache.clone(), i32([0, 0])
    q = ops.qk_norm_rope_kv_write(qkv, other, pos, perm, slots, table, qw, kw, 1e-6, inv, d if rotation else 0, nq, nkv, d, page, True, status,
                                  q_dtype=torch.bfloat16, angles=angles)
    want = torch.empty_like(q)
    ops.paged_attention_decode(q, want, other, None, T, pos, perm, slots, table, nq, nkv, d, page, None, d ** -0.5, splits, status)
    assert ops.decode_makes_its_rows(qkv, cache, d, nq // nkv, page)
    got = ops.paged_attention_decode_made(qkv, cache, pos, perm, slots, table, qw, kw, 1e-6, inv, angles, nq, nkv, d, page, d ** -0.5, splits, status)
    assert status.tolist() == [0, 0]
    assert torch.equal(cache, other) and torch.equal(got, want)


def test_what_is_not_taken():
    from litellmengine_b200.csrc import ops
    cache, qkv = torch.zeros(1, 2, 1, 16, 128, device=DEV, dtype=torch.bfloat16), torch.zeros(2, 384, device=DEV)
    assert ops.decode_makes_its_rows(qkv, cache, 128, 1, 16)
    assert not ops.decode_makes_its_rows(qkv, cache, 128, 1, 128) and not ops.decode_makes_its_rows(qkv, cache, 128, 17, 16)
    assert not ops.decode_makes_its_rows(qkv, cache.float(), 128, 1, 16) and not ops.decode_makes_its_rows(qkv, cache, 256, 1, 16)
    assert not ops.decode_makes_its_rows(ops.PartialSum(qkv[None], torch.bfloat16), cache, 128, 1, 16)
    sums = ops.PartialSum(qkv[None])
    assert ops.decode_makes_its_rows(sums, cache, 128, 1, 16, 4) and not ops.decode_makes_its_rows(sums, cache, 128, 1, 16, 5)
    assert ops.decode_makes_its_rows(qkv, cache, 128, 1, 16, 16)


def test_many_caches():
    """A process that makes caches at ever new addresses: what is taken once is taken again."""
    from litellmengine_b200.csrc import ops
    nq, nkv, page, d = 4, 2, 8, 64
    g = torch.Generator(device=DEV).manual_seed(1)
    caches = torch.randn(700, 1, 2, nkv, page, d, generator=g, device=DEV).to(torch.bfloat16)
    two = caches.clone()
    qkv = torch.randn(1, (nq + 2 * nkv) * d, generator=g, device=DEV)
    pos, zero = torch.tensor([5], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    table, status = torch.zeros(1, 1, dtype=torch.int32, device=DEV), torch.zeros(2, dtype=torch.int32, device=DEV)
    got = []
    for c in caches:
        assert ops.decode_makes_its_rows(qkv, c, d, nq // nkv, page)
        got.append(ops.paged_attention_decode_made(qkv, c, pos, zero, zero, table, None, None, 1e-6, None, None, nq, nkv, d, page, d ** -0.5, 1, status))
    for c, a in zip(two, got):
        q = ops.qk_norm_rope_kv_write(qkv, c, pos, zero, zero, table, None, None, 1e-6, None, 0, nq, nkv, d, page, True, status,
                                      q_dtype=torch.bfloat16)
        want = ops.paged_attention_decode(q, torch.empty_like(q), c, None, 1, pos, zero, zero, table, nq, nkv, d, page, None, d ** -0.5, 1, status)
        assert torch.equal(a, want)
    assert status.tolist() == [0, 0] and torch.equal(caches, two)
