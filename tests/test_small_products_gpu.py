"""Products whose weights the SMs hold all at once: against float64 at the edges of their tiles, and the rows and activations that
they make themselves against the kernels that make them otherwise, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from litellmengine_b200.csrc import ops as o
    return o


@pytest.mark.parametrize("N,K", [(16, 64), (1, 72), (100, 200), (1000, 1096), (4096, 1024), (1024, 2048), (1024, 3072)])
@pytest.mark.parametrize("tiled", [False, True])
def test_product(N, K, tiled):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    if tiled:
        o._tiled[w.data_ptr()] = o.tile_weight(w)
    try:
        for M in (1, 5, 8, 9, 16):
            x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
            assert o.small_product(M, w)
            want, carried = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
            got = o.linear_small(x, w, torch.float32)
            # K / 16 steps of products that are exact in float32 and sums cut or rounded at 2^-23 of what they hold
            assert bool(((got.double() - want).abs() <= (K / 16 + 24) * 2.0 ** -23 * carried).all()), (M, N, K)
            assert torch.equal(o.linear_small(x, w, torch.bfloat16), got.to(torch.bfloat16))
            assert torch.equal(o.linear(x, w, torch.float32), got)
    finally:
        o._tiled.pop(w.data_ptr(), None)
    assert o.stream_status(torch.device(DEV)).tolist() == [0, 0]


@pytest.mark.parametrize("N,K", [(16, 64), (48, 512), (1536, 520), (3072, 1024), (64, 2048)])
@pytest.mark.parametrize("parts", [0, 1, 3, 6])
def test_rows_made_on_the_way(N, K, parts):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(N + K + parts)
    w = (torch.randn(2 * N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)

    class Norm:
        products_apply_it, eps, weight = True, 1e-6, torch.randn(K, generator=g, device=DEV)
    for M in (1, 3, 8):
        h = torch.randn(M, K, generator=g, device=DEV)
        delta = None
        if parts:
            delta = torch.randn(parts, M, K, generator=g, device=DEV)
            delta = o.PartialSum(delta) if parts > 1 else delta[0]
        kept = h.clone()
        rows = o.pending_rows(h, delta, Norm, w, torch.bfloat16, True)
        assert rows is not None
        plain = o.linear(rows, w, torch.float32)
        gated = {a: o.linear_silu_mul(rows, w, torch.bfloat16, activation=a, limit=1.5) for a in o.ACTIVATIONS}
        assert torch.equal(h, kept)                              # the stream that others still read
        x = o.rmsnorm(h, Norm.weight, Norm.eps, torch.bfloat16, delta=delta, write_sum=delta is not None)
        assert torch.equal(rows.stream, h)
        assert torch.equal(o.linear_small(x, w, torch.float32), plain)
        for a, got in gated.items():
            assert torch.equal(o.silu_and_mul(plain.to(torch.bfloat16), activation=a, limit=1.5), got), a
            assert torch.equal(o.linear_silu_mul(x, w, torch.bfloat16, activation=a, limit=1.5), got), a
    assert o.stream_status(torch.device(DEV)).tolist() == [0, 0]


def test_what_is_not_taken():
    o = ops()
    bf = lambda *s: torch.zeros(*s, device=DEV, dtype=torch.bfloat16)
    assert not o.small_product(17, bf(64, 64)) and not o.small_product(0, bf(64, 64)) and not o.small_product(4, bf(64, 64).float())
    assert not o.small_product(1, bf(24576, 4096)) and not o.small_product(1, bf(4096, 4096))          # more than the SMs hold
    assert not o.small_product(1, bf(64, 36)) and not o.small_product(1, bf(64, 70))
    assert not o.small_product(9, bf(64, 64), normed=True) and not o.small_product(1, bf(64, 2056), normed=True) and not o.small_product(1, bf(40, 64), gated=True)

    class Norm:
        products_apply_it, eps, weight = True, 1e-6, torch.ones(64, device=DEV)
    h, w = torch.zeros(2, 64, device=DEV), bf(64, 64)
    assert o.pending_rows(h, None, Norm, w, torch.bfloat16, False) is not None
    assert o.pending_rows(h, None, Norm, w, torch.float32, False) is None
    assert o.pending_rows(h, o.PartialSum(torch.zeros(2, 2, 64, device=DEV), torch.bfloat16), Norm, w, torch.bfloat16, False) is None
    assert o.pending_rows(h, h.to(torch.bfloat16), Norm, w, torch.bfloat16, False) is None
    assert o.pending_rows(h.t().contiguous().t(), None, Norm, w, torch.bfloat16, False) is None
    assert o.pending_rows(h, None, object(), w, torch.bfloat16, False) is None


@pytest.mark.parametrize("form", ["rows", "tiled", "normed", "gated"])
def test_a_wait_that_runs_out(form):
    """A block that has no tries left for its weights records the status, lets its copies land and ends; the next products are right."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(5)
    w = (torch.randn(2048, 1024, generator=g, device=DEV) / 32).to(torch.bfloat16)
    x, h = torch.randn(5, 1024, generator=g, device=DEV).to(torch.bfloat16), torch.randn(5, 1024, generator=g, device=DEV)
    if form == "tiled":
        o._tiled[w.data_ptr()] = o.tile_weight(w)
    rows = o.PendingRows(h, None, torch.ones(1024, device=DEV), 1e-6, torch.bfloat16) if form == "normed" else x
    out = dict(out_dtype=torch.bfloat16, activation="silu") if form == "gated" else dict(out_dtype=torch.float32)
    status = o.stream_status(torch.device(DEV))
    try:
        want = o.linear_small(rows, w, **out)
        assert status.tolist() == [0, 0]
        o.linear_small(rows, w, waits=0, **out)
        assert status.tolist()[0] == 8
        status.zero_()
        for _ in range(3):
            assert torch.equal(o.linear_small(rows, w, **out), want)
        assert status.tolist() == [0, 0]
    finally:
        status.zero_()
        o._tiled.pop(w.data_ptr(), None)


def test_all_blocks_of_a_product_fit_at_once():
    """By registers as well as by shared memory: 148 SMs hold four blocks of 16 features for up to eight rows, three otherwise."""
    o = ops()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    takes = lambda rows, n, k, **f: o.small_product(rows, torch.empty(n, k, device=DEV, dtype=torch.bfloat16), **f)
    assert takes(8, 64 * sms, 256) and not takes(8, 64 * sms + 16, 256) and takes(16, 48 * sms, 256) and not takes(16, 48 * sms + 16, 256)
    assert takes(8, 2 * 48 * sms, 256, gated=True) and not takes(8, 2 * (48 * sms + 16), 256, gated=True)
    assert takes(8, 96 * sms, 256, normed=True) and not takes(8, 96 * sms + 32, 256, normed=True)
    assert takes(8, 64 * sms, 1024) and not takes(8, 64 * sms + 16, 1024)
    # where the streaming product leaves whole sums too, and has many features to do it with
    assert takes(8, 4096, 512) and not takes(8, 4112, 512) and not takes(8, 4112, 392) and takes(8, 4112, 384) and takes(8, 4112, 520)
