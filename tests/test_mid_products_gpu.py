"""Products of 17 to 48 rows: against float64 at the edges of their tiles and cuts, and the gated form against the activation
kernel on the same sums, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from litellmengine_b200.csrc import ops as o
    return o


@pytest.mark.parametrize("N,K", [(16, 64), (1, 72), (100, 200), (129, 4104), (1000, 1096), (9216, 1024), (4096, 4096), (2048, 6144),
                                 (40000, 264)])
def test_product(N, K):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    for M in (17, 31, 32, 33, 48):
        x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
        want, carried = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        got = o.linear_mid(x, w, torch.float32)
        # K / 16 steps of products that are exact in float32 and at most 8 parts, each sum cut or rounded at 2^-23 of what it holds
        assert bool(((got.double() - want).abs() <= (K / 16 + 24) * 2.0 ** -23 * carried).all()), (M, N, K)
        assert torch.equal(o.linear_mid(x, w, torch.float32), got)
        assert torch.equal(o.linear_mid(x, w, torch.bfloat16), got.to(torch.bfloat16))
        if o.mid_product(x, w, torch.float32):
            assert torch.equal(o.linear(x, w, torch.float32), got)
    assert o.mid_product(x[:32], w, torch.float32) and not o.mid_product(x[:16], w, torch.float32)
    assert not o.mid_product(x.t().contiguous().t(), w, torch.float32) and not o.mid_product(x, w, torch.float16)
    assert o.stream_status(torch.device(DEV)).tolist() == [0, 0]


@pytest.mark.parametrize("N,K", [(64, 64), (192, 520), (3072, 1024), (12288, 2048), (20480, 264)])
def test_gated(N, K):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w = (torch.randn(2 * N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    for M in (17, 32, 33, 48):
        x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
        product = o.linear_mid(x, w, torch.bfloat16)              # as many tiles and parts: the same sums
        for a in o.ACTIVATIONS:
            got = o.linear_silu_mul(x, w, torch.bfloat16, activation=a, limit=1.5)
            assert torch.equal(got, o.silu_and_mul(product, activation=a, limit=1.5)), (M, N, K, a)
    assert o.stream_status(torch.device(DEV)).tolist() == [0, 0]


def test_sizes_it_leaves():
    o = ops()
    x = torch.randn(20, 260, device=DEV).to(torch.bfloat16)       # rows that are no multiple of 16 bytes
    w = torch.randn(384, 260, device=DEV).to(torch.bfloat16)
    assert not o.mid_product(x, w, torch.float32)
    assert torch.allclose(o.linear(x, w, torch.float32), x.float() @ w.float().t(), rtol=1e-3, atol=1e-3)
    w = torch.randn(2 * 72, 256, device=DEV).to(torch.bfloat16)   # features that do not fill their tiles
    assert not o.mid_product(x[:, :256].contiguous(), w, torch.bfloat16, gated=True)
    assert o.linear_silu_mul(x[:, :256].contiguous(), w, torch.bfloat16).shape == (20, 72)


@pytest.mark.parametrize("N,K,gated", [(4096, 4096, False), (1024, 256, False), (24576, 1024, False), (512, 2048, True)])
def test_a_wait_that_runs_out(N, K, gated):
    """Waits without tries: the status is set, the copies land before the blocks end, and the next products are right."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(9)
    w = (torch.randn(2 * N if gated else N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    x = torch.randn(40, K, generator=g, device=DEV).to(torch.bfloat16)
    out = dict(out_dtype=torch.bfloat16, activation="silu") if gated else dict(out_dtype=torch.float32)
    status = o.stream_status(torch.device(DEV))
    try:
        want = o.linear_mid(x, w, **out)
        assert status.tolist() == [0, 0]
        o.linear_mid(x, w, waits=0, **out)
        assert status.tolist()[0] == 8
        status.zero_()
        for _ in range(3):
            assert torch.equal(o.linear_mid(x, w, **out), want)
        assert status.tolist() == [0, 0]
    finally:
        status.zero_()


@pytest.mark.parametrize("N,K,gated,rows,large,takes", [
    (8192, 4096, False, 17, 48, True), (8192, 4096, False, 17, 0, False), (8192, 4096, False, 48, 32, False), (8192, 4096, False, 32, 32, True),
    (1024, 1024, False, 32, 0, True), (1024, 1024, False, 33, 0, False), (1024, 1024, False, 33, 48, True),      # 32 rows: a small product
    (1536, 384, False, 32, 48, True), (1536, 384, False, 33, 48, False), (4096, 2048, False, 33, 48, False),
    (7168, 1536, True, 33, 48, True), (2048, 2560, True, 48, 48, True)])
def test_products_that_gain(N, K, gated, rows, large, takes):
    o = ops()
    x, w = torch.zeros(rows, K, dtype=torch.bfloat16, device=DEV), torch.zeros(N * (1 + gated), K, dtype=torch.bfloat16, device=DEV)
    assert o.mid_product(x, w, torch.bfloat16, gated, large) == takes
