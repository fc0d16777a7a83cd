"""The paired tcgen05 product at every kind of last token tile: a token's result does not depend on how many there are, and nothing
behind the last one is written."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N,K", [(528, 136), (256, 1024)])
def test_rows_at_the_end(N, K):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(1024, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    whole, gated = ops.linear_pair(x, w, torch.float32), ops.linear_pair_silu_mul(x, w)
    for T in (1, 127, 128, 129, 200, 255, 256, 257, 383, 384, 385, 511, 513, 640, 769, 1023):
        buf = torch.full((T + 300, N), 7.0, device=DEV)
        ops.linear_pair(x[:T], w, torch.float32, out=buf[:T])
        assert torch.equal(buf[:T], whole[:T]) and bool((buf[T:] == 7).all()), T
        ops.linear_pair(x[:T], w, torch.float32, out=buf[:T], accumulate=True)
        assert torch.equal(buf[:T], whole[:T] + whole[:T]) and bool((buf[T:] == 7).all()), T
        assert torch.equal(ops.linear_pair_silu_mul(x[:T], w), gated[:T]), T
    assert ops.stream_status(torch.device(DEV)).tolist() == [0, 0]
