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
