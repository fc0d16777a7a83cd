"""Both forms of the experts' router (a token a block for short steps, four for long ones) against the plain rule in float64: on
both sides of the switch, widths on both sides of the 1,024 columns that a lane fetches ahead and of sixteen-byte rows, more
than 32 choices a token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("T", [1, 296, 297, 603])
@pytest.mark.parametrize("W,E,top,score,groups", [(24, 5, 2, "sigmoid", None), (1024, 20, 3, "softmax", None), (1032, 16, 4, "sigmoid", (4, 2)),
                                                  (2056, 9, 9, "softmax", None), (1027, 70, 40, "sigmoid", None), (264, 64, 64, "sigmoid", None),
                                                  (40, 66, 33, "softmax", (3, 2))])
def test_router_against_the_plain_rule(T, W, E, top, score, groups):
    from litellmengine_b200.csrc import ops
    g = torch.Generator().manual_seed(T + W)
    x, wr = torch.randn(T, W, generator=g), torch.randn(E, W, generator=g) * W ** -0.5
    correction = torch.randn(E, generator=g) * 0.1 if score == "softmax" else None
    shared = torch.randn(W, generator=g) * W ** -0.5
    z = x.to(F64) @ wr.to(F64).T
    s = torch.softmax(z, -1) if score == "softmax" else torch.sigmoid(z)
    choose = s if correction is None else s + correction.to(F64)
    if groups:
        count, keep = groups
        best = choose.view(T, count, -1).topk(2, dim=-1).values.sum(-1).topk(keep, dim=-1).indices
        ok = torch.zeros(T, count, dtype=torch.bool).scatter_(1, best, True)
        choose = choose.masked_fill(~ok[:, :, None].expand(T, count, E // count).reshape(T, E), float("-inf"))
    pick = choose.topk(top, dim=-1).indices
    chosen = s.gather(1, pick)
    want = torch.zeros(T, E, dtype=F64).scatter_(1, pick, chosen / (chosen.sum(-1, keepdim=True) + 1e-20) * 1.5)
    dense, ids, wts, share = ops.moe_route(x.to(DEV), wr.to(DEV), top, groups, 1.5, lists=True, score=score,
                                           correction=None if correction is None else correction.to(DEV), shared_gate=shared.to(DEV))
    # A score's relative error is that of its logit's sum, some sqrt(W) roundings of 2^-24, and a few more; two experts, or two
    # groups, nearer than that at the edge of the choice may change places.
    tol = 2.0 ** -24 * (4 * W ** 0.5 + 16) * 1.5
    dense, ids, wts = dense.cpu().to(F64), ids.cpu().long(), wts.cpu().to(F64)
    assert bool((ids.sort(1).values[:, 1:] > ids.sort(1).values[:, :-1]).all()) and int(ids.min()) >= 0
    assert torch.equal(torch.zeros(T, E, dtype=F64).scatter_(1, ids, wts), dense)
    same = (ids.sort(1).values == pick.sort(1).values).all(1)
    assert float((dense - want)[same].abs().max()) < tol
    # the weights of a choice in another order of two experts that tie differ by as little
    assert int((~same).sum()) <= 1 + T // 200
    assert bool((choose.gather(1, ids).sum(1) >= choose.gather(1, pick).sum(1) - (0 if not groups else 1e-5) - top * tol)[~same].all())
    assert float((share.cpu().to(F64) - torch.sigmoid(x.to(F64) @ shared.to(F64))).abs().max()) < tol
