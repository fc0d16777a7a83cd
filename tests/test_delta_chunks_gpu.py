"""The delta rule's scan, eight tokens a chunk, against the token-by-token recurrence in 64 bits: portions that end anywhere in
a chunk and in a batch of sixteen, alone and beside others, for every layout of columns that the sizes choose."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("H,D,V,lens", [(2, 128, 128, [2, 3, 7, 8, 9]), (4, 128, 128, [15, 16]), (8, 128, 128, [17, 33]), (16, 128, 128, [40, 24, 9]),
                                        (3, 64, 20, [5, 23]), (2, 32, 33, [8, 31]), (2, 256, 64, [12, 18])])
def test_portions_end_anywhere(H, D, V, lens):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(H * 100 + D)
    taps, ra, rg, eps, T = 3, 4, 5, 1e-5, sum(lens)
    C = 2 * H * D + H * V
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, conv = rnd(T, C + H + ra + rg), rnd(C, taps) * 0.5
    wa, wg, dt, al, nw = rnd(ra, H * D) * 0.3, rnd(rg, H * V) * 0.3, rnd(H * D), rnd(H) * 0.5, 1 + 0.1 * rnd(V)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    b = types.SimpleNamespace(positions=i32([p for n in lens for p in range(n)]), token_entry=i32([e for e, n in enumerate(lens) for _ in range(n)]),
                              entry_slot=i32(list(range(len(lens)))), entry_q_start=i32(starts), entry_q_len=i32(lens), num_entries=len(lens))
    DP = ops.delta_padded(D)
    state = torch.zeros(len(lens), (H * V * DP + taps * C + 3) // 4 * 4, device=DEV)
    out = torch.zeros(T, H * V, device=DEV)
    ops.delta_rule(proj, (0, C, C + H, C + H + ra), (ra, rg), conv, wa, wg, dt, al, nw, eps, 1.0, out, 0, state, b, H, H, D, V, single=False)
    x = proj.to(F64)
    for e, n in enumerate(lens):
        u = x[starts[e]:starts[e] + n]
        mixed = sum(torch.nn.functional.pad(u[:, :C], (0, 0, taps - 1 - j, 0))[:n] * conv[:, j].to(F64) for j in range(taps))
        mixed = torch.nn.functional.silu(mixed)
        unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
        q, k = unit(mixed[:, :H * D].view(n, H, D)) * D ** -0.5, unit(mixed[:, H * D:2 * H * D].view(n, H, D))
        v, beta = mixed[:, 2 * H * D:].view(n, H, V), torch.sigmoid(u[:, C:C + H])
        decay = torch.exp(-torch.exp(al.to(F64))[None, :, None] * torch.nn.functional.softplus(u[:, C + H:C + H + ra] @ wa.to(F64) + dt.to(F64)).view(n, H, D))
        S, ref = torch.zeros(H, D, V, dtype=F64, device=DEV), torch.empty(n, H, V, dtype=F64, device=DEV)
        for t in range(n):
            S = decay[t][:, :, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None, :]
            ref[t] = torch.einsum("hdv,hd->hv", S, q[t])
        ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + eps) * nw.to(F64) * torch.sigmoid(u[:, C + H + ra:] @ wg.to(F64)).view(n, H, V)
        err = ((out[starts[e]:starts[e] + n].view(n, H, V).to(F64) - ref).abs() / (1 + ref.abs())).max()
        # a few dozen 32-bit roundings a token; the norm divides by o's size, which near a sequence's start is small
        assert float(err) < 1e-4, (n, float(err))
        got = state[e, :H * V * DP].view(H, V, DP)[..., :D].transpose(1, 2).to(F64)
        assert float((got - S).abs().max()) < 2e-5 * max(1.0, float(S.abs().max())), n
