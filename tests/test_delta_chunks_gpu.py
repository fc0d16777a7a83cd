"""The delta rule's scan, eight tokens a chunk, against the token-by-token recurrence in 64 bits: portions that end anywhere in
a chunk and in a batch of sixteen, alone and beside others, for every layout of columns that the sizes choose, up to 32 entries (walked longest first) and more."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("H,D,V,lens", [(2, 128, 128, [2, 3, 7, 8, 9]), (4, 128, 128, [15, 16]), (8, 128, 128, [17, 33]), (2, 128, 128, [1 + i % 19 for i in range(32)]), (1, 64, 16, [1 + i % 5 for i in range(40)]), (16, 128, 128, [40, 24, 9]),
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
                              entry_slot=i32(list(range(len(lens)))), entry_q_start=i32(starts), entry_q_len=i32(lens), num_entries=len(lens), max_q_len=max(lens))
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


@pytest.mark.parametrize("T,H,D,V,ra,rg", [(1 + 2, 1, 128, 128, 64, 33), (63, 2, 64, 24, 33, 80), (64, 3, 32, 20, 48, 64), (65, 1, 128, 64, 130, 1),
                                           (129, 5, 128, 33, 64, 64)])
def test_low_rank_products_on_the_tensor_cores(T, H, D, V, ra, rg):
    """bfloat16 weights (the split product) against the same weights as float32 (plain multiply-adds): edges of 64 tokens, 128
    channels, 64 and 16 ranks, widths with and without sixteen-byte rows, a token with an infinity and one with a NaN."""
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    taps, C = 2, 2 * H * D + H * V
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, conv = rnd(T, C + H + ra + rg), rnd(C, taps)
    proj[-1, C + H] = float("inf")
    proj[-2, C + H + ra] = float("nan")
    wa, wg = (rnd(ra, H * D) * 0.2).bfloat16(), (rnd(rg, H * V) * 0.2).bfloat16()
    dt, al, nw = rnd(H * D), rnd(H) * 0.5, torch.ones(V, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    b = types.SimpleNamespace(positions=i32(list(range(T))), token_entry=i32([0] * T), entry_slot=i32([0]), entry_q_start=i32([0]),
                              entry_q_len=i32([T]), num_entries=1)
    got = []
    for kind in (torch.bfloat16, torch.float32):
        state = torch.zeros(1, (H * V * ops.delta_padded(D) + taps * C + 3) // 4 * 4, device=DEV)
        out = torch.zeros(T, H * V, device=DEV)
        ops.delta_rule(proj, (0, C, C + H, C + H + ra), (ra, rg), conv, wa.to(kind), wg.to(kind), dt, al, nw, 1e-5, 1.0, out, 0, state, b,
                       H, H, D, V, single=False)
        got.append((out, state[:, :H * V * ops.delta_padded(D)].clone()))
    (a, sa), (w, sw) = got
    assert torch.equal(torch.isnan(a), torch.isnan(w)) and torch.isnan(w[-2]).all()
    # rank products of 32-bit rounding a number, through a logistic function or a decay; the norm divides by the outputs' size
    assert torch.allclose(a, w, rtol=2e-4, atol=2e-5, equal_nan=True)
    assert torch.allclose(sa, sw, rtol=1e-4, atol=2e-5, equal_nan=True)


@pytest.mark.parametrize("T,H,D,V,ra,rg", [(3, 1, 128, 128, 64, 33), (64, 2, 64, 24, 33, 80), (65, 5, 128, 33, 200, 64)])
def test_decays_and_gates_of_the_low_rank_products(T, H, D, V, ra, rg):
    """Each number alone against 64 bits: T requests of one token that write nothing (beta zero) leave the decay times the state they
    found, and two runs that differ in the gate's weights only have outputs whose ratio is the gate."""
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    taps, C = 2, 2 * H * D + H * V
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, conv = rnd(T, C + H + ra + rg), rnd(C, taps)
    proj[:, C:C + H] = -200.0
    wa, wg = (rnd(ra, H * D) * 0.2).bfloat16(), (rnd(rg, H * V) * 0.2).bfloat16()
    dt, al, nw = rnd(H * D), rnd(H) * 0.5 - 2, torch.ones(V, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    b = types.SimpleNamespace(positions=i32([0] * T), token_entry=i32(list(range(T))), entry_slot=i32(list(range(T))),
                              entry_q_start=i32(list(range(T))), entry_q_len=i32([1] * T), num_entries=T)
    DP, outs = ops.delta_padded(D), []
    for w in (wg, torch.zeros_like(wg)):
        state = torch.zeros(T, (H * V * DP + taps * C + 3) // 4 * 4, device=DEV)
        state[:, :H * V * DP] = 1.0
        out = torch.zeros(T, H * V, device=DEV)
        ops.delta_rule(proj, (0, C, C + H, C + H + ra), (ra, rg), conv, wa, w, dt, al, nw, 1e-5, 1.0, out, 0, state, b, H, H, D, V,
                       single=False)
        outs.append(out.to(F64))
    x = proj.to(F64)
    gate = torch.sigmoid(x[:, C + H + ra:] @ wg.to(F64))
    z = x[:, C + H:C + H + ra] @ wa.to(F64) + dt.to(F64)
    decay = torch.exp(-torch.exp(al.to(F64))[None, :, None] * torch.nn.functional.softplus(z).view(T, H, D))
    got = state[:, :H * V * DP].view(T, H, V, DP)[..., :D].to(F64)
    rms = lambda e: float(e.pow(2).mean().sqrt())
    # A few roundings of 2^-24 and the error of a sum of up to 200 exact products: 1e-7 to 2e-7.  Without the third part of the
    # inputs' split it is 2^-17 of the sum, above 5e-6 of a gate or a decay.
    assert rms(0.5 * outs[0] / outs[1] / gate - 1) < 1e-6
    assert rms(got / decay[:, :, None, :] - 1) < 1e-6


@pytest.mark.parametrize("D,V,H", [(128, 128, 2), (64, 20, 2), (128, 128, 16)])
def test_a_value_that_is_not_finite_reaches_only_later_tokens(D, V, H):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(D)
    T, bad, taps, ra, rg, C = 37, 14, 1, 4, 5, 2 * H * D + H * V
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, conv = rnd(T, C + H + ra + rg), rnd(C, taps)
    wa, wg, dt, al, nw = rnd(ra, H * D) * 0.3, rnd(rg, H * V) * 0.3, rnd(H * D), rnd(H) * 0.5, torch.ones(V, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    b = types.SimpleNamespace(positions=i32(list(range(T))), token_entry=i32([0] * T), entry_slot=i32([0]), entry_q_start=i32([0]),
                              entry_q_len=i32([T]), num_entries=1, max_q_len=T)
    outs = []
    for spoil in (False, True):
        x = proj.clone()
        if spoil:
            x[bad, 2 * H * D:C] = float("nan")
        state = torch.zeros(1, (H * V * ops.delta_padded(D) + taps * C + 3) // 4 * 4, device=DEV)
        out = torch.zeros(T, H * V, device=DEV)
        ops.delta_rule(x, (0, C, C + H, C + H + ra), (ra, rg), conv, wa, wg, dt, al, nw, 1e-5, 1.0, out, 0, state, b, H, H, D, V, single=False)
        outs.append(out)
    assert torch.equal(outs[0][:bad], outs[1][:bad]) and not bool(torch.isfinite(outs[1][bad:]).any())
