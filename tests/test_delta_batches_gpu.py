"""The delta rule in batches of sixteen tokens on the tensor cores against the token-by-token recurrence in 64 bits: portions that end
anywhere in a batch, blocks of 32 columns, heads that share keys, decays down to nothing, values that are not finite."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
TAPS, RA, RG, EPS = 3, 4, 5, 1e-5


def setup(H, G, V, lens, dt_std, seed):
    D, T, C = 128, sum(lens), 2 * G * 128 + H * V
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    w = dict(proj=rnd(T, C + H + RA + RG), conv=rnd(C, TAPS) * 0.5, wa=rnd(RA, H * D) * 0.3, wg=rnd(RG, H * V) * 0.3, dt=rnd(H * D) * dt_std,
             al=rnd(H) * 0.5, nw=1 + 0.1 * rnd(V), state=rnd(len(lens), (H * V * D + TAPS * C + 3) // 4 * 4))
    w["state"][:, H * V * D:] = 0                             # no tokens in front of these
    starts = [sum(lens[:i]) for i in range(len(lens))]
    batch = types.SimpleNamespace(positions=i32([p for n in lens for p in range(n)]), token_entry=i32([e for e, n in enumerate(lens) for _ in range(n)]),
                                  entry_slot=i32(list(range(len(lens)))), entry_q_start=i32(starts), entry_q_len=i32(lens), num_entries=len(lens),
                                  max_q_len=max(lens))
    return w, batch, starts


def run(w, batch, H, G, V, batched=True):
    """With the kernels of sixteen tokens a batch, or of eight, whatever the sizes would have chosen."""
    from litellmengine_b200.csrc import ops
    C = 2 * G * 128 + H * V
    state, out = w["state"].clone(), torch.zeros(w["proj"].shape[0], H * V, device=DEV)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(ops, "delta_batched", lambda *a: batched)
        ops.delta_rule(w["proj"], (0, C, C + H, C + H + RA), (RA, RG), w["conv"], w["wa"], w["wg"], w["dt"], w["al"], w["nw"], EPS, 1.0, out, 0,
                       state, batch, H, G, 128, V, single=False)
    assert ops.stream_status(DEV).tolist() == [0, 0]
    return out, state


@pytest.mark.parametrize("H,G,V,lens", [(12, 12, 128, [1, 2, 15]), (12, 6, 128, [16, 17]), (16, 16, 128, [33, 31]), (2, 2, 32, [1 + i for i in range(32)]),
                                        (24, 24, 64, [40]), (5, 5, 96, [16, 47, 3, 65])])
@pytest.mark.parametrize("dt_std", [1.0, 8.0])
def test_portions_end_anywhere(H, G, V, lens, dt_std):
    D = 128
    w, batch, starts = setup(H, G, V, lens, dt_std, H * 100 + V)
    out, state = run(w, batch, H, G, V)
    C, x = 2 * G * D + H * V, w["proj"].to(F64)
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    for e, n in enumerate(lens):
        u = x[starts[e]:starts[e] + n]
        mixed = torch.nn.functional.silu(sum(torch.nn.functional.pad(u[:, :C], (0, 0, TAPS - 1 - j, 0))[:n] * w["conv"][:, j].to(F64) for j in range(TAPS)))
        q, k = (unit(mixed[:, i * G * D:(i + 1) * G * D].view(n, G, D)).repeat_interleave(H // G, dim=1) for i in range(2))
        v, beta, q = mixed[:, 2 * G * D:].view(n, H, V), torch.sigmoid(u[:, C:C + H]), q * D ** -0.5
        decay = torch.exp(-torch.exp(w["al"].to(F64))[None, :, None] * torch.nn.functional.softplus(u[:, C + H:C + H + RA] @ w["wa"].to(F64) + w["dt"].to(F64)).view(n, H, D))
        S = w["state"][e, :H * V * D].view(H, V, D).transpose(1, 2).to(F64)
        ref = torch.empty(n, H, V, dtype=F64, device=DEV)
        for t in range(n):
            S = decay[t][:, :, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None, :]
            ref[t] = torch.einsum("hdv,hd->hv", S, q[t])
        ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + EPS) * w["nw"].to(F64) * torch.sigmoid(u[:, C + H + RA:] @ w["wg"].to(F64)).view(n, H, V)
        # a few dozen 32-bit roundings a token; the norm divides by o's size, which can be small
        assert float(((out[starts[e]:starts[e] + n].view(n, H, V).to(F64) - ref).abs() / (1 + ref.abs())).max()) < 1e-4, n
        got = state[e, :H * V * D].view(H, V, D).transpose(1, 2).to(F64)
        assert float((got - S).abs().max()) < 2e-5 * max(1.0, float(S.abs().max())), n


@pytest.mark.parametrize("at", [0, 14, 16, 36])
@pytest.mark.parametrize("piece", ["value", "key"])
def test_what_is_not_finite_reaches_only_its_own_and_later_tokens(at, piece):
    H = G = 12
    w, batch, _ = setup(H, G, 128, [37, 20], 1.0, 7)
    clean, _ = run(w, batch, H, G, 128)
    w["proj"][at, (2 if piece == "value" else 1) * G * 128 + 3] = float("nan")      # the first head's; values stand behind q and k
    out, state = run(w, batch, H, G, 128)
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[37:], clean[37:])
    assert torch.equal(out[:, 128:], clean[:, 128:]) and not bool(torch.isfinite(out[at:37, 3]).any())
    assert bool(torch.isfinite(state[1, :H * 128 * 128]).all())


def test_no_further_from_64_bits_than_the_kernels_of_eight_tokens():
    """Both forms on the same portions.  What both take in (unit norms, decays) is the larger part of their errors; the tensor cores
    cut sums off where multiply-adds round, which made this form's states 7 % worse before the rest of the largest product was added."""
    H, D, V, n = 12, 128, 128, 300
    C, err = 2 * H * D + H * V, {"batches": [0.0, 0.0], "eight": [0.0, 0.0]}
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    for seed in range(4):
        w, batch, _ = setup(H, H, V, [n], 1.0, seed)
        w["state"].zero_()
        x = w["proj"].to(F64)
        mixed = torch.nn.functional.silu(sum(torch.nn.functional.pad(x[:, :C], (0, 0, TAPS - 1 - j, 0))[:n] * w["conv"][:, j].to(F64) for j in range(TAPS)))
        q, k = (unit(mixed[:, i * H * D:(i + 1) * H * D].view(n, H, D)) for i in range(2))
        v, beta, q = mixed[:, 2 * H * D:].view(n, H, V), torch.sigmoid(x[:, C:C + H]), q * D ** -0.5
        decay = torch.exp(-torch.exp(w["al"].to(F64))[None, :, None] * torch.nn.functional.softplus(x[:, C + H:C + H + RA] @ w["wa"].to(F64) + w["dt"].to(F64)).view(n, H, D))
        S, ref = torch.zeros(H, D, V, dtype=F64, device=DEV), torch.empty(n, H, V, dtype=F64, device=DEV)
        for t in range(n):
            S = decay[t][:, :, None] * S
            S = torch.baddbmm(S, k[t][:, :, None], (beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0]))[:, None, :])
            ref[t] = (q[t][:, None, :] @ S)[:, 0]
        ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + EPS) * w["nw"].to(F64) * torch.sigmoid(x[:, C + H + RA:] @ w["wg"].to(F64)).view(n, H, V)
        for form in err:
            out, state = run(w, batch, H, H, V, form == "batches")
            got = state[0, :H * V * D].view(H, V, D).transpose(1, 2).to(F64)
            err[form][0] += float((out.view(n, H, V) - ref).norm() / ref.norm())
            err[form][1] += float((got - S).norm() / S.norm())
    assert err["batches"][0] <= err["eight"][0] and err["batches"][1] <= err["eight"][1], err


@pytest.mark.parametrize("H,V,entries,longest,want", [
    (16, 128, 3, 255, False), (16, 128, 3, 256, True), (16, 128, 1, 8000, False), (17, 128, 1, 256, True),       # 2,048 and 2,176 columns
    (6, 128, 2, 999, False), (6, 128, 2, 1000, True), (12, 128, 1, 1000, False), (11, 128, 1, 1000, False),        # 1,536: one request, two
    (37, 128, 2, 256, True), (38, 128, 2, 256, False), (16, 48, 6, 300, False), (16, 96, 6, 300, True), (16, 128, 0, 300, False)])
def test_which_kernels_a_step_takes(H, V, entries, longest, want):
    from litellmengine_b200.csrc import ops
    assert ops.delta_batched(types.SimpleNamespace(num_entries=entries, max_q_len=longest), H, 128, V) == want
    assert not ops.delta_batched(types.SimpleNamespace(num_entries=entries, max_q_len=longest), H, 64, V)


def test_a_portion_beside_single_tokens_and_states_that_are_not_finite():
    """Against the kernels of eight tokens, which take every column by itself: a portion beside decoding requests, decays of zero and one,
    and states that hold infinities, NaN and numbers beyond 2^60 in single places."""
    H, V, lens = 4, 64, [70, 1, 1, 33, 1]
    w, batch, starts = setup(H, H, V, lens, 1.0, 3)
    C = 2 * H * 128 + H * V
    w["dt"][:128:3], w["dt"][1:128:3] = -200.0, 3e4            # decays of one and of zero
    S = w["state"][:, :H * V * 128].view(len(lens), H, V, 128)
    S[0, 1, 5, 9], S[0, 2, 40, 100], S[1, 0, 3, 3], S[3, 3, 63, 127], S[3, 0, 0, 0] = float("inf"), float("nan"), 1e30, float("-inf"), 3e38
    out, state = run(w, batch, H, H, V)
    ref, end = run(w, batch, H, H, V, False)
    assert torch.equal(torch.isfinite(state), torch.isfinite(end))
    ok = torch.isfinite(end)
    assert float(((state - end).abs() / (1e-2 + end.abs()))[ok].max()) < 1e-3
    # outputs: what an infinity gives depends on the order of a sum, so those heads are left out
    for e, (a, n) in enumerate(zip(starts, lens)):
        for h in range(H):
            if (e, h) not in ((0, 1), (0, 2), (3, 0), (3, 3)):
                x, y = (t[a:a + n, h * V:(h + 1) * V] for t in (out, ref))
                assert float(((x - y).abs() / (1e-2 + y.abs())).max()) < 1e-3, (e, h)


def test_without_room_for_the_images_a_step_takes_the_kernels_of_eight_tokens():
    H, V = 12, 128
    w, batch, _ = setup(H, H, V, [300, 20], 1.0, 9)
    want = run(w, batch, H, H, V, False)
    real, refused = torch.empty, []

    def scarce(*a, **kw):
        if not refused and isinstance(a[0], int):
            refused.append(a[0])
            raise torch.cuda.OutOfMemoryError("no room for the images")
        return real(*a, **kw)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(torch, "empty", scarce)
        got = run(w, batch, H, H, V)
    assert refused and all(torch.equal(a, b) for a, b in zip(got, want))


def test_entries_without_tokens():
    """They keep their states and touch nobody's rows."""
    H, V, lens = 5, 32, [0, 40, 0, 17, 0]
    w, batch, _ = setup(H, H, V, lens, 1.0, 2)
    out, state = run(w, batch, H, H, V)
    full = [1, 3]
    short, _, _ = setup(H, H, V, [40, 17], 1.0, 2)
    short["state"] = w["state"][full].contiguous()
    _, other, _ = setup(H, H, V, [40, 17], 1.0, 2)
    for k in ("proj", "conv", "wa", "wg", "dt", "al", "nw"):
        short[k] = w[k]
    want, end = run(short, other, H, H, V)
    assert torch.equal(out, want) and torch.equal(state[full], end)
    assert torch.equal(state[[0, 2, 4]], w["state"][[0, 2, 4]])
