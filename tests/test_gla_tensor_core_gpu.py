"""The tensor-core scan of gated linear attention (states of 128 x 128) against float64: at the edges of its batches of 32 and 64
tokens and blocks of 16, with decays strong enough to leave the batched form, and with values that are not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64
D = 128


def ops():
    from litellmengine_b200.csrc import ops as o
    return o


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def inputs(lens, H, low, g):
    """proj [T, 4 H D + 4], decays between `low` and 1, a state per entry."""
    T = sum(lens)
    proj = torch.randn(T, 4 * H * D + 4, generator=g, device=DEV)
    alpha = low + (1 - low) * torch.rand(T, H * D, generator=g, device=DEV)
    return proj, alpha, torch.randn(len(lens), H, D, D, generator=g, device=DEV)


def plain(proj, alpha, state, lens, H):
    T, end = sum(lens), state.to(F64).clone()
    q, k, v, gate = (proj[:, i * H * D:(i + 1) * H * D].view(T, H, D).to(F64) for i in range(4))
    out, at = torch.empty(T, H, D, dtype=F64, device=DEV), 0
    for e, n in enumerate(lens):
        S = end[e]
        for t in range(at, at + n):
            S = alpha[t].view(H, D, 1).to(F64) * S + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t]) * D ** -0.5
        end[e], at = S, at + n
    return out * torch.rsqrt(out.pow(2).mean(-1, keepdim=True) + 1e-5) * torch.nn.functional.silu(gate), end


def run(proj, alpha, state, lens, H, chunk, longest=0, tau=0.0):
    """One pass over whole entries (chunk None) or over pieces of `chunk` tokens; float32 outputs and the states after."""
    T, B, o = sum(lens), len(lens), ops()
    starts = [sum(lens[:i]) for i in range(B)]
    out, state = torch.full((T, H * D + 4), 7.0, device=DEV), state.clone()
    a = (proj, (0, H * D, 2 * H * D, 3 * H * D), alpha, torch.ones(D, device=DEV), 1e-5, D ** -0.5, 1.0, out, 4, state,
         i32(list(range(B))), i32(starts), i32(lens))
    if chunk is None:
        o.gla_scan(*a, None, B, o.GLA_FULL, None, None, H, D, D, longest=longest, tau=tau)
    else:
        items, chains = [], []
        for e, n in enumerate(lens):
            chains.append((e, len(items), -(-n // chunk)))
            items += [(e, starts[e] + at, min(chunk, n - at), len(items) + i) for i, at in enumerate(range(0, n, chunk))]
        n = len(items)
        ss, sa = torch.empty(n, H, D, D, device=DEV), torch.empty(n, H, D, device=DEV)
        rows = i32(items + [(-1, 0, 0, 0)])
        o.gla_scan(*a, rows, n + 1, o.GLA_LOCAL, ss, sa, H, D, D, longest=longest, tau=tau)
        o.gla_chain(state, ss, sa, i32(chains), B, i32(list(range(B))), H, D, D)
        o.gla_scan(*a, rows, n + 1, o.GLA_OUT, ss, sa, H, D, D, longest=longest, tau=tau)
    assert bool((out[:, :4] == 7).all())
    return out[:, 4:].view(T, H, D), state


@pytest.mark.parametrize("H", [1, 19])
@pytest.mark.parametrize("low", [0.9, 0.5, 0.0])
@pytest.mark.parametrize("chunk,longest", [(None, 0), (None, 1), (64, 0), (100, 0)])
def test_every_mode(H, low, chunk, longest):
    lens = [1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 100, 129]
    x = inputs(lens, H, low, torch.Generator(device=DEV).manual_seed(H))
    ref, end = plain(*x, lens, H)
    out, state = run(*x, lens, H, chunk, longest)
    # a state's element carries a rounding (2^-24) of each of the few dozen tokens it remembers and one more a batch; an output is a
    # sum of 128 products with it, divided by a norm: a handful of 2^-24 relative in the 2-norm
    assert float((state - end).norm() / end.norm()) < 4 * 2.0 ** -24
    assert float((out - ref).norm() / ref.norm()) < 8 * 2.0 ** -24


@pytest.mark.parametrize("chunk", [None, 64])
@pytest.mark.parametrize("what", [float("nan"), float("inf"), 3e38])
def test_a_value_that_is_not_finite_reaches_only_its_own_and_later_tokens(chunk, what):
    lens, H, at = [100, 70], 2, 45
    x = inputs(lens, H, 0.9, torch.Generator(device=DEV).manual_seed(5))
    clean, _ = run(*x, lens, H, chunk)
    x[0][at, 2 * H * D + 3] = what                            # column 3 of the first head's values
    out, state = run(*x, lens, H, chunk)
    first = out[:at]
    assert bool(torch.isfinite(first).all()) and float((first - clean[:at]).abs().max()) < 1e-4
    assert float((out[lens[0]:] - clean[lens[0]:]).abs().max()) < 1e-4        # the other entry
    assert float((out[:, 1] - clean[:, 1]).abs().max()) < 1e-4                 # the other head
    assert not bool(torch.isfinite(state[0, 0, :, 3]).all()) or what == 3e38
    assert bool(torch.isfinite(state[0, 0, :, 4:]).all())


@pytest.mark.parametrize("tau", [2.0, 8.0, 32.0])
@pytest.mark.parametrize("lens,chunk", [([30] * 6, None), ([100] * 3, None), ([512], 64)])
def test_no_further_from_64_bits_than_the_register_tiled_kernel(tau, lens, chunk):
    """The tensor cores cut sums off where multiply-adds round: before the rest of the newest tokens' product was added, states with
    decays of sigmoid(z)^(1/2) were 18 % further off."""
    H, g = 8, torch.Generator(device=DEV).manual_seed(3)
    proj = torch.randn(sum(lens), 4 * H * D + 4, generator=g, device=DEV)
    alpha = torch.sigmoid(torch.randn(sum(lens), H * D, generator=g, device=DEV)) ** (1 / tau)
    state = torch.zeros(len(lens), H, D, D, device=DEV)
    ref, end = plain(proj, alpha, state, lens, H)
    err = []
    for longest in (0, 1):                                    # 1: items too short for the tensor-core kernel, if it were true
        out, got = run(proj, alpha, state, lens, H, chunk, longest)
        err.append((float((out - ref).norm() / ref.norm()), float((got - end).norm() / end.norm())))
    assert err[0][0] <= err[1][0] and err[0][1] <= err[1][1], err


@pytest.mark.parametrize("chunk", [None, 64])
def test_gates_of_any_size(chunk):
    """silu from the lowest to the largest number, infinities and NaN; every other column has an ordinary one."""
    lens, H = [70], 2
    x = inputs(lens, H, 0.9, torch.Generator(device=DEV).manual_seed(11))
    top = 3.4028234663852886e38
    odd = [-top, -1e35, -1e30, -1e10, -1e4, -1000.0, -200.0, -100.0, -89.0, -88.0, -87.0, -80.0, -20.0, -1e-30, 0.0, 1e-30, 20.0, 88.0, 1e4, 1e30,
           top, float("inf"), float("-inf"), float("nan")]
    gates = x[0][:, 3 * H * D:4 * H * D]
    gates[:, 0:2 * len(odd):2] = torch.tensor(odd, device=DEV)
    ref, _ = plain(*x, lens, H)
    # in 64 bits too, silu of minus infinity is minus infinity times zero
    out = run(*x, lens, H, chunk)[0].to(F64)
    want = torch.where(ref.abs() > top, ref.sign() * float("inf"), ref)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
    fine = torch.isfinite(want)
    # a head's outputs have a root mean square of 1 in front of the gate and are a few dozen 2^-24 of that off, the small ones among them
    # too; below 1e-36 silu is zero in 32 bits, since exp(-g) is infinite
    size = torch.nn.functional.silu(gates.view(sum(lens), H, D).to(F64)).abs()
    assert float(((out - want).abs()[fine] / (1e-30 + size[fine])).max()) < 1e-5


@pytest.mark.parametrize("chunk", [None, 64])
@pytest.mark.parametrize("what", [float("inf"), float("-inf"), float("nan"), 3.4e38])
def test_a_state_that_is_not_finite_or_does_not_split(chunk, what):
    """Infinite, or too large for three bfloat16 values: the same numbers, zeros and NaN as the register-tiled kernel gives."""
    lens, H = [40, 20], 2
    x = inputs(lens, H, 0.9, torch.Generator(device=DEV).manual_seed(17))
    x[2][0, 1, 5, 7] = what
    out, state = run(*x, lens, H, chunk)
    want, end = run(*x, lens, H, chunk, longest=1)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isfinite(state), torch.isfinite(end))
    assert not bool(torch.isnan(out[:, 0]).any()) and not bool(torch.isnan(out[40:]).any())        # the other head, the other entry
    near = lambda a, b: float(((a - b).abs() / (1e-3 + b.abs()))[torch.isfinite(b)].max()) < 1e-3
    assert near(out, want) and near(state, end)


@pytest.mark.parametrize("chunk", [None, 64])
def test_strong_decays_stay_with_the_register_tiled_kernel(chunk):
    """Below tau = 2 the passes with outputs are the register-tiled kernel's, from 2 on (or unknown) the tensor cores'."""
    lens, H = [100, 64], 3
    x = inputs(lens, H, 0.5, torch.Generator(device=DEV).manual_seed(23))
    tensor, tiled = run(*x, lens, H, chunk), run(*x, lens, H, chunk, longest=1)
    assert not torch.equal(tensor[0], tiled[0])
    same = lambda a, b: all(torch.equal(i, j) for i, j in zip(a, b))
    assert same(run(*x, lens, H, chunk, tau=2.0), tensor) and same(run(*x, lens, H, chunk, tau=64.0), tensor)
    for tau in (0.1, 1.0, 1.99):
        got = run(*x, lens, H, chunk, tau=tau)
        if chunk is None:
            assert same(got, tiled)
        else:                                                 # the local pass takes any decays
            assert torch.equal(got[1], tensor[1]) and not torch.equal(got[0], tensor[0])
            assert float((got[0] - tiled[0]).abs().max()) < 1e-4
