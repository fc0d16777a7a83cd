"""What stands in front of the delta rule's scan, read sixteen bytes at a time: portions that start and end anywhere in a block of four
tokens, with a cached context and without, and one to four taps, against the same rows one float further on, which such loads
cannot take and the other kernel prepares."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lens,contexts", [([9], [0]), ([5, 1, 2, 70], [0, 3, 1, 2]), ([1, 1, 1, 30], [7, 0, 2, 64]), ([33, 64], [1, 0])])
@pytest.mark.parametrize("D,V,taps", [(128, 128, 4), (128, 128, 1), (100, 36, 2), (104, 260, 3)])
def test_rows_from_anywhere(lens, contexts, D, V, taps):
    from litellmengine_b200.csrc import ops
    G, H, ra, rg = 3, 3, 16, 16
    C, T, n = 2 * G * D + H * V, sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(T + D + taps)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = types.SimpleNamespace(
        positions=i32([c + j for c, l in zip(contexts, lens) for j in range(l)]), token_entry=i32([i for i, l in enumerate(lens) for _ in range(l)]),
        entry_slot=i32([n - i for i in range(n)]), entry_q_start=i32([sum(lens[:i]) for i in range(n)]), entry_q_len=i32(lens), num_entries=n,
        max_q_len=max(lens))
    width = C + H + ra + rg
    stride = (width + 4) // 4 * 4
    rows, conv, wa, wg = rand(T, width), rand(C, taps) * 0.5, rand(ra, H * D) * 0.3, rand(rg, H * V) * 0.3
    dt, al, nw = rand(H * D), rand(H) * 0.5, 1 + 0.1 * rand(V)
    state0 = rand(n + 1, (H * V * ops.delta_padded(D) + taps * C + 3) // 4 * 4) * 0.1
    outs = []
    for shift in (0, 1):
        proj = torch.full((T * stride + 4,), float("nan"), device=DEV)[shift:shift + T * stride].view(T, stride)[:, :width]
        proj.copy_(rows)
        state, out = state0.clone(), torch.zeros(T, H * V, device=DEV)
        ops.delta_rule(proj, (0, C, C + H, C + H + ra), (ra, rg), conv, wa, wg, dt, al, nw, 1e-5, 1.0, out, 0, state, batch, H, G, D, V)
        outs.append((out, state))
    (a, sa), (b, sb) = outs
    assert bool(torch.isfinite(a).all()) and bool(torch.isfinite(sa).all())
    # the same convolutions; the squares of a head are added in another order: at most 12 roundings of 2^-24 in a norm of q and of k, half
    # of that in the unit vectors, and every token of a portion adds its own to the state that the next ones read
    bound = 12 * 2.0 ** -24 * (2 + max(lens))
    assert float((a - b).norm()) <= bound * float(b.norm()) and float((sa - sb).norm()) <= bound * float(sb.norm())
    assert ops.stream_status(torch.device(DEV)).tolist() == [0, 0]
