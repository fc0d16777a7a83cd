"""latent_prepare's two forms (latents held in registers, and read twice where they are too wide for that) against each other, bit for
bit, and against 64 bits: the norms' sums keep one order, so that a row in the cache does not depend on how wide its neighbours are."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def prepare(proj, Q, R, P, wq, wkv, off=0):
    from litellmengine_b200.csrc import ops
    T, page = proj.shape[0], 16
    keys = torch.zeros(-(-T // page), 1, page, R + P, device=DEV)
    status = i32([0, 0])
    batch = types.SimpleNamespace(positions=i32(list(range(T))), token_entry=i32([0] * T), entry_slot=i32([0]))
    cq = ops.latent_prepare(proj, off, off + Q, Q, R, P, 0, wq, wkv, 1e-5, None, keys, batch, i32([list(range(keys.shape[0]))]), page, status,
                            torch.float32)
    assert status.tolist() == [0, 0]
    return cq, keys.view(-1, R + P)[:T]


@pytest.mark.parametrize("Q,R,off", [(1536, 512, 0), (8, 4, 0), (255, 257, 3), (2048, 1024, 1), (300, 1000, 0), (2049, 512, 0), (512, 1030, 2)])
def test_norms_of_both_latents(Q, R, off):
    P, T = 4, 19
    g = torch.Generator(device=DEV).manual_seed(Q + R)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, wq, wkv = rnd(T, off + Q + R + P), 1 + 0.1 * rnd(Q), 1 + 0.1 * rnd(R)
    cq, rows = prepare(proj, Q, R, P, wq, wkv, off)
    rms = lambda x, w: x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w.to(F64)
    x = proj.to(F64)
    # a mean of squares of one sign (a few 2^-24), its root, a division and two products: some roundings each
    tol = 12 * 2.0 ** -24
    assert float(((cq - rms(x[:, off:off + Q], wq)).abs() / (1e-3 + cq.abs())).max()) < tol
    assert float(((rows[:, :R] - rms(x[:, off + Q:off + Q + R], wkv)).abs() / (1e-3 + rows[:, :R].abs())).max()) < tol
    assert torch.equal(rows[:, R:], proj[:, off + Q + R:])


def test_a_latent_is_normed_alike_in_both_forms():
    """The other latent's width chooses the form."""
    P, T, Q, R = 4, 11, 1536, 512
    g = torch.Generator(device=DEV).manual_seed(2)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    dq, dkv, kr, wq, wkv = rnd(T, Q), rnd(T, R), rnd(T, P), 1 + 0.1 * rnd(Q), 1 + 0.1 * rnd(R)
    held = prepare(torch.cat([dq, dkv, kr], 1), Q, R, P, wq, wkv)
    wide_q = prepare(torch.cat([rnd(T, 4096), dkv, kr], 1), 4096, R, P, torch.ones(4096, device=DEV), wkv)
    wide_kv = prepare(torch.cat([dq, rnd(T, 2048), kr], 1), Q, 2048, P, wq, torch.ones(2048, device=DEV))
    assert torch.equal(held[1], wide_q[1]) and torch.equal(held[0], wide_kv[0])
