"""The register-tiled scan of gated linear attention and the tiled decay kernel against float64, over every state size they
take, at the edges of their batches of 16 tokens and chunks of 64, in each mode, with a block an SM and with several.  (States of 128 x
128 are told that their items are short, which keeps them from the tensor-core kernel.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("D,V,H", [(64, 32, 3), (64, 128, 3), (128, 32, 3), (128, 64, 3), (128, 128, 3), (64, 64, 20), (128, 128, 20)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_scan_in_one_pass_and_over_chunks(D, V, H, out_dtype):
    from litellmengine_b200.csrc import ops
    g = torch.Generator(device=DEV).manual_seed(D + V)
    rank, eps, C = 20, 1e-5, 64
    lens, tau = [1, 15, 16, 17, 63, 64, 65, 130], 4.0
    T = sum(lens)
    W = 2 * H * D + 2 * H * V + rank
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj = rnd(T, W)
    offs = (0, H * D, 2 * H * D, 2 * H * D + H * V)
    w2t, b2, norm = rnd(rank, H * D), rnd(H * D) * 2, 1 + 0.1 * rnd(V)
    b2[0], b2[1] = 200.0, -300.0                              # never forgets; forgets at once
    w2t[:, 0] = w2t[:, 1] = 0.0
    alpha = ops.gla_decay(proj, 2 * H * D + 2 * H * V, rank, w2t, b2, tau)
    z = proj[:, -rank:].to(F64) @ w2t.to(F64) + b2.to(F64)
    want = torch.exp(torch.nn.functional.logsigmoid(z) / tau)
    assert float((alpha.to(F64) - want).abs().max()) < 3e-6
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    slots = list(range(len(lens)))[::-1]
    state0 = rnd(len(lens), H, D, V)
    q, k = (proj[:, o:o + H * D].view(T, H, D).to(F64) for o in offs[:2])
    v, gate = (proj[:, o:o + H * V].view(T, H, V).to(F64) for o in offs[2:])
    ref, end = torch.empty(T, H, V, dtype=F64, device=DEV), state0.to(F64).clone()
    for e, n in enumerate(lens):
        S = end[slots[e]]
        for t in range(starts[e], starts[e] + n):
            S = alpha[t].view(H, D, 1).to(F64) * S + k[t][:, :, None] * v[t][:, None, :]
            ref[t] = torch.einsum("hdv,hd->hv", S, q[t]) * D ** -0.5
        end[slots[e]] = S
    ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + eps) * norm.to(F64) * torch.nn.functional.silu(gate) * 0.5
    tol = 2e-4 if out_dtype == torch.float32 else 2e-2       # 130 tokens of 32-bit sums; 2^-9 of values up to about 10
    for chunked in (False, True):
        state, out = state0.clone(), torch.full((T, H * V + 8), 7.0, device=DEV, dtype=out_dtype)
        a = (proj, offs, alpha, norm, eps, D ** -0.5, 0.5, out, 4, state, i32(slots), i32(starts), i32(lens))
        if not chunked:
            ops.gla_scan(*a, None, len(lens), ops.GLA_FULL, None, None, H, D, V, longest=1)
        else:
            chunks, chains = [], []
            for e, n in enumerate(lens):
                chains.append((e, len(chunks), -(-n // C)))
                for at in range(0, n, C):
                    chunks.append((e, starts[e] + at, min(C, n - at), len(chunks)))
            n = len(chunks)
            chunks, chains = i32(chunks + [(-1, 0, 0, 0)]), i32(chains)
            ss, sa = torch.empty(n, H, D, V, device=DEV), torch.empty(n, H, D, device=DEV)
            ops.gla_scan(*a, chunks, n + 1, ops.GLA_LOCAL, ss, sa, H, D, V, longest=1)
            ops.gla_chain(state, ss, sa, chains, len(lens), i32(slots), H, D, V)
            ops.gla_scan(*a, chunks, n + 1, ops.GLA_OUT, ss, sa, H, D, V, longest=1)
        got = out[:, 4:4 + H * V].view(T, H, V).to(F64)
        assert float(((got - ref).abs() / (1 + ref.abs())).max()) < tol, chunked
        assert float((state.to(F64) - end).abs().max()) < 2e-4 * float(end.abs().max())
        assert float((out[:, :4].float() - 7).abs().max()) == 0 and float((out[:, 4 + H * V:].float() - 7).abs().max()) == 0
