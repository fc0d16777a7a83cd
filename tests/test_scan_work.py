"""How steps of several prompt portions are cut for the recurrence kernels: short of 256 tokens only while the chunks find SMs."""
import types

import numpy as np
import pytest

from litellmengine_b200.parts.context import StepFacts
from litellmengine_b200.parts.linear_attention import ScanWork


def cut(lens, heads):
    work, q_len = ScanWork(heads), np.array(lens, dtype=np.int64)
    facts = StepFacts(q_start=np.cumsum(q_len) - q_len, q_len=q_len, past=np.zeros(len(lens), np.int64), slot=np.arange(len(lens), dtype=np.int32),
                      num_tokens=int(q_len.sum()))
    out = {k: np.full(n, -7, np.int32) for k, n in work.sections(int(q_len.sum()), len(lens)).items()}
    ns, nc, nh = work.fill(facts, out)
    chunks, short = out["chunks"][:4 * nc].reshape(nc, 4), out["short"][:4 * ns].reshape(ns, 4)
    rows = sorted(r for _, q0, n, _ in chunks.tolist() + short.tolist() for r in range(q0, q0 + n))
    assert rows == list(range(int(q_len.sum())))              # every token once
    views = ScanWork.Views(None, None, None, ns, nc, nh)
    batch = types.SimpleNamespace(entries=[types.SimpleNamespace(tokens=[0] * n) for n in lens])
    assert views.longest(batch) == (int(short[:, 2].max()) if ns else 0)
    return sorted(lens[e] for e in out["chains"][:3 * nh].reshape(nh, 3)[:, 0].tolist())


@pytest.mark.parametrize("lens,heads,want", [
    ([127], 1, []), ([128], 1, [128]), ([128], 74, [128]), ([128], 75, []),                       # 2 chunks: 148 and 150 blocks
    ([130] * 3, 16, [130] * 3), ([130] * 4, 16, []), ([191] * 4, 16, []), ([192] * 4, 16, [192] * 4),
    ([250] * 4, 16, [250] * 4), ([250] * 5, 16, []), ([255] * 2, 37, [255] * 2), ([255] * 2, 38, []),     # 296 and 304 blocks
    ([130, 250, 1, 7], 16, [130, 250]), ([128, 128, 250, 250], 16, []),       # 12 chunks: 189 tokens on average
    ([256], 500, [256]), ([300, 255, 3], 400, [300]), ([130] * 60 + [1000], 16, [1000]),
])
def test_portions_are_cut_while_their_chunks_find_sms(lens, heads, want):
    assert cut(lens, heads) == want
