"""How a long prompt step of latent attention is cut into portions whose rows are mapped to keys and values and tokens that
attend over the rows themselves."""
import numpy as np
import pytest

from litellmengine_b200.csrc import ops
from litellmengine_b200.parts.context import StepFacts
from litellmengine_b200.parts.latent_attention import LatentWork


def cut(past, q_len, window=None, most_rows=1 << 20):
    past, q_len = np.asarray(past, dtype=np.int64), np.asarray(q_len, dtype=np.int64)
    T = int(q_len.sum())
    work = LatentWork(window, most_rows)
    out = {k: np.full(n, -7, dtype=np.int32) for k, n in work.sections(T, len(q_len)).items()}
    start = np.cumsum(q_len) - q_len
    n_tiles, n_segs, n_rest, gathered, longest = work.fill(
        StepFacts(q_start=start, q_len=q_len, past=past, slot=np.arange(len(past)), num_tokens=T), out)
    segs, tiles = out["segs"][:4 * n_segs].reshape(-1, 4), out["tiles"][:2 * n_tiles].reshape(-1, 2)
    # every token in exactly one place
    seen = np.zeros(T, dtype=int)
    seen[out["rows"][:n_rest]] += 1
    for s, q0 in tiles:
        e = segs[s, 0]
        seen[start[e] + q0:start[e] + min(q_len[e], q0 + ops.LATENT_TILE_ROWS)] += 1
    assert (seen == 1).all()
    assert gathered == segs[:, 3].sum() and longest == segs[:, 3].max(initial=0)
    assert (segs[:, 2] == np.cumsum(segs[:, 3]) - segs[:, 3]).all() and (segs[:, 3] % ops.LATENT_TILE_KEYS == 0).all()
    return segs, out["rows"][:n_rest]


@pytest.mark.parametrize("window", [None, 100])
def test_only_portions_of_many_queries_are_expanded(window):
    L = LatentWork.LEAST
    segs, rest = cut([0, 5000, 40, 900, 7], [1200, 2, 1, L, L - 1], window)
    assert segs[:, 0].tolist() == [0, 3]
    assert len(rest) == 2 + 1 + L - 1
    assert segs[1, 1] == (900 - window + 1 if window else 0)


def test_a_step_of_short_portions_expands_nothing():
    segs, rest = cut([300] * 600, [2] * 600)
    assert len(segs) == 0 and rest.tolist() == list(range(1200))


def test_short_portions_that_leave_no_other_token():
    """They go with the long one where their rows are few, and not where a single token, or a long past, takes the other path anyway."""
    assert cut([0, 500, 0], [1200, 2, 5])[0][:, 0].tolist() == [0, 1, 2]
    assert cut([0, 500, 0, 40], [1200, 2, 5, 1])[0][:, 0].tolist() == [0]
    assert cut([0, 4000, 0], [1200, 2, 5])[0][:, 0].tolist() == [0]


def test_a_request_with_a_long_past_leaves_the_others_alone():
    """What does not fit is left out; the fewest rows a query come first, whatever the order in the step."""
    for order in ([0, 1, 2], [2, 1, 0], [1, 2, 0]):
        past, new = [9000, 0, 100], [500, 700, 300]
        segs, _ = cut([past[i] for i in order], [new[i] for i in order], most_rows=2000)
        assert sorted(order[e] for e in segs[:, 0]) == [1, 2]
    assert len(cut([9000, 0], [500, 700], most_rows=10)[0]) == 0
