"""Steps of recurrent mixers that are replayed as graphs leave the very states that the same steps leave when their kernels are launched
one by one, also when the graph was captured from a step that divided the same number of tokens otherwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W = 256


def runner_of(kind, heads):
    from litellmengine_b200.config import config_from_dict
    from litellmengine_b200.engine import ModelRunner
    mixer = {"heads": heads, "dim": 128, "vdim": 128}
    if kind == "gla":
        mixer.update(tau=8.0, rank=16)
    else:
        mixer.update(kv_heads=heads, conv=4, decay_rank=16, gate_rank=16)
    config = config_from_dict({"architecture": "Vugedra" if kind == "gla" else "Pukatar", "vocab": 64, "width": W, "norm": {"eps": 1e-5},
                               "layers": [{"type": kind, "mixer": mixer, "mlp": None}]})
    return ModelRunner.from_config(config, dtype="bfloat16", device=DEV, page_size=16, max_total_tokens=2048, max_requests=4, max_tokens_per_step=1024)


def states_after(runner, slots, lens):
    """The states after one step from fresh ones; nothing is committed, so that the same step can run again."""
    from litellmengine_b200.engine import StepEntry
    kept = [t for k, t in runner.cache.state.items() if not isinstance(k, str)]
    for t in kept:
        t.zero_()
    entries = [StepEntry(s, [(7 * i + s) % 64 for i in range(n)], [n - 1]) for s, n in zip(slots, lens)]
    runner.forward(runner.prepare(entries))
    torch.cuda.synchronize()
    return [t.clone() for t in kept]


@pytest.mark.parametrize("kind,heads,lens,other", [
    ("gla", 2, [1, 1, 1, 25], [7, 7, 7, 7]),                   # one pass, items on both sides of the tensor-core kernel's line
    ("gla", 2, [7, 7, 7, 7], [1, 1, 1, 25]),
    ("channel_delta", 12, [300, 1], [150, 151]),               # portions on both sides of the tensor-core kernels' line
    ("channel_delta", 12, [150, 151], [300, 1]),
])
def test_replayed_steps_launch_what_the_step_would(kind, heads, lens, other):
    runner = runner_of(kind, heads)
    slots = [runner.admit() for _ in lens]
    first = states_after(runner, slots, lens)                  # kernel by kernel
    states_after(runner, slots, other)
    states_after(runner, slots, other)                         # captured from this division
    replays = runner.graph_replays
    for _ in range(3):
        again = states_after(runner, slots, lens)
        assert all(torch.equal(a, b) for a, b in zip(first, again))
    assert runner.graph_replays >= replays + 2
