"""Layers whose kernels are chosen by the step: the shorter way is taken where its rule says so, and gives what the general way gives
over the options that its conditions admit.  The general way is had by answering the rule's question with no."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def qwen(**over):
    c = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=1, hidden_size=256, num_attention_heads=8,
             num_key_value_heads=4, head_dim=128, intermediate_size=512, vocab_size=512, rope_theta=1e6, rms_norm_eps=1e-6,
             max_position_embeddings=4096, tie_word_embeddings=True, torch_dtype="bfloat16")
    return dict(c, **over)


def windowed(rot, mask):
    mixer = {"heads": 8, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": mask}
    if rot:
        mixer["rot"] = {"base": 10000.0, "dims": rot}
    return {"architecture": "Pukatar", "vocab": 64, "width": 256, "norm": {"eps": 1e-5},
            "layers": [{"type": "attention", "mixer": mixer, "mlp": None}]}


def latent(rot):
    mixer = {"heads": 8, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 96, "kv_rank": 512, "scale": 192 ** -0.5}
    if rot:
        mixer["rot"] = {"base": 10000.0, "dims": 64}
    return {"architecture": "Vugedra", "vocab": 64, "width": 256, "norm": {"eps": 1e-5},
            "layers": [{"type": "latent_attention", "mixer": mixer, "mlp": None}]}


def make(config, requests, room):
    from litellmengine_b200.config import config_from_dict
    from litellmengine_b200.engine import ModelRunner
    from litellmengine_b200.parts.model import model_parameters
    from litellmengine_b200.weights import DictSource
    g = torch.Generator(device=DEV).manual_seed(3)
    cfg, w = config_from_dict(config), {}
    for name, spec in model_parameters(cfg.plan()).items():
        if spec.optional_alias is None:
            t = torch.randn(spec.shape, generator=g, device=DEV)
            w[name] = 1.0 + 0.1 * t if spec.role == "scale" else (t * spec.shape[-1] ** -0.5).to(torch.bfloat16)
    return ModelRunner.from_config(cfg, dtype="bfloat16", device=DEV, source=DictSource(w), page_size=16, max_total_tokens=room,
                                   max_requests=requests, max_tokens_per_step=4096)


def layer(config, portions):
    """One mixer over portions of two prompts, the second half of each behind the cached first: its output and its pages."""
    from litellmengine_b200.engine import StepEntry
    runner = make(config, len(portions), 2 * sum(portions) + 64)
    g = torch.Generator(device=DEV).manual_seed(4)
    slots, block = [runner.admit() for _ in portions], runner.model.blocks[0]
    for _ in range(2):
        batch = runner.prepare([StepEntry(s, [0] * n) for s, n in zip(slots, portions)])
        ctx = runner.model.stage_context(0, batch, runner.cache)
        y = block.mixer.forward(torch.randn(sum(portions), 256, generator=g, device=DEV).to(torch.bfloat16), ctx)
        runner.finish(batch)
    runner.check_status()
    return y, (ctx.cache if ctx.cache is not None else ctx.cache_keys).clone()


def both_ways(monkeypatch, rule, answer, op, run, counts=lambda *a: True):
    """run() as it is, which has to call ops.<op> (with arguments that `counts`), and with ops.<rule> answering `answer`, which must not."""
    from litellmengine_b200.csrc import ops
    calls, real = [], getattr(ops, op)

    def called(*a, **k):
        if counts(*a):
            calls.append(1)
        return real(*a, **k)
    monkeypatch.setattr(ops, op, called)
    one, taken = run(), len(calls)
    assert taken
    monkeypatch.setattr(ops, rule, lambda *a, **k: answer)
    two = run()
    assert len(calls) == taken
    return one, two


def near(a, b, most):
    # roundings to bfloat16 of values that another order of sums left a few 2^-24 apart: few entries differ, each by a rounding
    # or, behind attention, by what a handful of rounded keys moves
    for x, y in zip(a, b):
        x, y = x.double(), y.double()
        assert float((x - y).norm()) <= most * float(y.norm())


@pytest.mark.parametrize("config", [qwen(), windowed(64, {"size": 512, "keep_first": 4}), windowed(128, None), windowed(64, None),
                                    windowed(None, {"size": 100, "keep_first": 0})])
def test_prompts_through_the_heads_product(monkeypatch, config):
    one, two = both_ways(monkeypatch, "heads_product", False, "linear_pair_heads", lambda: layer(config, [1500, 548]))
    near(one, two, 2e-3)


def test_prompts_that_the_heads_product_would_slow_down(monkeypatch):
    """1,024 tokens of 2,048 x 256: fewer values than the saved kernel is worth."""
    from litellmengine_b200.csrc import ops
    calls, real = [], ops.linear_pair_heads
    monkeypatch.setattr(ops, "linear_pair_heads", lambda *a, **k: calls.append(1) or real(*a, **k))
    for config in (qwen(), windowed(64, None)):
        layer(config, [800, 224])
    assert not calls
    w = lambda n, k: torch.empty(n, k, device=DEV, dtype=torch.bfloat16)
    big = w(6144, 4096)
    assert [t for t in (640, 768, 1024, 1200, 1536, 1600, 2048, 2900) if ops.heads_pay(t, big)] == [1536, 2048, 2900]
    assert [t for t in (768, 1024, 1100, 1280, 2048) if ops.heads_pay(t, w(4096, 2048))] == [1024, 2048]
    assert [t for t in (1024, 1800) if ops.heads_pay(t, w(2048, 1024))] == [1800]


@pytest.mark.parametrize("rot", [True, False])
def test_prompts_whose_latent_queries_are_packed(monkeypatch, rot):
    one, two = both_ways(monkeypatch, "latent_q_product", False, "linear_pair_latent_q", lambda: layer(latent(rot), [900, 380]))
    near(one, two, 2e-3)


def steps(config, requests, times=3):
    """Logits and pages of a few decode steps behind short prompts, launched kernel by kernel."""
    from litellmengine_b200.engine import StepEntry
    runner = make(config, requests, 176 * requests)
    runner.use_graphs = False
    slots = [runner.admit() for _ in range(requests)]
    runner.step([StepEntry(s, list(range(5 + 7 * i)), [4 + 7 * i]) for i, s in enumerate(slots)])
    out = []
    for t in range(times):
        batch = runner.prepare([StepEntry(s, [t + i], [0]) for i, s in enumerate(slots)])
        out.append(runner.forward(batch).clone())
        runner.finish(batch)
    runner.check_status()
    return out + [g.kv.clone() for g in runner.cache.groups]


@pytest.mark.parametrize("requests", [1, 5, 8])
def test_decode_steps_whose_products_make_their_rows(monkeypatch, requests):
    """Norm and residual add in the product are the norm kernel's numbers: the same bits."""
    from litellmengine_b200.csrc import ops
    config = qwen(num_hidden_layers=3)
    one, two = both_ways(monkeypatch, "pending_rows", None, "linear_small", lambda: steps(config, requests),
                         lambda x, *a: isinstance(x, ops.PendingRows))
    assert all(torch.equal(a, b) for a, b in zip(one, two))


@pytest.mark.parametrize("requests", [1, 5, 20])
def test_decode_steps_whose_attention_makes_its_rows(monkeypatch, requests):
    """And so are queries, keys and values made in the attention kernel."""
    config = qwen(num_hidden_layers=3)
    one, two = both_ways(monkeypatch, "decode_makes_its_rows", False, "paged_attention_decode_made", lambda: steps(config, requests))
    assert all(torch.equal(a, b) for a, b in zip(one, two))
