"""Choices the product path makes on the host, checked without a GPU: which products may take the
engine's own kernels, and when a position part offers a table for the step."""
import types

import pytest

import torch

from litellmengine_b200.config.specs import PositionSpec
from litellmengine_b200.csrc import ops
from litellmengine_b200.parts.position import NoPosition, RotaryPosition


def test_the_paired_product_is_never_chosen_for_host_tensors_or_other_types():
    x = torch.zeros(300, 64, dtype=torch.bfloat16)
    w = torch.zeros(128, 64, dtype=torch.bfloat16)
    for kind in ("plain", "silu", "into"):
        assert ops._pair_takes(x, w, 64, kind) is False
    assert ops._pair_takes(x.float(), w.float(), 64, "silu") is False
    assert ops.linear_into(x, w, torch.zeros(300, 128)) is False


def test_only_the_gate_up_product_takes_the_paired_kernel_by_default():
    assert ops._PAIR_NEEDS["silu"] is not None
    assert ops._PAIR_NEEDS["plain"] is None and ops._PAIR_NEEDS["into"] is None


def test_a_position_part_offers_its_table_only_for_steps_its_kernel_reads_it_in():
    rope = RotaryPosition(PositionSpec(kind="rope", theta=10000.0, rotary_dim=None), 128, "cpu")
    small = types.SimpleNamespace(num_tokens=8, tables={}, positions=None)
    large = types.SimpleNamespace(num_tokens=4096, tables={}, positions=None)
    assert rope.angles(small) is None
    assert rope.angles(large) is None                      # tables live on the GPU only
    assert NoPosition(PositionSpec(kind="none"), 128, "cpu").rotation(large) is None
    assert rope.rotation(large).inv_freq is rope.inv_freq and rope.rotation(large).angles is None
    odd = RotaryPosition(PositionSpec(kind="rope", theta=10000.0, rotary_dim=32), 48, "cpu")
    assert odd._table_ok is False and rope._table_ok is True


def test_partial_sums_add_up_and_round_once():
    parts = torch.tensor([[[1.0, 2.0]], [[0.5, 0.25]], [[1e-3, 0.0]]])
    total = ops.as_tensor(ops.PartialSum(parts, None))
    assert torch.equal(total, (parts[0] + parts[1]) + parts[2])
    rounded = ops.as_tensor(ops.PartialSum(parts, torch.bfloat16))
    assert rounded.dtype == torch.bfloat16 and torch.equal(rounded, total.to(torch.bfloat16))


def test_decode_key_splits_follow_the_length_and_the_wave_fill():
    """On a device of 148 SMs (296 CTA slots).  Few rows: the square-root rule, in steps, never under
    64 keys a split.  More rows: the fewest splits that fill 0.85 of the waves they start."""
    from litellmengine_b200.parts import attention
    dev = torch.device("cpu")
    attention._slots[dev] = 296
    attention._split_choice.clear()
    try:
        pick = lambda rows, kv, nkv=8: attention.decode_key_splits(dev, rows, nkv, kv)
        assert [pick(1, kv) for kv in (1, 64, 65, 300, 1024, 2304, 4096, 8192, 32768)] == [1, 1, 2, 4, 8, 12, 16, 16, 32]
        assert [pick(rows, 4096) for rows in (2, 4, 8, 12, 16, 20, 24, 32, 40, 48, 64, 128)] == [16, 8, 4, 3, 2, 5, 3, 1, 4, 2, 1, 1]
        assert pick(40, 100) == 1 and pick(40, 1000) == 1 and pick(40, 2048) == 4   # evening out the waves pays from 512 keys a split
        assert pick(4, 100) == 2 and pick(4, 64) == 1                   # fewer CTAs than slots: a short context caps the splits
        assert pick(1, 1300, nkv=2) == 8 and pick(1, 201, nkv=2) == 4
    finally:
        del attention._slots[dev]
        attention._split_choice.clear()


@pytest.mark.gpu
def test_small_products_take_the_streaming_kernel_up_to_32_rows():
    """On the GPU (the rule reads the device's SM count): the products of a 0.6B-sized layer are small,
    those of an 8B-sized layer and an output head are not; `linear` follows."""
    assert all(ops.skinny_small(n, k) for n, k in ((4096, 1024), (1024, 2048), (6144, 1024), (1024, 3072)))
    assert not any(ops.skinny_small(n, k) for n, k in ((6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288), (151936, 1024)))
    before = ops.launch_count
    x = torch.randn(24, 1024, device="cuda:0").bfloat16()
    w = (torch.randn(4096, 1024, device="cuda:0") * 0.05).bfloat16()
    y = ops.linear(x, w, out_dtype=torch.float32)
    assert ops.launch_count > before                              # the engine's own kernel ran, not the library's
    assert float((y - x.float() @ w.float().t()).abs().max()) < 1e-4


def test_rows_are_left_to_a_product_only_by_parts_that_say_so_of_their_own_forward(monkeypatch):
    """`products_apply_it` and `first_product` speak for the forward of the class that states them: a part that derives from
    such a one and has a forward of its own is called, and is given a tensor."""
    from litellmengine_b200.config.specs import NormSpec
    from litellmengine_b200.parts import block
    from litellmengine_b200.parts.attention import AttentionMixer
    from litellmengine_b200.parts.feed_forward import SwiGLU
    from litellmengine_b200.parts.norms import RMSNorm

    class Own(RMSNorm):
        def forward(self, *a, **k):
            return "own"

    class Again(Own):
        products_apply_it = True

    class Kept(RMSNorm):
        def load(self, tensors):
            self.weight = 1.0 + tensors[self.name]

    class Mixer(AttentionMixer):
        def forward(self, x, ctx):
            return x.shape

    rows = types.SimpleNamespace(stream="stream")
    monkeypatch.setattr(ops, "pending_rows", lambda *a: rows)
    monkeypatch.setattr(RMSNorm, "forward", lambda self, *a, **k: "normed")
    h = types.SimpleNamespace(is_cuda=True, shape=(4, 8))
    spec = NormSpec("rmsnorm", 1e-6)
    new = lambda cls: cls.__new__(cls)
    mixer, ff = new(AttentionMixer), new(SwiGLU)
    mixer.w_qkv = ff.w_gate_up = None
    normed = lambda norm, part: block._normed(norm, part, h, None, torch.bfloat16)
    assert normed(RMSNorm(spec, 8), mixer) == normed(Kept(spec, 8), ff) == normed(Again(spec, 8), ff) == ("stream", rows)
    assert normed(Own(spec, 8), mixer) == (h, "own")
    other = new(Mixer)
    other.w_qkv = None
    assert normed(RMSNorm(spec, 8), other) == (h, "normed")
    patched = RMSNorm(spec, 8)
    patched.forward = lambda *a, **k: "patched"
    assert normed(patched, mixer) == (h, "patched")


def test_a_mixer_that_mixes_in_its_own_way_is_asked_to(monkeypatch):
    """The q/k/v product that prepares attention itself stands for `GatedAttentionMixer.mix` only."""
    from litellmengine_b200.config.specs import MixerSpec
    from litellmengine_b200.parts.attention import GatedAttentionMixer

    class Own(GatedAttentionMixer):
        def mix(self, proj, col0, ctx, out, out_col0, out_scale):
            out.fill_(3.0)

    spec = MixerSpec("gated_attention", num_heads=1, num_kv_heads=1, head_dim=128, position=PositionSpec(kind="none"))
    monkeypatch.setattr(ops, "heads_product", lambda *a: True)
    monkeypatch.setattr(ops, "heads_pay", lambda *a: True)
    monkeypatch.setattr(ops, "linear", lambda x, w, **k: x.float() @ w.float().t())
    x, ctx = torch.ones(4, 8, dtype=torch.bfloat16), types.SimpleNamespace(batch=types.SimpleNamespace(tables={}, positions=None, token_entry=None,
              entry_slot=None), writes_cache=True, cache=torch.zeros(1), block_table=None, page_size=16, status=None)
    asked = []
    monkeypatch.setattr(ops, "linear_pair_heads", lambda *a: asked.append(a) or torch.zeros(4, 128))
    monkeypatch.setattr(GatedAttentionMixer, "_attend", lambda self, q, proj, col0, ctx, out, at, scale: out.fill_(5.0))
    for cls, value, times in ((GatedAttentionMixer, 5.0, 1), (Own, 3.0, 1)):
        m = cls(spec, 8, torch.bfloat16, "cpu")
        m.w_in, m.w_o = torch.ones(384, 8), torch.ones(1, 128)
        assert torch.equal(m.forward(x, ctx), torch.full((4, 1), 128 * value)) and len(asked) == times


def test_branch_mixers_say_where_middling_products_gain(monkeypatch):
    from litellmengine_b200.parts.attention import BranchMixer, GatedAttentionMixer
    from litellmengine_b200.parts.delta_rule import DeltaRuleMixer
    from litellmengine_b200.parts.linear_attention import GatedLinearAttention, RetentionMixer
    from litellmengine_b200.parts.parallel import ParallelMixer
    asked = []
    monkeypatch.setattr(ops, "linear", lambda x, w, large_mid_rows, small=True, **k: asked.append(large_mid_rows) or torch.zeros(x.shape[0], w.shape[0]))
    alone = types.SimpleNamespace(partials_ok=False, residual=None)
    between = (types.SimpleNamespace(partials_ok=True, residual=None), types.SimpleNamespace(partials_ok=False, residual=torch.zeros(1)))
    for cls, n, k, rows, inside in ((GatedAttentionMixer, 8, 4096, [0, 0], [32, 32]), (GatedAttentionMixer, 8, 4088, [0, 0], [32, 48]),
                                    (GatedLinearAttention, 8, 8, [0, 0], [0, 0]), (RetentionMixer, 8, 8, [0, 0], [0, 0]),
                                    (DeltaRuleMixer, 8, 8, [32, 32], [48, 32]), (DeltaRuleMixer, 12, 8, [48, 32], [48, 32])):
        m = cls.__new__(cls)
        m.w_in, m.w_o, m.out_width, m.dtype, m.mix = torch.ones(n, 8), torch.ones(8, k), k, torch.bfloat16, lambda *a: None
        for ctx, want in ((alone, rows), (types.SimpleNamespace(), rows), (between[0], inside), (between[1], inside)):
            BranchMixer.forward(m, torch.ones(20, 8), ctx)
            assert asked == want, cls
            asked.clear()
    m = ParallelMixer.__new__(ParallelMixer)
    m.w_in, m.w_o, m.dtype, m.branches, m.scales, m.in_cols, m.out_cols = torch.ones(6, 8), torch.ones(8, 4), torch.bfloat16, [], [], [], []
    m.forward(torch.ones(20, 8), types.SimpleNamespace())
    assert asked == [0, 0]


@pytest.mark.parametrize("heads,hidden,rows", [(16, 2048, 16), (8, 512, 8), (8, 392, 8), (8, 384, 16), (8, 520, 16), (5, 1280, 16), (5, 1288, 0), (6, 1288, 16)])
def test_the_delta_rule_says_where_small_products_gain(monkeypatch, heads, hidden, rows):
    from litellmengine_b200.config.specs import MixerSpec
    from litellmengine_b200.parts.delta_rule import DeltaRuleMixer
    asked = []
    m = DeltaRuleMixer(MixerSpec("channel_delta", num_heads=heads, head_dim=32, params=(("taps", 1), ("decay_rank", 4), ("gate_rank", 4))), hidden,
                       torch.bfloat16, "cpu")
    m.load({n: torch.zeros(p.shape) for n, p in m.parameters().items()})
    assert m.w_in.shape == (m.in_width, hidden) and m.in_width % 2 == heads % 2
    monkeypatch.setattr(ops, "linear", lambda x, w, small=True, **k: asked.append(small) or torch.zeros(x.shape[0], w.shape[0]))
    m.mix = lambda *a: None
    for n in (1, 8, 9, 16):
        m.forward(torch.ones(n, hidden), types.SimpleNamespace())
    assert asked[::2] == [n <= rows for n in (1, 8, 9, 16)] and all(asked[1::2])


@pytest.mark.parametrize("rows,group,pending,worth", [(1, 4, False, True), (16, 1, False, True), (8, 4, True, False), (8, 16, True, False),
                                                      (9, 4, True, True), (9, 3, True, False), (15, 2, True, False), (16, 2, True, True)])
def test_rows_are_made_in_the_attention_kernel_where_that_pays(monkeypatch, rows, group, pending, worth):
    qkv = torch.zeros(rows, 384)
    qkv = ops.PartialSum(torch.stack([qkv, qkv])) if pending else qkv
    for captured in (True, False):
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: captured)
        assert ops.rows_worth_making(qkv, group) == (worth or not captured)


def test_tables_of_angles_go_by_the_spec(monkeypatch):
    """Layers of equal specs share a step's table, others do not, and a spec may hold its numbers in a list."""
    from litellmengine_b200.config.specs import MixerSpec
    from litellmengine_b200.parts.latent_attention import LatentAttentionMixer
    made = []
    monkeypatch.setattr(ops, "rope_angles", lambda positions, inv_freq: made.append(inv_freq) or len(made))

    def mixer(numbers, theta=10000.0):
        position = PositionSpec(kind="rope_pairs", theta=theta, rotary_dim=64, params=(("wavelengths", numbers),))
        return LatentAttentionMixer(MixerSpec("latent_attention", num_heads=2, head_dim=128, value_dim=128, position=position,
                                              params=(("q_rank", 16), ("kv_rank", 512), ("rot_dim", 64))), 32, torch.bfloat16, "cpu")

    step = types.SimpleNamespace(tables={}, positions=None)
    first = mixer([8.0, 1.0, 4.0, 8192.0])
    assert first._angles(step) == 1 and first._angles(step) == 1 and mixer([8.0, 1.0, 4.0, 8192.0])._angles(step) == 1
    assert mixer([4.0, 1.0, 4.0, 8192.0])._angles(step) == 2 and mixer([8.0, 1.0, 4.0, 8192.0], 5000.0)._angles(step) == 3
    assert first._angles(types.SimpleNamespace(positions=None)) == 4 and len(made) == 4           # a batch that keeps no tables


def test_rows_of_wide_streams_and_pending_splits_are_the_norm_kernels(monkeypatch):
    """Each block of a product that makes its rows reads all they are made of: that pays for whole sums of up to 1,024 values only."""
    from litellmengine_b200.config.specs import NormSpec
    from litellmengine_b200.parts import block
    from litellmengine_b200.parts.attention import AttentionMixer
    from litellmengine_b200.parts.norms import RMSNorm
    rows = types.SimpleNamespace(stream="stream")
    monkeypatch.setattr(ops, "pending_rows", lambda *a: rows)
    monkeypatch.setattr(RMSNorm, "forward", lambda self, *a, **k: "normed")
    norm, part = RMSNorm(NormSpec("rmsnorm", 1e-6), 8), AttentionMixer.__new__(AttentionMixer)
    part.w_qkv = None
    for width, delta, left in ((1024, None, True), (512, torch.zeros(4, 512), True), (1032, None, False),
                               (1024, ops.PartialSum(torch.zeros(2, 4, 1024)), False)):
        h = types.SimpleNamespace(is_cuda=True, shape=(4, width))
        assert block._normed(norm, part, h, delta, torch.bfloat16) == (("stream", rows) if left else (h, "normed"))
