"""Latent attention: softmax attention whose keys and values are linear maps of a small cached latent."""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import Dict, Optional

import numpy as np
import torch

from ..cache import PagedNeed
from ..config.specs import MixerSpec
from ..csrc import ops
from ..weights.loader import ParamSpec
from .context import StageContext, StepPrelude
from .position import step_angles
from .registry import lookup, register_mixer


class LatentWork(StepPrelude):
    """How a long prompt step of latent attention is cut: the portions that are worth it as segments (entry, first position
    some query of it sees, first gathered row, rows padded to whole key tiles) and tiles of 256 query rows of them, longest
    walk first; the rows of all other entries.  Filled only for steps of at least `FROM` tokens."""
    # Shorter steps are replayed as captured graphs that serve any division of their tokens among requests, and what is
    # allocated here depends on how many rows the requests have cached (a step that is being captured never takes the lists).
    # (At 1,024 tokens of one request the cached-row kernel takes 340 us, the expanded path about 90.)
    FROM = 1025
    # Queries a portion needs: mapping a row costs the same for two queries as for two thousand.  Four portions beside a prompt
    # of 1,100 tokens, the layer at 32 heads (us, expanded and on the cached rows): 4,000 cached rows each, 8 queries 377, 275; 16:
    # 379, 390; 32: 387, 542; 128: 393, 1,595; 500 rows, 16 queries: 191, 226; 8 heads, 4,000 rows, 8 queries 206, 187; 16: 207, 300.
    LEAST = 16
    # With fewer, a portion is expanded only where that leaves no token to the other path, whose launches cost about 50 us, and
    # these have few rows together (of portions as above, 8 queries each: no cached rows 152, 195; 500 each 185, 210).
    FEW_ROWS = 3072

    @dataclass
    class Views:
        tiles: torch.Tensor              # int32 [n, 2]
        segs: torch.Tensor               # int32 [n, 4]
        rows: torch.Tensor               # int32 [n] rows of the batch that belong to no segment
        num_tiles: int
        num_segs: int
        num_rest: int
        gathered: int                    # rows of all segments
        longest: int                     # and of the longest

    def __init__(self, window: Optional[int], most_rows: int):
        """`most_rows`: gathered rows of a step that may be expanded at once."""
        self.window, self.most_rows = window, most_rows
        self.name = f"latent_work:{window or 0}:{most_rows}"

    def sections(self, max_tokens: int, max_entries: int):
        return {"tiles": 2 * (max_tokens // ops.LATENT_TILE_ROWS + max_entries + 1), "segs": 4 * max_entries, "rows": max_tokens}

    def fill(self, facts, out):
        if facts.num_tokens < self.FROM:
            return 0, 0, 0, 0, 0
        K, R = ops.LATENT_TILE_KEYS, ops.LATENT_TILE_ROWS
        first = np.maximum(facts.past - self.window + 1, 0) if self.window else np.zeros_like(facts.past)
        rows = -(-(facts.past + facts.q_len - first) // K) * K
        chosen = facts.q_len >= self.LEAST
        if not chosen.all() and (facts.q_len > 1).all() and rows[~chosen].sum() <= self.FEW_ROWS:
            chosen[:] = True
        # those with the fewest rows a query first, while there is room: one request with a long past leaves the others alone
        long = np.nonzero(chosen)[0]
        long = long[np.argsort(rows[long] / facts.q_len[long], kind="stable")]
        long = np.sort(long[np.cumsum(rows[long]) <= self.most_rows])
        rest = np.ones(len(facts.q_len), dtype=bool)
        rest[long] = False
        token_rest = np.repeat(rest, facts.q_len)
        num_rest = int(token_rest.sum())
        out["rows"][:num_rest] = np.nonzero(token_rest)[0]
        past, n, first, rows = facts.past[long], facts.q_len[long], first[long], rows[long]
        start = np.cumsum(rows) - rows
        out["segs"][:4 * len(long)] = np.stack([long, first, start, rows], axis=1).reshape(-1)
        tiles = [(i, q0) for i in range(len(long)) for q0 in range(0, int(n[i]), R)]
        tiles.sort(key=lambda t: -(int(past[t[0]] - first[t[0]]) + t[1]))
        out["tiles"][:2 * len(tiles)] = np.asarray(tiles, dtype=np.int64).reshape(-1)
        return len(tiles), len(long), num_rest, int(rows.sum()), int(rows.max()) if len(rows) else 0

    def views(self, dev, filled):
        n, segs, rest, gathered, longest = filled
        return LatentWork.Views(dev["tiles"][:2 * n].view(n, 2), dev["segs"][:4 * segs].view(segs, 4), dev["rows"][:rest], n, segs,
                                rest, gathered, longest)


@register_mixer("latent_attention")
class LatentAttentionMixer:
    """H heads; per head D unrotated and P rotated query/key entries and V value entries; latents of Q (queries) and
    R (keys and values) entries.  For a token with layer input x:

        cq = rmsnorm(W_dq x) * w_dq             q[h] = W_uq[h] cq = [qn[h] (D) | qr[h] (P)],  qr rotated by position
        [d | kr] = W_dkv x                      c = rmsnorm(d) * w_dkv (R),  kr (P) rotated by position, shared by all heads
        key[h] = [W_uk[h] c | kr]               value[h] = W_uv[h] c
        score(i, j) = (qn_i[h] . W_uk[h] c_j + qr_i[h] . kr_j) * scale        over the keys of the window, softmax
        out = W_o (concat_h(sum_j p_j value_j[h]) * sigmoid(W_g x))      (the gate one value per channel, or per head)

    Only the row [c | kr] (R + P entries, ONE "kv head") goes to the pages.  The per-head maps are folded into the
    query and the output, q_abs[h] = W_uk[h]^T qn[h] and sum_j p_j value_j[h] = W_uv[h] sum_j p_j c_j, so attention
    runs straight over the cached rows with key width R + P and the values the first R entries of the same rows:
    nothing per head is ever materialised per key, in prompts or in decoding.  A mixer whose spec says `has_kv`
    False has no W_dkv and reads the rows another stage cached (the stage's `cache_from`), with maps, queries,
    window and everything else of its own.

    One product yields [dq | dkv | g] per token in float32; `latent_prepare` norms both latents, rotates kr and
    writes the page row; W_uq; `latent_q_split` rotates qr and lays qn out head-major; a batched product with
    W_uk^T fills q_abs; attention (bfloat16: the tensor-core kernel in which all heads of a token share each staged
    tile of rows; float32: the general kernel); a batched product with W_uv^T; the gate; W_o.

    Long prompt steps (bfloat16, heads of 128 + 64 and 128) turn that around: where many queries meet every row it is
    cheaper to map the rows to per-head keys and values once, and attend to those (`_expanded`)."""

    graph_safe = True           # kernels and library products on the current stream only
    any_division_safe = True    # nothing is shaped by the number of entries

    _DEFAULT_NAMES = {"dq": "q_down.weight", "dq_norm": "q_down_norm.weight", "uq": "q_up.weight",
                      "dkv": "kv_down.weight", "dkv_norm": "kv_down_norm.weight", "uk": "k_up.weight",
                      "uv": "v_up.weight", "g": "g_proj.weight", "o": "o_proj.weight"}

    def __init__(self, spec: MixerSpec, hidden_size: int, compute_dtype: torch.dtype, device):
        p = dict(spec.params)
        self.H, self.D, self.V = spec.num_heads, spec.head_dim, spec.value_dim or spec.head_dim
        self.Q, self.R, self.P = int(p["q_rank"]), int(p["kv_rank"]), int(p.get("rot_dim", 0))
        if min(self.H, self.D, self.V, self.Q, self.R) <= 0 or self.P < 0:
            raise ValueError("latent attention needs positive heads, widths and ranks")
        if self.R > 512 or self.R + self.P > 1024:
            raise ValueError("latent attention: the attention kernel takes latents up to 512 and rows up to 1024 entries")
        if spec.output_gate not in (None, "sigmoid"):
            raise ValueError(f"output_gate {spec.output_gate!r}: 'sigmoid' or None")
        if spec.window is not None and spec.window <= 0:
            raise ValueError("an attention window must be positive")
        self.eps = float(p.get("eps", 1e-6))
        self.keep_window = p.get("keep_window", spec.window)
        self.spec, self.hidden, self.dtype, self.device = spec, hidden_size, compute_dtype, torch.device(device)
        self.scale = spec.scale if spec.scale is not None else 1.0 / math.sqrt(float(self.D + self.P))
        self.names = dict(self._DEFAULT_NAMES, **dict(spec.tensor_names))
        self.rot_dims, self.inv_freq, self.rot_pairs, self.rot_mag, pos = 0, None, False, 1.0, None
        if spec.position.kind == "rope" and self.P:
            pos = lookup("position", "rope")(spec.position, self.P, device)       # the rotation's frequencies, float32
            self.rot_dims, self.inv_freq = pos.rotary_dim, pos.inv_freq
        elif spec.position.kind == "rope_pairs" and self.P:                       # neighbouring pairs, stretched frequencies
            pos = lookup("position", "rope_pairs")(spec.position, self.P, device)
            self.inv_freq, self.rot_dims, self.rot_mag, self.rot_pairs = pos.kernel_args()
        elif spec.position.kind != "none":
            raise ValueError("latent attention rotates by 'rope', by 'rope_pairs' or not at all")
        self.table_key = getattr(pos, "table_key", None)
        if spec.output_gate_scope not in ("channel", "head"):
            raise ValueError(f"output_gate_scope {spec.output_gate_scope!r}: 'channel' or 'head'")
        self.gate_per_head = bool(spec.output_gate) and spec.output_gate_scope == "head"
        self.dq_off = 0
        self.dkv_off = self.Q
        self.g_off = self.Q + (self.R + self.P if spec.has_kv else 0)
        self.gate_width = 0 if not spec.output_gate else (self.H if self.gate_per_head else self.H * self.V)
        # bfloat16 on the tensor-core kernel over the cached rows; float32 (and other latent sizes) on the general kernel
        self.tensor_core = (compute_dtype == torch.bfloat16 and self.device.type == "cuda"
                            and ops.latent_attention_supported(self.R, self.P))
        self.expands = (self.tensor_core and self.scale > 0 and ops.latent_prefill_supported(self.D, self.V, self.R, self.P))
        self._work = LatentWork(spec.window, self.EXPANDED_BYTES // (2 * self.H * (self.D + self.V))) if self.expands else None
        self._expand = None         # (W_ukv [H * (D + V), R],): per head the key map, then the value map, for long prompt steps
        self.w_in = self.w_uq = self.w_uk_t = self.w_uv_t = self.w_o = None
        self.wq_norm = self.wkv_norm = None

    def parameters(self) -> Dict[str, ParamSpec]:
        n, s = self.names, self.spec
        p = {n["dq"]: ParamSpec((self.Q, self.hidden)),
             n["dq_norm"]: ParamSpec((self.Q,), role="scale", init=("one_plus_normal", 0.01)),
             n["uq"]: ParamSpec((self.H * (self.D + self.P), self.Q)),
             n["uk"]: ParamSpec((self.H * self.D, self.R)), n["uv"]: ParamSpec((self.H * self.V, self.R)),
             n["o"]: ParamSpec((self.hidden, self.H * self.V))}
        if s.has_kv:
            p[n["dkv"]] = ParamSpec((self.R + self.P, self.hidden))
            p[n["dkv_norm"]] = ParamSpec((self.R,), role="scale", init=("one_plus_normal", 0.01))
        if s.output_gate:
            p[n["g"]] = ParamSpec((self.gate_width, self.hidden))
        return p

    def load(self, t: Dict[str, torch.Tensor]) -> None:
        n, s = self.names, self.spec
        rows = [t[n["dq"]]] + ([t[n["dkv"]]] if s.has_kv else []) + ([t[n["g"]]] if s.output_gate else [])
        dt = torch.float32 if any(x.dtype == torch.float32 for x in rows) else rows[0].dtype
        self.w_in = torch.cat([x.to(dt) for x in rows], dim=0).contiguous()
        self.w_uq, self.w_o = t[n["uq"]].contiguous(), t[n["o"]].contiguous()
        # per head: [D, R] (q_abs = qn W_uk) and [R, V] (value = latent sum times W_uv^T), the batched products' right sides
        self.w_uk_t = t[n["uk"]].view(self.H, self.D, self.R).contiguous()
        self.w_uv_t = t[n["uv"]].view(self.H, self.V, self.R).transpose(1, 2).contiguous()
        if self.expands and t[n["uk"]].dtype == t[n["uv"]].dtype == torch.bfloat16:
            both = torch.cat([self.w_uk_t, t[n["uv"]].view(self.H, self.V, self.R)], dim=1)
            self._expand = (both.view(-1, self.R),)
            self.w_uk_t = both[:, :self.D]              # the key map is kept once
        self.wq_norm = t[n["dq_norm"]].float().contiguous()
        if s.has_kv:
            self.wkv_norm = t[n["dkv_norm"]].float().contiguous()
        for w in (self.w_in, self.w_uq, self.w_o):
            ops.prepare_streaming(w)

    def cache_need(self):
        if not self.spec.has_kv:
            return None
        return PagedNeed(1, self.R + self.P, self.keep_window, 0)       # keys only: the values are part of the key rows

    # Keys and values of all rows of a step that are made at once at most (65,536 rows at 32 heads); portions beyond that stay
    # on the cached-row kernel, which needs nothing per row.
    EXPANDED_BYTES = 1 << 30

    def step_prelude(self):
        return self._work

    def _absorbed(self, q: torch.Tensor, positions: torch.Tensor, token_entry: torch.Tensor, ctx: StageContext) -> torch.Tensor:
        """Attention over the cached rows themselves: q float32 [n, H * (D + P)] of n tokens -> [n, H * V]."""
        b, s = ctx.batch, self.spec
        H, D, P, R, V, T = self.H, self.D, self.P, self.R, self.V, q.shape[0]
        qn, packed = ops.latent_q_split(q, positions, self.inv_freq, H, D, P, R, self.rot_dims, self.dtype,
                                        rot_pairs=self.rot_pairs, rot_mag=self.rot_mag)
        # q_abs[h] = qn[h] W_uk[h], written into the first R columns of head h of the packed query
        torch.bmm(qn, self.w_uk_t if self.w_uk_t.dtype == qn.dtype else self.w_uk_t.to(qn.dtype),
                  out=packed.view(T, H, R + P)[:, :, :R].permute(1, 0, 2))
        lat = torch.empty((T, H * R), dtype=self.dtype, device=q.device)
        if self.tensor_core:
            ops.latent_attention(packed, ctx.cache_keys, positions, token_entry, b.entry_slot, ctx.block_table, H, R, P,
                                 ctx.page_size, s.window, self.scale, ctx.status, lat)
        else:
            ops.paged_attention_generic_kv(packed, ctx.cache_keys, None, positions, token_entry, b.entry_slot,
                                           ctx.block_table, H, 1, R + P, R, ctx.page_size, s.window, self.scale, ctx.status,
                                           lat, values_in_keys=True)
        heads = torch.empty((T, H * V), dtype=self.dtype, device=q.device)
        torch.bmm(lat.view(T, H, R).permute(1, 0, 2), self.w_uv_t if self.w_uv_t.dtype == lat.dtype else self.w_uv_t.to(lat.dtype),
                  out=heads.view(T, H, V).permute(1, 0, 2))
        return heads

    def _gated(self, heads: torch.Tensor, gates: torch.Tensor, off: int) -> torch.Tensor:
        if self.spec.output_gate:
            ops.gate_mul(heads, gates, off, heads, 0, self.spec.output_gate, per_head=self.V if self.gate_per_head else 0)
        return heads

    def _angles(self, b) -> Optional[torch.Tensor]:
        """The step's table of angles, shared by all layers of the same rotation."""
        return step_angles(b, self.inv_freq, self.table_key) if self.rot_dims else None

    def _portions(self, q: torch.Tensor, proj: torch.Tensor, work: LatentWork.Views, ctx: StageContext) -> torch.Tensor:
        """[T, H * V] whose rows that belong to segments hold their attention over per-head keys and values (a gate per head is
        applied as the kernel stores).  q: float32, or packed already (bfloat16)."""
        b, s = ctx.batch, self.spec
        H, D, P, R, V, T = self.H, self.D, self.P, self.R, self.V, q.shape[0]
        heads = torch.empty((T, H * V), dtype=self.dtype, device=q.device)
        rows = ops.latent_gather(ctx.cache_keys, work.segs, work.num_segs, work.gathered, work.longest, b.entry_slot, b.entry_kv_len,
                                 ctx.block_table, ctx.page_size, ctx.status)
        kv = torch.mm(rows[:, :R], self._expand[0].t())
        packed = q if q.dtype == torch.bfloat16 else ops.latent_q_pack(q, b.positions, self.inv_freq, H, D, P, self.rot_dims,
                                                                       rot_pairs=self.rot_pairs, rot_mag=self.rot_mag)
        ops.latent_prefill(packed, kv, rows, heads, work.tiles, work.num_tiles, work.segs, b.entry_q_start, b.entry_q_len,
                           b.entry_kv_len, H, R, s.window, self.scale, ctx.status, gate=proj if self.gate_per_head else None,
                           gate_off=self.g_off)
        return heads if self.gate_per_head else self._gated(heads, proj, self.g_off)

    def _expanded(self, q: torch.Tensor, proj: torch.Tensor, work: LatentWork.Views, ctx: StageContext) -> torch.Tensor:
        """Long portions over per-head keys and values made from their requests' rows; the other tokens of the same step over
        the rows themselves."""
        b = ctx.batch
        heads = self._portions(q, proj, work, ctx)
        if work.num_rest:
            pick = work.rows.long()
            one = self._absorbed(q.index_select(0, pick), b.positions.index_select(0, pick), b.token_entry.index_select(0, pick), ctx)
            gate = proj.narrow(1, self.g_off, self.gate_width).index_select(0, pick)
            heads.index_copy_(0, pick, self._gated(one, gate, 0))
        return heads

    def forward(self, x: torch.Tensor, ctx: StageContext):
        b, s = ctx.batch, self.spec
        if s.has_kv != ctx.writes_cache:
            raise RuntimeError("a latent attention mixer keeps its own latent, or reads another stage's, as its spec says")
        H, D, P, R, V, T = self.H, self.D, self.P, self.R, self.V, x.shape[0]
        proj = ops.as_tensor(ops.linear(x, self.w_in, out_dtype=torch.float32))
        cq = ops.latent_prepare(proj, self.dq_off, self.dkv_off, self.Q, R, P, self.rot_dims, self.wq_norm, self.wkv_norm,
                                self.eps, self.inv_freq, ctx.cache_keys if s.has_kv else None, b, ctx.block_table,
                                ctx.page_size, ctx.status, self.dtype, rot_pairs=self.rot_pairs, rot_mag=self.rot_mag)
        q = None
        work = b.preludes.get(self._work.name) if self._expand is not None and not getattr(b, "any_division", False) else None
        heads = None
        if work is not None and work.num_tiles and 2 * work.gathered * H * (D + V) <= self.EXPANDED_BYTES:
            try:
                if (not work.num_rest and (not self.rot_dims or (self.rot_pairs and self.rot_mag == 1.0 and self.rot_dims == P))
                        and ops.latent_q_product(cq, self.w_uq)):
                    # every token belongs to a portion: the queries leave their product as the attention kernel reads them
                    heads = self._portions(ops.linear_pair_latent_q(cq, self.w_uq, self._angles(b), H), proj, work, ctx)
                else:
                    q = ops.as_tensor(ops.linear(cq, self.w_uq, out_dtype=torch.float32))
                    heads = self._expanded(q, proj, work, ctx)
            except torch.cuda.OutOfMemoryError:
                pass                                  # what it holds grows with the cached rows; the other path's does not
        if heads is None:
            if q is None:
                q = ops.as_tensor(ops.linear(cq, self.w_uq, out_dtype=torch.float32))
            heads = self._gated(self._absorbed(q, b.positions, b.token_entry, ctx), proj, self.g_off)
        return ops.linear(heads, self.w_o, out_dtype=torch.float32, partials_ok=getattr(ctx, "partials_ok", False))
