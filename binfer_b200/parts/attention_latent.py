"""Attention over a cached latent vector per token, as a mixer part.

A down projection of the mixer's input yields ``rank + dr`` numbers per token: the first
``rank``, RMS-normed with a weight, are the latent ``c``; the last ``dr``, rotated by the
token's position, are a key part that all heads share.  Head h's key is ``[W_uk,h c | shared
part]``, its value ``W_uv,h c``, its query ``[d plain | dr rotated]``; scores are scaled,
masked causally and pass an ordinary softmax (whose denominator may hold a learned logit per
head, ``sinks``); each head's output may be multiplied by the
sigmoid of one projected number per head; the output projection follows.

Only ``c`` and the shared key part are cached: one cache "head" of ``rank + dr`` numbers per
token and no values.  Keys and values are never expanded.  Because ``q_h . (W_uk,h c) =
(W_uk,h^T q_h) . c``, each query head's plain part is first carried into latent coordinates
(a product per head against ``W_uk,h^T``), the attention then runs with one shared key head
of ``rank + dr`` numbers whose first ``rank`` are also the value, and each head's result, a
mixture of latents, is expanded by ``W_uv,h`` afterwards.  The float32 engine runs every step so,
and the logits cannot depend on how a prompt was cut.

In bfloat16, prompt portions long enough to pay for it run expanded: the latents of their whole
context are gathered from the pages, one product against ``[W_uk,h | W_uv,h]`` of all heads makes
keys and values of them, and a tcgen05 kernel attends with 192 + 128 multiply-adds per score and
head instead of ``rank + 64 + rank``.  Single tokens in the same step stay in latent coordinates.

With ``q_rank`` the queries go through a latent of their own: the stacked product yields
``W_dq h`` in place of the queries, an RMS norm with a weight follows (float arithmetic), and
a second product ``W_uq`` gives the query heads.
"""
from __future__ import annotations

import dataclasses
import os
from typing import Callable, List, Optional

import torch

from ..cache.manager import KVNeed
from ..config.specs import LatentAttentionSpec
from ..csrc import ops
from ..weights.loader import ParamSpec
from .base import (BuildEnv, EntryView, Mixer, StackedOut, StepContext, build_position,
                   register_mixer)
from .linear import linear, linear_heads

# BINFER_B200_LATENT_TENSOR_CORES=0: the one-warp-per-row kernel also in bfloat16 (the float32
# path), to tell the two apart when something differs
TENSOR_CORES = os.environ.get("BINFER_B200_LATENT_TENSOR_CORES", "1") != "0"


# BINFER_B200_LATENT_EXPAND=0: prompt portions in latent coordinates too
EXPAND = os.environ.get("BINFER_B200_LATENT_EXPAND", "1") != "0"
# most bytes of expanded keys and values a step may take
EXPAND_MAX_BYTES = 768 << 20


class LatentAttention(Mixer, StackedOut):
    def __init__(self, spec: LatentAttentionSpec, hidden_size: int, prefix: str, env: BuildEnv):
        s = spec
        if min(s.num_heads, s.head_dim, s.value_dim, s.kv_rank) <= 0 or s.rot_dim < 0:
            raise ValueError("latent attention: heads and sizes must be positive")
        if s.kv_rank + s.rot_dim > ops.GENERIC_MAX_HEAD_DIM or s.kv_rank > ops.GENERIC_MAX_VALUE_DIM:
            raise ValueError(f"latent attention: a latent of {s.kv_rank} with a rotated part of "
                             f"{s.rot_dim} is not supported (latent at most "
                             f"{ops.GENERIC_MAX_VALUE_DIM}, together at most "
                             f"{ops.GENERIC_MAX_HEAD_DIM})")
        self.spec, self.hidden, self.prefix, self.env = spec, hidden_size, prefix, env
        self.H, self.d, self.dr, self.dv, self.rank = (s.num_heads, s.head_dim, s.rot_dim,
                                                       s.value_dim, s.kv_rank)
        self.q_size = self.H * (self.d + self.dr)
        self.kv_size = self.rank + self.dr
        self.q_rank = int(getattr(s, "q_rank", 0) or 0)
        # rows of the stacked product in front: the queries, or their latent
        self.q_rows = self.q_rank if self.q_rank else self.q_size
        self.position = None
        if s.position is not None and self.dr:
            # the rotated sizes are a vector of their own: dr numbers, rotated from its start
            self.position = build_position(dataclasses.replace(s.position, offset=0), self.dr, env)
            if self.position.inv_freq is None:
                raise ValueError("latent attention takes rotary encodings only")
        self.names = dict(s.names)
        self.gate_off = self.q_rows + self.kv_size
        self.out_cols = self.H * self.dv
        self.w_proj = self.w_ukT = self.w_uv = self.w_out = self.norm_w = None
        self.w_uq = self.q_norm_w = self.sinks = self.w_ukv = None
        self.expands = EXPAND and ops.latent_expand_takes(env.dtype, self.d, self.dr, self.dv,
                                                          self.rank)

    # ----------------------------------------------------------------- weights
    def _spec(self, role: str) -> ParamSpec:
        shape = {"q": (self.q_size, self.hidden), "dkv": (self.kv_size, self.hidden),
                 "dkv_norm": (self.rank,), "uk": (self.H * self.d, self.rank),
                 "uv": (self.H * self.dv, self.rank), "g": (self.H, self.hidden),
                 "o": (self.hidden, self.H * self.dv), "dq": (self.q_rank, self.hidden),
                 "dq_norm": (self.q_rank,), "uq": (self.q_size, self.q_rank),
                 "sink": (self.H,)}[role]
        n = self.prefix + self.names[role]
        if role == "sink":
            return ParamSpec(n, shape, init="around_zero", role="vector")
        if role in ("dkv_norm", "dq_norm"):
            return ParamSpec(n, shape, init="norm", role="vector")
        return ParamSpec(n, shape)

    def _roles(self) -> List[str]:
        q = ["dq", "dq_norm", "uq"] if self.q_rank else ["q"]
        return (q + ["dkv", "dkv_norm", "uk", "uv"] + (["g"] if self.spec.head_gate else [])
                + (["sink"] if self.spec.sinks else []) + ["o"])

    def param_specs(self) -> List[ParamSpec]:
        return [self._spec(r) for r in self._roles()]

    def load(self, get: Callable[[ParamSpec], torch.Tensor]) -> None:
        g = lambda role: get(self._spec(role))          # noqa: E731
        rows = [g("dq") if self.q_rank else g("q"), g("dkv")] + (
            [g("g")] if self.spec.head_gate else [])
        self.w_proj = torch.cat(rows, dim=0).contiguous()
        if self.q_rank:
            self.w_uq, self.q_norm_w = g("uq"), g("dq_norm")
        self.norm_w = g("dkv_norm")
        # per head: W_uk,h^T [rank, d] carries a query into latent coordinates; W_uv,h
        # [dv, rank] expands a mixture of latents into the head's value
        self.w_ukT = g("uk").view(self.H, self.d, self.rank).transpose(1, 2).contiguous()
        self.w_uv = g("uv").view(self.H, self.dv, self.rank).contiguous()
        if self.expands:       # per head [W_uk,h ; W_uv,h]: rows of keys, then of values
            both = torch.cat([g("uk").view(self.H, self.d, self.rank), self.w_uv], dim=1)
            self.w_ukv = both.reshape(-1, self.rank)
            self.w_uv = both[:, self.d:]         # (the values' rows are kept once)
        self.w_out = g("o")
        if self.spec.sinks:
            self.sinks = g("sink")

    # ------------------------------------------------------------------- cache
    def kv_need(self) -> Optional[KVNeed]:
        return KVNeed(1, self.kv_size, None, 0)      # one head per token, no values

    # ----------------------------------------------------------------- forward
    def forward(self, x: torch.Tensor, ctx: StepContext, view: EntryView) -> torch.Tensor:
        out = torch.empty((x.shape[0], self.out_cols), dtype=x.dtype, device=x.device)
        self.forward_inner(x, ctx, view, out)
        return linear(out, self.w_out)

    def forward_inner(self, x: torch.Tensor, ctx: StepContext, view: EntryView,
                      out: torch.Tensor) -> bool:
        """Everything but the output projection, into ``out [T, heads * value_dim]`` (which may be
        a column block of a wider buffer)."""
        s, T, H = self.spec, x.shape[0], self.H
        if not view.writes_cache:
            raise ValueError("latent attention keeps a cache of its own")
        g = view.group
        proj = linear(x, self.w_proj)
        if self.q_rank:
            c_q = torch.empty((T, self.q_rank), dtype=x.dtype, device=x.device)
            ops.section_norm(proj, 0, self.q_rank, self.q_norm_w, s.norm_eps, c_q)
            q = linear(c_q, self.w_uq)
        else:
            q = proj[:, :self.q_size]
        rows = self._expanded_rows(q, out, ctx)
        cache, lead = view.k_cache, 0
        if not rows:
            self._in_latent_coordinates(q, proj, out, ctx, view, T)
        elif ctx.n_decode:
            # single tokens in front of the portions, as the scheduler puts them, are a step of
            # their own; elsewhere all rows go through the products and the attention takes theirs
            lead = next(b for b, n in enumerate(ctx.q_lens) if n != 1)
            lead = lead if lead == ctx.n_decode else 0
            self._in_latent_coordinates(q, proj, out, ctx, view, lead or T, n_max=1)
            if not lead:
                cache = None                     # (stored)
        if rows:
            self._encode(proj, q, None, cache, ctx, g, lead, T)
            lat, rot, base = ops.latent_gather(view.k_cache, ctx.block_tables[g],
                                               ctx.prefill_items, ctx.n_prefill, rows, self.rank,
                                               ctx.err)
            gate = proj[:, self.gate_off:self.gate_off + H] if s.head_gate else None
            ops.latent_attention_prefill(q, linear(lat, self.w_ukv), rot, base, ctx.prefill_items,
                                         ctx.n_prefill, ctx.max_prefill_rows, out, H,
                                         s.softmax_scale, ctx.err, gate=gate, sinks=self.sinks)
        return True

    def _expanded_rows(self, q: torch.Tensor, out: torch.Tensor, ctx: StepContext) -> int:
        """Rows of expanded keys and values (contexts of the step's prompt portions, each rounded up
        to 64), or 0 where the step stays in latent coordinates.  There a pair of a row and a key
        that it sees costs about 24 ps a head (1,800 rows behind 500 keys, 16 heads: 964 us); the
        expansion costs 0.22 ns a head and key and 30 us for its launches, and the pairs then next
        to nothing (the same rows: 60 us, 16 for gathering and expanding)."""
        if (not self.expands or not ctx.n_prefill or self.spec.softmax_scale <= 0
                or q.stride(0) % 8 or q.data_ptr() % 16 or out.stride(0) % 8
                or out.data_ptr() % 16):
            return 0
        if self.H * 2.4e-11 * q.shape[0] * ctx.max_ctx_len < 3e-5:
            return 0
        rows = pairs = 0
        for n, c in zip(ctx.q_lens, ctx.ctx_lens_host):
            if n > 1:
                rows += -(-c // 64) * 64
                pairs += n * (c - n) + n * (n + 1) // 2
        if (self.H * (2.4e-11 * pairs - 2.2e-10 * rows) < 3e-5
                or rows * self.H * 2 * (self.d + self.dv) > EXPAND_MAX_BYTES):
            return 0
        return rows

    def _encode(self, proj, q, q_abs, cache, ctx: StepContext, group, first: int,
                last: int) -> None:
        """Rows ``first .. last - 1`` of the step; ``q_abs`` (None: in place) begins with the first."""
        s, pos = self.spec, self.position
        positions, slots = ctx.positions, ctx.slots[group]
        if last - first < ctx.T:                 # (a view of each costs the host a microsecond)
            proj, q, positions, slots = (x[first:last] for x in (proj, q, positions, slots))
        ops.latent_encode(proj, 0, self.q_rows, self.norm_w, s.norm_eps,
                          pos.inv_freq if pos is not None else None,
                          bool(pos is not None and pos.interleaved),
                          pos.magnitude if pos is not None else 1.0, positions, slots, q_abs, cache,
                          self.H, self.d, self.dr, self.rank, ctx.err, q=q)

    def _in_latent_coordinates(self, q, proj, out, ctx: StepContext, view: EntryView, T: int,
                               n_max: int = 0) -> None:
        """The step's first ``T`` rows (``n_max`` > 0: those of requests with at most so many tokens;
        what ``out`` holds for the others says nothing) with the queries carried into latent
        coordinates; ``q`` is left as it is."""
        s, H, g = self.spec, self.H, view.group
        B = ctx.B
        q_abs = torch.empty((T, H, self.kv_size), dtype=q.dtype, device=q.device)
        self._encode(proj, q, q_abs, view.k_cache, ctx, g, 0, T)
        if T < q.shape[0]:                       # fewer rows than the step's: single tokens
            B, q, proj, out = T, q[:T], proj[:T], out[:T]
        q_heads = q.view(T, H, self.d + self.dr)
        linear_heads(q_heads[:, :, :self.d], self.w_ukT, q_abs[:, :, :self.rank])
        # (rows that the attention leaves alone go through the product behind it as zeros)
        o_lat = (torch.zeros if n_max and B < T else torch.empty)(
            (T, H, self.rank), dtype=q.dtype, device=q.device)
        if (TENSOR_CORES and s.softmax_scale > 0
                and ops.latent_attention_takes(q.dtype, self.rank, self.dr)):
            # bfloat16: tiles of (token, head) rows against tiles of cache rows, each fetched
            # once as keys and values, on the tensor cores
            few = ctx.decode_only or n_max == 1
            ops.latent_attention(q_abs, view.k_cache, ctx.q_start, ctx.positions,
                                 ctx.block_tables[g], o_lat, B,
                                 1 if few else ctx.max_q_len, H, self.rank,
                                 s.softmax_scale, ctx.err,
                                 max_ctx=ctx.max_decode_ctx if n_max == 1 else ctx.max_ctx_len,
                                 sinks=self.sinks, n_max=n_max)
        else:
            ops.paged_attention_generic(
                q_abs.view(T, H * self.kv_size), view.k_cache, view.k_cache, ctx.seq_of_token,
                ctx.positions, ctx.block_tables[g], o_lat.view(T, H * self.rank), H, 1,
                self.kv_size, None, s.softmax_scale, ctx.err, value_dim=self.rank,
                v_stride=self.kv_size, sinks=self.sinks)
        heads = out.unflatten(1, (H, self.dv))
        if not s.head_gate or out.is_contiguous():
            linear_heads(o_lat, self.w_uv, heads)
            if s.head_gate:
                ops.head_gate_mul(out, proj[:, self.gate_off:self.gate_off + H], H, self.dv)
            return
        own = torch.empty((T, H, self.dv), dtype=q.dtype, device=q.device)
        linear_heads(o_lat, self.w_uv, own)
        own = own.view(T, H * self.dv)
        ops.head_gate_mul(own, proj[:, self.gate_off:self.gate_off + H], H, self.dv)
        out.copy_(own)


register_mixer("latent_attention", LatentAttention)
