"""Attention whose keys and values come from one low-rank latent per token.

From the layer input x: q = W_q x, laid out head by head as [``dim`` unrotated ; ``rot_dim`` rotated]; W_dkv x has
``kv_rank + rot_dim`` rows, the first kv_rank RMS-normed (plain weight) are the latent c, the last rot_dim, rotated,
are a key part r that all heads share.  Head j's key is [W_uk_j c ; r] and its value W_uv_j c; causal softmax with
the given scale (with ``sink`` a learned number per head, ``sink_name``, whose exponential is added to the softmax's denominator:
it has neither key nor value); the heads' outputs are optionally multiplied by sigmoid(W_g x), element by element (``gate=True``) or
with one gate per head (``gate="head"``, W_g has ``heads`` rows), then projected by W_o.  With ``q_rank`` the queries are
made in two steps: the rows W_dq x of that width, RMS-normed and multiplied by a weight, then W_uq on the result.

Only c and r are cached (one row of kv_rank + rot_dim elements per token: a cache group with one key head and no
values).  The queries are folded through W_uk (a_j = W_uk_j^T q_j, one batched product), attention runs over the
latent rows with their first kv_rank elements as values, and W_uv is applied to the result (another batched
product): the same arithmetic regrouped, in which no per-head key or value is ever made.  Scores, softmax
weights, their sums and the folded queries are fp32.  In bfloat16, prompt portions of some length run the other way round:
their per-head keys and values are made from the cached rows by one product and used once (:class:`_Plan`).  Rotary pairs are (2i, 2i + 1) (``pairing="interleaved"``) or
(i, i + rot_dims / 2) (``pairing="half"``) over the first ``rot_dims`` elements of the rotated part, angle = position *
rot_base^(-2i / rot_dims).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Mapping, Sequence

import torch

from torchinferno_b200.engine.batch import EntryPlacement
from torchinferno_b200.kernels import ops
from torchinferno_b200.kernels.gemm import LinearWeight, linear
from torchinferno_b200.parts.base import CacheSpec, LayerContext, Mixer, WeightSpec, register_part


class LatentAttention(Mixer):
    def __init__(self, *, hidden_size: int, heads: int, dim: int, rot_dim: int, value_dim: int, kv_rank: int, scale: float,
                 rot_base: float, rot_dims: int | None = None, eps: float = 1e-6, gate: bool | str = True, sink: bool = False,
                 q_rank: int | None = None, pairing: str = "interleaved",
                 q_name: str = "q", dkv_name: str = "dkv", latent_norm_name: str = "dkv.norm", uk_name: str = "uk",
                 uv_name: str = "uv", g_name: str = "g", o_name: str = "o", dq_name: str = "dq", q_norm_name: str = "dq.norm",
                 uq_name: str = "uq", sink_name: str = "sink", dtype: torch.dtype, device: torch.device) -> None:
        super().__init__(dtype=dtype, device=device)
        if gate not in (True, False, "element", "head") or pairing not in ("interleaved", "half"):
            raise ValueError(f"unknown gate {gate!r} or pairing {pairing!r}")
        self.hidden_size, self.heads, self.dim, self.rot_dim = hidden_size, heads, dim, rot_dim
        self.value_dim, self.kv_rank, self.scale, self.eps, self.gate = value_dim, kv_rank, float(scale), float(eps), bool(gate)
        self.gate_per_head = gate == "head"
        self.q_rank, self.half_pairs = (int(q_rank) if q_rank else 0), pairing == "half"
        self.rot_dims = rot_dim if rot_dims is None else int(rot_dims)
        if self.rot_dims % 2 or self.rot_dims > rot_dim:
            raise ValueError("rot_dims must be even and at most rot_dim")
        i = torch.arange(self.rot_dims // 2, dtype=torch.float64)
        self.inv_freq = (torch.tensor(float(rot_base), dtype=torch.float64) ** (-2.0 * i / max(self.rot_dims, 1))) \
            .to(torch.float32).to(device)
        self.names = {"q": q_name, "dkv": dkv_name, "norm": latent_norm_name, "uk": uk_name, "uv": uv_name, "g": g_name,
                      "o": o_name, "dq": dq_name, "q_norm": q_norm_name, "uq": uq_name, "sink": sink_name}
        self.has_sink = bool(sink)
        self.sink: torch.Tensor | None = None
        self.in_weight: LinearWeight | None = None
        self.uq_weight: LinearWeight | None = None
        self.o_weight: LinearWeight | None = None
        self.unfold: LinearWeight | None = None

    def weight_specs(self) -> list[WeightSpec]:
        n, h, w = self.names, self.heads, self.hidden_size
        std, rank_std = w ** -0.5, self.kv_rank ** -0.5      # (random weights: rows of about unit size)
        if self.q_rank:
            specs = [WeightSpec(n["dq"], (self.q_rank, w), std=std),
                     WeightSpec(n["q_norm"], (self.q_rank,), init="about_one", std=0.1, role="vector"),
                     WeightSpec(n["uq"], (h * (self.dim + self.rot_dim), self.q_rank), std=self.q_rank ** -0.5)]
        else:
            specs = [WeightSpec(n["q"], (h * (self.dim + self.rot_dim), w), std=std)]
        specs += [WeightSpec(n["dkv"], (self.kv_rank + self.rot_dim, w), std=std),
                 WeightSpec(n["norm"], (self.kv_rank,), init="ones", role="vector"),
                 WeightSpec(n["uk"], (h * self.dim, self.kv_rank), std=rank_std),
                 WeightSpec(n["uv"], (h * self.value_dim, self.kv_rank), std=rank_std)]
        if self.has_sink:
            specs.append(WeightSpec(n["sink"], (h,), std=1.0, role="vector"))
        if self.gate:
            specs.append(WeightSpec(n["g"], (h if self.gate_per_head else h * self.value_dim, w), std=std))
        specs.append(WeightSpec(n["o"], (w, h * self.value_dim), std=(h * self.value_dim) ** -0.5))
        return specs

    def bind(self, weights: Mapping[str, torch.Tensor]) -> None:
        n, h = self.names, self.heads
        rows = [weights[n["dq"] if self.q_rank else n["q"]], weights[n["dkv"]]] + ([weights[n["g"]]] if self.gate else [])
        total = sum(r.shape[0] for r in rows)
        if total % 8:       # (rows of the product's output then start on 16-byte boundaries in bfloat16)
            rows.append(torch.zeros((8 - total % 8, self.hidden_size), dtype=rows[0].dtype, device=rows[0].device))
        self.in_weight = LinearWeight(torch.cat(rows, dim=0), few_rows_tcgen05=None)
        if self.q_rank:
            self.uq_weight = LinearWeight(weights[n["uq"]], few_rows_tcgen05=None)
            self.q_norm_weight = weights[n["q_norm"]].to(torch.float32).contiguous()
        self.o_weight = LinearWeight(weights[n["o"]], few_rows_tcgen05=None)
        self.latent_norm_weight = weights[n["norm"]].to(torch.float32).contiguous()
        if self.has_sink:
            self.sink = weights[n["sink"]].to(torch.float32).contiguous()
        uk = weights[n["uk"]].view(h, self.dim, self.kv_rank)              # per head [in = dim, out = kv_rank]
        self.uv_weight = weights[n["uv"]].view(h, self.value_dim, self.kv_rank).contiguous()   # per head [out, in]
        if uk.dtype == torch.float32:
            self.uk_weight = uk.transpose(1, 2).contiguous()               # the fp32 product wants [out, in]
        else:
            self.uk_weight = uk.contiguous()

        # W_uk and W_uv head by head: the step's keys and values for prompts, of all heads or a run of them.  The folded form's two weights
        # are views of it.
        self.unfold = None
        if uk.dtype == torch.bfloat16 and uk.is_cuda and self.scale > 0 \
                and ops.latent_prefill_supports(self.dim, self.value_dim, self.kv_rank, self.rot_dim):
            both = torch.cat([self.uk_weight, self.uv_weight], dim=1)
            self.unfold = LinearWeight(both.flatten(0, 1), allow_transpose=False)
            self.uk_weight, self.uv_weight = both[:, :self.dim], both[:, self.dim:]

    def cache_spec(self) -> CacheSpec:
        return CacheSpec(1, self.kv_rank + self.rot_dim, None, value_dim=0)

    # The unfolded form multiplies 2 (dim + value_dim) rank numbers a head and key once, and saves some two thirds of the folded
    # kernel's products on every (query, key) pair, which run at a tenth of the library's rate: it wins from about six
    # queries a key, and is taken from sixteen (the layer on two prompts of 1,667 and 833 tokens, 16 heads: 1,226 us
    # folded, 165 unfolded; error against 64 bits 0.0048 and 0.0045).  A step of prompts alone unfolds them all, a step of shorter
    # portions none; a step that mixes them takes what :func:`_plan` finds cheapest.
    UNFOLD_QUERIES = 16
    # Room for the rows, keys and values made at a time (two prompts of 1,667 and 833 tokens take 24 MB at 16 heads of 128 + 128): what
    # is above the bound goes entry by entry, and some heads at a time.
    UNFOLD_BYTES = 256 << 20

    def _plan(self, batch) -> "_Plan | None":
        """Which entries of the step run on keys and values made for it; None: none, or the entries are not known."""
        if self.unfold is None or batch.n_multi == 0 or len(batch.entries) != batch.n_entries:
            return None
        row_bytes = 2 * (self.dim + self.value_dim + self.kv_rank + self.rot_dim)      # (with one head's key and value)
        key = (self.UNFOLD_QUERIES, self.UNFOLD_BYTES // row_bytes, self.heads, self.dim + self.value_dim, self.kv_rank, self.rot_dim)
        if key not in batch.plans:
            batch.plans[key] = _plan(batch.entries, *key)
        return batch.plans[key]

    def _unfolded_rows(self, batch) -> int:
        """Rows of keys and values to make for this step, 0 where the folded form is to run throughout."""
        plan = self._plan(batch)
        return plan.rows if plan else 0

    def _unfolded(self, plan: "_Plan", q: torch.Tensor, dkv: torch.Tensor, gate: torch.Tensor | None, out: torch.Tensor, ctx: LayerContext) -> None:
        """The portions of the plan's groups, on keys and values made for them."""
        kv, batch, h, width = ctx.kv, ctx.batch, self.heads, self.dim + self.value_dim
        rows_dkv, rows_q, positions, token_slot = dkv, q, batch.positions, batch.token_slot
        if not plan.whole:
            tokens = slice(*plan.long_tokens)
            rows_dkv, rows_q, positions, token_slot = dkv[tokens], q[tokens], positions[tokens], token_slot[tokens]
        ops.latent_append(rows_dkv, rows_q, None, kv.keys if kv.writes else None, positions, token_slot, kv.block_table,
                          self.latent_norm_weight, self.eps, self.inv_freq, h, self.dim, self.kv_rank, self.rot_dim,
                          ctx.error_word, half_pairs=self.half_pairs)
        for first, end, rows, longest, longest_kv in plan.groups:
            q_start, kv_start, slots = batch.q_start, batch.kv_start, batch.slots
            if not plan.whole:
                q_start, kv_start, slots = q_start[first:end + 1], kv_start[first:end], slots[first:end]
            at_a_time = min(h, max(1, (self.UNFOLD_BYTES - 2 * rows * (self.kv_rank + self.rot_dim)) // (2 * rows * width)))
            latent = torch.empty((rows, self.kv_rank), dtype=q.dtype, device=q.device)
            rotated = torch.empty((rows, self.rot_dim), dtype=q.dtype, device=q.device)
            ops.latent_gather(kv.keys, kv.block_table, q_start, kv_start, slots, end - first, longest_kv, latent, rotated, ctx.error_word)
            for head in range(0, h, at_a_time):
                heads = self.unfold if at_a_time == h else self.unfold.rows(head * width, min(h, head + at_a_time) * width)
                ops.latent_prefill(q, linear(latent, heads), rotated, out, q_start, kv_start, end - first, longest, h, self.dim, self.value_dim,
                                   self.scale, plan.shortest, head, gate, self.gate_per_head, self.sink, ctx.error_word)

    def _folded(self, q: torch.Tensor, dkv: torch.Tensor, gate: torch.Tensor | None, heads_out: torch.Tensor, ctx: LayerContext,
                plan: "_Plan | None") -> None:
        """The whole step folded, or the short portions of the plan."""
        kv, batch, h, c, r = ctx.kv, ctx.batch, self.heads, self.kv_rank, self.rot_dim
        positions, token_slot, q_start, kv_start, slots = batch.positions, batch.token_slot, batch.q_start, batch.kv_start, batch.slots
        first_row, entries, max_q_len, max_kv_len = 0, batch.n_entries, batch.max_q_len, batch.max_kv_len
        if plan is not None:
            tokens, (first, end) = slice(*plan.short_tokens), plan.short
            q, dkv, heads_out, gate = q[tokens], dkv[tokens], heads_out[tokens], None if gate is None else gate[tokens]
            positions, token_slot = positions[tokens], token_slot[tokens]
            q_start, kv_start, slots = q_start[first:end + 1], kv_start[first:end], slots[first:end]
            first_row, entries, max_q_len, max_kv_len = tokens.start, end - first, plan.short_q_len, plan.short_kv_len
        n, width = q.shape[0], c + r
        folded = torch.empty((n, h, width), dtype=torch.float32, device=q.device)
        ops.latent_append(dkv, q, folded, kv.keys if kv.writes else None, positions, token_slot, kv.block_table,
                          self.latent_norm_weight, self.eps, self.inv_freq, h, self.dim, c, r, ctx.error_word,
                          half_pairs=self.half_pairs)
        q_plain = q.as_strided((n, h, self.dim), (q.stride(0), self.dim + r, 1))
        if q.dtype == torch.float32:
            for j in range(h):
                ops.gemm_f32(q_plain[:, j], self.uk_weight[j], folded[:, j, :c])
        else:
            ops.library_gemm_batched(q_plain, self.uk_weight, folded[:, :, :c], w_kn=True)
        latent_out = torch.empty((n, h, c), dtype=torch.float32, device=q.device)
        rows = torch.empty((n, h, c), dtype=q.dtype, device=q.device) if q.dtype != torch.float32 else None
        mixed = ops.latent_attention(folded, kv.keys, latent_out, q_start, kv_start, slots, kv.block_table, entries, max_q_len, h, c, r,
                                     self.scale, ctx.error_word, max_kv_len=max_kv_len, sink=self.sink, merged=rows, first_row=first_row)
        if q.dtype == torch.float32:
            for j in range(h):
                ops.gemm_f32(latent_out[:, j], self.uv_weight[j], heads_out[:, j])
        else:
            if mixed is not rows:
                ops.cast(mixed, rows)
            ops.library_gemm_batched(rows, self.uv_weight, heads_out, w_kn=False)
        if gate is not None:
            flat = heads_out.view(n, h * self.value_dim)
            ops.sigmoid_gate(flat, gate, flat, group=self.value_dim if self.gate_per_head else 1)

    def forward(self, x: torch.Tensor, ctx: LayerContext) -> torch.Tensor:
        kv, batch = ctx.kv, ctx.batch
        if kv is None or kv.keys is None:
            raise RuntimeError("latent attention needs a cache binding with key pages")
        n, h, c, r = x.shape[0], self.heads, self.kv_rank, self.rot_dim
        width = c + r
        q_width = self.q_rank if self.q_rank else h * (self.dim + r)      # columns of the first projection's q part
        proj = linear(x, self.in_weight)
        q, dkv = proj[:, :q_width], proj[:, q_width:q_width + width]
        if self.q_rank:
            latent_q = ops.rmsnorm(q, self.q_norm_weight, self.eps, torch.empty((n, self.q_rank), dtype=x.dtype, device=x.device))
            q = linear(latent_q, self.uq_weight)
        gates = (h if self.gate_per_head else h * self.value_dim) if self.gate else 0
        gate = proj[:, q_width + width:q_width + width + gates] if self.gate else None
        heads_out = torch.empty((n, h, self.value_dim), dtype=x.dtype, device=x.device)
        # (the kernels copy rows from 16-byte boundaries; a projection of an odd width leaves the gate's rows off them)
        plan = self._plan(batch) if x.dtype == torch.bfloat16 and self._unfolded_rows(batch) else None
        if plan and q.stride(0) % 8 == 0 and q.data_ptr() % 16 == 0 and kv.keys.stride(0) % 8 == 0 and kv.keys.data_ptr() % 16 == 0 \
                and (gate is None or self.gate_per_head or gate.data_ptr() % 16 == 0):
            if plan.short:      # (first: where long portions lie between, their rows are written here too, and again below)
                self._folded(q, dkv, gate, heads_out, ctx, plan)
            self._unfolded(plan, q, dkv, gate, heads_out, ctx)
        else:
            self._folded(q, dkv, gate, heads_out, ctx, None)
        return linear(heads_out.view(n, h * self.value_dim), self.o_weight)


@dataclass(frozen=True)
class _Plan:
    """How a step is shared out between the two forms."""
    # entries first .. end - 1 whose keys and values are made together, their rows, their longest portion and context
    groups: tuple[tuple[int, int, int, int, int], ...]
    rows: int                                     # of all groups
    whole: bool                                   # one group holds the step
    shortest: int                                 # portion among them that runs on these
    long_tokens: tuple[int, int]                  # the tokens from the first to the last of the groups' entries
    short: tuple[int, int] | None                 # the entries from the first to the last that stay folded, and their tokens
    short_tokens: tuple[int, int]
    short_q_len: int                              # their longest portion and context
    short_kv_len: int


# What the folded form's launches, and those of both forms in one step, take the host that issues a prompt's layer call by call beyond
# the unfolded form's, in us (100 a layer unfolded, 117 folded, 206 with both; the differences were the same when a call took the interpreter longer:
# 126, 144 and 245).
FOLDED_HOST_US, BOTH_FORMS_US = 15.0, 110.0


def _folded_us(entries: Sequence[EntryPlacement], heads: int, rank: int, rot: int) -> float:
    """Roughly what the folded form takes the device: products at 45 TFLOP/s, but a block walks its context 64 keys in 8 us, unless the
    step has single tokens only, whose contexts are shared out."""
    pairs = sum(e.q_len * (e.kv_start + (e.q_len + 1) / 2) for e in entries)
    chain = 0.0 if all(e.q_len == 1 for e in entries) else max(8.0 * (e.kv_start + e.q_len) / 64 for e in entries)
    return max(pairs * heads * 2 * (2 * rank + rot) / 45e6, chain)


def _unfolded_us(entries: Sequence[EntryPlacement], heads: int, width: int, rank: int) -> float:
    """The same of the unfolded form: keys and values at 1,100 TFLOP/s, then a block per head and 128 tokens (8 us, and 2 for every 128
    keys), 148 of them side by side."""
    rows = sum(e.kv_start + e.q_len + 64 for e in entries)
    each = [8.0 + 2.0 * (e.kv_start + e.q_len) / 128 for e in entries]
    blocks = sum(us * -(-e.q_len // 128) for us, e in zip(each, entries))
    return rows * heads * width * rank * 2 / 1.1e9 + max(blocks * heads / 148, max(each))


def _plan(entries: Sequence[EntryPlacement], queries: int, most_rows: int, heads: int, width: int, rank: int, rot: int) -> _Plan | None:
    """Portions of at least ``queries`` tokens run on keys and values made for the step, shorter ones folded.  Where a step has both,
    they run in one form, or each in its own, by what that takes (64 single tokens at 4,000 beside a prompt of 512: 673 us folded, 352 apart;
    eight at 1,000 beside it: 122 unfolded and 89 apart, which the second set of launches costs the host).  Neighbours share a product
    up to ``most_rows`` rows, across folded portions too where these add no more rows than there are."""
    padded = [-(-(e.kv_start + e.q_len) // ops.LATENT_TILE) * ops.LATENT_TILE for e in entries]
    long = [i for i, e in enumerate(entries) if e.q_len >= queries]
    if not long:
        return None
    if len(long) < len(entries):
        folded, unfolded = _folded_us(entries, heads, rank, rot) + FOLDED_HOST_US, _unfolded_us(entries, heads, width, rank)
        apart = _unfolded_us([e for e in entries if e.q_len >= queries], heads, width, rank) + BOTH_FORMS_US \
            + _folded_us([e for e in entries if e.q_len < queries], heads, rank, rot)
        if folded < min(unfolded, apart):
            return None
        if unfolded <= apart:
            long, queries = list(range(len(entries))), 1
    groups = []
    for i in long:
        between = sum(padded[groups[-1][1]:i]) if groups else 0
        if groups and between <= groups[-1][2] and groups[-1][2] + between + padded[i] <= most_rows:
            groups[-1] = (groups[-1][0], i + 1, groups[-1][2] + between + padded[i])
        else:
            groups.append((i, i + 1, padded[i]))
    taken = set(long)
    longest = lambda part: (max(e.q_len for e in part), max(e.kv_start + e.q_len for e in part))
    groups = tuple((first, end, rows, *longest(entries[first:end])) for first, end, rows in groups)
    short = [i for i in range(len(entries)) if i not in taken]
    tokens = lambda first, last: (entries[first].q_start, entries[last].q_start + entries[last].q_len)
    return _Plan(groups, sum(g[2] for g in groups), groups[0][:2] == (0, len(entries)), queries, tokens(long[0], long[-1]),
                 (short[0], short[-1] + 1) if short else None, tokens(short[0], short[-1]) if short else (0, 0),
                 *(longest([entries[i] for i in short]) if short else (0, 0)))


register_part("mixer", "latent_attention", LatentAttention)
