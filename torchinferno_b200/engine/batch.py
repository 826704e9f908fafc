"""The ragged batch one step runs.

The reference's unified step pads rows to the longest entry and carries
``q_lens``, ``seq_lens``, ``write_positions`` and ``logit_positions``
(src/torchinferno/runtime/serving.py:2587-2600).  Here nothing is padded: all
tokens of the step lie on one axis, and an entry (one request's next tokens) is
a range of it.

Device arrays (int32, views into one uploaded buffer):
  token_ids[t], positions[t], token_slot[t]     per token
  q_start[e] (n_entries + 1), kv_start[e], slots[e]   per entry
  logit_rows[i], logit_slots[i]                 token rows whose logits are wanted, and the slot of their request
"""
from __future__ import annotations

from collections import Counter
from dataclasses import dataclass, field
from typing import Hashable, Sequence

import torch


@dataclass(frozen=True)
class StepEntry:
    """One request's share of a step: its next tokens and where logits are wanted."""
    request_id: Hashable
    tokens: Sequence[int]
    want: Sequence[int] = ()      # indices into ``tokens``
    seed: int = 0                 # sampling parameters, written into the request's record when this step opens it
    temperature: float = 0.0


@dataclass
class EntryPlacement:
    request_id: Hashable
    slot: int
    q_start: int
    q_len: int
    kv_start: int                 # tokens the request held before this step


@dataclass
class StepBatch:
    token_ids: torch.Tensor
    positions: torch.Tensor
    token_slot: torch.Tensor
    q_start: torch.Tensor
    kv_start: torch.Tensor
    slots: torch.Tensor
    logit_rows: torch.Tensor
    logit_slots: torch.Tensor
    n_tokens: int
    n_entries: int
    n_logits: int
    max_q_len: int
    max_kv_len: int               # bound on the longest context (cached + new tokens) of an entry
    n_single: int = 0             # entries that bring one token
    n_multi: int = 0              # entries that bring more
    entries: list[EntryPlacement] = field(default_factory=list)
    portions: dict[int, int] = field(default_factory=dict)      # how many entries bring that many tokens (empty: not known)
    h2d_bytes: int = 0
    plans: dict = field(default_factory=dict)      # what the parts worked out from the entries, for their other layers


def build_batch(placements: list[EntryPlacement], tokens: list[Sequence[int]], wants: list[Sequence[int]],
                table_updates: list[tuple[list[int], list[int]]], device: torch.device
                ) -> tuple[StepBatch, list[tuple[torch.Tensor, torch.Tensor]]]:
    """Pack the step's integers into one host buffer, upload it once, and slice it."""
    n = sum(place.q_len for place in placements)
    entries = len(placements)
    q_start, kv_start, slots = [0], [], []
    logit_rows: list[int] = []
    logit_slots: list[int] = []
    for place, want in zip(placements, wants):
        q_start.append(place.q_start + place.q_len)
        kv_start.append(place.kv_start)
        slots.append(place.slot)
        logit_rows.extend(place.q_start + int(w) for w in want)
        logit_slots.extend([place.slot] * len(want))
    small = [q_start, kv_start, slots, logit_rows, logit_slots]
    for index, value in table_updates:
        small.extend((index, value))
    lengths = [n, n, n] + [len(section) for section in small]
    total = sum(lengths)
    use_cuda = device.type == "cuda"
    host = torch.empty(max(total, 1), dtype=torch.int32, pin_memory=use_cuda)
    # the three arrays of one number per token are filled entry by entry where they lie (a Python list of a prompt's numbers
    # three times over took most of the time before the step's first launch); the short ones go in as one list
    if entries and all(place.q_len == 1 for place in placements):      # single tokens
        host[:3 * n] = torch.tensor([int(toks[0]) for toks in tokens] + kv_start + slots, dtype=torch.int32)
    else:
        row = 0
        for place, toks in zip(placements, tokens):
            end = row + place.q_len
            plain = isinstance(toks, list) and set(map(type, toks)) == {int}
            host[row:end] = torch.tensor(toks if plain else [int(t) for t in toks], dtype=torch.int32)
            torch.arange(place.kv_start, place.kv_start + place.q_len, dtype=torch.int32, out=host[n + row:n + end])
            host[2 * n + row:2 * n + end].fill_(place.slot)
            row = end
    flat: list[int] = []
    for section in small:
        flat.extend(section)
    if flat:
        host[3 * n:total] = torch.tensor(flat, dtype=torch.int32)
    dev = host.to(device, non_blocking=use_cuda)
    views: list[torch.Tensor] = []
    offset = 0
    for length in lengths:
        views.append(dev[offset: offset + length])
        offset += length
    batch = StepBatch(
        token_ids=views[0], positions=views[1], token_slot=views[2], q_start=views[3], kv_start=views[4],
        slots=views[5], logit_rows=views[6], logit_slots=views[7], n_tokens=n, n_entries=entries,
        n_logits=len(logit_rows), max_q_len=max((p.q_len for p in placements), default=0),
        max_kv_len=max((p.kv_start + p.q_len for p in placements), default=0),
        n_single=sum(1 for p in placements if p.q_len == 1), n_multi=sum(1 for p in placements if p.q_len > 1),
        entries=placements, portions=dict(Counter(p.q_len for p in placements)), h2d_bytes=total * 4)
    updates = [(views[8 + 2 * i], views[9 + 2 * i]) for i in range(len(table_updates))]
    return batch, updates
