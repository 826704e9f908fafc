"""How a step is shared out between the two forms of the latent attention."""
import pytest

from torchinferno_b200.engine.batch import EntryPlacement
from torchinferno_b200.parts import latent_attention
from torchinferno_b200.parts.latent_attention import _plan

SIZES = (16, 256, 512, 64)      # heads, dim + value_dim, rank, rotated


def _entries(pairs):
    row, out = 0, []
    for i, (new, past) in enumerate(pairs):
        out.append(EntryPlacement(i, i, row, new, past))
        row += new
    return out


@pytest.mark.parametrize("pairs, groups, short", [
    ([(1, 4000)] * 3, None, None),
    ([(15, 0), (16, 0)], ((1, 2, 128),), (0, 1)),
    ([(1, 4000)] * 8 + [(2048, 0)], ((8, 9, 2048),), (0, 8)),                          # (decoding contexts are not unfolded)
    ([(512, 0)] + [(1, 4000)] * 64, ((0, 1, 512),), (1, 65)),                          # (many of them do not fold the prompt)
    ([(109, 20), (1, 127), (30, 0)], ((0, 3, 512),), (1, 2)),                          # (a small one between is carried along)
    ([(109, 20), (1, 1000), (30, 0)], ((0, 1, 256), (2, 3, 128)), (1, 2)),
    ([(900, 0), (900, 0), (900, 0)], ((0, 2, 2048), (2, 3, 1024)), None),              # (as many together as there is room for)
    ([(64, 3000), (64, 100)], ((0, 1, 3072), (1, 2, 256)), None)])                     # (one that needs more room than there is)
def test_each_portion_in_its_own_form(pairs, groups, short, monkeypatch):
    monkeypatch.setattr(latent_attention, "BOTH_FORMS_US", -1e9)      # (apart wherever a step has both)
    entries = _entries(pairs)
    plan = _plan(entries, 16, 2048, *SIZES)
    if groups is None:
        assert plan is None
        return
    assert tuple(g[:3] for g in plan.groups) == groups and plan.short == short and plan.shortest == 16
    assert plan.rows == sum(g[2] for g in groups) and plan.whole == (len(groups) == 1 and groups[0][:2] == (0, len(entries)))
    for a, b, _, longest, longest_kv in plan.groups:
        assert (longest, longest_kv) == (max(e.q_len for e in entries[a:b]), max(e.q_len + e.kv_start for e in entries[a:b]))
    first, last = entries[groups[0][0]], entries[groups[-1][1] - 1]
    assert plan.long_tokens == (first.q_start, last.q_start + last.q_len)
    if short:
        inside = [e for i, e in enumerate(entries) if short[0] <= i < short[1] and not any(a <= i < b and e.q_len >= 16 for a, b, _ in groups)]
        assert plan.short_tokens == (entries[short[0]].q_start, entries[short[1] - 1].q_start + entries[short[1] - 1].q_len)
        assert (plan.short_q_len, plan.short_kv_len) == (max(e.q_len for e in inside), max(e.q_len + e.kv_start for e in inside))


@pytest.mark.parametrize("pairs, form", [
    ([(1, 4000)] * 64 + [(512, 0)], "apart"), ([(1, 4000)] * 8 + [(2048, 0)], "apart"), ([(1, 4000)] * 64 + [(64, 0)], "apart"),
    ([(30, 1), (14, 1)], "unfolded"), ([(1, 1000)] * 8 + [(512, 0)], "unfolded"), ([(512, 0), (1, 100)], "unfolded"), ([(1, 300)] * 4 + [(64, 0)], "unfolded"),
    ([(1, 500)] * 64 + [(16, 0)], "folded"), ([(15, 100)], "folded"), ([(2000, 0), (16, 4000)], "unfolded")])
def test_the_cheapest_form_of_a_mixed_step(pairs, form):
    plan = _plan(_entries(pairs), 16, 1 << 20, *SIZES)
    assert form == ("folded" if plan is None else "apart" if plan.short else "unfolded")
    if form == "unfolded":
        assert plan.whole and plan.long_tokens == (0, sum(n for n, _ in pairs)) and plan.shortest == (1 if min(n for n, _ in pairs) < 16 else 16)
