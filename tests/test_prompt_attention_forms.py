"""The fused prompt attention in every form a design may ask for, against plain float64 attention over the same cache rows."""
from __future__ import annotations

import pytest
import torch

from mdi_llm_b200.ops import hybrid as H
from mdi_llm_b200.ops.hybrid import BatchPlan


def _plain(q, k, v, p0, scale, cap, mask, W, sink, rep):
    """``q [n, H, D]`` at positions ``p0 ..`` over ``k [S, G, D]``, ``v [S, G, V]`` in float64."""
    n, keys = q.size(0), p0 + q.size(0)
    j, p = torch.arange(keys)[None], (p0 + torch.arange(n))[:, None]
    hidden = j > p
    if W:
        hidden = hidden | ((j < p // W * W) if mask == "chunk" else (p - j >= W))
    s = torch.einsum("nhd,khd->hnk", q, k[:keys].repeat_interleave(rep, 1)) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(hidden[None], float("-inf"))
    if sink is not None:
        s = torch.cat((s, sink[:, None, None].expand(-1, n, 1)), -1)
    return torch.einsum("hnk,khv->nhv", torch.softmax(s, -1)[..., :keys], v[:keys].repeat_interleave(rep, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("mask,W", [("window", 0), ("window", 40), ("chunk", 0), ("chunk", 33), ("chunk", 64), ("chunk", 100)])
@pytest.mark.parametrize("cap", [0.0, 5.0])
@pytest.mark.parametrize("sink", ["none", "zero", "learned"])
@pytest.mark.parametrize("split", [False, True])
def test_forms_against_float64(mask, W, cap, sink, split):
    g = torch.Generator().manual_seed(W + int(cap))
    G, rep, D, V, S, slots = 2, 3, 32, 48, 260, 4
    Hh = G * rep
    cache = torch.randn(slots, S, G * (D + V), generator=g).bfloat16()
    lengths, at, starts = [70, 1, 130, 65], [2, 0, 3, 1], [0, 0, 0, 97]
    N = sum(lengths)
    q = (torch.randn(N, Hh * D, generator=g) * 2.0).bfloat16()
    sv = {"none": None, "zero": torch.zeros(Hh), "learned": torch.randn(Hh, generator=g) * 2.0}[sink]
    plan = BatchPlan.make(lengths, at, starts, torch.device("cuda"))
    table = H.span_table(plan, W, S, mask)
    spans = []
    for r0, n, slot, p0 in plan.seqs:
        first = 0 if W <= 0 else p0 // W * W if mask == "chunk" else max(0, p0 - W + 1)
        spans.append((r0, n, slot * S + first, p0, first))
    assert table.cpu().tolist() == [list(s) for s in spans]
    got = H.prompt_attn(q.cuda(), cache.cuda().view(-1, cache.size(2)), spans, Hh, D, V, 0.25, W, split, table=table, kv_heads=G,
                        sink=None if sv is None else sv.cuda(), cap=cap, mask=mask).float().cpu()
    want = torch.empty(N, Hh, V, dtype=torch.float64)
    for r0, n, slot, p0 in plan.seqs:
        k, v = (t.double() for t in (cache[slot, :, :G * D].view(S, G, D), cache[slot, :, G * D:].view(S, G, V)))
        want[r0:r0 + n] = _plain(q[r0:r0 + n].double().view(n, Hh, D), k, v, p0, 0.25, cap, mask, W, None if sv is None else sv.double(), rep)
    # the output is rounded to bf16 once (2^-9); without the remainders the weights are too, each by itself
    assert (got - want).norm() / want.norm() < (2.5e-3 if split else 5e-3)
    assert (got - want).abs().max() < (1.5e-2 if split else 3e-2) * max(1.0, want.abs().max().item())


@pytest.mark.gpu
@pytest.mark.parametrize("each", [False, True], ids=["per head", "per value"])
@pytest.mark.parametrize("V", [16, 48, 128])
def test_gates_cost_no_rounding_of_their_own(V, each):
    """The output is rounded to bf16 once, behind the gate: no further from float64 than float64 rounded that way, but for the weights'
    2^-17.  (With a rounding in front of the gate it is 1.4 times as far.)"""
    g = torch.Generator().manual_seed(V)
    n, Hh, D = 200, 2, 32
    cache = torch.randn(1, n, D + V, generator=g).bfloat16()
    q = torch.randn(n, Hh * D, generator=g).bfloat16()
    wide = torch.randn(n, Hh * V + 7, generator=g).bfloat16()
    gate = wide[:, 3:3 + (Hh * V if each else Hh)]  # a column slice that starts anywhere
    plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
    gd = wide.cuda()[:, 3:3 + gate.size(1)]
    got = H.prompt_attn(q.cuda(), cache.cuda().view(-1, D + V), [(0, n, 0, 0, 0)], Hh, D, V, 0.25, 0, True, table=H.span_table(plan, 0, n),
                        kv_heads=1, gate=gd).double().cpu()
    k, v = cache[0, :, :D].double().view(n, 1, D), cache[0, :, D:].double().view(n, 1, V)
    want = _plain(q.double().view(n, Hh, D), k, v, 0, 0.25, 0.0, "window", 0, None, Hh) * torch.sigmoid(gate.double()).view(n, Hh, -1)
    once = (want.bfloat16().double() - want).norm()
    assert (got - want).norm() < 1.1 * once


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [5.0, 50.0, 1000.0, 10000.0])
def test_the_cap_is_exact_for_scores_far_below_it(cap):
    """Each row sees two keys with scores of up to 6 that differ by some 0.006, with values of +1 and -1: the output is
    tanh(difference / 2), so an error of a score shows as it is.  Scores and cap are fp32 (a few units of 2^-24 * 6 each: 0.1 % of
    outputs of 0.003), the weights keep 16 bits (2^-17: 0.3 %) and the output is rounded once (2^-9 of it: 0.2 %)."""
    g = torch.Generator().manual_seed(3)
    n, Hh, D, V = 192, 2, 16, 16
    base = torch.randn(1, D, generator=g)
    key = base + 2.0 ** -9 * torch.randn(n, D, generator=g)
    value = torch.where(torch.arange(n)[:, None] % 2 == 0, 1.0, -1.0).expand(n, V)
    cache = torch.zeros(1, n, D + V)
    cache[0, :, :D], cache[0, :, D:] = key, value
    cache = cache.bfloat16()
    q = torch.randn(n, Hh * D, generator=g)
    q = (q / q.view(n, Hh, D).norm(dim=-1).repeat_interleave(D, 1) * 8.0 / base.norm()).bfloat16()
    plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
    got = H.prompt_attn(q.cuda(), cache.cuda().view(-1, D + V), [(0, n, 0, 0, 0)], Hh, D, V, 1.0, 2, True, table=H.span_table(plan, 2, n),
                        kv_heads=1, cap=cap).double().cpu()
    k, v = cache[0, :, :D].double().view(n, 1, D), cache[0, :, D:].double().view(n, 1, V)
    want = _plain(q.double().view(n, Hh, D), k, v, 0, 1.0, cap, "window", 2, None, Hh)
    assert 2e-3 < want[1:].abs().median() < 5e-3
    assert (got - want)[1:].norm() / want[1:].norm() < 6e-3


def test_forms_are_chosen_by_type_and_size_only():
    q = torch.zeros(4, 64, dtype=torch.bfloat16)
    assert not H.prompt_attn_takes(q, 2, 32, 32)  # not on the CPU: the plain bodies serve there


def test_short_prompts_beside_a_longer_one_keep_the_decoding_form_until_the_fused_one_pays():
    """By what the step's tokens see; prompts of their own, and plain forms as always, go fused."""
    from mdi_llm_b200.models.hybrid import WindowAttention

    def layer(heads, window=0, **traits):
        return WindowAttention(64, dict(heads=heads, kv_heads=2, dim=16, vdim=16, scale=0.25, mask=dict(size=window) if window else None,
                                        softcap=traits.pop("softcap", 0.0)), 1e-5, traits)

    def pays(m, lengths, starts=None):
        return m._fused_pays(BatchPlan.make(lengths, list(range(len(lengths))), starts or [0] * len(lengths), torch.device("cpu")))

    capped = layer(8, softcap=50.0)
    assert not pays(capped, [2, 13, 129, 292, 3]) and not pays(capped, [64, 3]) and not pays(capped, [400, 3])
    assert pays(capped, [600, 3]) and pays(capped, [64]) and pays(capped, [64, 100]) and pays(capped, [300, 3], [1000, 0])
    assert pays(layer(16, softcap=50.0), [400, 3])
    block = layer(8, window=64, mask="chunk", sink=True)
    assert not pays(block, [2000, 3]) and pays(block, [5000, 3])
    assert pays(layer(8, window=64), [64, 3]) and pays(layer(8), [64, 3])
