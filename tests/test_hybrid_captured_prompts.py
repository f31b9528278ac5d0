"""Prompt kernels whose launches are laid out from the step's list of sequences, inside a CUDA graph."""
from __future__ import annotations

import pytest
import torch

from mdi_llm_b200.ops import hybrid as H
from mdi_llm_b200.ops.hybrid import BatchPlan


def _case(kind):
    """A plan and a call on it that starts from the same state every time; returns its outputs."""
    g = torch.Generator().manual_seed(7)
    lengths = [70, 3, 130]
    N = sum(lengths)

    def rnd(*s):
        return torch.randn(*s, generator=g).bfloat16().cuda()

    plan = BatchPlan.make(lengths, [1, 0, 2], [0, 5, 0], torch.device("cuda"))
    heads, D, V, S = 2, 32, 16, 144
    if kind == "attention":
        q, cache = rnd(N, heads * D), rnd(3, S, heads * (D + V))
        spans = [(r0, n, slot * S + max(0, p0 - 39), p0, max(0, p0 - 39)) for r0, n, slot, p0 in plan.seqs]
        return plan, lambda: [H.prompt_attn(q, cache.view(-1, cache.size(2)), spans, heads, D, V, 0.2, 40, table=H.span_table(plan, 40, S))]
    if kind == "packed attention":
        keys = sum(n + p0 for _, n, _, p0 in plan.seqs)
        q, kv, spans, at = rnd(N, heads * D), rnd(keys, heads * (D + V)), [], 0
        for r0, n, _, p0 in plan.seqs:
            spans.append((r0, n, at, p0, 0))
            at += n + p0
        return plan, lambda: [H.prompt_attn(q, kv, spans, heads, D, V, 0.2, table=H.span_table(plan, 0))]
    first = torch.randn(3, heads, D, V, generator=g).cuda()
    state = torch.empty_like(first)
    if kind == "lightning":
        q, k, v, decay = rnd(N, heads * D), rnd(N, heads * D), rnd(N, heads * V), torch.tensor([0.9, 0.99], device="cuda")

        def call():
            state.copy_(first)
            return [H.lightning_recurrence(q, k, v, decay, state, plan, heads, D, V, variant=2), state]
    else:
        xbc, dt, d = rnd(N, heads * V + 2 * D), rnd(N, heads), torch.ones(heads, device="cuda")

        def call():
            state.copy_(first)
            return [H.ssd_recurrence(xbc, dt, d, d, d, state, plan, heads, 1, D, V, variant=2), state]
    return plan, call


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["attention", "packed attention", "lightning", "state space"])
def test_a_plan_that_has_run_can_be_captured(kind):
    plan, call = _case(kind)
    want = [t.clone() for t in call()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # on another stream than the pass before
        got = call()
    for t in got:
        t.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["attention", "lightning"])
def test_a_plan_that_has_not_run_is_refused(kind):
    plan, call = _case(kind)
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(H.HybridOpsError):
        with torch.cuda.graph(graph):
            call()


@pytest.mark.gpu
def test_streams_have_tables_of_their_own():
    plan, call = _case("attention")
    want = call()[0]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = call()[0]
    side.synchronize()
    assert torch.equal(got, want)
    tables = [t for k, v in plan.shared.items() if k.startswith("table_") for t in v.values()]
    assert len({t.data_ptr() for t in tables}) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("window,mask,cap", [(40, "window", 0.0), (0, "window", 30.0), (48, "chunk", 0.0)])
def test_prompt_attention_on_tcgen05_can_be_captured(window, mask, cap, monkeypatch):
    """Heads of 128, which run on tensor memory with maps of the call's tensors: a captured call reads what they hold when it is replayed."""
    monkeypatch.setattr(H, "_tc_pays", lambda *a: True)
    g = torch.Generator().manual_seed(8)
    lengths, starts, heads, D, S = [70, 3, 130], [0, 5, 0], 2, 128, 144
    plan = BatchPlan.make(lengths, [1, 0, 2], starts, torch.device("cuda"))
    data = [[torch.randn(*s, generator=g).bfloat16().cuda() for s in ((sum(lengths), heads * D), (3, S, heads * 2 * D))] for _ in range(2)]
    (q, cache), other = [t.clone() for t in data[0]], data[1]
    low = [0 if not window else p0 // window * window if mask == "chunk" else max(0, p0 - window + 1) for _, _, _, p0 in plan.seqs]
    spans = [(r0, n, slot * S + f, p0, f) for (r0, n, slot, p0), f in zip(plan.seqs, low)]

    def call():
        return H.prompt_attn(q, cache.view(-1, cache.size(2)), spans, heads, D, D, 0.1, window, True, table=H.span_table(plan, window, S, mask),
                             cap=cap, mask=mask, status=plan.status)

    first = call().clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = call()
    for inputs in (other, data[0]):
        q.copy_(inputs[0])
        cache.copy_(inputs[1])
        want = call().clone()
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    assert torch.equal(got, first)
