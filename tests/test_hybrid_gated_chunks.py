"""The chunked prompt form of the gated recurrences against the recurrence itself in float64, token by token."""
from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

from mdi_llm_b200.ops.hybrid import BatchPlan


def _exact(t, state, lengths, slots, heads, kv, D, V, mode, tau, eps):
    """Outputs and final states in float64 from the float64 copies in ``t``."""
    N, rep = sum(lengths), heads // kv
    z = t["z"].view(N, heads, D) + t["zb"].view(heads, D)
    q, k = (t[n].reshape(N, kv, D).repeat_interleave(rep, 1) for n in ("q", "k"))
    if mode == "delta":
        a = torch.exp(-torch.exp(t["a_log"])[None, :, None] * torch.clamp(z, min=0).add(torch.log1p(torch.exp(-z.abs()))))
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        b = torch.sigmoid(t["beta"])
        gate = torch.sigmoid(t["gate"])
    else:
        a = torch.exp(F.logsigmoid(z) / tau)
        gate = F.silu(t["gate"])
    q, v, out, S = q * D ** -0.5, t["v"].view(N, heads, V), torch.empty(N, heads, V, dtype=torch.float64), state.clone()
    r = 0
    for n, slot in zip(lengths, slots):
        s = S[slot]
        for i in range(r, r + n):
            s.mul_(a[i][:, :, None])
            u = v[i] if mode == "gla" else b[i][:, None] * (v[i] - torch.einsum("hdv,hd->hv", s, k[i]))
            s += k[i][:, :, None] * u[:, None]
            out[i] = torch.einsum("hdv,hd->hv", s, q[i])
        r += n
    out = out / torch.sqrt((out * out).mean(-1, keepdim=True) + eps) * t["w"]
    return (out.reshape(N, heads * V) * gate), S


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("decay", ["slow", "mixed", "spikes"])
@pytest.mark.parametrize("heads,kv,D,V,lengths", [
    (2, 1, 128, 128, (64, 1, 200)), (3, 3, 64, 48, (15, 129, 63, 2)), (2, 2, 32, 16, (65, 16, 17, 128)), (1, 1, 128, 112, (24,)),
], ids=str)
@pytest.mark.parametrize("mode", ["gla", "delta"])
def test_chunks_against_float64(mode, heads, kv, D, V, lengths, decay, dtype):
    """The chunks' sums run in another order than the scan's, both in fp32 from the same values: neither may be further from
    float64 than a few times the other (or than fp32 sums of this length are at all)."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(len(lengths) * D + V)
    N = sum(lengths)

    def rnd(*s, scale=1.0):
        return (torch.randn(*s, generator=g) * scale).to(torch.bfloat16)

    sign = 1.0 if mode == "gla" else -1.0  # the direction of z that keeps the state
    z = rnd(N, heads * D, scale=2.0)
    if decay == "slow":
        z = (z.float() * 0.25 + 6.0 * sign).to(torch.bfloat16)
    if decay == "spikes":
        z = torch.where(torch.rand(N, 1, generator=g) < 0.1, torch.tensor(-90.0 * sign), z.float() + 5.0 * sign).to(torch.bfloat16)
    t = dict(q=rnd(N, kv * D), k=rnd(N, kv * D), v=rnd(N, heads * V), z=z, gate=rnd(N, heads * V), w=1 + rnd(V, scale=0.1).float(),
             zb=rnd(heads * D, scale=0.3), beta=rnd(N, heads, scale=2.0), a_log=rnd(heads, scale=0.3))
    t["w"] = t["w"].to(torch.bfloat16)
    if decay == "slow":  # repeated keys that are read back in full: the hardest triangular systems
        t["k"][N // 2:] = t["k"][N // 2]
        t["beta"][N // 2:] = 8.0
    slots = list(range(len(lengths)))[::-1]
    state = rnd(len(lengths), heads, D, V, scale=0.3).float()
    want_y, want_s = _exact({n: x.double() for n, x in t.items()}, state.double(), lengths, slots, heads, kv, D, V, mode, 5.0, 1e-5)
    err = {}
    for variant in (3, 4):
        x = {n: v.to("cuda", dtype) for n, v in t.items()}
        wide = torch.zeros(N, heads * D + 3, device="cuda", dtype=dtype)  # rows that start at odd places
        wide[:, 3:] = x["z"]
        st = state.cuda()
        kw = dict(beta=x["beta"], a_log=x["a_log"]) if mode == "delta" else dict(tau=5.0)
        plan = BatchPlan.make(lengths, slots, [0] * len(lengths), torch.device("cuda"))
        y = H.gated_recurrence(x["q"], x["k"], x["v"], wide[:, 3:], x["gate"], x["w"], st, plan, heads=heads, kv_heads=kv, dim=D,
                               vdim=V, mode=mode, eps=1e-5, zb=x["zb"], variant=variant, **kw)
        err[variant] = ((y.double().cpu() - want_y).norm() / want_y.norm(), (st.double().cpu() - want_s).norm() / want_s.norm())
    print(mode, D, V, decay, dtype, {v: tuple("%.2g" % float(x) for x in e) for v, e in err.items()})
    # outputs are rounded to `dtype` once (2^-9 for bf16), the state is fp32: sums of up to 128 + 64 terms of like size, twice
    floor_y, floor_s = (2e-6 if dtype == torch.float32 else 2e-3), 2e-6
    assert err[4][0] <= 1.5 * err[3][0] + floor_y
    assert err[4][1] <= 1.5 * err[3][1] + floor_s


@pytest.mark.gpu
def test_sizes_without_a_chunked_form_keep_the_scan():
    from mdi_llm_b200.ops import hybrid as H

    assert [H.lib().hyb_gated_chunk_floats(D, V, 1) > 0 for D, V in ((128, 128), (128, 129), (96, 64), (64, 144), (32, 16), (256, 64))] \
        == [True, False, False, False, True, False]


@pytest.mark.gpu
def test_a_captured_prompt_keeps_the_scan():
    """A capture of a long step is accepted as before, and replays follow the state it was captured on."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(5)
    heads, D, V, n = 2, 32, 16, 200
    q, k, z = (torch.randn(n, heads * D, generator=g).bfloat16().cuda() for _ in range(3))
    v, gate = (torch.randn(n, heads * V, generator=g).bfloat16().cuda() for _ in range(2))
    w = torch.ones(V, device="cuda", dtype=torch.bfloat16)
    plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
    state = torch.zeros(1, heads, D, V, device="cuda")

    def run(variant=0):
        return H.gated_recurrence(q, k, v, z, gate, w, state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode="gla", eps=1e-5, tau=4.0,
                                  variant=variant)

    want = run().clone()
    end = state.clone()
    state.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    graph.replay()
    torch.cuda.synchronize()
    # scan and chunks: fp32 sums of 200 terms in another order, the output rounded to bf16 (one unit in the last place)
    assert (got.float() - want.float()).abs().max() <= 2.0 ** -7 * want.float().abs().max()
    assert (state - end).abs().max() <= 1e-5 * end.abs().max()
    with pytest.raises(H.HybridOpsError):  # asked for by number it is refused
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            run(variant=4)


@pytest.mark.gpu
@pytest.mark.parametrize("what", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("place", [0, 5, 31, 32, 47, 63, 64, 90])
@pytest.mark.parametrize("mode", ["gla", "delta"])
@pytest.mark.parametrize("variant", [0, 4])
def test_a_value_that_is_not_finite_leaves_earlier_tokens_alone(variant, mode, place, what):
    """Outputs before a token with such a value are bit for bit those of a prompt without it; from it on none is a number."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(place)
    heads, D, V, n = 2, 64, 48, 130

    def rnd(*s):
        return torch.randn(*s, generator=g).bfloat16().cuda()

    q, k, z, v, gate = rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * V), rnd(n, heads * V)
    beta, a_log, w = rnd(n, heads), rnd(heads), torch.ones(V, device="cuda", dtype=torch.bfloat16)
    kw = dict(beta=beta, a_log=a_log) if mode == "delta" else dict(tau=4.0)
    out = []
    for values in (v, v.clone()):
        if out:
            values[place, V:] = what  # the second head's
        state = torch.zeros(1, heads, D, V, device="cuda")
        plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
        out.append(H.gated_recurrence(q, k, values, z, gate, w, state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode=mode,
                                      eps=1e-5, variant=variant, **kw).cpu())
    assert torch.isfinite(out[0]).all()
    assert torch.equal(out[1][:place], out[0][:place]) and torch.equal(out[1][:, :V], out[0][:, :V])
    assert not torch.isfinite(out[1][place:, V:]).any()


@pytest.mark.gpu
def test_a_call_is_three_launches():
    """Short prompts are bound by the host: the chunks take as many launches as the scan, with nothing to tabulate before them."""
    from torch.profiler import ProfilerActivity, profile

    from mdi_llm_b200.ops import hybrid as H

    heads, D, V, n = 2, 32, 16, 100
    q, k, z = (torch.randn(n, heads * D, device="cuda").bfloat16() for _ in range(3))
    v, gate = (torch.randn(n, heads * V, device="cuda").bfloat16() for _ in range(2))
    w, state = torch.ones(V, device="cuda", dtype=torch.bfloat16), torch.zeros(1, heads, D, V, device="cuda")
    names = {}
    for variant in (3, 4):
        for _ in range(2):  # the first pass loads the kernels
            plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
            torch.cuda.synchronize()
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                H.gated_recurrence(q, k, v, z, gate, w, state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode="gla", eps=1e-5,
                                   tau=4.0, variant=variant)
                torch.cuda.synchronize()
        names[variant] = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    assert len(names[4]) == len(names[3]) == 3, names


def test_which_sequences_of_a_step_go_in_chunks():
    """Short prompts and one-token streams keep the scan; a few of them ride along with a prompt, many do not."""
    from mdi_llm_b200.ops import hybrid as H

    for mode in ("gla", "delta"):
        T, B = H.gated_chunk_rule[mode]["from"], H.gated_chunk_rule[mode]["beside"]
        assert 0 < T <= B
        assert H.gated_chunk_least([T - 1], 16, 128, mode) == H.gated_chunk_least([1] * 64 + [T - 1], 16, 128, mode) == 0
        assert H.gated_chunk_least([T], 16, 128, mode) == H.gated_chunk_least([1, T, 1], 16, 128, mode) == 1
        assert H.gated_chunk_least([T] * 64, 16, 128, mode) == 1  # nobody is short
        assert H.gated_chunk_least([1] * 64 + [B - 1], 16, 128, mode) == 0
        assert H.gated_chunk_least([1] * 64 + [B], 16, 128, mode) == T
        assert H.gated_chunk_least([T - 1] * 9 + [2048], 16, 128, mode) == T
        assert H.gated_chunk_least([T - 1] * 9 + [2048], 2, 16, mode) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [(1,) * 20 + (150,) + (1,) * 20, (300, 1, 30) + (1,) * 34 + (20, 150, 2), (47,) * 38 + (200,)], ids=["streams", "mixed", "short prompts"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("mode", ["gla", "delta"])
def test_a_step_of_streams_and_prompts(mode, dtype, lengths):
    """Prompts in chunks and the rest by the scan, in any order, on slots in any order, against float64."""
    from mdi_llm_b200.ops import hybrid as H

    heads, kv, D, V = 4, 2, 64, 128
    g = torch.Generator().manual_seed(len(lengths))
    N = sum(lengths)

    def rnd(*s, scale=1.0):
        return (torch.randn(*s, generator=g) * scale).to(torch.bfloat16)

    sign = 1.0 if mode == "gla" else -1.0
    t = dict(q=rnd(N, kv * D), k=rnd(N, kv * D), v=rnd(N, heads * V), z=(rnd(N, heads * D).float() + 3.0 * sign).to(torch.bfloat16), gate=rnd(N, heads * V),
             w=(1 + rnd(V, scale=0.1).float()).to(torch.bfloat16), zb=rnd(heads * D, scale=0.3), beta=rnd(N, heads, scale=2.0), a_log=rnd(heads, scale=0.3))
    slots = torch.randperm(len(lengths), generator=g).tolist()
    state = rnd(len(lengths), heads, D, V, scale=0.3).float()
    want_y, want_s = _exact({n: x.double() for n, x in t.items()}, state.double(), lengths, slots, heads, kv, D, V, mode, 5.0, 1e-5)
    assert H.gated_chunk_least(lengths, heads, V, mode) > 1
    err = {}
    for variant in (3, 0):
        x = {n: v.to("cuda", dtype) for n, v in t.items()}
        st = state.cuda()
        kw = dict(beta=x["beta"], a_log=x["a_log"]) if mode == "delta" else dict(tau=5.0)
        plan = BatchPlan.make(lengths, slots, [0] * len(lengths), torch.device("cuda"))
        y = H.gated_recurrence(x["q"], x["k"], x["v"], x["z"], x["gate"], x["w"], st, plan, heads=heads, kv_heads=kv, dim=D, vdim=V,
                               mode=mode, eps=1e-5, zb=x["zb"], variant=variant, **kw)
        err[variant] = ((y.double().cpu() - want_y).norm() / want_y.norm(), (st.double().cpu() - want_s).norm() / want_s.norm())
    # as above: neither form further from float64 than the other or than fp32 sums of this length are
    assert err[0][0] <= 1.5 * err[3][0] + (2e-6 if dtype == torch.float32 else 2e-3)
    assert err[0][1] <= 1.5 * err[3][1] + 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["gla", "delta"])
def test_heads_in_turns_within_the_work_space(mode, monkeypatch):
    """Work space has a limit; heads that do not fit into it run one group after the other, with the same results."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(2)
    heads, kv, D, V, lengths = 6, 3, 32, 32, [130, 70]
    N = sum(lengths)

    def rnd(*s):
        return torch.randn(*s, generator=g).bfloat16().cuda()

    q, k, z, v, gate = rnd(N, kv * D), rnd(N, kv * D), rnd(N, heads * D), rnd(N, heads * V), rnd(N, heads * V)
    beta, a_log, w = rnd(N, heads), rnd(heads), torch.ones(V, device="cuda", dtype=torch.bfloat16)
    kw = dict(beta=beta, a_log=a_log) if mode == "delta" else dict(tau=4.0)
    nchunks, floats = 5, H._gated_chunk_floats(D, V, int(mode == "delta"))
    got = []
    for at_once in (heads, 4, 1, 0):  # none fits: one at a time all the same
        monkeypatch.setattr(H, "gated_chunk_work", at_once * nchunks * floats + 1)
        state = torch.zeros(2, heads, D, V, device="cuda")
        plan = BatchPlan.make(lengths, [1, 0], [0, 0], torch.device("cuda"))
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        y = H.gated_recurrence(q, k, v, z, gate, w, state, plan, heads=heads, kv_heads=kv, dim=D, vdim=V, mode=mode, eps=1e-5, variant=4, **kw)
        assert torch.cuda.max_memory_allocated() - before < 4 * (max(1, at_once) * nchunks * floats) + (1 << 18)
        got.append((y, state))
    for y, state in got[1:]:
        assert torch.equal(y, got[0][0]) and torch.equal(state, got[0][1])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("D,V,n", [(32, 16, 17), (64, 128, 64), (128, 48, 129), (128, 128, 72)])
@pytest.mark.parametrize("mode", ["gla", "delta"])
def test_rows_at_odd_places_and_a_key_that_is_not_finite(mode, D, V, n, dtype):
    """Loads of single values bring what wide ones do, bit for bit; a key that is not finite reaches no row before its own."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(D + V)
    heads = 2

    def rnd(*s):
        return torch.randn(*s, generator=g).bfloat16().to("cuda", dtype)

    def odd(x):
        wide = torch.zeros(x.size(0), x.size(1) + 3, device="cuda", dtype=dtype)
        wide[:, 1:-2] = x
        return wide[:, 1:-2]

    q, k, z, v, gate = rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * V), rnd(n, heads * V)
    kw = dict(beta=rnd(n, heads), a_log=rnd(heads)) if mode == "delta" else dict(tau=4.0)
    w, place, out = rnd(V), n // 2 + 1, []
    for turn in range(3):
        x = [odd(t) if turn == 1 else t for t in (q, k, v, z, gate)]
        if turn == 2:
            x[1] = k.clone()
            x[1][place, 3] = float("inf")
        state = torch.zeros(1, heads, D, V, device="cuda")
        plan = BatchPlan.make([n], [0], [0], torch.device("cuda"))
        y = H.gated_recurrence(*x, w, state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode=mode, eps=1e-5, variant=4, **kw)
        out.append((y, state))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert torch.equal(out[0][0][:place], out[2][0][:place])
    assert torch.equal(out[0][0][:, V:], out[2][0][:, V:]) and not torch.isfinite(out[2][0][place:, :V]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("through", ["logit", "bias"])
@pytest.mark.parametrize("mode,tau", [("gla", 5.0), ("gla", 1e-3), ("delta", 1.0)])
def test_gate_logits_without_bounds(mode, tau, through, dtype):
    """A logit that is infinite, or so large that its quotient by tau is, closes its channel (decay 0) or leaves it as it is (decay 1), in
    every form alike: chunks, scan, registers, shared memory and the CPU."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(11)
    heads, D, V, n = 2, 32, 16, 100

    def rnd(*s):
        return torch.randn(*s, generator=g).to(torch.bfloat16).to(dtype)

    q, k, z, v, gate, w, zb = rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * V), rnd(n, heads * V), rnd(V), rnd(heads * D)
    special = torch.tensor([float("inf"), float("-inf"), 3e38, -3e38, 1e5, -1e5, 200.0, -200.0]).to(dtype)
    if through == "bias":
        zb[3:11] = special
    else:
        for i in range(8):
            z[11 * i + 3::17, 5 + i] = special[i]
    kw = dict(beta=rnd(n, heads), a_log=rnd(heads)) if mode == "delta" else dict(tau=tau)
    got = {}
    for variant in ("cpu", 1, 2, 3, 4):
        dev = torch.device("cpu" if variant == "cpu" else "cuda")
        state = torch.ones(1, heads, D, V, device=dev)
        plan = BatchPlan.make([n], [0], [0], dev)
        y = H.gated_recurrence(*(t.to(dev) for t in (q, k, v, z, gate, w)), state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode=mode, eps=1e-5,
                               zb=zb.to(dev), variant=0 if variant == "cpu" else variant, **{a: b.to(dev) if torch.is_tensor(b) else b for a, b in kw.items()})
        got[variant] = (y.double().cpu(), state.double().cpu())
    for variant, (y, state) in got.items():
        assert torch.isfinite(y).all() and torch.isfinite(state).all(), variant
        # fp32 sums of up to 100 + 64 terms; outputs are rounded to `dtype` (bf16: half of 2^-8)
        assert (state - got["cpu"][1]).norm() <= 1e-5 * got["cpu"][1].norm(), variant
        assert (y - got["cpu"][0]).norm() <= (1e-5 if dtype == torch.float32 else 2.0 ** -8) * got["cpu"][0].norm(), variant
