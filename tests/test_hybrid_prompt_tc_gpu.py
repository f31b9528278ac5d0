"""The tcgen05 form of the hybrid family's prompt attention at the edges of its tiles (128 rows, 64 or 128 keys), for every combination of
sizes, masks, cap, sink, gates and split weights that it has a kernel for, against fp64 and against the warp-level kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _on_tcgen05(monkeypatch):
    """These tests are of that form, at sizes for which the rule may choose the other one."""
    from mdi_llm_b200.ops import hybrid as H_

    monkeypatch.setattr(H_, "_tc_pays", lambda *a: True)


def _reference(q, kv, spans, H, G, DK, V, scale, W, sink, gate, cap, chunk):
    out = torch.zeros(q.size(0), H, V, device=q.device, dtype=torch.double)
    for r0, n, k0, p0, first in spans:
        keys = p0 + n - first
        k = kv[k0:k0 + keys, :G * DK].double().view(keys, G, DK).repeat_interleave(H // G, 1)
        v = kv[k0:k0 + keys, G * DK:].double().view(keys, G, V).repeat_interleave(H // G, 1)
        s = torch.einsum("ihd,jhd->hij", q[r0:r0 + n].double().view(n, H, DK), k) * scale
        if cap > 0:
            s = cap * torch.tanh(s / cap)
        i, j = p0 + torch.arange(n, device=q.device)[:, None], first + torch.arange(keys, device=q.device)[None]
        hidden = j > i
        if W > 0:
            hidden = hidden | ((j < i // W * W) if chunk else (i - j >= W))
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.double()[:, None, None].expand(H, n, 1)), -1)
        o = torch.einsum("hij,jhv->ihv", torch.softmax(s, -1)[..., :keys], v)
        out[r0:r0 + n] = o if gate is None else o * torch.sigmoid(gate[r0:r0 + n].double()).view(n, H, -1)
    return out


def _step(lengths, starts, H, G, DK, V, W, chunk, hold=0):
    """Queries, keys and spans of a step; ``hold``: rows between the sequences' keys that belong to nobody."""
    g = torch.Generator(device="cuda").manual_seed(sum(lengths) + DK + V + W)
    spans, r, k0 = [], 0, hold
    for n, p0 in zip(lengths, starts):
        first = 0 if W <= 0 else p0 // W * W if chunk else max(0, p0 - W + 1)
        spans.append((r, n, k0, p0, first))
        r, k0 = r + n, k0 + p0 + n - first + hold
    q = torch.randn(r, H * DK, generator=g, device="cuda").bfloat16()
    return q, torch.randn(k0, G * (DK + V), generator=g, device="cuda").bfloat16(), spans, g


LENGTHS = [((128,), (0,)), ((129, 33), (0, 500)), ((300, 1, 127), (77, 3, 64)), ((65,), (191,)), ((257,), (0,))]


@pytest.mark.parametrize("lengths,starts", LENGTHS)
@pytest.mark.parametrize("DK,V", [(64, 64), (64, 128), (128, 64), (128, 128), (192, 64), (192, 128)])
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("cap", [0.0, 20.0])
@pytest.mark.parametrize("W,chunk", [(0, 0), (100, 0), (96, 1)])
def test_prompt_attention_tiles(lengths, starts, DK, V, split, cap, W, chunk):
    from mdi_llm_b200.ops import hybrid as H_

    H, G = 4, 2
    q, kv, spans, g = _step(lengths, starts, H, G, DK, V, W, chunk)
    kind = (sum(lengths) + V) % 3  # no gate, a gate per head, a gate per value
    gate = None if kind == 0 else torch.randn(q.size(0), H if kind == 1 else H * V, generator=g, device="cuda").bfloat16()
    sink = torch.randn(H, generator=g, device="cuda") if split else None
    args = (q, kv, spans, H, DK, V, 3 * DK ** -0.5, W, bool(split))
    more = dict(kv_heads=G, sink=sink, gate=gate, cap=cap, mask="chunk" if chunk else "window")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = H_.prompt_attn(*args, **more, status=status).double()
    ref = _reference(q, kv, spans, H, G, DK, V, 3 * DK ** -0.5, W, sink, gate, cap, chunk)
    # rounding of the result (2^-9 at most, 0.29 of that in the mean) and, without split, of the weights: 2^-9 times two
    assert int(status) == 0 and (got - ref).norm() <= 2.0 ** -8 * ref.norm()
    assert (got - ref).abs().max() <= 2.0 ** -7 * ref.abs().max()


def test_no_more_error_than_the_warp_level_kernel():
    """Whole prompts, against that kernel with the 64 keys a step that it ran these sizes with (it rounds a row's largest weight so far to
    exactly one, so its error depends on the keys per step): both round the same weights, the sums differ in order only."""
    from mdi_llm_b200.ops import hybrid as H_

    for DK, split in ((128, False), (128, True), (192, False)):
        q, kv, spans, _ = _step((1024, 300), (0, 100), 8, 2, DK, 128, 0, 0)
        ref = _reference(q, kv, spans, 8, 2, DK, 128, DK ** -0.5, 0, None, None, 0.0, 0)
        new = H_.prompt_attn(q, kv, spans, 8, DK, 128, DK ** -0.5, 0, split, kv_heads=2).double()
        old, table = torch.empty(q.size(0), 8, 128, device="cuda", dtype=q.dtype), torch.tensor(spans, dtype=torch.int32, device="cuda")
        H_._check(H_.lib().hyb_prompt_attn_mma(q.data_ptr(), q.stride(0), kv.data_ptr(), kv.stride(0), old.data_ptr(), table.data_ptr(), 2, 1024, 8, 2,
                                               DK, 128, 0, DK ** -0.5, int(split), 64, None, None, 0, 0, 0.0, 0, H_._st()), "prompt_attn_mma")
        assert (new - ref).norm() <= 1.003 * (old.double() - ref).norm()


@pytest.mark.parametrize("bad", [math.inf, math.nan])
@pytest.mark.parametrize("W,chunk", [(0, 0), (100, 0), (96, 1)])
def test_rows_of_other_sequences_stay_out(bad, W, chunk):
    """Keys and values around a sequence's own that are not finite change nothing, bit for bit."""
    from mdi_llm_b200.ops import hybrid as H_

    q, kv, spans, _ = _step((130, 40), (33, 200), 4, 2, 128, 128, W, chunk, hold=140)
    args, more = (spans, 4, 128, 128, 0.1, W, True), dict(kv_heads=2, mask="chunk" if chunk else "window")
    clean = H_.prompt_attn(q, kv, *args, **more)
    own = torch.zeros(kv.size(0), dtype=torch.bool, device="cuda")
    for _, n, k0, p0, first in spans:
        own[k0:k0 + p0 + n - first] = True
    dirty = torch.where(own[:, None], kv, torch.full_like(kv, bad))
    assert torch.equal(H_.prompt_attn(q, dirty, *args, **more), clean)


@pytest.mark.parametrize("bad", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("DK,V,split,cap", [(128, 128, 1, 0.0), (64, 64, 0, 20.0), (192, 128, 0, 0.0)])
@pytest.mark.parametrize("W,chunk", [(0, 0), (100, 0), (300, 0), (96, 1), (300, 1)])
def test_values_that_are_not_finite_reach_the_rows_that_see_their_key(bad, DK, V, split, cap, W, chunk):
    """... and no other: those are what they are with zeros in their place, bit for bit.  Keys at both ends of the diagonal's tiles, in
    tiles that every row of a block sees whole, and around a window's or a block's start."""
    from mdi_llm_b200.ops import hybrid as H_

    H, G = 4, 2
    q, kv, spans, g = _step((500, 70), (40, 150), H, G, DK, V, W, chunk)
    gate = torch.randn(q.size(0), H, generator=g, device="cuda").bfloat16()
    args, more = (spans, H, DK, V, DK ** -0.5, W, bool(split)), dict(kv_heads=G, gate=gate, cap=cap, mask="chunk" if chunk else "window")
    clean, dirty = kv.clone(), kv.clone()
    expect = torch.zeros(q.size(0), H, V, dtype=torch.bool, device="cuda")
    for r0, n, k0, p0, first in spans:
        for pos in (first, p0 + 1, p0 + 63, p0 + 127, p0 + 128, p0 + 290, p0 + n - 1):
            head, column = pos % G, (7 * pos) % V
            if pos >= p0 + n:
                continue
            at = k0 + pos - first, G * DK + head * V + column
            clean[at], dirty[at] = 0, bad
            i = p0 + torch.arange(n, device="cuda")
            sees = (i >= pos) & ((i // W * W <= pos) if chunk else (i - pos < W) if W > 0 else (i >= 0))
            expect[r0:r0 + n, head * (H // G):(head + 1) * (H // G), column] |= sees[:, None]
    assert expect.any() and not expect.all()
    want, got = H_.prompt_attn(q, clean, *args, **more), H_.prompt_attn(q, dirty, *args, **more)
    assert torch.equal(~torch.isfinite(got), expect)
    assert torch.equal(got[~expect], want[~expect])


def test_rows_that_overlap_are_the_warp_level_kernels():
    """One row of keys and values for all positions (a stride of zero), queries that share columns: what a tensor map does not describe."""
    from mdi_llm_b200.ops import hybrid as H_

    g = torch.Generator(device="cuda").manual_seed(4)
    q, kv = (torch.randn(40, 4 * 128, generator=g, device="cuda").bfloat16(), torch.randn(1, 2 * 256, generator=g, device="cuda").bfloat16().expand(40, -1))
    shared = torch.randn(39 * 64 + 512, generator=g, device="cuda").bfloat16().as_strided((40, 512), (64, 1))
    spans = [(0, 40, 0, 0, 0)]
    for a, b in ((q, kv), (shared, torch.randn(40, 512, generator=g, device="cuda").bfloat16())):
        got = H_.prompt_attn(a, b, spans, 4, 128, 128, 0.1, 0, True, kv_heads=2).double()
        want = _reference(a, b.contiguous(), spans, 4, 2, 128, 128, 0.1, 0, None, None, 0.0, 0)
        assert (got - want).norm() <= 2.0 ** -8 * want.norm()
