"""Kernels of one-token steps at the sizes where their layout changes, against the same functions on the CPU in fp32."""
from __future__ import annotations

import pytest
import torch

from mdi_llm_b200.ops.hybrid import BatchPlan, NextInput


@pytest.mark.gpu
@pytest.mark.parametrize("C", [4, 1020, 1024, 1028, 2048, 4096, 4100, 1023])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("kind,parts", [("layer", "y b copy next"), ("rms", "y next"), ("layer", "next b"), ("rms", "y copy")], ids=str)
def test_row_update(kind, parts, dtype, C):
    """Rows in registers (up to 4096 values in groups of four) and in shared memory."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(C)
    n = 5
    x, y, w, b, w2, b2 = (torch.randn(*s, generator=g).to(dtype) for s in ((n, C), (n, C), (C,), (C,), (C,), (C,)))
    got = []
    for dev in ("cpu", "cuda"):
        plan = BatchPlan.make([1] * n, list(range(n)), [3] * n, torch.device(dev))
        xx = x.float().to(dev).clone()
        copy = torch.empty(n, C, device=dev, dtype=dtype) if "copy" in parts else None
        bias = lambda t: t.to(dev) if "b" in parts.split() else None  # noqa: E731
        nxt = NextInput(w2.to(dev), bias(b2), 1e-6, kind, None, None) if "next" in parts else None
        yy = y.to(dev) if "y" in parts.split() else None
        h = H.row_update(xx, yy, None if yy is None else w.to(dev), None if yy is None else bias(b), 1e-6, kind, 0.5, copy=copy, nxt=nxt, plan=plan, out_dtype=dtype)
        got.append([t.double().cpu() for t in (xx, copy, h) if t is not None])
    # fp32 sums of up to 4100 squares, a rounding to `dtype` of copy and h (half a unit in the last place of values up to 20, twice)
    for a, c, stored in zip(got[0], got[1], (torch.float32, dtype, dtype)):
        assert (a - c).abs().max() <= (2e-5 if stored == torch.float32 else 2.0 ** -8 * a.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("C,n", [(2052, 5), (3072, 5), (3076, 5), (4096, 592), (4096, 593), (2052, 887), (4096, 888)])
def test_row_update_by_rows(C, n):
    """Widths around the registers that are kept, and row counts around those where fp32 rows keep the kernel in shared memory."""
    from mdi_llm_b200.ops import hybrid as H

    for dtype in (torch.float32, torch.bfloat16):
        g = torch.Generator().manual_seed(C + n)
        x, y, w, b, w2, b2 = (torch.randn(*s, generator=g).to(dtype) for s in ((n, C), (n, C), (C,), (C,), (C,), (C,)))
        got = []
        for dev in ("cpu", "cuda"):
            plan = BatchPlan.make([n], [0], [3], torch.device(dev))
            xx, copy = x.float().to(dev).clone(), torch.empty(n, C, device=dev, dtype=dtype)
            h = H.row_update(xx, y.to(dev), w.to(dev), b.to(dev), 1e-6, "layer", 0.5, copy=copy, nxt=NextInput(w2.to(dev), b2.to(dev), 1e-6, "layer", None, None),
                             plan=plan, out_dtype=dtype)
            got.append([t.double().cpu() for t in (xx, copy, h)])
        for a, c, stored in zip(got[0], got[1], (torch.float32, dtype, dtype)):  # (the bounds of test_row_update)
            assert (a - c).abs().max() <= (2e-5 if stored == torch.float32 else 2.0 ** -8 * a.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("contexts", [(0, 62, 63, 64), (65, 126, 127, 128, 300, 1, 17, 191), (2048,)], ids=str)
@pytest.mark.parametrize("heads,L,R,window", [(16, 512, 64, 0), (3, 32, 16, 0), (17, 96, 32, 100), (8, 128, 64, 64), (16, 512, 144, 0)], ids=str)
def test_latent_decode(heads, L, R, window, contexts):
    """Edges of the tiles of 64 keys, of the shares, of the warps' latent columns; the longest rows of which two tiles fit shared memory."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(L + R + heads)
    D, n, seq = 32, len(contexts), max(contexts) + 1
    qlat = torch.randn(heads, n, L, generator=g)
    q = torch.randn(n, heads * (D + R), generator=g).bfloat16()
    cache = torch.randn(n, seq, L + R, generator=g).bfloat16()
    sink = torch.randn(heads, generator=g)
    slots = list(range(n))[::-1]
    got = []
    for dev in ("cpu", "cuda"):
        plan = BatchPlan.make([1] * n, slots, list(contexts), torch.device(dev))
        got.append(H.latent_attn(qlat.to(dev), q.to(dev), cache.to(dev), plan, heads, D, R, L, (L + R) ** -0.5, window=window, sink=sink.to(dev)).float().cpu())
    # weights and queries as two bf16 numbers (2^-17), the output rounded to bf16 in both
    assert (got[0] - got[1]).abs().max() <= 2.0 ** -7 * got[0].abs().max()
    assert (got[0] - got[1]).norm() <= 4e-3 * got[0].norm()


@pytest.mark.gpu
@pytest.mark.parametrize("split", [0, 1], ids=["shares", "one share"])
@pytest.mark.parametrize("R,nrot", [(160, 0), (160, 64), (208, 208)])
def test_latent_decode_of_rows_too_long_for_two_tiles(R, nrot, split):
    """One tile in shared memory, refilled between the products: one to six tiles a share, the angles' place behind the tiles."""
    from mdi_llm_b200.ops import hybrid as H

    heads, L, D, contexts = 17, 512, 32, (5, 63, 64, 191, 355)
    assert 2 * (32 + 2 * 64) * (L + R + 8) > 210 * 1024  # two tiles do not fit
    g = torch.Generator().manual_seed(R + nrot)
    n, seq = len(contexts), max(contexts) + 1
    qlat = torch.randn(heads, n, L, generator=g)
    q = torch.randn(n, heads * (D + R), generator=g).bfloat16()
    cache = torch.randn(n, seq, L + R, generator=g).bfloat16()
    freq = 1e4 ** (-torch.arange(0, max(nrot, 2), 2).float() / max(nrot, 2))
    got = []
    for dev in ("cpu", "cuda"):
        plan = BatchPlan.make([1] * n, list(range(n)), list(contexts), torch.device(dev))
        got.append(H.latent_attn(qlat.to(dev), q.to(dev), cache.to(dev), plan, heads, D, R, L, (L + R) ** -0.5, split=split, nrot=nrot,
                                 inv_freq=freq.to(dev) if nrot else None).float().cpu())
    # (the bounds of test_latent_decode)
    assert (got[0] - got[1]).abs().max() <= 2.0 ** -7 * got[0].abs().max()
    assert (got[0] - got[1]).norm() <= 4e-3 * got[0].norm()


@pytest.mark.gpu
@pytest.mark.parametrize("D,V", [(128, 128), (64, 128), (32, 16), (128, 48), (100, 64), (130, 64)])
@pytest.mark.parametrize("mode", ["gla", "delta"])
def test_one_token_recurrence(mode, D, V):
    """The register kernel's lanes per column (sixteen, four) against the kernel with its state in shared memory."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(D * V)
    heads, n = 3, 4

    def rnd(*s):
        return torch.randn(*s, generator=g).bfloat16().cuda()

    q, k, z, v, gate, w = rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * D), rnd(n, heads * V), rnd(n, heads * V), rnd(V)
    kw = dict(beta=rnd(n, heads), a_log=rnd(heads)) if mode == "delta" else dict(tau=4.0)
    first, got = torch.randn(n, heads, D, V, generator=g).cuda(), []
    for variant in (1, 2):
        state = first.clone()
        plan = BatchPlan.make([1] * n, list(range(n)), [7] * n, torch.device("cuda"))
        y = H.gated_recurrence(q, k, v, z, gate, w, state, plan, heads=heads, kv_heads=heads, dim=D, vdim=V, mode=mode, eps=1e-5, variant=variant, **kw)
        got.append((y.float(), state))
    # sums of up to 130 terms in another order; the output rounded to bf16
    assert (got[0][1] - got[1][1]).abs().max() <= 2e-6 * got[0][1].abs().max() * 8
    assert (got[0][0] - got[1][0]).abs().max() <= 2.0 ** -7 * got[0][0].abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("Q,L,R", [(8, 8, 8), (1536, 512, 64), (2048, 2048, 8), (2056, 512, 64)])
def test_latent_prepare_by_rows(Q, L, R, dtype):
    """Rows that are asked for at once (up to 444 of up to 2048 values) and rows that are not: the same bits."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator().manual_seed(Q + L)
    p = torch.randn(445, Q + L + R, generator=g).to("cuda", dtype)
    qw, w, f = torch.randn(Q, generator=g).to("cuda", dtype), torch.randn(L, generator=g).to("cuda", dtype), torch.rand(R // 2, generator=g).cuda()
    got = []
    for n in (445, 444, 3):
        cache = torch.zeros(1, 450, L + R, device="cuda", dtype=dtype)
        plan = BatchPlan.make([n], [0], [2], torch.device("cuda"))
        cq = H.latent_prepare(p[:n, :Q], qw, p[:n, Q:], w, f, cache, plan, R, L, R, 1e-6)
        got.append((cq, cache[0, 2:2 + n]))
    for cq, rows in got[1:]:
        assert torch.equal(cq, got[0][0][:cq.size(0)]) and torch.equal(rows, got[0][1][:rows.size(0)])
    want = p[:, :Q].double() / (p[:, :Q].double().square().mean(-1, keepdim=True) + 1e-6).sqrt() * qw.double()
    # fp32 sums of up to 2056 squares, the result rounded to `dtype`
    assert (got[0][0].double() - want).norm() <= (1e-6 if dtype == torch.float32 else 2.0 ** -8) * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("width", [8, 576, 100, 33])
@pytest.mark.parametrize("window", [0, 5, 64])
def test_gathered_keys(width, window):
    """The rows that each sequence sees, whole 16-byte groups or not, of slots in any order."""
    from mdi_llm_b200.ops import hybrid as H

    lengths, slots, starts = [9, 1, 70, 3], [2, 0, 4, 1], [0, 63, 7, 5]
    cache = torch.randn(5, 80, width, generator=torch.Generator().manual_seed(width)).bfloat16().cuda()
    plan = BatchPlan.make(lengths, slots, starts, torch.device("cuda"))
    spans, at, want = [], 0, []
    for (r0, n, slot, p0) in plan.seqs:
        first = max(0, p0 - window + 1) if window else 0
        spans.append((r0, n, at, p0, first))
        at += p0 + n - first
        want.append(cache[slot, first:p0 + n])
    assert torch.equal(H.gather_keys(cache, plan, spans, H.span_table(plan, window)), torch.cat(want))
    with pytest.raises(H.HybridOpsError):
        H.gather_keys(cache[:, :70], plan, spans, H.span_table(plan, window))
    for other in (cache.half(), cache[:, :, :width - 1], torch.randn(5, width, 80, device="cuda").bfloat16().transpose(1, 2)):
        with pytest.raises(H.HybridOpsError):
            H.gather_keys(other, plan, spans, H.span_table(plan, window))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.02, 1.0, 30.0, 300.0])
def test_capped_scores_small_and_large(scale):
    """Scores within three quarters of the cap, on both sides of it in one tile, and far beyond it."""
    from mdi_llm_b200.ops import hybrid as H

    g = torch.Generator(device="cuda").manual_seed(3)
    n, heads, G, D, cap = 300, 2, 1, 128, 20.0
    q = (torch.randn(n, heads * D, generator=g, device="cuda") * torch.logspace(-1, 0, n, device="cuda")[:, None] * scale).bfloat16()
    kv = torch.randn(n, G * 2 * D, generator=g, device="cuda").bfloat16()
    y = H.prompt_attn(q, kv, [(0, n, 0, 0, 0)], heads, D, D, D ** -0.5, split=True, kv_heads=G, cap=cap).double()
    k, v = kv[:, :D].double(), kv[:, D:].double()
    s = cap * torch.tanh(torch.einsum("nhd,md->hnm", q.view(n, heads, D).double(), k) * D ** -0.5 / cap)
    s = s.masked_fill(torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ref = torch.einsum("hnm,md->nhd", torch.softmax(s, -1), v)
    # weights as two bf16 numbers, sums in fp32, one rounding to bf16 (2^-9) at the end
    assert (y - ref).norm() / ref.norm() < 2.5e-3
