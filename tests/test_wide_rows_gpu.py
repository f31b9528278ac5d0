"""Row kernels of the hybrid family that read whole 16-byte groups, at the edges of what they take, against the plain bodies."""
from __future__ import annotations

import pytest
import torch

from mdi_llm_b200.ops import hybrid as H
from mdi_llm_b200.ops.hybrid import BatchPlan

pytestmark = pytest.mark.gpu


def _tol(dtype):
    # fp32: sums of up to 8192 terms in another order; bf16: one rounding (2^-9 of the value) that may fall to the other side
    return dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2.0 ** -7, atol=2.0 ** -7)


@pytest.mark.parametrize("n", [8, 12, 2040, 2048, 2056, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("kind", ["layer", "rms", "none"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("odd", [False, True])
def test_norm_rows(n, kind, dtype, odd):
    g = torch.Generator().manual_seed(n)
    x = torch.randn(5, n + 1, generator=g)[:, odd:n + odd] * 3 + 1  # a row that starts on a 16-byte boundary or not
    w, b = (1 + 0.1 * torch.randn(n, generator=g)).to(dtype), torch.randn(n, generator=g).to(dtype)
    bias = b if kind == "layer" else None
    xd = torch.empty(5, n + 8, device="cuda")[:, odd:n + odd]
    xd.copy_(x)
    if kind != "none":
        got = H.norm_rows(xd, w.cuda(), None if bias is None else bias.cuda(), 1e-6, kind, dtype).cpu()
        torch.testing.assert_close(got.float(), H.norm_rows(x, w, bias, 1e-6, kind, dtype).float(), **_tol(dtype))
    y, r = torch.randn(5, n, generator=g).to(dtype), torch.randn(5, n, generator=g)
    rd = r.cuda()
    ww, bb = (None, None) if kind == "none" else (w, bias)
    H.norm_accumulate(rd, y.cuda(), None if ww is None else ww.cuda(), None if bb is None else bb.cuda(), 1e-6, kind, 0.5)
    H.norm_accumulate(r, y, ww, bb, 1e-6, kind, 0.5)
    torch.testing.assert_close(rd.cpu(), r, rtol=2e-5, atol=2e-5)


@pytest.mark.parametrize("heads,kv,D,V,nrot", [(16, 4, 128, 128, 64), (2, 1, 24, 16, 8), (3, 3, 20, 12, 6), (17, 1, 128, 8, 128), (40, 8, 128, 64, 0),
                                               (64, 2, 128, 128, 32), (65, 1, 128, 128, 32)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("borrows", [False, True])
def test_full_norm_append(heads, kv, D, V, nrot, dtype, borrows):
    g = torch.Generator().manual_seed(heads)
    lengths, slots, starts = [3, 1, 9], [2, 0, 1], [0, 5, 700]
    N, S = sum(lengths), 720
    p = torch.randn(N, heads * D + kv * (D + V) + 8, generator=g).to(dtype)
    cols = (0, heads * D, heads * D + kv * D, heads * D + kv * (D + V))
    qw, kw = ((1 + 0.1 * torch.randn(c, generator=g)).to(dtype) for c in (heads * D, kv * D))
    inv = H.rotary_inv_freq(nrot, 10000.0, torch.device("cpu")) if nrot else None
    cache = torch.zeros(3, S, kv * (D + V), dtype=dtype)

    def run(dev):
        x, c = p.clone().to(dev), cache.clone().to(dev)
        plan = BatchPlan.make(lengths, slots, starts, torch.device(dev))
        q, k, v = (x[:, a:b] for a, b in zip(cols, cols[1:]))
        H.full_norm_append(q, None if borrows else k, None if borrows else v, None if inv is None else inv.to(dev), c, plan, heads, kv, D, V,
                           nrot, 1e-6, qw.to(dev), None if borrows else kw.to(dev))
        return x.float().cpu(), c.float().cpu()

    for got, want in zip(run("cuda"), run("cpu")):
        torch.testing.assert_close(got, want, **_tol(dtype))


@pytest.mark.parametrize("M,K", [(1, 128), (5, 2048), (128, 2176), (129, 4096), (3, 4224), (256, 14336)])
@pytest.mark.parametrize("off", [0, 4])
def test_quantize_rows(M, K, off):
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator().manual_seed(K)
    flat = (torch.randn(M * K + off, generator=g) * 3).bfloat16()
    flat[off:off + 128] = 0  # an empty block keeps scale 1
    x = flat.cuda()[off:].view(M, K)
    ld = (M + 127) // 128 * 128 + 5
    q, st = torch.empty(M, K, dtype=torch.uint8, device="cuda"), torch.full((K // 128, ld), float("nan"), device="cuda")
    ops.check(ops.lib().mdi_quantize_rows_fp8(ops.ptr(x), ops.ptr(q), ops.ptr(st), M, K, ld, ops.stream_ptr()), "quantize_rows_fp8")
    q2, st2 = ops.quantize_rows_fp8(x)
    assert torch.equal(q, q2) and torch.equal(st[:, :M], st2[:, :M]) and (st2[:, M:] == 0).all()
    xf = flat[off:].float().view(M, K // 128, 128)
    scale = xf.abs().amax(-1) / 448.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    torch.testing.assert_close(st[:, :M].t().cpu(), scale, rtol=1e-6, atol=0)
    assert (st[:, M:] == 0).all()  # every entry is written: the table held NaN
    back = q.view(torch.float8_e4m3fn).float().cpu().view(M, K // 128, 128) * scale[..., None]
    assert ((back - xf).abs() <= 0.5 * 2.0 ** -3 * xf.abs() * 1.001 + scale[..., None] * 2.0 ** -10 * 1.001).all()  # half a unit of e4m3


@pytest.mark.parametrize("rows", [1, 147, 148])
@pytest.mark.parametrize("heads,hv", [(1, 1), (3, 85), (2, 128), (5, 103)])
def test_headmajor_gate(rows, heads, hv):
    g = torch.Generator().manual_seed(rows)
    a, gate = torch.randn(heads, rows, hv, generator=g), torch.randn(rows, heads * hv + 3, generator=g)[:, 1:heads * hv + 1]
    got = H.headmajor_gate(a.cuda(), gate.cuda()).cpu()
    torch.testing.assert_close(got, H.headmajor_gate(a, gate), rtol=2e-6, atol=1e-7)  # expf and a division, 2 units each
