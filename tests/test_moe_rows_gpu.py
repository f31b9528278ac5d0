"""The routed feed-forward of a prompt on the device against the eager formulation."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,top", [(1, 8, 2), (33, 8, 2), (300, 8, 2), (257, 3, 1), (130, 40, 4), (64, 256, 8)])
def test_rows_are_sorted_and_combined(T, E, top):
    from mdi_llm_b200 import ops

    g = torch.Generator().manual_seed(T + E)
    C = 256
    logits = torch.randn(T, E, generator=g).bfloat16()
    logits[0, : min(E, 4)] = 9.0  # equal logits: the lower expert first
    h = torch.randn(T, C, generator=g).bfloat16()
    wts, counts, where, rows = (t.cpu() for t in ops.moe_rows_sort(logits.cuda(), h.cuda(), top))
    order = torch.argsort(-logits.float(), dim=-1, stable=True)[:, :top]
    val = torch.gather(logits.float(), 1, order)
    assert torch.equal(counts.long(), torch.bincount(order.reshape(-1), minlength=E))
    pos = torch.argsort(order.reshape(-1), stable=True)
    want = torch.empty_like(pos)
    want[pos] = torch.arange(T * top)
    assert torch.equal(where.long().reshape(-1), want) and torch.equal(rows, h[pos // top])
    # the softmax in fp32, rounded to bf16 once: one unit in the last place
    assert (wts.float() - torch.softmax(val, -1)).abs().max() <= 2.0 ** -8
    x, y = torch.randn(T, C, generator=g).bfloat16(), torch.randn(T * top, C, generator=g).bfloat16()
    got = ops.moe_rows_combine(x.cuda(), y.cuda(), where.cuda(), wts.cuda()).cpu()
    s = torch.zeros(T, C).bfloat16()
    for k in range(top):
        s = s + wts[:, k:k + 1] * y[where[:, k].long()]
    assert torch.equal(got, x + s)


@pytest.mark.parametrize("T,E,top", [(128, 8, 2), (129, 8, 2), (900, 1, 1), (700, 16, 2), (1, 16, 8), (300, 17, 1), (513, 32, 1), (33, 33, 2), (800, 256, 8)])
def test_rows_are_sorted_at_the_edges(T, E, top):
    """Pairs around those from which an expert's are counted in parts, experts around a warp each, whole blocks of 256 pairs and what is left."""
    test_rows_are_sorted_and_combined(T, E, top)


@pytest.mark.parametrize("counts", [(5, 0, 256, 257, 1), (0, 0, 300), (1, 2, 3, 4, 5, 6, 7, 8, 9, 513)])
@pytest.mark.parametrize("N,K,gated", [(384, 512, True), (384, 512, False), (200, 72, True), (520, 256, False)])
def test_grouped_gemm_matches_one_product_per_group(counts, N, K, gated):
    from mdi_llm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N + K)
    M = sum(counts)

    def r(*s):
        return torch.randn(*s, generator=g, device="cuda").bfloat16()

    a, w = r(M, K), [r(N, K) * K ** -0.5 for _ in counts]
    w2 = [r(N, K) * K ** -0.5 for _ in counts] if gated else None
    got = ops.gemm_grouped(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), w2=w2)
    at = 0
    for e, n in enumerate(counts):
        y = a[at:at + n].float() @ w[e].float().T
        if gated:
            y = torch.nn.functional.silu(y) * (a[at:at + n].float() @ w2[e].float().T)
        # gate, up and their product are each rounded to bf16: three roundings of half a unit in the last place (2^-9)
        torch.testing.assert_close(got[at:at + n].float(), y, rtol=2e-2, atol=2e-2)
        at += n


@pytest.mark.parametrize("M,N", [(256, 4096), (448, 4096), (448, 6144), (300, 1000), (1000, 14336)])
@pytest.mark.parametrize("gated", [False, True])
def test_pair_gemm_tile_widths(M, N, gated):
    """Shapes that take the 128-, 192- and 256-column tiles of the CTA-pair kernel."""
    from mdi_llm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N)
    K = 320
    a, w, w2 = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N, N))
    w, w2 = w * K ** -0.5, w2 * K ** -0.5
    res = None if gated else torch.randn(M, N, generator=g, device="cuda").bfloat16()
    got = ops.gemm(a, w, w2=w2 if gated else None, residual=res, block_n=512)
    y = a.float() @ w.float().T
    y = torch.nn.functional.silu(y) * (a.float() @ w2.float().T) if gated else y + res.float()
    torch.testing.assert_close(got.float(), y, rtol=2e-2, atol=3e-2)
