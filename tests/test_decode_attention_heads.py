"""Decode attention for every head size and number of query heads, at the edges of its tiles, from queries at any place."""
from __future__ import annotations

import math

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("qpk,hs", [(q, hs) for hs in (64, 128) for q in (1, 2, 4, 8)] + [(1, 256), (2, 256)])
@pytest.mark.parametrize("L", [1, 8, 9, 16, 17, 128, 129, 257, 1100])
@pytest.mark.parametrize("odd", [0, 1], ids=["aligned", "odd"])
def test_heads(qpk, hs, L, odd):
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(L + hs)
    G, S, n_split = 3, 1152, 16
    H = G * qpk
    q = torch.zeros(H * hs + 1, device="cuda", dtype=torch.bfloat16)[odd:][:H * hs]
    q.copy_(torch.randn(H * hs, generator=g, device="cuda"))
    kv = torch.randn(1, 2, G, S, hs, generator=g, device="cuda").bfloat16()
    kv[:, :, :, L:] = float("nan")  # nothing behind the newest position is read into a result
    y, tickets = torch.zeros(H * hs, device="cuda", dtype=torch.bfloat16), torch.zeros(G, device="cuda", dtype=torch.int32)
    part = torch.full((H * n_split * (hs + 2),), float("nan"), device="cuda")
    ctx = torch.zeros(8, device="cuda", dtype=torch.int32)
    ctx[ops.CTX_POS] = L - 1
    ops.attn_decode(q, kv, y, part, tickets, ctx, n_head=H, n_groups=G, head_size=hs, max_seq=S, n_split=n_split)
    k, v = (kv[0, i, :, :L].double().repeat_interleave(qpk, 0) for i in (0, 1))
    ref = torch.softmax((q.view(H, 1, hs).double() @ k.transpose(1, 2)) / math.sqrt(hs), -1) @ v
    # exact products, fp32 sums of up to 256 terms, weights in fp32; one rounding to bf16 (2^-9) at the end
    assert (y.view(H, 1, hs).double() - ref).norm() / ref.norm() < 2.5e-3
    assert tickets.abs().sum() == 0
