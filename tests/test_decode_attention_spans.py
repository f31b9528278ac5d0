"""Where the spans of a decode step's attention meet: in one cluster, or in global memory."""
from __future__ import annotations

import math

import pytest
import torch


def test_the_limits_of_the_cluster_form():
    """Tiles a warp up to which a group's spans stay in a cluster, by head size, query heads per group and groups (the library needs no GPU to be
    asked).  They say what is chosen, not what is faster: the split form, which is taken beyond them, no longer is."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.ops import build

    if build.nvcc_path() is None and not build.is_fresh():
        pytest.skip("the kernel library is not built here")
    tiles = ops.lib().mdi_attn_cluster_tiles
    assert [tiles(128, 4, g) for g in (1, 2, 3, 4, 8, 12, 16, 32)] == [3, 3, 3, 8, 8, 8, 4, 4]
    assert [tiles(128, 2, g) for g in (1, 3, 4, 32)] == [2, 2, 8, 8]
    assert [tiles(256, 1, g) for g in (1, 4, 8, 12, 16)] == [1, 1, 8, 8, 1]
    assert all(tiles(hs, q, g) == 8 for g in (1, 4, 8, 32) for hs, q in ((64, 1), (64, 8), (128, 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,hs", [(32, 8, 128), (4, 1, 128), (64, 16, 128), (8, 4, 128), (16, 2, 64), (16, 16, 256), (8, 8, 256)])
@pytest.mark.parametrize("L", [1025, 2048, 2049, 3072, 3073, 4096, 4097, 8192, 8193, 8300])
def test_spans_against_plain_attention(H, G, hs, L):
    """At every limit of the cluster form, with as many spans as a stage takes (a multiple of the cluster's eight)."""
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(L)
    S = 8320
    n_split = max(8, min(64, 296 // G) // 8 * 8)
    q = torch.randn(H * hs, generator=g, device="cuda").bfloat16()
    kv = torch.randn(1, 2, G, S, hs, generator=g, device="cuda").bfloat16()
    y = torch.zeros(H * hs, device="cuda", dtype=torch.bfloat16)
    tickets = torch.zeros(G, device="cuda", dtype=torch.int32)
    part = torch.full((H * n_split * (hs + 2),), float("nan"), device="cuda")
    ctx = torch.zeros(8, device="cuda", dtype=torch.int32)
    ctx[ops.CTX_POS] = L - 1
    ops.attn_decode(q, kv, y, part, tickets, ctx, n_head=H, n_groups=G, head_size=hs, max_seq=S, n_split=n_split)
    k, v = (kv[0, i, :, :L].double().repeat_interleave(H // G, 0) for i in (0, 1))
    ref = torch.softmax((q.view(H, 1, hs).double() @ k.transpose(1, 2)) / math.sqrt(hs), -1) @ v
    # fp32 throughout, one rounding to bf16 (2^-9) at the end; exponentials are approximate (2^-22)
    assert (y.view(H, 1, hs).double() - ref).norm() / ref.norm() < 2.5e-3
    assert tickets.abs().sum() == 0
