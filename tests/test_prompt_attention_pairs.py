"""The prompt attention of the transformer stages with two query tiles per block (prompts whose pairs of tiles fill the GPU)."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,hs", [(32, 8, 128), (32, 4, 64), (40, 40, 128)])
@pytest.mark.parametrize("T", [1025, 1152, 1153, 1280, 1300, 2048])
def test_two_tiles_match_plain_attention(H, G, hs, T):
    """Sizes whose last block has a full, a partial or no second tile.  Scratch holds NaN: whatever is read has been written."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.models.gpt import build_rope_cache

    ops.require()
    assert (T + 255) // 256 * H >= 148  # else a block has one tile
    g = torch.Generator(device="cuda").manual_seed(T + hs)
    S, n_slots, slot = T + 77, 2, 1
    qkv = (torch.randn(T, (H + 2 * G) * hs, generator=g, device="cuda") * 0.7).bfloat16()
    cos, sin = (t.float().contiguous() for t in build_rope_cache(S, hs, device=torch.device("cuda")))
    pool = torch.full((n_slots, 2, G, S, hs), float("nan"), device="cuda", dtype=torch.bfloat16)
    T_pad = (T + 127) // 128 * 128
    scratch = tuple(torch.full(s, float("nan"), device="cuda", dtype=torch.bfloat16) for s in ((H, T_pad, hs), (G, hs, T_pad)))
    status = torch.zeros(4, device="cuda", dtype=torch.int32)
    y = ops.attn_prefill(qkv, cos, sin, pool, slot, n_head=H, n_groups=G, head_size=hs, rope_n_elem=hs, scratch=scratch, status=status)
    assert status.tolist() == [0, 0, 0, 0]
    rows = qkv.view(T, G, H // G + 2, hs).float()

    def turned(x):  # [T, heads, hs]
        a, b = x[..., : hs // 2], x[..., hs // 2:]
        return x * cos[:T, None] + torch.cat((-b, a), -1) * sin[:T, None]

    q = turned(rows[:, :, :-2].reshape(T, H, hs)).bfloat16().float()
    k, v = turned(rows[:, :, -2]).bfloat16().float(), rows[:, :, -1]
    ref = torch.empty(T, H, hs, device="cuda")
    hidden = torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1)
    for h in range(H):
        s = (q[:, h].double() @ k[:, h // (H // G)].double().T) / math.sqrt(hs)
        ref[:, h] = (torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v[:, h // (H // G)].double()).float()
    # weights and outputs are rounded to bf16 (2^-9 each), and q and k to bf16 on values that may differ in the last place of fp32
    assert (y.view(T, H, hs).float() - ref).norm() / ref.norm() < 6e-3
    torch.testing.assert_close(y.view(T, H, hs).float(), ref, rtol=2e-2, atol=1e-2)
    torch.testing.assert_close(pool[slot, 0, :, :T].float(), k.transpose(0, 1), rtol=2.0 ** -7, atol=1e-3)
    assert torch.equal(pool[slot, 1, :, :T].float(), v.transpose(0, 1))
    assert torch.isnan(pool[0]).all() and torch.isnan(pool[slot, :, :, T:]).all()
