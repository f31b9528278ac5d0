"""Decode products whose items are too few for the warps: two or four warps share an item's columns."""
from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("gated", [False, True], ids=["plain", "gated"])
@pytest.mark.parametrize("N", [1, 7, 886, 1776, 1777, 3554])
@pytest.mark.parametrize("K", [8, 1024, 1032, 2048, 3000, 4096, 5000, 9216])
def test_products(K, N, gated, variant):
    """One to nine chunks of 1024 columns in one, two or four parts (the last one shorter), rows in pairs and alone."""
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(N + K)
    W, W2 = ((torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    x, res = torch.randn(K, generator=g, device="cuda").bfloat16(), torch.randn(N, generator=g, device="cuda").bfloat16()
    ctx = torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
    y = torch.empty(N, device="cuda", dtype=torch.bfloat16)
    a = W.double() @ x.double()
    if gated:
        ops.linear_decode(W, x, y, ctx, W2=W2, act="silu_gate", variant=variant)
        ref = torch.nn.functional.silu(a) * (W2.double() @ x.double())
    else:
        ops.linear_decode(W, x, y, ctx, residual=res, variant=variant)
        ref = a + res.double()
    # fp32 sums.  bf16 keeps 8 bits, so a rounding moves a value by up to 2^-8 of it.  Plain: the product and the result are rounded.
    # Gated: both products, the activation and the result, and a rounded argument g moves SiLU by up to |1 + g (1 - sigmoid(g))| <= 6
    # times its share for |g| <= 5: (6 + 3) 2^-8.
    limit = 9 * 2.0 ** -8 * ref.norm() if gated else 2.0 ** -8 * (a.norm() + ref.norm())
    assert (y.double() - ref).norm() <= 1.01 * limit + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("residual", [False, True], ids=["plain", "residual"])
@pytest.mark.parametrize("K", [128, 4096, 6272])
@pytest.mark.parametrize("N", [5, 28416, 28419])
def test_fp8_products(N, K, residual):
    """One to four chunks of 2048 columns, one item and several to a warp, rows that fill the ring from the row count on that takes fewer CTAs."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(N + K)
    q, s = quantize_fp8_block(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5)
    x, res = torch.randn(K, generator=g, device="cuda").bfloat16(), torch.randn(N, generator=g, device="cuda").bfloat16()
    ctx = torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
    y = torch.empty(N, device="cuda", dtype=torch.bfloat16)
    ops.linear_decode(q, x, y, ctx, wscale=s, residual=res if residual else None)
    a = dequantize_fp8_block(q, s, torch.float64) @ x.double()
    ref = a + res.double() if residual else a
    # fp16 sums of eight exact products (2^-11 a step: up to 8 of them), fp32 beyond; the product and the result are rounded to bf16 (2^-8)
    assert (y.double() - ref).norm() <= 1.01 * 2.0 ** -8 * (a.norm() + ref.norm()) + 8 * 2.0 ** -11 * a.norm() + 1e-6
