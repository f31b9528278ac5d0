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
