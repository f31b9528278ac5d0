"""bf16 products of up to 64 rows, whose stages hold no more (the instruction reads 128): alone and with shared K ranges, from fewer K blocks than
there are stages to many, several tiles to a CTA, and the first row count of the tall stages."""
from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("gated", [False, True], ids=["plain", "gated"])
@pytest.mark.parametrize("K", [8, 320, 640, 2056, 4096])
@pytest.mark.parametrize("N", [8, 300, 2052, 19200])
@pytest.mark.parametrize("M", [1, 32, 33, 63, 64, 65])
def test_products(M, N, K, gated):
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, r = (torch.randn(M, n, generator=g, device="cuda").bfloat16() for n in (K, N))
    w, w2 = ((torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    b, b2 = (torch.randn(N, generator=g, device="cuda").bfloat16() for _ in range(2))
    lin = [a.double() @ x.double().T + y.double() for x, y in ((w, b), (w2, b2))]
    # bf16 keeps 8 bits: a rounding moves a value by up to 2^-8 of it.  Plain: the product and the sum are rounded.  Gated: both products, the
    # activation and the result, and a rounded argument g moves SiLU by up to |1 + g (1 - sigmoid(g))| <= 8 times its share for |g| <= 7: (8 + 3) 2^-8.
    if gated:
        y, ref = ops.gemm(a, w, bias=b, w2=w2, bias2=b2, act="silu_gate", block_n=128), torch.nn.functional.silu(lin[0]) * lin[1]
        limit = 11 * 2.0 ** -8 * ref.norm()
    else:
        y, ref = ops.gemm(a, w, bias=b, residual=r, block_n=128), lin[0] + r.double()
        limit = 2.0 ** -8 * (lin[0].norm() + ref.norm())
    assert (y.double() - ref).norm() <= 1.01 * limit
