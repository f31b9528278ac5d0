"""The product of every group of rows with its own weight: rows a group around the steps of the tile width, more groups than a launch takes,
output columns that end inside a tile, rows of another group that are not finite."""
from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [(31, 32, 33, 0, 64, 65, 160, 161), (255, 256, 257, 511, 512, 513, 1, 2049), (40,) * 17, (0, 0, 7), (3000,)])
@pytest.mark.parametrize("N,K,gated", [(127, 64, True), (129, 200, True), (1025, 1000, True), (255, 64, False), (257, 200, False), (2049, 1000, False)])
def test_groups(counts, N, K, gated):
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(N + K + len(counts))
    M, E = sum(counts), len(counts)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    last = sum(counts[:-1])
    a[last] = float("nan")  # the first row of the last group: it reaches no other row
    w, w2 = ([(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(E)] for _ in range(2))
    y = ops.gemm_grouped(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), w2=w2 if gated else None).double()
    assert y[last].isnan().all()
    at = 0
    for e, n in enumerate(counts):
        rows = [i for i in range(at, at + n) if i != last]
        at += n
        if not rows:
            continue
        ref = a[rows].double() @ w[e].double().T
        if gated:
            ref = torch.nn.functional.silu(ref) * (a[rows].double() @ w2[e].double().T)
        # bf16 keeps 8 bits: a rounding moves a value by up to 2^-8 of it.  Plain: the result is rounded.  Gated: both products, the activation
        # and the result, and a rounded argument g moves SiLU by up to |1 + g (1 - sigmoid(g))| <= 6 times its share for |g| <= 5: (6 + 3) 2^-8.
        # The fp32 sums of 1000 terms add less than 2^-10 of the product's norm.
        limit = (9 if gated else 1) * 2.0 ** -8 * ref.norm() + 2.0 ** -10 * ref.norm()
        assert (y[rows] - ref).norm() <= limit


@pytest.mark.gpu
@pytest.mark.parametrize("act", ["silu_gate", "gelu_tanh_gate", "gelu_erf_gate"])
def test_activations(act):
    """Each of the three stands in a loop of its own."""
    from mdi_llm_b200 import ops

    ops.require()
    g = torch.Generator(device="cuda").manual_seed(5)
    counts, N, K = (5, 70, 33), 130, 72
    a = torch.randn(sum(counts), K, generator=g, device="cuda").bfloat16()
    w, w2 = ([(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in counts] for _ in range(2))
    y = ops.gemm_grouped(a, w, torch.tensor(counts, dtype=torch.int32, device="cuda"), w2=w2, act=act).double()
    f = torch.nn.functional.silu if act == "silu_gate" else lambda x: torch.nn.functional.gelu(x, approximate="tanh" if "tanh" in act else "none")
    ref = torch.cat([f(x.double() @ u.double().T) * (x.double() @ v.double().T) for x, u, v in zip(a.split(counts), w, w2)])
    # four roundings to bf16 and what the first does to the activation's argument, as above (the slope of GELU is smaller than SiLU's share)
    assert (y - ref).norm() <= 9 * 2.0 ** -8 * ref.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,gated", [(129, 200, True), (257, 200, False)])
def test_every_width(N, K, gated):
    """Tiles of 32 to 256 columns, whose rows come in one box or two; the one of 224 loads rows of the next group, one of them not finite."""
    test_groups((3, 40, 70, 100, 130, 170, 250, 200, 9), N, K, gated)
