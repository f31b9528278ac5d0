"""Products of up to eight rows (``csrc/hybrid_linear.cu``) and what is left to the library."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,O,bias", [(1, 8, 1, False), (8, 16, 2048, False), (3, 2056, 33, True), (5, 4104, 48, True), (8, 4096, 2368, False),
                                        (2, 64, 17, True), (7, 1536, 6000, False), (8, 8192, 16, True)])
def test_few_rows_linear(N, K, O, bias):
    """Products of up to eight rows: odd sizes, both splits, rows that are part of wider ones.  Bound: one rounding to bf16 of a fp32 sum."""
    from mdi_llm_b200.ops import hybrid as H_

    g = torch.Generator(device="cuda").manual_seed(N + K + O)
    x = torch.randn(N, K + 24, generator=g, device="cuda").bfloat16()[:, 8:8 + K]
    w = (torch.randn(O, K + 8, generator=g, device="cuda") * K ** -0.5).bfloat16()[:, :K]
    b = torch.randn(O, generator=g, device="cuda").bfloat16() if bias else None
    assert H_._few_rows(x, w, b)
    got = H_.linear(x, w, b).double()
    ref = x.double() @ w.double().T + (0 if b is None else b.double())
    assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)).all()


def test_what_few_rows_leaves_to_the_library():
    from mdi_llm_b200.ops import hybrid as H_

    x, w = torch.randn(4, 64, device="cuda").bfloat16(), torch.randn(32, 64, device="cuda").bfloat16()
    assert H_._few_rows(x, w, None)
    assert not H_._few_rows(x.repeat(3, 1), w, None) and not H_._few_rows(x.float(), w.float(), None)
    assert not H_._few_rows(x[:, 1:57], w[:, 1:57], None) and not H_._few_rows(x, w.t().contiguous().t(), None)
    wg = w.clone().requires_grad_()
    H_.linear(x, wg).sum().backward()
    assert wg.grad is not None
    torch.testing.assert_close(torch.func.vmap(lambda r: H_.linear(r[None], w)[0])(x), torch.nn.functional.linear(x, w), rtol=2e-2, atol=2e-1)
    with torch.autograd.forward_ad.dual_level():
        d = torch.autograd.forward_ad.make_dual(x, x)
        assert torch.autograd.forward_ad.unpack_dual(H_.linear(d, w)).tangent is not None
