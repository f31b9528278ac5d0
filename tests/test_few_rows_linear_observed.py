"""What records or rewrites calls keeps the library's product: a kernel launched past the dispatcher would be missing in it."""
import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from mdi_llm_b200.ops import hybrid as H


class _Dispatch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Function(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_calls_that_are_recorded_or_rewritten_are_noticed():
    seen = []

    def call(x):
        seen.append(H._observed())
        return x * 2

    x = torch.ones(3)
    call(x)
    with torch.device("cpu"):  # a default device only says where new tensors go
        call(x)
    assert seen == [False, False]
    seen.clear()
    torch.jit.trace(call, x, check_trace=False)
    make_fx(call)(x)
    torch.func.vmap(call)(x)
    torch.func.jvp(call, (x,), (x,))
    with _Dispatch():
        call(x)
    with _Function():
        call(x)
    with torch.autograd.forward_ad.dual_level():
        call(x)
    assert seen and all(seen) and not H._observed()


@pytest.mark.gpu
def test_a_trace_of_a_product_of_few_rows_computes_it():
    w = torch.randn(32, 64, device="cuda").bfloat16()
    x, y = (torch.randn(4, 64, device="cuda").bfloat16() for _ in range(2))
    want = torch.nn.functional.linear(y, w)
    assert torch.equal(torch.jit.trace(lambda v: H.linear(v, w), x, check_trace=False)(y), want)
    assert torch.equal(make_fx(lambda v: H.linear(v, w))(x)(y), want)
    counted = []

    class Count(_Dispatch):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            counted.append(func)
            return func(*args, **(kwargs or {}))

    with Count():
        assert torch.equal(H.linear(y, w), want)
    assert any("mm" in str(f) or "linear" in str(f) for f in counted)
    assert H._few_rows(x, w, None) and not H._few_rows(x, w.to_sparse(), None)
