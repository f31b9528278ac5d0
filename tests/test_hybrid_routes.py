"""Which of two kernels a call of the hybrid family takes, on sizes alone: lines drawn where the two were measured to meet."""
import pytest
import torch

from mdi_llm_b200.ops import hybrid as H


def _spans(lengths, start, window, chunk):
    spans, r, k = [], 0, 0
    for n in lengths:
        first = 0 if window <= 0 else start // window * window if chunk else max(0, start - window + 1)
        spans.append((r, n, k, start, first))
        r, k = r + n, k + start + n - first
    return spans


@pytest.mark.parametrize("lengths,start,window,chunk,DK,V,split,cap,tc", [
    ([2048], 0, 0, False, 128, 128, True, True, True),
    ([1411, 501, 136], 0, 0, False, 192, 128, False, False, True),
    ([128], 0, 0, False, 64, 64, True, True, True),
    ([300], 0, 0, False, 64, 64, True, False, True),
    ([40], 8000, 0, False, 128, 128, True, False, True),
    ([48] * 100, 3000, 0, False, 128, 128, True, False, True),
    ([1000] + [1] * 40, 1000, 0, False, 128, 128, False, False, True),
    ([33] * 40, 0, 0, False, 64, 64, True, False, False),
    ([33] * 40, 0, 0, False, 64, 64, True, True, False),
    ([33] + [1] * 40, 2000, 128, False, 64, 64, True, False, False),
    ([300] + [1] * 40, 500, 128, False, 128, 128, True, True, False),
    ([180, 17, 124, 87], 0, 0, False, 192, 64, True, True, True),
    ([208] + [1] * 17, 90, 0, False, 128, 128, True, True, True),
    ([129], 0, 128, False, 64, 64, True, True, False),
])
def test_short_prompts_take_the_kernel_that_is_faster_for_them(lengths, start, window, chunk, DK, V, split, cap, tc):
    assert H._tc_pays(_spans(lengths, start, window, chunk), min(lengths), window, chunk, DK, V, split, cap) is tc


@pytest.mark.gpu
@pytest.mark.parametrize("window,mask", [(0, "window"), (50, "window"), (64, "chunk")])
@pytest.mark.parametrize("split,cap", [(True, 0.0), (False, 0.0), (True, 20.0)])
def test_both_kernels_give_a_short_prompts_result(window, mask, split, cap, monkeypatch):
    """A step around the line, by one and by the other: both round the same weights and the result, so they differ by a rounding of each."""
    lengths, g = [33, 1, 64, 65, 128], torch.Generator(device="cuda").manual_seed(3)
    spans = _spans(lengths, 70, window, mask == "chunk")
    q = torch.randn(sum(lengths), 4 * 64, generator=g, device="cuda").bfloat16()
    kv = torch.randn(spans[-1][2] + 70 + 128 - spans[-1][4], 2 * 128, generator=g, device="cuda").bfloat16()
    out = []
    for tc in (False, True):
        monkeypatch.setattr(H, "_tc_pays", lambda *a: tc)
        out.append(H.prompt_attn(q, kv, spans, 4, 64, 64, 0.2, window, split, kv_heads=2, cap=cap, mask=mask).double())
    assert (out[0] - out[1]).norm() <= 2.0 ** -7 * out[0].norm() and not torch.equal(out[0], out[1])


@pytest.mark.parametrize("N,K,O,own", [(1, 8, 1, True), (8, 64, 4096, True), (8, 2048, 4160, True), (8, 16384, 4096, True), (8, 2048, 8192, True),
                                       (8, 2048, 32000, True), (1, 1536, 6000, True), (4, 4096, 128256, True), (8, 64, 32000, False), (1, 512, 11008, False),
                                       (8, 3072, 8192, False), (2, 14336, 8192, False), (1, 14336, 1, False), (9, 2048, 2048, False), (4, 60, 64, False)])
def test_products_of_few_rows_take_the_kernel_that_is_faster_for_them(N, K, O, own):
    assert H._few_rows_pay(N, K, O) is own
