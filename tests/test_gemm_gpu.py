"""tcgen05/TMEM/TMA GEMM (prefill linears) against an fp32 PyTorch reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from mdi_llm_b200 import ops

    ops.require()
    return ops


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (128, 256, 256), (64, 6144, 4096), (200, 4096, 4096), (1000, 14336, 4096),
                                   (37, 4096, 14336), (512, 1000, 520)])
@pytest.mark.parametrize("block_n", [64, 128, 256])
def test_gemm_matches_fp32_reference(M, N, K, block_n):
    ops = _ops()
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    out = ops.gemm(a, w, block_n=block_n)
    ref = a.float() @ w.float().T
    err = (out.float() - ref).abs().max().item()
    assert err <= 0.02 * ref.abs().max().item() + 0.05, f"max err {err}"


def test_gemm_bias_and_residual_epilogue():
    ops = _ops()
    torch.manual_seed(0)
    M, N, K = 300, 2048, 1024
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    res = torch.randn(M, N, device="cuda").bfloat16()
    out = ops.gemm(a, w, bias=bias, residual=res)
    ref = (a.float() @ w.float().T + bias.float()).bfloat16().float() + res.float()
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=6e-2)


def test_gemm_throughput_smoke():
    """Not a benchmark (profiles/ has those) — just checks the kernel is in the tensor-core regime."""
    ops = _ops()
    M, N, K = 2048, 14336, 4096
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.randn(N, K, device="cuda").bfloat16()
    out = ops.gemm(a, w, block_n=256)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(10):
        ops.gemm(a, w, out=out, block_n=256)
    e1.record()
    torch.cuda.synchronize()
    tflops = 10 * 2 * M * N * K / (e0.elapsed_time(e1) * 1e-3) / 1e12
    print(f"tcgen05 gemm {M}x{N}x{K}: {tflops:.0f} TFLOP/s")
    assert tflops > 100  # CUDA-core bf16 FMA tops out far below this


@pytest.mark.parametrize("M,N,K", [(64, 14336, 4096), (300, 5632, 2048), (129, 1000, 520)])
@pytest.mark.parametrize("act", ["silu_gate", "gelu_tanh_gate"])
@pytest.mark.parametrize("block_n", [64, 128])
def test_gated_gemm_dual_accumulator(M, N, K, act, block_n):
    """act(a w1^T + b1) * (a w2^T + b2) from two TMEM accumulators in one pass."""
    ops = _ops()
    torch.manual_seed(M + N)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w1 = (torch.randn(N, K, device="cuda") * 0.03).bfloat16()
    w2 = (torch.randn(N, K, device="cuda") * 0.03).bfloat16()
    b1, b2 = torch.randn(N, device="cuda").bfloat16(), torch.randn(N, device="cuda").bfloat16()
    out = ops.gemm(a, w1, bias=b1, w2=w2, bias2=b2, act=act, block_n=block_n)
    g = (a.float() @ w1.float().T + b1.float()).bfloat16().float()
    u = (a.float() @ w2.float().T + b2.float()).bfloat16().float()
    gate = torch.nn.functional.silu(g) if act == "silu_gate" else torch.nn.functional.gelu(g, approximate="tanh")
    ref = gate.bfloat16().float() * u
    torch.testing.assert_close(out.float(), ref, rtol=3e-2, atol=8e-2)


def test_gemm_fused_hop_signal_local():
    """Epilogue stores into a raw destination pointer and the last CTA publishes flag[slot] = signal."""
    ops = _ops()
    torch.manual_seed(1)
    M, N, K = 200, 4096, 1024
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    res = torch.randn(M, N, device="cuda").bfloat16()
    dst = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    flags = torch.zeros(4, dtype=torch.int32, device="cuda")
    ctr = torch.zeros(1, dtype=torch.int32, device="cuda")
    ctx = torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
    ctx[0], ctx[3] = 2, 7  # slot 2, signal value 7
    assert ops.gemm(a, w, residual=res, out_ptr=dst.data_ptr(), signal_flag=flags.data_ptr(), done_ctr=ctr, ctx=ctx) is None
    torch.cuda.synchronize()
    assert flags.tolist() == [0, 0, 7, 0] and int(ctr) == 0
    ref = (a.float() @ w.float().T).bfloat16().float() + res.float()
    torch.testing.assert_close(dst.float(), ref, rtol=2e-2, atol=6e-2)


def _deq_rows(q8, scale_t, M):
    """e4m3 bytes + transposed block scales -> fp32."""
    K = q8.shape[1]
    return (q8.view(torch.float8_e4m3fn).float().view(M, K // 128, 128) * scale_t[:, :M].t().unsqueeze(-1)).view(M, K)


def test_quantize_rows_fp8_matches_torch():
    from mdi_llm_b200 import ops

    ops.require()
    torch.manual_seed(0)
    x = (torch.randn(70, 512, device="cuda") * 3).bfloat16()
    x[3] = 0  # an all-zero row keeps scale 1 and zeros
    q, st = ops.quantize_rows_fp8(x)
    assert q.shape == (70, 512) and st.shape == (4, 128)
    xf = x.float().view(70, 4, 128)
    scale = xf.abs().amax(-1) / 448.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    torch.testing.assert_close(st[:, :70].t(), scale, rtol=1e-6, atol=0)
    ref = (xf / scale.unsqueeze(-1)).clamp(-448, 448).to(torch.float8_e4m3fn).view(70, 512)
    assert (q.view(torch.float8_e4m3fn).float() - ref.float()).abs().max().item() <= 32.0 * 0.07  # <= 1 ulp at the top binade
    assert (q.view(torch.float8_e4m3fn).float() == ref.float()).float().mean().item() > 0.99


@pytest.mark.parametrize("M,N,K,bias,res", [(128, 128, 128, False, False), (200, 384, 512, True, True), (64, 4096, 4096, False, True),
                                             (300, 1000, 1792, True, False), (1024, 6144, 4096, False, False)])
def test_gemm_fp8_blockscaled_matches_dequantised_reference(M, N, K, bias, res):
    """tcgen05.mma kind::f8f6f4 with per-128-K block scales on both operands against the same product computed in
    fp32 from the dequantised operands (identical rounding of the inputs, only the accumulation order differs)."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    ops.require()
    torch.manual_seed(1)
    a = (torch.randn(M, K, device="cuda") * 0.7).bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    w[:, 128:256] *= 8.0 if K > 128 else 1.0  # block scales that really differ along K
    b = (torch.randn(N, device="cuda") * 0.3).bfloat16() if bias else None
    r = (torch.randn(M, N, device="cuda") * 0.5).bfloat16() if res else None
    q, s = quantize_fp8_block(w)
    a8, a_st = ops.quantize_rows_fp8(a)
    out = ops.gemm_fp8(a8, a_st, q.view(torch.uint8), s.t().contiguous(), bias=b, residual=r)
    ref = _deq_rows(a8, a_st, M) @ dequantize_fp8_block(q, s, torch.float32).t()
    if b is not None:
        ref = ref + b.float()
    ref = ref.bfloat16().float()
    if r is not None:
        ref = ref + r.float()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 0.01 * scale + 0.02, f"max err {err} (scale {scale})"
    # and it is a faithful fp8 GEMM of the ORIGINAL operands (quantisation error only)
    full = a.float() @ w.float().t() + (b.float() if b is not None else 0) + (r.float() if r is not None else 0)
    assert (out.float() - full).norm().item() <= 0.06 * full.norm().item()


@pytest.mark.parametrize("M,I,K", [(128, 64, 128), (130, 448, 512), (512, 3584, 4096)])
def test_gemm_fp8_gated_mlp_one_pass(M, I, K):
    """SwiGLU in one fp8 GEMM: fc_1 and fc_2 rows share a B tile, act(g) * u in the epilogue."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    ops.require()
    torch.manual_seed(2)
    a = (torch.randn(M, K, device="cuda") * 0.6).bfloat16()
    w1 = (torch.randn(I, K, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn(I, K, device="cuda") * 0.05).bfloat16()
    (q1, s1), (q2, s2) = quantize_fp8_block(w1), quantize_fp8_block(w2)
    a8, a_st = ops.quantize_rows_fp8(a)
    out = ops.gemm_fp8(a8, a_st, q1.view(torch.uint8), s1.t().contiguous(), w2_8=q2.view(torch.uint8), w2_scale_t=s2.t().contiguous(),
                       act="silu_gate")
    ad = _deq_rows(a8, a_st, M)
    g = (ad @ dequantize_fp8_block(q1, s1, torch.float32).t()).bfloat16().float()
    u = (ad @ dequantize_fp8_block(q2, s2, torch.float32).t()).bfloat16().float()
    ref = torch.nn.functional.silu(g).bfloat16().float() * u
    err = (out.float() - ref).abs().max().item()
    assert out.shape == (M, I) and err <= 0.02 * ref.abs().max().item() + 0.02, err


@pytest.mark.parametrize("M,N,K,bias,res", [(256, 256, 64, False, False), (256, 256, 512, False, False), (512, 768, 1024, True, True),
                                             (2048, 6144, 4096, False, False), (1000, 4096, 14336, False, True), (300, 1000, 520, True, False)])
def test_gemm_cta_pair_kernel_matches_reference(M, N, K, bias, res):
    """cta_group::2: two CTAs of a cluster share one 256 x 256 tile (each loads its A rows and half of B, the
    leader issues M = 256 MMAs, commits are multicast to the pair)."""
    import os

    if os.environ.get("MDI_TEST_PAIR", "1") == "0":
        pytest.skip("CTA-pair GEMM disabled")
    ops = _ops()
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.05).bfloat16()
    b = torch.randn(N, device="cuda").bfloat16() if bias else None
    r = torch.randn(M, N, device="cuda").bfloat16() if res else None
    out = ops.gemm(a, w, bias=b, residual=r, block_n=512)
    ref = a.float() @ w.float().T + (b.float() if bias else 0)
    ref = ref.bfloat16().float() + (r.float() if res else 0)
    err = (out.float() - ref).abs().max().item()
    assert err <= 0.02 * ref.abs().max().item() + 0.06, f"max err {err}"


@pytest.mark.parametrize("M,I,K", [(256, 128, 64), (300, 1000, 520), (2048, 14336, 4096)])
def test_gemm_cta_pair_gated_matches_reference(M, I, K):
    """Gated MLP on the CTA-pair kernel: rank 0 loads the fc_1 half of the B tile, rank 1 the fc_2 half."""
    ops = _ops()
    torch.manual_seed(M + I + K)
    a = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    w1 = (torch.randn(I, K, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn(I, K, device="cuda") * 0.05).bfloat16()
    out = ops.gemm(a, w1, w2=w2, act="silu_gate", block_n=512)
    g = (a.float() @ w1.float().T).bfloat16().float()
    u = (a.float() @ w2.float().T).bfloat16().float()
    ref = torch.nn.functional.silu(g).bfloat16().float() * u
    err = (out.float() - ref).abs().max().item()
    assert out.shape == (M, I) and err <= 0.02 * ref.abs().max().item() + 0.05, err


@pytest.mark.parametrize("M,N,K,gated", [(1, 132, 128, False), (129, 1004, 384, False), (257, 260, 1152, False), (1, 68, 128, True), (130, 132, 640, True),
                                         (70, 4096, 4096, False), (128, 4100, 5120, False), (256, 4096, 5248, False), (65, 2048, 4224, True), (40, 4096, 5120, True)])
def test_gemm_fp8_edges_of_tiles(M, N, K, gated):
    """Columns in fours that are not eights, single rows, fewer and more K blocks than there are partial accumulators, K blocks shared by
    four and by two CTAs; biases, a residual.
    Bound: every K block's sum is exact to fp32, the result is rounded to bf16 once per step of the eager order (2^-8 of its size each)."""
    from mdi_llm_b200 import ops
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    ops.require()
    torch.manual_seed(M + N + K)
    a = (torch.randn(M, K, device="cuda") * 0.7).bfloat16()
    a8, a_st = ops.quantize_rows_fp8(a)
    ad = _deq_rows(a8, a_st, M)
    ws = [(torch.randn(N, K, device="cuda") * 0.05).bfloat16() for _ in range(1 + gated)]
    bs = [(torch.randn(N, device="cuda") * 0.3).bfloat16() for _ in ws]
    qs = [quantize_fp8_block(w) for w in ws]
    lins = [(ad @ dequantize_fp8_block(q, s, torch.float32).t() + b.float()).bfloat16().float() for (q, s), b in zip(qs, bs)]
    args = (a8, a_st, qs[0][0].view(torch.uint8), qs[0][1].t().contiguous())
    if gated:
        out = ops.gemm_fp8(*args, bias=bs[0], w2_8=qs[1][0].view(torch.uint8), w2_scale_t=qs[1][1].t().contiguous(), bias2=bs[1], act="silu_gate")
        ref = torch.nn.functional.silu(lins[0]).bfloat16().float() * lins[1]
    else:
        r = (torch.randn(M, N, device="cuda") * 0.5).bfloat16()
        out = ops.gemm_fp8(*args, bias=bs[0], residual=r)
        ref = lins[0] + r.float()
    assert (out.float() - ref).abs().max().item() <= 4 * 2.0 ** -8 * ref.abs().max().item()


@pytest.mark.parametrize("M,N,K", [(1, 8, 1024), (33, 4096, 2056), (100, 4100, 4096), (128, 6144, 1032), (129, 2048, 1600), (300, 2560, 2048), (512, 2046, 1088)])
@pytest.mark.parametrize("gated", [False, True])
def test_gemm_with_a_shared_k_range(M, N, K, gated):
    """Few tiles: four and two CTAs share a tile's K range; odd columns, K blocks that do not divide, biases, a residual.  Bound: one rounding
    to bf16 per step of the eager order (2^-8 of the largest value each, the products' inputs being exact)."""
    ops = _ops()
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w, w2 = ((torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    b, b2 = (torch.randn(N, device="cuda").bfloat16() for _ in range(2))
    lin = [(a.double() @ x.double().T + y.double()).bfloat16().double() for x, y in ((w, b), (w2, b2))]
    if gated:
        out = ops.gemm(a, w, bias=b, w2=w2, bias2=b2, act="silu_gate", block_n=128)
        ref = torch.nn.functional.silu(lin[0]).bfloat16().double() * lin[1]
    else:
        r = torch.randn(M, N, device="cuda").bfloat16()
        out = ops.gemm(a, w, bias=b, residual=r, block_n=512)
        ref = lin[0] + r.double()
    assert (out.double() - ref).abs().max() <= 4 * 2.0 ** -8 * ref.abs().max()
    assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


def test_a_shared_tile_signals_its_hop():
    ops = _ops()
    torch.manual_seed(3)
    a, w = torch.randn(64, 2048, device="cuda").bfloat16(), (torch.randn(2048, 2048, device="cuda") * 0.02).bfloat16()
    dst, flags = torch.zeros(64, 2048, device="cuda", dtype=torch.bfloat16), torch.zeros(4, dtype=torch.int32, device="cuda")
    ctr, ctx = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
    ctx[0], ctx[3] = 1, 9
    assert ops.gemm(a, w, out_ptr=dst.data_ptr(), signal_flag=flags.data_ptr(), done_ctr=ctr, ctx=ctx) is None
    torch.cuda.synchronize()
    assert flags.tolist() == [0, 9, 0, 0] and int(ctr) == 0
    torch.testing.assert_close(dst.float(), a.float() @ w.float().T, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("N", [8, 24])
def test_a_shared_tile_of_few_columns_in_rows_that_start_anywhere(N):
    """Output and residual on 2-byte boundaries, which the other tiles take for fewer than 32 columns."""
    ops = _ops()
    torch.manual_seed(N)
    M, K = 130, 4104
    a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    r, out = (torch.randn(M * N + 8, device="cuda").bfloat16()[1:1 + M * N].view(M, N) for _ in range(2))
    around = out.untyped_storage().nbytes() // 2
    assert r.data_ptr() % 16 == 2 and out.data_ptr() % 16 == 2
    whole = torch.as_strided(out, (around,), (1,), 0)
    before = whole.clone()
    ops.gemm(a, w, residual=r, out=out)
    ref = (a.double() @ w.double().T).bfloat16().double() + r.double()
    assert (out.double() - ref).abs().max() <= 4 * 2.0 ** -8 * ref.abs().max()
    assert torch.equal(whole[:1], before[:1]) and torch.equal(whole[1 + M * N:], before[1 + M * N:])


def _hop_args(ops):
    flags, ctr = torch.zeros(4, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ctx = torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
    ctx[0], ctx[3] = 2, 7  # slot 2, signal value 7
    return flags, dict(signal_flag=flags.data_ptr(), done_ctr=ctr, ctx=ctx, status=torch.zeros(4, dtype=torch.int32, device="cuda"))


# sizes at which no K range is shared: short ones, and more than 64 tiles of 128 x 128
@pytest.mark.parametrize("M,N,K", [(300, 2048, 520), (70, 1000, 1016), (600, 2048, 1088), (1100, 1032, 1152)])
@pytest.mark.parametrize("block_n", [64, 128, 256, 512])
@pytest.mark.parametrize("hop", [False, True])
def test_every_width_of_tile_has_its_bias_residual_and_hop(M, N, K, block_n, hop):
    """The kernel that ``block_n`` names, with bias and residual together, into a tensor and through a hop; gated where it has no residual.
    Bounds as for the shared form."""
    ops = _ops()
    assert ops.lib().mdi_gemm_k_shares(M, N, K, 0, block_n) == ops.lib().mdi_gemm_k_shares(M, N, K, 1, block_n) == 1
    torch.manual_seed(M + N + K)
    a, r = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    w, w2 = ((torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    b, b2 = (torch.randn(N, device="cuda").bfloat16() for _ in range(2))
    lin = [(a.double() @ x.double().T + y.double()).bfloat16().double() for x, y in ((w, b), (w2, b2))]
    for args, ref in ((dict(residual=r), lin[0] + r.double()), (dict(w2=w2, bias2=b2, act="silu_gate"), torch.nn.functional.silu(lin[0]).bfloat16().double() * lin[1])):
        flags, to = _hop_args(ops)
        out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        if hop:
            assert ops.gemm(a, w, bias=b, block_n=block_n, out_ptr=out.data_ptr(), **to, **args) is None
            torch.cuda.synchronize()
            assert flags.tolist() == [0, 0, 7, 0] and int(to["done_ctr"]) == 0
        else:
            ops.gemm(a, w, bias=b, block_n=block_n, out=out, **args)
        assert (out.double() - ref).abs().max() <= 4 * 2.0 ** -8 * ref.abs().max()
        assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("M,N,K,shares", [(100, 4096, 4096, 4), (250, 4096, 5120, 2), (100, 4096, 2048, 1), (1000, 1536, 4096, 1)])
def test_fp8_products_signal_their_hop(M, N, K, shares):
    """Alone and with shared K blocks: the last CTA, of a cluster or not, releases the flag; an aborted stage poisons it."""
    ops = _ops()
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    assert ops.lib().mdi_gemm_fp8_shares(M, N, K, 0) == shares
    torch.manual_seed(M + N + K)
    a, r = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    w8, ws = quantize_fp8_block((torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16())
    a8, a_s = ops.quantize_rows_fp8(a)
    ref = (_deq_rows(a8, a_s, M).double() @ dequantize_fp8_block(w8, ws, torch.float32).double().T).bfloat16().double() + r.double()
    for aborted in (False, True):
        flags, to = _hop_args(ops)
        to["status"][1] = int(aborted)
        out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        assert ops.gemm_fp8(a8, a_s, w8, ws.t().contiguous(), residual=r, out_ptr=out.data_ptr(), **to) is None
        torch.cuda.synchronize()
        assert int(to["done_ctr"]) == 0 and flags.tolist() == [0, 0, ops.POISON if aborted else 7, 0]
        assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("M,N,K,gated,shares", [(1, 8, 2056, 0, 4), (33, 4096, 2080, 0, 4), (100, 6140, 4096, 0, 2), (128, 4100, 3208, 1, 2), (40, 1000, 1416, 1, 4),
                                                (129, 2048, 3080, 0, 4), (300, 2556, 4104, 0, 2), (512, 2046, 4168, 1, 2)])
def test_products_that_share_their_k_range(M, N, K, gated, shares):
    """As above, at sizes for which the rule chooses it: ranges that do not divide by the CTAs, a last block of eight columns, odd output columns."""
    ops = _ops()
    assert all(ops.lib().mdi_gemm_k_shares(M, N, K, gated, n) == shares for n in (128, 256, 512))
    torch.manual_seed(M + N + K)
    a, r = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    w, w2 = ((torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16() for _ in range(2))
    b, b2 = (torch.randn(N, device="cuda").bfloat16() for _ in range(2))
    lin = [(a.double() @ x.double().T + y.double()).bfloat16().double() for x, y in ((w, b), (w2, b2))]
    if gated:
        out, ref = ops.gemm(a, w, bias=b, w2=w2, bias2=b2, act="silu_gate", block_n=128), torch.nn.functional.silu(lin[0]).bfloat16().double() * lin[1]
    else:
        out, ref = ops.gemm(a, w, bias=b, residual=r, block_n=512), lin[0] + r.double()
    assert (out.double() - ref).abs().max() <= 4 * 2.0 ** -8 * ref.abs().max()
    assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()


@pytest.mark.parametrize("M,N,K,gated", [(33, 3072, 1024, 0), (512, 1024, 1024, 0), (64, 8192, 2048, 0), (200, 2048, 2048, 0), (900, 768, 3072, 1), (300, 4096, 4096, 0)])
def test_products_whose_exchange_would_cost_more_than_it_saves_stay_whole(M, N, K, gated):
    assert _ops().lib().mdi_gemm_k_shares(M, N, K, gated, 128 if M <= 128 else 512) == 1


@pytest.mark.parametrize("N", [264, 260])
@pytest.mark.parametrize("K", [256, 5120])
@pytest.mark.parametrize("biases", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("act", [None, "silu_gate", "gelu_tanh_gate", "gelu_erf_gate"])
def test_fp8_epilogues(N, K, biases, act):
    """Every branch of the epilogue: a bias of one product or of both, each activation, plain products with (second of ``biases``) and without a
    residual, columns that are eights and not, with and without shared K blocks.  Bound as above."""
    ops = _ops()
    from mdi_llm_b200.utils.quantize import dequantize_fp8_block, quantize_fp8_block

    M = 200
    assert (ops.lib().mdi_gemm_fp8_shares(M, N, K, int(act is not None)) > 1) == (K > 256)
    torch.manual_seed(N + K)
    a8, a_s = ops.quantize_rows_fp8((torch.randn(M, K, device="cuda") * 0.7).bfloat16())
    qs = [quantize_fp8_block((torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()) for _ in range(2)]
    bs = [(torch.randn(N, device="cuda") * 0.3).bfloat16() if on else None for on in biases]
    lins = [_deq_rows(a8, a_s, M).double() @ dequantize_fp8_block(q, s, torch.float32).double().T for q, s in qs]
    args = (a8, a_s, qs[0][0].view(torch.uint8), qs[0][1].t().contiguous())
    add = lambda x, b: (x if b is None else x + b.double()).bfloat16().double()  # noqa: E731
    if act is None:
        r = (torch.randn(M, N, device="cuda") * 0.5).bfloat16() if biases[1] else None
        out, ref = ops.gemm_fp8(*args, bias=bs[0], residual=r), add(lins[0], bs[0]) + (0 if r is None else r.double())
    else:
        out = ops.gemm_fp8(*args, bias=bs[0], w2_8=qs[1][0].view(torch.uint8), w2_scale_t=qs[1][1].t().contiguous(), bias2=bs[1], act=act)
        f = torch.nn.functional.silu if act == "silu_gate" else lambda x: torch.nn.functional.gelu(x, approximate="tanh" if "tanh" in act else "none")
        ref = f(add(lins[0], bs[0])).bfloat16().double() * add(lins[1], bs[1])
    assert (out.double() - ref).abs().max() <= 4 * 2.0 ** -8 * ref.abs().max()
    assert (out.double() - ref).norm() <= 2.0 ** -8 * ref.norm()
