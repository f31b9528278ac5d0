#!/usr/bin/env python3
"""Small deterministic workloads for ncu captures (scripts/capture_ncu.sh):
   decode: the Llama-3-8B gate/up weight-streaming kernel (+RMSNorm, SiLU*mul epilogue), 235 MB of weights
   decode_fp8: the same on block-scaled fp8 weights, 117 MB
   gemm  : the tcgen05 CTA-pair prefill GEMM 2048 x 14336 x 4096
   attn  : decode attention at 470 live positions (cluster merge), Llama-3-8B heads
   attnp : tcgen05 prefill attention, 2048-token prompt, Llama-3-8B heads
   gemm_fp8: the block-scaled fp8 GEMM (tcgen05 kind::f8f6f4) 2048 x 6144 x 4096
   gemm_shared: the GEMM of a prompt's down projection, whose tiles share their K range in clusters, 100 x 4096 x 14336
   few_rows: the product of eight rows with 2048 x 8192 weights of the hybrid family, two CTAs to a tile
   grouped: the grouped GEMM of eight experts, 1994 rows x 14336 x 4096, gated
   chunks: the three chunk kernels of the delta rule, 2048 tokens, 16 heads of 128
   capped: prompt attention of the hybrid family with capped scores, 2048 tokens, 16 heads of 128 on 4 key heads"""
import os
import sys

import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from mdi_llm_b200 import ops  # noqa: E402

what = sys.argv[1] if len(sys.argv) > 1 else "decode"
ops.require()
ctx = torch.zeros(ops.CTX_INTS, dtype=torch.int32, device="cuda")
if what == "decode":
    variant = int(sys.argv[2]) if len(sys.argv) > 2 else 2
    C, I = 4096, 14336
    Ws = [torch.randn(I, C, device="cuda", dtype=torch.bfloat16) * 0.02 for _ in range(4)]
    x = torch.randn(C, device="cuda", dtype=torch.bfloat16)
    nw = torch.ones(C, device="cuda", dtype=torch.bfloat16)
    y = torch.empty(I, device="cuda", dtype=torch.bfloat16)
    for i in range(6):
        ops.linear_decode(Ws[(2 * i) % 4], x, y, ctx, W2=Ws[(2 * i + 1) % 4], norm_w=nw, act="silu_gate", variant=variant, ctas_per_sm=3)
elif what == "decode_fp8":
    from mdi_llm_b200.utils.quantize import quantize_fp8_block

    C, I = 4096, 14336
    Ws = [quantize_fp8_block((torch.randn(I, C, device="cuda") * 0.02).bfloat16()) for _ in range(4)]
    x, nw, y = torch.randn(C, device="cuda").bfloat16(), torch.ones(C, device="cuda").bfloat16(), torch.empty(I, device="cuda").bfloat16()
    for i in range(6):
        (w1, s1), (w2, s2) = Ws[(2 * i) % 4], Ws[(2 * i + 1) % 4]
        ops.linear_decode(w1, x, y, ctx, W2=w2, norm_w=nw, act="silu_gate", wscale=s1, wscale2=s2, ctas_per_sm=3)
elif what == "gemm":
    M, N, K = 2048, 14336, 4096
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.randn(N, K, device="cuda").bfloat16()
    for _ in range(4):
        ops.gemm(a, w, block_n=512)  # the CTA-pair kernel (cta_group::2)
elif what == "gemm_shared":
    a = torch.randn(100, 14336, device="cuda").bfloat16()
    ws = [torch.randn(4096, 14336, device="cuda").bfloat16() for _ in range(2)]
    for i in range(4):
        ops.gemm(a, ws[i % 2])
elif what == "few_rows":
    from mdi_llm_b200.ops import hybrid as hy

    x, ws = torch.randn(8, 8192, device="cuda").bfloat16(), [torch.randn(2048, 8192, device="cuda").bfloat16() for _ in range(6)]
    for w in ws:
        hy.linear(x, w)
elif what == "attn":
    H, G, hs, S = 32, 8, 128, 4096
    q = torch.randn(H * hs, device="cuda").bfloat16()
    kv = torch.randn(1, 2, G, S, hs, device="cuda").bfloat16()
    y = torch.zeros(H * hs, device="cuda", dtype=torch.bfloat16)
    part = torch.zeros(H * 40 * (hs + 2), device="cuda")
    tickets = torch.zeros(G, dtype=torch.int32, device="cuda")
    ctx[1] = int(sys.argv[2]) - 1 if len(sys.argv) > 2 else 469  # live context: 470 positions -> 4 spans, cluster (DSMEM) merge
    for _ in range(4):
        ops.attn_decode(q, kv, y, part, tickets, ctx, n_head=H, n_groups=G, head_size=hs, max_seq=S, n_split=40)
elif what == "gemm_fp8":
    from mdi_llm_b200.utils.quantize import quantize_fp8_block

    M, N, K = 2048, 6144, 4096
    a = torch.randn(M, K, device="cuda").bfloat16()
    q, s = quantize_fp8_block((torch.randn(N, K, device="cuda") * 0.02).bfloat16())
    a8, a_st = ops.quantize_rows_fp8(a)
    st = s.t().contiguous()
    for _ in range(4):
        ops.gemm_fp8(a8, a_st, q.view(torch.uint8), st)
elif what == "grouped":
    counts = torch.tensor([249, 250, 249, 249, 250, 249, 249, 249], dtype=torch.int32, device="cuda")
    a = torch.randn(1994, 4096, device="cuda").bfloat16()
    w, w2 = ([torch.randn(14336, 4096, device="cuda").bfloat16() for _ in range(8)] for _ in range(2))
    for _ in range(3):
        ops.gemm_grouped(a, w, counts, w2=w2)
elif what in ("chunks", "capped"):
    from mdi_llm_b200.ops import hybrid as hy

    T, heads, dim = 2048, 16, 128
    plan = hy.BatchPlan.make([T], [0], [0], torch.device("cuda"))
    rows = lambda n: torch.randn(T, n, device="cuda").bfloat16()  # noqa: E731
    if what == "chunks":
        q, k, v, z, g = rows(8 * dim), rows(8 * dim), rows(heads * dim), rows(heads * dim), rows(heads * dim)
        state = torch.zeros(1, heads, dim, dim, device="cuda")
        for _ in range(3):
            hy.gated_recurrence(q, k, v, z, g, rows(dim)[0], state, plan, heads=heads, kv_heads=8, dim=dim, vdim=dim, mode="delta", eps=1e-5,
                                beta=rows(heads), a_log=rows(heads)[0], variant=4)
    else:
        q, cache = rows(heads * dim), torch.randn(1, T, 4 * 2 * dim, device="cuda").bfloat16()
        for _ in range(3):
            hy.prompt_attn(q, cache.view(T, -1), [(0, T, 0, 0, 0)], heads, dim, dim, dim ** -0.5, 0, True, table=hy.span_table(plan, 0, T),
                           kv_heads=4, cap=50.0, sink=torch.zeros(heads, device="cuda"))
torch.cuda.synchronize()
print("done", what)

if what == "attnp":
    from mdi_llm_b200.models.gpt import build_rope_cache

    H, G, hs, S, T = 32, 8, 128, 2048, 2048
    qkv = (torch.randn(T, (H + 2 * G) * hs, device="cuda") * 0.5).bfloat16()
    cos, sin = build_rope_cache(S, hs, device=torch.device("cuda"))
    cos, sin = cos.float().contiguous(), sin.float().contiguous()
    pool = torch.zeros(1, 2, G, S, hs, device="cuda", dtype=torch.bfloat16)
    for _ in range(4):
        ops.attn_prefill(qkv, cos, sin, pool, 0, n_head=H, n_groups=G, head_size=hs, rope_n_elem=hs)
torch.cuda.synchronize()
