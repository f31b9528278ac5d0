// Causal flash attention for the prefill (T > 1) on the 5th-generation tensor cores, sm_100a.
//
// Reference behaviour being replaced, at prefill: view/permute/split of the fused QKV
// output, RoPE as ~8 elementwise launches, index_copy_ into a cache expanded to n_head heads, then
// F.scaled_dot_product_attention with an explicit mask (model.py:693-751).  Here:
//
//   rope_split_kernel     one pass over the QKV GEMM's output [T, (H+2G)*hs]: RoPE on q and k, q written
//                         head-major for TMA, k/v appended to the slot KV pool (G group heads only) and v
//                         additionally transposed to [G, hs, T] so that P.V sees a K-major B operand;
//   attn_prefill_tcgen05  grid (T/128 query tiles, H heads).  Per 128-key tile:
//                         S = Q K^T      tcgen05.mma, operands staged by TMA (SWIZZLE_128B), S in TMEM
//                         softmax        4 warps, one query row per thread: tcgen05.ld, scale, causal
//                                        mask, online max/sum in registers, P (bf16) written to shared
//                                        memory in the same swizzled K-major layout TMA would produce
//                         O_t = P V      tcgen05.mma into a second TMEM region, added to the register
//                                        accumulator (already rescaled by exp2(m_old - m_new))
//                         one elected thread issues every TMA and MMA; mbarriers carry all hand-offs.
//
// GQA: the q heads of a group read the same K / V^T tiles (L2 hits after the first head).
#include "tcgen05.cuh"

namespace mdi {

constexpr int PA_BM = 128;       // query rows per CTA  (= TMEM lanes)
constexpr int PA_BN = 128;       // keys per tile
constexpr int PA_THREADS = 192;  // warps 0-3 softmax / epilogue, warp 4 TMA + MMA issue, warp 5 TMEM alloc

struct PrefillAttnParams {
  CUtensorMap map_q;   // [H * T_pad, hs]
  CUtensorMap map_k;   // this layer's KV pool viewed as [n_slots * 2 * G * S, hs]
  CUtensorMap map_vt;  // [G * hs, T_pad]
  bf16* y;             // [T, H * hs]
  int T, T_pad, n_head, q_per_kv, n_groups, max_seq, slot;
  float scale_log2;    // (1 / sqrt(hs)) * log2(e)
  int* status;         // the stage's status words (common.cuh), may be null: [0] |= 8, [1] = 1 when a wait ran out
};

// ---- RoPE + split ------------------------------------------------------------------------------------
struct RopeSplitArgs {
  const bf16* qkv;   // [T, (H + 2G) * hs], litGPT group-interleaved columns
  const float* cos;  // [S, ne]
  const float* sin;
  bf16* q_out;       // [H, T_pad, hs]
  bf16* kv;          // layer pool [n_slots, 2, G, S, hs]
  bf16* vt;          // [G, hs, T_pad]
  int T, T_pad, slot, n_head, n_groups, hs, ne, max_seq;
};

// grid (T_pad / 16, G * ceil((H/G + 2) / RS_SLOTS)): 16 tokens for up to three head slots (q heads, k head or v head) of a group.
// A thread owns 8 consecutive dims of one token: 16-byte loads / stores everywhere, the slots' loads together, and one read
// of its 64 bytes of cosines and sines for all of them (with a block per slot the tables were four times the traffic of the
// data: 35 us at 4096 tokens, 48 slots of 128, now 27).  V is additionally transposed through shared memory so that V^T
// rows are written 16 tokens (32 B) at a time; rows behind T become zeros.
constexpr int RS_TOK = 16, RS_SLOTS = 3;
__global__ void __launch_bounds__(256) rope_split_kernel(const RopeSplitArgs a) {
  __shared__ __align__(16) bf16 vt_tile[128][RS_TOK];
  const int hs = a.hs, ne = a.ne, half_ne = ne / 2;
  const int chunks = hs / 8;                       // 8-dim chunks per head (8 or 16)
  const int tt = threadIdx.x / chunks, ch = threadIdx.x % chunks;
  const int t = blockIdx.x * RS_TOK + tt;
  const int qpk = a.n_head / a.n_groups, per = (qpk + 2 + RS_SLOTS - 1) / RS_SLOTS;
  const int g = blockIdx.y / per, sl0 = (blockIdx.y % per) * RS_SLOTS;
  const bool active = tt < RS_TOK && t < a.T;
  const int d0 = ch * 8;
  const bool rot = d0 < ne, lo = d0 < half_ne;
  uint4 xv[RS_SLOTS], pv[RS_SLOTS];
  float cs[8], sn[8];
  const bf16* row = a.qkv + ((size_t)t * (a.n_head + 2 * a.n_groups) + g * (qpk + 2)) * hs;
#pragma unroll
  for (int i = 0; i < RS_SLOTS; ++i) {
    const int sl = sl0 + i;
    xv[i] = pv[i] = make_uint4(0, 0, 0, 0);
    if (active && sl < qpk + 2) {
      xv[i] = *reinterpret_cast<const uint4*>(row + (size_t)sl * hs + d0);
      if (sl <= qpk && rot) pv[i] = *reinterpret_cast<const uint4*>(row + (size_t)sl * hs + (lo ? d0 + half_ne : d0 - half_ne));
    }
  }
  if (active && rot && sl0 <= qpk) {
    const float* c = a.cos + (size_t)t * ne + d0;
    const float* s = a.sin + (size_t)t * ne + d0;
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
      *reinterpret_cast<float4*>(cs + e) = *reinterpret_cast<const float4*>(c + e);
      *reinterpret_cast<float4*>(sn + e) = *reinterpret_cast<const float4*>(s + e);
    }
  }
#pragma unroll
  for (int i = 0; i < RS_SLOTS; ++i) {
    const int sl = sl0 + i;
    if (sl >= qpk + 2) break;  // the same for the whole block
    uint4 out = xv[i];
    if (active) {
      if (sl <= qpk && rot) {  // q and k heads: NeoX half rotation on the first `ne` dims (model.py:881-891)
        const uint32_t xw[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w}, pw[4] = {pv[i].x, pv[i].y, pv[i].z, pv[i].w};
        uint32_t ow[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float x0 = bf16lo(xw[q]), x1 = bf16hi(xw[q]);
          const float r0 = lo ? -bf16lo(pw[q]) : bf16lo(pw[q]), r1 = lo ? -bf16hi(pw[q]) : bf16hi(pw[q]);
          ow[q] = pack_bf16x2(fmaf(x0, cs[2 * q], r0 * sn[2 * q]), fmaf(x1, cs[2 * q + 1], r1 * sn[2 * q + 1]));
        }
        out = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
      if (sl < qpk) {
        *reinterpret_cast<uint4*>(a.q_out + ((size_t)(g * qpk + sl) * a.T_pad + t) * hs + d0) = out;
      } else {
        const size_t which = (sl == qpk) ? 0 : 1;
        *reinterpret_cast<uint4*>(a.kv + ((((size_t)a.slot * 2 + which) * a.n_groups + g) * a.max_seq + t) * hs + d0) = out;
      }
    }
    if (sl != qpk + 1) continue;  // only the V slot transposes (the last slot of its block)
    if (tt < RS_TOK) {
      const uint32_t w[4] = {out.x, out.y, out.z, out.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        vt_tile[d0 + 2 * q][tt] = __ushort_as_bfloat16((unsigned short)(w[q] & 0xffffu));
        vt_tile[d0 + 2 * q + 1][tt] = __ushort_as_bfloat16((unsigned short)(w[q] >> 16));
      }
    }
    __syncthreads();
    const int d = threadIdx.x / 2, part = threadIdx.x % 2;  // two threads per V^T row, 8 tokens (16 B) each
    if (d < hs)
      *reinterpret_cast<uint4*>(a.vt + ((size_t)g * hs + d) * a.T_pad + blockIdx.x * RS_TOK + part * 8) =
          *reinterpret_cast<const uint4*>(&vt_tile[d][part * 8]);
  }
}

// ---- attention -----------------------------------------------------------------------------------------
template <int HS>
__global__ void __launch_bounds__(PA_THREADS, 1) attn_prefill_tcgen05_kernel(const __grid_constant__ PrefillAttnParams p) {
  extern __shared__ __align__(1024) unsigned char pa_smem[];
  constexpr int KA = HS / 64;                  // 64-column swizzle atoms along the head dimension
  constexpr int ROW_ATOM = 128 * 128;          // bytes of one [128 rows x 128 B] atom
  constexpr int Q_BYTES = KA * ROW_ATOM;
  constexpr int K_BYTES = KA * ROW_ATOM;
  constexpr int VT_ATOM = HS * 128;            // [HS rows x 64 keys]
  constexpr int VT_BYTES = 2 * VT_ATOM;
  constexpr int P_BYTES = 2 * ROW_ATOM;
  constexpr int TMEM_COLS = 256;               // S: columns [0,128), O_t: [128, 128 + HS)
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pa_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* q_s = base;
  unsigned char* k_s = q_s + Q_BYTES;
  unsigned char* vt_s = k_s + K_BYTES;
  unsigned char* p_s = vt_s + VT_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_s + P_BYTES);
  uint64_t *q_full = bars, *kv_full = bars + 1, *s_full = bars + 2, *p_ready = bars + 3, *o_full = bars + 4, *o_done = bars + 5;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 6);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tile = blockIdx.x, h = blockIdx.y, g = h / p.q_per_kv;
  const int m0 = m_tile * PA_BM;
  const int n_tiles = m_tile + 1;  // causal: keys [0, m0 + 128)

  if (warp == 4 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_vt) : "memory");
    mbar_init(q_full, 1); mbar_init(kv_full, 1); mbar_init(s_full, 1); mbar_init(o_full, 1);
    mbar_init(p_ready, 128); mbar_init(o_done, 128);
    mbar_fence_init();
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_s = *tmem_ptr_smem, tmem_o = tmem_s + 128;

  if (warp == 4) {
    if (lane == 0) {
      // ===== TMA + MMA issue =====
      const uint32_t idesc_s = umma_idesc_bf16(PA_BM, PA_BN), idesc_o = umma_idesc_bf16(PA_BM, HS);
      const int q_row0 = h * p.T_pad + m0;
      const int k_row0 = ((p.slot * 2 + 0) * p.n_groups + g) * p.max_seq;
      mbar_expect_tx(q_full, Q_BYTES);
#pragma unroll
      for (int a = 0; a < KA; ++a) tma_load_2d(q_s + a * ROW_ATOM, &p.map_q, q_full, a * 64, q_row0);
      for (int t = 0; t < n_tiles; ++t) {
        const int j0 = t * PA_BN;
        if (t > 0) mbar_wait(o_full, (t - 1) & 1);  // previous P.V retired: K, V^T and P buffers are free
        mbar_expect_tx(kv_full, K_BYTES + VT_BYTES);
#pragma unroll
        for (int a = 0; a < KA; ++a) tma_load_2d(k_s + a * ROW_ATOM, &p.map_k, kv_full, a * 64, k_row0 + j0);
#pragma unroll
        for (int a = 0; a < 2; ++a) tma_load_2d(vt_s + a * VT_ATOM, &p.map_vt, kv_full, j0 + a * 64, g * HS);
        if (t == 0) mbar_wait(q_full, 0);
        mbar_wait(kv_full, t & 1);
        tcgen05_fence_after();
        // S = Q K^T : K dimension = head size
#pragma unroll
        for (int k = 0; k < HS / 16; ++k) {
          const uint32_t off = (uint32_t)(k / 4) * ROW_ATOM + (uint32_t)(k % 4) * 32;
          tcgen05_mma_f16(tmem_s, umma_desc_sw128(smem_u32(q_s) + off), umma_desc_sw128(smem_u32(k_s) + off), idesc_s, k ? 1u : 0u);
        }
        tcgen05_commit(s_full);
        mbar_wait(p_ready, t & 1);                  // P is in shared memory, S has been read
        if (t > 0) mbar_wait(o_done, (t - 1) & 1);  // previous O_t has been read out of TMEM
        tcgen05_fence_after();
        // O_t = P V : K dimension = the 128 keys of this tile
#pragma unroll
        for (int k = 0; k < PA_BN / 16; ++k) {
          const uint32_t offp = (uint32_t)(k / 4) * ROW_ATOM + (uint32_t)(k % 4) * 32;
          const uint32_t offv = (uint32_t)(k / 4) * VT_ATOM + (uint32_t)(k % 4) * 32;
          tcgen05_mma_f16(tmem_o, umma_desc_sw128(smem_u32(p_s) + offp), umma_desc_sw128(smem_u32(vt_s) + offv), idesc_o, k ? 1u : 0u);
        }
        tcgen05_commit(o_full);
      }
    }
  } else if (warp < 4) {
    // ===== softmax + output: thread <-> query row <-> TMEM lane =====
    const int r = threadIdx.x;
    const int q_idx = m0 + r;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    float O[HS];
#pragma unroll
    for (int d = 0; d < HS; ++d) O[d] = 0.f;
    float m_run = -INFINITY, l_run = 0.f;
    for (int t = 0; t < n_tiles; ++t) {
      const int j0 = t * PA_BN;
      mbar_wait(s_full, t & 1);
      tcgen05_fence_after();
      // pass 1: row maximum of the masked, scaled scores
      float mx = -INFINITY;
#pragma unroll 1
      for (int c = 0; c < PA_BN / 32; ++c) {
        uint32_t sv[32];
        tmem_ld_32x32(tmem_s + lane_off + (uint32_t)(c * 32), sv);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int j = j0 + c * 32 + i;
          if (j <= q_idx && j < p.T) mx = fmaxf(mx, __uint_as_float(sv[i]) * p.scale_log2);
        }
      }
      const float m_new = fmaxf(m_run, mx);
      const float corr = (m_run == -INFINITY) ? 0.f : exp2f(m_run - m_new);
      // pass 2: probabilities -> bf16 -> swizzled K-major tile in shared memory
      float psum = 0.f;
#pragma unroll 1
      for (int c = 0; c < PA_BN / 32; ++c) {
        uint32_t sv[32];
        tmem_ld_32x32(tmem_s + lane_off + (uint32_t)(c * 32), sv);
        float pf[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int j = j0 + c * 32 + i;
          const float pv = (j <= q_idx && j < p.T && m_new != -INFINITY) ? exp2f(__uint_as_float(sv[i]) * p.scale_log2 - m_new) : 0.f;
          pf[i] = pv;
          psum += pv;
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {  // 4 x 16 B = keys [c*32 + 8v, c*32 + 8v + 8)
          const int key = c * 32 + v * 8;
          const int atom = key >> 6, chunk = (key & 63) >> 3;
          uint4 o;
          o.x = pack_bf16x2(pf[v * 8 + 0], pf[v * 8 + 1]); o.y = pack_bf16x2(pf[v * 8 + 2], pf[v * 8 + 3]);
          o.z = pack_bf16x2(pf[v * 8 + 4], pf[v * 8 + 5]); o.w = pack_bf16x2(pf[v * 8 + 6], pf[v * 8 + 7]);
          *reinterpret_cast<uint4*>(p_s + atom * ROW_ATOM + r * 128 + ((chunk ^ (r & 7)) << 4)) = o;
        }
      }
      l_run = l_run * corr + psum;
      m_run = m_new;
#pragma unroll
      for (int d = 0; d < HS; ++d) O[d] *= corr;
      fence_proxy_async_smem();  // P stores (generic proxy) -> visible to the MMA's operand reads (async proxy)
      tcgen05_fence_before();
      mbar_arrive(p_ready);
      mbar_wait(o_full, t & 1);
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < HS / 32; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32(tmem_o + lane_off + (uint32_t)(c * 32), ov);
#pragma unroll
        for (int i = 0; i < 32; ++i) O[c * 32 + i] += __uint_as_float(ov[i]);
      }
      tcgen05_fence_before();
      mbar_arrive(o_done);
    }
    if (q_idx < p.T) {
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      bf16* dst = p.y + (size_t)q_idx * p.n_head * HS + (size_t)h * HS;
#pragma unroll
      for (int v = 0; v < HS / 8; ++v) {
        uint4 o;
        o.x = pack_bf16x2(O[v * 8 + 0] * inv, O[v * 8 + 1] * inv); o.y = pack_bf16x2(O[v * 8 + 2] * inv, O[v * 8 + 3] * inv);
        o.z = pack_bf16x2(O[v * 8 + 4] * inv, O[v * 8 + 5] * inv); o.w = pack_bf16x2(O[v * 8 + 6] * inv, O[v * 8 + 7] * inv);
        *reinterpret_cast<uint4*>(dst + v * 8) = o;
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 5) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_s), "n"(TMEM_COLS) : "memory");
  }
}

// ---- pipelined variant ------------------------------------------------------------------------------------
// Same math, deeper overlap: K / V^T tiles are double-buffered in shared memory (the TMA of tile t+2 is in
// flight while tile t+1 is being used) and the score matrix is double-buffered in TMEM (S[t+1] = Q K^T is
// computed by the tensor cores WHILE the softmax warps work on S[t]).  Per tile only the softmax, the
// P.V MMA and the O_t read-out remain on the serial chain.
template <int HS>
__global__ void __launch_bounds__(PA_THREADS, 1) attn_prefill_tcgen05_pipe_kernel(const __grid_constant__ PrefillAttnParams p) {
  extern __shared__ __align__(1024) unsigned char pa_smem[];
  constexpr int KA = HS / 64;
  constexpr int ROW_ATOM = 128 * 128;
  constexpr int Q_BYTES = KA * ROW_ATOM;
  constexpr int K_BYTES = KA * ROW_ATOM;
  constexpr int VT_ATOM = HS * 128;
  constexpr int VT_BYTES = 2 * VT_ATOM;
  constexpr int P_BYTES = 2 * ROW_ATOM;
  constexpr int TMEM_COLS = 512;  // S0: [0,128)  S1: [128,256)  O_t: [256, 256 + HS)
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pa_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* q_s = base;
  unsigned char* k_s = q_s + Q_BYTES;            // [2][K_BYTES]
  unsigned char* vt_s = k_s + 2 * K_BYTES;       // [2][VT_BYTES]
  unsigned char* p_s = vt_s + 2 * VT_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(p_s + P_BYTES);
  uint64_t *q_full = bars, *kv_full = bars + 1 /* [2] */, *s_full = bars + 3 /* [2] */, *p_ready = bars + 5,
           *o_full = bars + 6, *o_done = bars + 7;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tile = blockIdx.x, h = blockIdx.y, g = h / p.q_per_kv;
  const int m0 = m_tile * PA_BM;
  const int n_tiles = m_tile + 1;

  if (warp == 4 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_vt) : "memory");
    mbar_init(q_full, 1); mbar_init(o_full, 1);
    for (int b = 0; b < 2; ++b) { mbar_init(&kv_full[b], 1); mbar_init(&s_full[b], 1); }
    mbar_init(p_ready, 128); mbar_init(o_done, 128);
    mbar_fence_init();
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem, tmem_o = tmem_base + 256;

  if (warp == 4) {
    if (lane == 0) {
      const uint32_t idesc_s = umma_idesc_bf16(PA_BM, PA_BN), idesc_o = umma_idesc_bf16(PA_BM, HS);
      const int q_row0 = h * p.T_pad + m0;
      const int k_row0 = ((p.slot * 2 + 0) * p.n_groups + g) * p.max_seq;
      auto load_tile = [&](int t) {  // K and V^T of key tile t into buffer t & 1
        const int b = t & 1, j0 = t * PA_BN;
        mbar_expect_tx(&kv_full[b], K_BYTES + VT_BYTES);
#pragma unroll
        for (int a = 0; a < KA; ++a) tma_load_2d(k_s + b * K_BYTES + a * ROW_ATOM, &p.map_k, &kv_full[b], a * 64, k_row0 + j0);
#pragma unroll
        for (int a = 0; a < 2; ++a) tma_load_2d(vt_s + b * VT_BYTES + a * VT_ATOM, &p.map_vt, &kv_full[b], j0 + a * 64, g * HS);
      };
      auto mma_s = [&](int t) {  // S[t & 1] = Q K_t^T
        const int b = t & 1;
        mbar_wait(&kv_full[b], (t >> 1) & 1);
        tcgen05_fence_after();
#pragma unroll
        for (int k = 0; k < HS / 16; ++k) {
          const uint32_t off = (uint32_t)(k / 4) * ROW_ATOM + (uint32_t)(k % 4) * 32;
          tcgen05_mma_f16(tmem_base + (uint32_t)(b * 128), umma_desc_sw128(smem_u32(q_s) + off),
                          umma_desc_sw128(smem_u32(k_s + b * K_BYTES) + off), idesc_s, k ? 1u : 0u);
        }
        tcgen05_commit(&s_full[b]);
      };
      mbar_expect_tx(q_full, Q_BYTES);
#pragma unroll
      for (int a = 0; a < KA; ++a) tma_load_2d(q_s + a * ROW_ATOM, &p.map_q, q_full, a * 64, q_row0);
      load_tile(0);
      if (n_tiles > 1) load_tile(1);
      mbar_wait(q_full, 0);
      mma_s(0);
      for (int t = 0; t < n_tiles; ++t) {
        const int b = t & 1;
        // (A) scores of the NEXT tile while the softmax warps are busy with this one.  S[(t+1)&1] is free:
        //     its previous reader (softmax of tile t-1) arrived on p_ready(t-1), waited for in (B) below.
        if (t + 1 < n_tiles) mma_s(t + 1);
        // (B) O_t = P V_t
        mbar_wait(p_ready, t & 1);
        if (t > 0) mbar_wait(o_done, (t - 1) & 1);
        tcgen05_fence_after();
#pragma unroll
        for (int k = 0; k < PA_BN / 16; ++k) {
          const uint32_t offp = (uint32_t)(k / 4) * ROW_ATOM + (uint32_t)(k % 4) * 32;
          const uint32_t offv = (uint32_t)(k / 4) * VT_ATOM + (uint32_t)(k % 4) * 32;
          tcgen05_mma_f16(tmem_o, umma_desc_sw128(smem_u32(p_s) + offp), umma_desc_sw128(smem_u32(vt_s + b * VT_BYTES) + offv),
                          idesc_o, k ? 1u : 0u);
        }
        tcgen05_commit(o_full);
        // (C) buffer b is free once P V_t has retired (K_t was consumed by S[t] long ago): fetch tile t + 2
        if (t + 2 < n_tiles) {
          mbar_wait(o_full, t & 1);
          load_tile(t + 2);
        }
      }
    }
  } else if (warp < 4) {
    const int r = threadIdx.x;
    const int q_idx = m0 + r;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    float O[HS];
#pragma unroll
    for (int d = 0; d < HS; ++d) O[d] = 0.f;
    float m_run = -INFINITY, l_run = 0.f;
    for (int t = 0; t < n_tiles; ++t) {
      const int j0 = t * PA_BN;
      const uint32_t tmem_s = tmem_base + (uint32_t)((t & 1) * 128) + lane_off;
      mbar_wait(&s_full[t & 1], (t >> 1) & 1);
      tcgen05_fence_after();
      // only the diagonal tile (and a ragged last one) needs the causal / length mask; four independent
      // max / sum chains keep the single warp per scheduler from serialising on FP latency
      const bool full = (j0 + PA_BN - 1 <= m0) && (j0 + PA_BN <= p.T);
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int c = 0; c < PA_BN / 32; ++c) {
        uint32_t sv[32];
        tmem_ld_32x32(tmem_s + (uint32_t)(c * 32), sv);
        if (full) {
#pragma unroll
          for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int j = j0 + c * 32 + i;
            if (j <= q_idx && j < p.T) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
          }
        }
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;  // scale > 0: max commutes
      const float m_new = fmaxf(m_run, mx);
      const float corr = (m_run == -INFINITY) ? 0.f : exp2f(m_run - m_new);
      float ps4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int c = 0; c < PA_BN / 32; ++c) {
        uint32_t sv[32];
        tmem_ld_32x32(tmem_s + (uint32_t)(c * 32), sv);
        float pf[32];
        if (full) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            pf[i] = exp2f(fmaf(__uint_as_float(sv[i]), p.scale_log2, -m_new));
            ps4[i & 3] += pf[i];
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int j = j0 + c * 32 + i;
            pf[i] = (j <= q_idx && j < p.T && m_new != -INFINITY) ? exp2f(fmaf(__uint_as_float(sv[i]), p.scale_log2, -m_new)) : 0.f;
            ps4[i & 3] += pf[i];
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int key = c * 32 + v * 8;
          const int atom = key >> 6, chunk = (key & 63) >> 3;
          uint4 o;
          o.x = pack_bf16x2(pf[v * 8 + 0], pf[v * 8 + 1]); o.y = pack_bf16x2(pf[v * 8 + 2], pf[v * 8 + 3]);
          o.z = pack_bf16x2(pf[v * 8 + 4], pf[v * 8 + 5]); o.w = pack_bf16x2(pf[v * 8 + 6], pf[v * 8 + 7]);
          *reinterpret_cast<uint4*>(p_s + atom * ROW_ATOM + r * 128 + ((chunk ^ (r & 7)) << 4)) = o;
        }
      }
      l_run = l_run * corr + ((ps4[0] + ps4[1]) + (ps4[2] + ps4[3]));
      m_run = m_new;
#pragma unroll
      for (int d = 0; d < HS; ++d) O[d] *= corr;
      fence_proxy_async_smem();
      tcgen05_fence_before();
      mbar_arrive(p_ready);
      mbar_wait(o_full, t & 1);  // also guarantees P is free before the next tile's softmax overwrites it
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < HS / 32; ++c) {
        uint32_t ov[32];
        tmem_ld_32x32(tmem_o + lane_off + (uint32_t)(c * 32), ov);
#pragma unroll
        for (int i = 0; i < 32; ++i) O[c * 32 + i] += __uint_as_float(ov[i]);
      }
      tcgen05_fence_before();
      mbar_arrive(o_done);
    }
    if (q_idx < p.T) {
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      bf16* dst = p.y + (size_t)q_idx * p.n_head * HS + (size_t)h * HS;
#pragma unroll
      for (int v = 0; v < HS / 8; ++v) {
        uint4 o;
        o.x = pack_bf16x2(O[v * 8 + 0] * inv, O[v * 8 + 1] * inv); o.y = pack_bf16x2(O[v * 8 + 2] * inv, O[v * 8 + 3] * inv);
        o.z = pack_bf16x2(O[v * 8 + 4] * inv, O[v * 8 + 5] * inv); o.w = pack_bf16x2(O[v * 8 + 6] * inv, O[v * 8 + 7] * inv);
        *reinterpret_cast<uint4*>(dst + v * 8) = o;
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 5) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
}

// ---- two query tiles in ping-pong, output in TMEM (mode 2, the default) ------------------------------------
// A CTA owns 256 query rows of one head as two tiles A and B that share every K / V^T tile.  While the softmax warps of A
// work on S_A(t), the tensor core runs P_B V(t-1) and S_B(t), and the other way round, so that the exponentials hide behind the
// products instead of standing in line with them:
//
//   warps 0-3 / 4-7  softmax of tile A / B: a thread holds a whole row of scores in registers (one TMEM read), writes the row
//                    of P (bf16) over the first 64 columns of its scores, half by half, and adds up the row sum.  When a row's
//                    maximum moves, the warp rescales its rows of O in TMEM (O is stable: s_full(t) is committed behind
//                    P V(t-1)).  Moving it only by large steps saves 10 % at 4096 tokens, but then the largest weight of a row is
//                    no longer exactly one and is rounded like the others: 1 % more error against float64, not taken.
//   warps 8 / 10     one thread each issues the MMAs of A / B (one thread for both would keep A waiting for B's exponentials); both
//                    operands of S from shared memory, P as the A operand of P V from TMEM
//   warp 9           one thread issues the TMA loads, two stages each of K and V^T
//
// TMEM: S_A / P_A [0,128)  S_B / P_B [128,256)  O_A [256, 256 + HS)  O_B [384, 384 + HS).
// The MMAs of one thread run in the order they are issued: S(t+1) may follow P V(t) that reads P from the same columns.
// What bounds it: a step of two tiles takes 4100 cycles, 2600 of them products (a 128 x 128 x 16 MMA takes 93 cycles with both
// operands in shared memory, 69 with one in TMEM) and 2048 exponentials (16 a cycle), which overlap by half; three eighths of the
// exponentials on the FMA units changed nothing.  Blocks start with the longest rows: the last ones of a causal grid are
// then the short ones.  A grid of pairs that does not fill the SMs (`single`) is cut into CTAs of one tile.
constexpr int PP_THREADS = 384;  // three warpgroups: the third gives registers up to the first two (see setmaxnreg below)
// packed pairs of fp32
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void up2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2_(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2_(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {  // a NaN anywhere stays one
  float r;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
template <int HS>
__global__ void __launch_bounds__(PP_THREADS, 1) attn_prefill_tcgen05_pingpong_kernel(const __grid_constant__ PrefillAttnParams p, int single) {
  extern __shared__ __align__(1024) unsigned char pa_smem[];
  constexpr int KA = HS / 64;
  constexpr int ROW_ATOM = 128 * 128;
  constexpr int Q_BYTES = KA * ROW_ATOM;  // one query tile
  constexpr int K_BYTES = KA * ROW_ATOM;
  constexpr int VT_ATOM = HS * 128;
  constexpr int VT_BYTES = 2 * VT_ATOM;
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pa_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* q_s = base;                 // [2][Q_BYTES]
  unsigned char* k_s = q_s + 2 * Q_BYTES;    // [2][K_BYTES]
  unsigned char* vt_s = k_s + 2 * K_BYTES;   // [2][VT_BYTES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(vt_s + 2 * VT_BYTES);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 3, *v_full = bars + 5, *v_empty = bars + 7, *s_full = bars + 9,
           *p_ready = bars + 11 /* [tile][half] */, *o_full = bars + 15;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 17);
  const WaitLimit lim{reinterpret_cast<volatile int*>(tmem_ptr_smem + 1), p.status};

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int unit = (int)(gridDim.y - 1 - blockIdx.y), h = blockIdx.x, g = h / p.q_per_kv;
  const int m0 = unit * (single ? PA_BM : 2 * PA_BM);
  const int nA = m0 / PA_BM + 1, nB = !single && m0 + PA_BM < p.T ? nA + 1 : 0;  // key tiles of A and of B (0: no rows there)
  const int n_tiles = nB ? nB : nA;

  if (warp == 8 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_vt) : "memory");
    *lim.lost = 0;
    mbar_init(q_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&k_full[b], 1); mbar_init(&k_empty[b], nB ? 2 : 1); mbar_init(&v_full[b], 1); mbar_init(&v_empty[b], nB ? 2 : 1);
      mbar_init(&s_full[b], 1); mbar_init(&p_ready[2 * b], 128); mbar_init(&p_ready[2 * b + 1], 128); mbar_init(&o_full[b], 1);
    }
    mbar_fence_init();
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);

  // 384 threads are launched with 168 registers (64512 in all): 128 x 40 + 256 x 232 is the same sum
  if (warp >= 8) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  if (warp == 9) {
    if (elect_one()) {
      const int q_row0 = h * p.T_pad + m0;
      const int k_row0 = ((p.slot * 2 + 0) * p.n_groups + g) * p.max_seq;
      mbar_expect_tx(q_full, nB ? 2 * Q_BYTES : Q_BYTES);
#pragma unroll
      for (int a = 0; a < KA; ++a) tma_load_2d(q_s + a * ROW_ATOM, &p.map_q, q_full, a * 64, q_row0);
      if (nB)
#pragma unroll
        for (int a = 0; a < KA; ++a) tma_load_2d(q_s + Q_BYTES + a * ROW_ATOM, &p.map_q, q_full, a * 64, q_row0 + PA_BM);
      for (int t = 0; t < n_tiles; ++t) {
        const int b = t & 1, j0 = t * PA_BN;
        const uint32_t par = ((t >> 1) & 1) ^ 1;  // the buffer's previous use has been read (passes at once the first time)
        limited_wait(&k_empty[b], par, lim);
        mbar_expect_tx(&k_full[b], K_BYTES);
#pragma unroll
        for (int a = 0; a < KA; ++a) tma_load_2d(k_s + b * K_BYTES + a * ROW_ATOM, &p.map_k, &k_full[b], a * 64, k_row0 + j0);
        limited_wait(&v_empty[b], par, lim);
        mbar_expect_tx(&v_full[b], VT_BYTES);
#pragma unroll
        for (int a = 0; a < 2; ++a) tma_load_2d(vt_s + b * VT_BYTES + a * VT_ATOM, &p.map_vt, &v_full[b], j0 + a * 64, g * HS);
      }
    }
  } else if (warp == 8 || (warp == 10 && nB)) {
    if (elect_one()) {
      const int x = warp == 10, n = x ? nB : nA;
      const uint32_t idesc_s = umma_idesc_bf16(PA_BM, PA_BN), idesc_o = umma_idesc_bf16(PA_BM, HS);
      const uint32_t s_at = tmem + (uint32_t)(x * 128), o_at = tmem + 256u + (uint32_t)(x * 128);
      auto mma_s = [&](int t) {  // S_x = Q_x K_t^T
        const int b = t & 1;
        limited_wait(&k_full[b], (t >> 1) & 1, lim);
        tcgen05_fence_after();
#pragma unroll
        for (int k = 0; k < HS / 16; ++k) {
          const uint32_t off = (uint32_t)(k / 4) * ROW_ATOM + (uint32_t)(k % 4) * 32;
          tcgen05_mma_f16(s_at, umma_desc_sw128(smem_u32(q_s + x * Q_BYTES) + off), umma_desc_sw128(smem_u32(k_s + b * K_BYTES) + off),
                          idesc_s, k ? 1u : 0u);
        }
        tcgen05_commit(&s_full[x]);
        tcgen05_commit(&k_empty[b]);
        if (t >= nA) tcgen05_commit(&k_empty[b]);  // A has no use for these keys: B speaks for it
      };
      limited_wait(q_full, 0, lim);
      mma_s(0);
      for (int t = 0; t < n; ++t) {
        const int b = t & 1;
        limited_wait(&v_full[b], (t >> 1) & 1, lim);
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // O_x += P_x V_t, 64 keys at a time as the softmax warps finish them
          limited_wait(&p_ready[2 * x + half], t & 1, lim);
          tcgen05_fence_after();
#pragma unroll
          for (int k = 4 * half; k < 4 * half + 4; ++k) {
            const uint32_t offv = (uint32_t)(k / 4) * VT_ATOM + (uint32_t)(k % 4) * 32;
            tcgen05_mma_f16_ts(o_at, s_at + (uint32_t)(k * 8), umma_desc_sw128(smem_u32(vt_s + b * VT_BYTES) + offv), idesc_o,
                               (t | k) ? 1u : 0u);
          }
        }
        if (t + 1 < n) mma_s(t + 1);
        else tcgen05_commit(&o_full[x]);
        tcgen05_commit(&v_empty[b]);
        if (t >= nA) tcgen05_commit(&v_empty[b]);
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    const int x = warp >> 2, n = x ? nB : nA;
    const int r = threadIdx.x & 127;               // query row == TMEM lane
    const int q_idx = m0 + x * PA_BM + r;
    const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s_at = row + (uint32_t)(x * 128), o_at = row + 256u + (uint32_t)(x * 128);
    const f32x2 scale2 = pk2(p.scale_log2, p.scale_log2);
    float m_run = -INFINITY, l_run = 0.f;
    for (int t = 0; t < n; ++t) {
      limited_wait(&s_full[x], t & 1, lim);
      tcgen05_fence_after();
      uint32_t sv[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32_nowait(s_at + (uint32_t)(c * 32), sv + c * 32);
      tmem_wait_ld();
      if (t == n - 1) {  // the tile on the diagonal (rows before it end before p.T, so does what they see)
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i > r) sv[i] = 0xff800000u;
      }
      float mx8[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) mx8[e] = __uint_as_float(sv[e]);
#pragma unroll
      for (int i = 8; i < 120; i += 16)
#pragma unroll
        for (int e = 0; e < 8; ++e) mx8[e] = max3_nan(mx8[e], __uint_as_float(sv[i + e]), __uint_as_float(sv[i + 8 + e]));
#pragma unroll
      for (int e = 0; e < 4; ++e) mx8[e] = max3_nan(max3_nan(mx8[e], mx8[e + 4], __uint_as_float(sv[120 + e])), __uint_as_float(sv[124 + e]), -INFINITY);
      const float mx = max3_nan(max3_nan(mx8[0], mx8[1], mx8[2]), mx8[3], -INFINITY)
                       * p.scale_log2;  // scale > 0: max commutes
      const bool move = t == 0 || !(mx <= m_run);  // a NaN moves too, and stays
      float corr = 1.f;
      if (move) {
        corr = m_run == -INFINITY ? 0.f : exp2f(m_run - mx);
        m_run = mx;
        l_run *= corr;
      }
      if (t > 0 && __any_sync(0xffffffffu, move)) {
#pragma unroll 1
        for (int c = 0; c < HS / 64; ++c) {
          uint32_t ov[64];
          tmem_ld32_nowait(o_at + (uint32_t)(c * 64), ov);
          tmem_ld32_nowait(o_at + (uint32_t)(c * 64 + 32), ov + 32);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 64; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
          tmem_st32(o_at + (uint32_t)(c * 64), ov);
          tmem_st32(o_at + (uint32_t)(c * 64 + 32), ov + 32);
        }
      }
      // a row that has seen nothing finite yet has no weights; one with an infinite score has no value
      const float m_use = m_run == -INFINITY ? 0.f : m_run == INFINITY ? __int_as_float(0x7fffffff) : m_run;
      const f32x2 neg = pk2(-m_use, -m_use);
      f32x2 ps[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const f32x2 xx = fma2_(pk2(__uint_as_float(sv[c * 64 + 2 * i]), __uint_as_float(sv[c * 64 + 2 * i + 1])), scale2, neg);
          float a, b;
          up2(xx, a, b);
          a = exp2f(a);
          b = exp2f(b);
          ps[i & 3] = add2_(ps[i & 3], pk2(a, b));
          pk[i] = pack_bf16x2(a, b);
        }
        tmem_st32(s_at + (uint32_t)(c * 32), pk);
        tmem_wait_st();
        tcgen05_fence_before();
        mbar_arrive(&p_ready[2 * x + c]);
      }
      float s0, s1;
      up2(add2_(add2_(ps[0], ps[1]), add2_(ps[2], ps[3])), s0, s1);
      l_run += s0 + s1;
    }
    if (n > 0) {
      limited_wait(&o_full[x], 0, lim);
      tcgen05_fence_after();
      const float inv = *lim.lost ? __int_as_float(0x7fffffff) : l_run > 0.f ? 1.f / l_run : l_run == 0.f ? 0.f : l_run;
      bf16* dst = p.y + (size_t)q_idx * p.n_head * HS + (size_t)h * HS;
#pragma unroll 1
      for (int c = 0; c < HS / 32; ++c) {
        uint32_t ov[32];
        tmem_ld32_nowait(o_at + (uint32_t)(c * 32), ov);
        tmem_wait_ld();
        if (q_idx < p.T) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(ov[v * 8 + 0]) * inv, __uint_as_float(ov[v * 8 + 1]) * inv);
            o.y = pack_bf16x2(__uint_as_float(ov[v * 8 + 2]) * inv, __uint_as_float(ov[v * 8 + 3]) * inv);
            o.z = pack_bf16x2(__uint_as_float(ov[v * 8 + 4]) * inv, __uint_as_float(ov[v * 8 + 5]) * inv);
            o.w = pack_bf16x2(__uint_as_float(ov[v * 8 + 6]) * inv, __uint_as_float(ov[v * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = o;
          }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 8) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}

static int g_prefill_attn_pipe = 2;  // two query tiles in ping-pong; see mdi_set_prefill_attn_pipe

template <int HS>
static int launch_prefill_attn_pipe(const PrefillAttnParams& p, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)((HS / 64) * 128 * 128 * 3 + 2 * 2 * HS * 128 + 2 * 128 * 128) + 128;
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_tcgen05_pipe_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  dim3 grid((p.T + PA_BM - 1) / PA_BM, p.n_head);
  attn_prefill_tcgen05_pipe_kernel<HS><<<grid, PA_THREADS, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

template <int HS>
static int launch_prefill_attn_pingpong(const PrefillAttnParams& p, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)((HS / 64) * 128 * 128 * 4 + 2 * 2 * HS * 128) + 160;
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_tcgen05_pingpong_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int pairs = (p.T + 2 * PA_BM - 1) / (2 * PA_BM), tiles = (p.T + PA_BM - 1) / PA_BM;
  const bool single = pairs * p.n_head < device_sm_count();
  attn_prefill_tcgen05_pingpong_kernel<HS><<<dim3(p.n_head, single ? tiles : pairs), PP_THREADS, smem, stream>>>(p, single);
  return (int)cudaGetLastError();
}

template <int HS>
static int launch_prefill_attn(const PrefillAttnParams& p, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)(2 * (HS / 64) * 128 * 128 + 2 * HS * 128 + 2 * 128 * 128) + 128;
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_tcgen05_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  dim3 grid((p.T + PA_BM - 1) / PA_BM, p.n_head);
  attn_prefill_tcgen05_kernel<HS><<<grid, PA_THREADS, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace mdi

using namespace mdi;

// qkv: [T, (H + 2G) * hs] bf16 (output of the QKV GEMM), positions 0..T-1.  q_scratch: [H, T_pad, hs],
// vt_scratch: [G, hs, T_pad] (T_pad = T rounded up to 128; need no initialisation: V^T is written up to T_pad, and a query
// row behind T only reaches its own output, which is not stored),
// kv: the layer's pool [n_slots, 2, G, S, hs], y: [T, H * hs].  status: the stage's status words or null.
extern "C" int mdi_attn_prefill(const void* qkv, const float* cos, const float* sin, void* kv, void* q_scratch,
                                void* vt_scratch, void* y, int T, int T_pad, int slot, int n_slots, int n_head,
                                int n_groups, int head_size, int rope_n_elem, int max_seq, int* status, cudaStream_t stream) {
  if (T <= 0 || T > max_seq || T_pad % PA_BN != 0 || T_pad < T || n_head % n_groups != 0) return -2;
  if (head_size != 64 && head_size != 128) return -3;
  if (rope_n_elem % 16 != 0 || rope_n_elem > head_size) return -2;  // the vectorised pre-pass rotates 8-dim chunks
  RopeSplitArgs r;
  r.qkv = (const bf16*)qkv; r.cos = cos; r.sin = sin; r.q_out = (bf16*)q_scratch; r.kv = (bf16*)kv; r.vt = (bf16*)vt_scratch;
  r.T = T; r.T_pad = T_pad; r.slot = slot; r.n_head = n_head; r.n_groups = n_groups; r.hs = head_size; r.ne = rope_n_elem;
  r.max_seq = max_seq;
  rope_split_kernel<<<dim3(T_pad / RS_TOK, n_groups * ((n_head / n_groups + 2 + RS_SLOTS - 1) / RS_SLOTS)), 256, 0, stream>>>(r);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;

  PrefillAttnParams p;
  p.y = (bf16*)y; p.T = T; p.T_pad = T_pad; p.n_head = n_head; p.n_groups = n_groups; p.q_per_kv = n_head / n_groups;
  p.max_seq = max_seq; p.slot = slot; p.status = status;
  p.scale_log2 = 1.4426950408889634f / sqrtf((float)head_size);
  int rc = make_map(&p.map_q, q_scratch, (long long)n_head * T_pad, head_size, PA_BM);
  if (rc) return rc;
  rc = make_map(&p.map_k, kv, (long long)n_slots * 2 * n_groups * max_seq, head_size, PA_BN);
  if (rc) return rc;
  rc = make_map(&p.map_vt, vt_scratch, (long long)n_groups * head_size, T_pad, head_size);
  if (rc) return rc;
  if (g_prefill_attn_pipe == 2) return head_size == 128 ? launch_prefill_attn_pingpong<128>(p, stream) : launch_prefill_attn_pingpong<64>(p, stream);
  if (g_prefill_attn_pipe) return head_size == 128 ? launch_prefill_attn_pipe<128>(p, stream) : launch_prefill_attn_pipe<64>(p, stream);
  return head_size == 128 ? launch_prefill_attn<128>(p, stream) : launch_prefill_attn<64>(p, stream);
}

// 0 = simple sequential kernel, 1 = pipelined (double-buffered K/V^T tiles and score matrix), 2 = two query tiles in
// ping-pong with the output in TMEM (default)
extern "C" void mdi_set_prefill_attn_pipe(int on) { g_prefill_attn_pipe = on; }
extern "C" int mdi_get_prefill_attn_pipe() { return g_prefill_attn_pipe; }
