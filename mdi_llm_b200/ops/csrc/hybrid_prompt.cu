// Prompt attention of the hybrid family on the 5th-generation tensor cores (heads of 64, 128 or 192 key and 64 or 128 value channels in
// bf16; other sizes keep prompt_attn_mma_kernel, whose arguments and results these are).
//
// A CTA owns 128 query rows of one head; two CTAs share an SM, so that one multiplies while the other's softmax warps work:
//
//   warps 0-7  softmax: two threads share a row of scores, exchange its maximum, write its weights over the scores as bf16, with SPLIT
//              what the rounding dropped behind them, and rescale half a row of O each when the maximum moves
//   warp 8     one thread issues the products: S = Q K^T from shared memory, O += P V with P from TMEM and V as it lies in the cache (a row
//              of V per key: the MN-major form of the operand, so nothing is transposed before)
//   warp 9     one thread loads Q, K and V by TMA straight from the packed rows
//   10, 11     look through V in the key tiles that not every row sees whole: a weight of zero would not keep an infinite value out.  Rows
//              outside the sequence become zero, and values that are not finite, which the softmax warps then add themselves to
//              the rows that see them (a layer over 2048 tokens, 16 heads of 128, capped: 131 us without and 133 with it)
//
// TMEM: S / P [0, KEYS), O [128, 128 + V).  Key tiles are laid so that the last one ends with the CTA's last row.
// What bounds it: the softmax warps (with a cap on the scores: its tanh), hence two threads to a row and a barrier per step for it.
// us a launch, prompt_attn_mma_kernel and this, 16 heads: 2048 tokens, 128 on 4 key heads, capped 173 and 66 (78 where scores pass 0.75 of the cap), causal 146 and 47, window of
// 1024 112 and 35, block mask 98 and 36; heads of 192, window, 1411 + 501 + 136 tokens 84 and 41; 64 tokens 8.9 and 7.0.  Tried: two
// query tiles in ping-pong in one CTA of 4 (115 and 55 for the first two) and 8 softmax warps a tile (113 and 66): few CTAs of unequal
// length; one CTA of one tile on an SM 73 and 50, window 50.
#include "hybrid_math.cuh"
#include "tcgen05.cuh"

namespace hyb {

using namespace mdi;

constexpr int PT_THREADS = 384, PT_ROWS = 128;

struct PromptTcParams {
  CUtensorMap map_q, map_kv;  // boxes of 64 columns x 128 rows, 64 columns x the rows of a key tile
  const bf16* kv;
  bf16* out;
  const int* spans;
  const float* sink;
  const bf16* gate;
  int* status;  // becomes 1 when a wait ran out (the rows of that CTA are NaN then)
  long long kv_stride, gate_stride;
  int gate_each, H, G, window;
  float scale_log2e, cap_log2e;
};

__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t group_bytes) {  // 64-column groups `group_bytes` apart
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | ((uint64_t)(group_bytes >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 2^x for x <= 0: exp2f without its steps for results below 2^-126, which are zero here
__device__ __forceinline__ float pt_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Keys of a tile.  Heads of 192 leave room for two CTAs on an SM only with 64.  Weights of 16 bits keep the 64 of the warp-level kernel too: a
// row's largest weight so far is exactly one and loses nothing in rounding, so fewer and longer tiles add 0.5 % of error.  Else
// 128: half the barriers (2048 tokens, 16 heads of 128, us with 64 and 128: causal 54 and 47, block mask 40 and 36).
__host__ __device__ constexpr int pt_keys(int DK, bool split) { return DK > 128 || !split ? 64 : 128; }

template <int DK, int V, bool SPLIT, bool CAP, bool CHUNK>
__global__ void __launch_bounds__(PT_THREADS, 2) prompt_attn_tc_kernel(const __grid_constant__ PromptTcParams p) {
  extern __shared__ __align__(1024) unsigned char pt_smem[];
  constexpr int KEYS = pt_keys(DK, SPLIT), HK = KEYS / 2;           // keys of a tile, of a softmax thread
  constexpr int KG = DK / 64, VG = V / 64;                   // groups of 64 columns
  constexpr int QGROUP = PT_ROWS * 128, GROUP = KEYS * 128;  // bytes of one in Q, in K and V
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(pt_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* q_s = base;               // [KG][QGROUP]
  unsigned char* k_s = q_s + KG * QGROUP;  // [KG][GROUP]
  unsigned char* v_s = k_s + KG * GROUP;   // [VG][GROUP]
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + VG * GROUP);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = bars + 2, *v_full = bars + 3, *v_empty = bars + 4, *s_full = bars + 5, *p_ready = bars + 6,
           *o_full = bars + 7, *v_fixed = bars + 8, *v_tail = bars + 9;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* stray = reinterpret_cast<volatile int*>(bars + 11);  // values that are not finite were taken out of V
  float* red = reinterpret_cast<float*>(bars + 12);  // [step parity][half][row]: maxima, at the end sums
  const WaitLimit lim{reinterpret_cast<volatile int*>(tmem_ptr_smem + 1), nullptr};

  const int* sp = p.spans + 5 * blockIdx.z;
  const int n = sp[1], p0 = sp[3], first = sp[4], units = (n + PT_ROWS - 1) / PT_ROWS;
  if ((int)blockIdx.y >= units) return;
  const int h = blockIdx.x, hk = h / (p.H / p.G), m0 = (units - 1 - (int)blockIdx.y) * PT_ROWS;  // long rows of work first
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int off = p0 - first;  // key index of row 0
  auto low = [&](int i) {  // first key that row i sees
    return CHUNK ? (p0 + i) / p.window * p.window - first : p.window > 0 ? max(0, off + i - p.window + 1) : 0;
  };
  // key tile t holds the keys kb + KEYS t ..; the last one ends with row m0 + 127; those without a key that a row of the sequence sees
  // are left out, and rows of V outside [0, ke) become zero.  In the tiles [0, lead) and [tail, used) some row misses a key.
  const int end = off + m0 + PT_ROWS, kb = end - (end - low(m0) + KEYS - 1) / KEYS * KEYS;
  const int ke = off + min(n, m0 + PT_ROWS), used = (ke - kb + KEYS - 1) / KEYS;
  const int lead = min(used, (low(min(n, m0 + PT_ROWS) - 1) - kb + KEYS - 1) / KEYS), tail = (off + m0 - kb) / KEYS;

  if (warp == 8) {
    if (lane == 0) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_q) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&p.map_kv) : "memory");
      *lim.lost = 0;
      *stray = 0;
      for (int b = 0; b < 10; ++b) mbar_init(bars + b, bars + b == p_ready ? 256 : bars + b == v_fixed ? 2 : 1);
      mbar_fence_init();
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_ptr_smem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);

  // 384 threads are launched with 80 registers (30720 in all): 128 x 32 + 256 x 104 is the same sum
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == 9) {
      if (elect_one()) {
        mbar_expect_tx(q_full, KG * QGROUP);
#pragma unroll
        for (int a = 0; a < KG; ++a) tma_load_2d(q_s + a * QGROUP, &p.map_q, q_full, h * DK + a * 64, sp[0] + m0);
        for (int t = 0; t < used; ++t) {
          const int row = sp[2] + kb + t * KEYS;
          limited_wait(k_empty, (t & 1) ^ 1, lim);  // the buffer's previous use has been read
          mbar_expect_tx(k_full, KG * GROUP);
#pragma unroll
          for (int a = 0; a < KG; ++a) tma_load_2d(k_s + a * GROUP, &p.map_kv, k_full, hk * DK + a * 64, row);
          limited_wait(v_empty, (t & 1) ^ 1, lim);
          if (t == tail) mbar_arrive(v_tail);
          mbar_expect_tx(v_full, VG * GROUP);
#pragma unroll
          for (int a = 0; a < VG; ++a) tma_load_2d(v_s + a * GROUP, &p.map_kv, v_full, p.G * DK + hk * V + a * 64, row);
        }
      }
    } else if (warp == 8) {
      if (elect_one()) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(PT_ROWS, KEYS), idesc_o = umma_idesc_bf16(PT_ROWS, V) | (1u << 16);  // V: MN-major
        const uint32_t o_at = tmem + 128u;
        auto mma_s = [&](int t) {  // S = Q K_t^T
          limited_wait(k_full, t & 1, lim);
          tcgen05_fence_after();
#pragma unroll
          for (int k = 0; k < DK / 16; ++k)
            tcgen05_mma_f16(tmem, umma_desc_sw128(smem_u32(q_s) + (uint32_t)(k / 4) * QGROUP + (uint32_t)(k % 4) * 32),
                            umma_desc_sw128(smem_u32(k_s) + (uint32_t)(k / 4) * GROUP + (uint32_t)(k % 4) * 32), idesc_s, k ? 1u : 0u);
          tcgen05_commit(s_full);
          tcgen05_commit(k_empty);
        };
        limited_wait(q_full, 0, lim);
        mma_s(0);
        int edge = 0;
        for (int t = 0; t < used; ++t) {
          limited_wait(v_full, t & 1, lim);
          if (t < lead || t >= tail) limited_wait(v_fixed, edge++ & 1, lim);
          limited_wait(p_ready, t & 1, lim);
          tcgen05_fence_after();
#pragma unroll
          for (int u = 0; u < (SPLIT ? 2 : 1); ++u)  // O += P V_t
#pragma unroll
            for (int k = 0; k < KEYS / 16; ++k)
              tcgen05_mma_f16_ts(o_at, tmem + (uint32_t)(u * HK + k * 8), umma_desc_mn_sw128(smem_u32(v_s) + (uint32_t)(k * 2048), GROUP), idesc_o,
                                 t || k || u ? 1u : 0u);
          tcgen05_commit(v_empty);
          if (t + 1 < used) mma_s(t + 1);  // runs behind the product that reads P from the same columns
          else tcgen05_commit(o_full);
        }
      }
    } else {
      auto finite = [](uint32_t w) {  // two bf16, the ones that are not finite as zero
        return ((w & 0x7f80u) == 0x7f80u ? 0u : w & 0xffffu) | ((w & 0x7f800000u) == 0x7f800000u ? 0u : w & 0xffff0000u);
      };
      auto look = [&](int t) {  // 16 bytes of a row at a time, every other 32 of them for this warp
        const int r0 = -(kb + t * KEYS), r1 = ke + r0;  // rows of the sequence in the tile
        limited_wait(v_full, t & 1, lim);
        __nv_bfloat162 odd[2] = {};  // NaN once something that is not finite was multiplied with zero
#pragma unroll 2
        for (int i = (warp - 10) * 32 + lane; i < KEYS * 8; i += 64)
#pragma unroll
          for (int a = 0; a < VG; ++a) {
            uint4* at = reinterpret_cast<uint4*>(v_s + a * GROUP + i * 16);
            if ((i >> 3) < r0 || (i >> 3) >= r1) {
              *at = make_uint4(0, 0, 0, 0);
            } else {
              const uint4 v = *at;
              const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                odd[e & 1] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]), __nv_bfloat162{}, odd[e & 1]);
            }
          }
        const __nv_bfloat162 o = __hadd2(odd[0], odd[1]);
        if (__any_sync(0xffffffffu, __hisnan(o.x) || __hisnan(o.y))) {
#pragma unroll 1
          for (int i = (warp - 10) * 32 + lane; i < KEYS * 8 * VG; i += 64) {
            uint4* at = reinterpret_cast<uint4*>(v_s + i * 16);
            const uint4 v = *at;
            *at = make_uint4(finite(v.x), finite(v.y), finite(v.z), finite(v.w));
          }
          *stray = 1;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(v_fixed);
      };
      for (int t = 0; t < min(lead, tail); ++t) look(t);
      if (lead < tail) limited_wait(v_tail, 0, lim);  // from here on the buffer's phase is that of tile `tail`
      for (int t = tail; t < used; ++t) look(t);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int half = warp >> 2, r = threadIdx.x & 127, i = m0 + r;  // query row, TMEM lane r; this thread has a tile's keys HK half ..
    const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16), s_at = at + (uint32_t)(half * HK), o_at = at + 128u + (uint32_t)(half * (V / 2));
    float* mine = red + half * 128 + r;
    const float* other = red + (half ^ 1) * 128 + r;
    float m_run = -INFINITY, l_run = 0.f;
    const int hi = off + i - HK * half, lo = low(i) - HK * half;  // keys that the row sees
#pragma unroll 1
    for (int t = 0; t < used; ++t) {
      limited_wait(s_full, t & 1, lim);
      __syncwarp();
      tcgen05_fence_after();
      float s[HK];
      uint32_t* sv = reinterpret_cast<uint32_t*>(s);
#pragma unroll
      for (int c = 0; c < HK; c += 32) tmem_ld32_nowait(s_at + (uint32_t)c, sv + c);
      tmem_wait_ld();
      const int j0 = kb + t * KEYS;
      if (CAP) {
        float big[4] = {};
#pragma unroll
        for (int j = 0; j < HK; j += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) big[e] = fmaxf(fmaxf(big[e], fabsf(s[j + e])), fabsf(s[j + 4 + e]));
        const float most = fmaxf(fmaxf(big[0], big[1]), fmaxf(big[2], big[3])) * p.scale_log2e;
        if (__all_sync(0xffffffffu, most <= 0.75f)) {  // (tanhf asks for each value whether it is small)
#pragma unroll
          for (int j = 0; j < HK; ++j) s[j] = p.cap_log2e * small_tanh(s[j] * p.scale_log2e);
        } else {
#pragma unroll
          for (int j = 0; j < HK; ++j) s[j] = p.cap_log2e * tanhf(s[j] * p.scale_log2e);
        }
      }
      if (__any_sync(0xffffffffu, hi - j0 < HK - 1 || lo > j0)) {
#pragma unroll
        for (int j = 0; j < HK; ++j)
          if (j > hi - j0 || j < lo - j0) s[j] = -INFINITY;
      }
      float mx4[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) mx4[e] = fmaxf(s[e], s[e + 4]);
#pragma unroll
      for (int j = 8; j < HK; j += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx4[e] = fmaxf(fmaxf(mx4[e], s[j + e]), s[j + 4 + e]);
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      if (!CAP) mx *= p.scale_log2e;  // scale > 0: the maximum commutes
      // the other half's maximum.  Behind this barrier both halves have read their scores, over which the weights go
      const int turn = (t & 1) * 256;
      mine[turn] = mx;
      tcgen05_fence_before();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      tcgen05_fence_after();
      mx = fmaxf(mx, other[turn]);
      const float m_new = fmaxf(m_run, mx), m_use = m_new == -INFINITY ? 0.f : m_new;  // a row that has seen no key yet
      const float corr = pt_exp2(m_run - m_use);
      const bool move = m_new != m_run;
      m_run = m_new;
      l_run *= corr;
      if (t > 0 && __any_sync(0xffffffffu, move)) {
#pragma unroll
        for (int c = 0; c < V / 2; c += 16) {
          uint32_t ov[16];
          tmem_ld16(o_at + (uint32_t)c, ov);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * corr);
          tmem_st16(o_at + (uint32_t)c, ov);
        }
      }
      float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < HK / 32; ++c) {
        uint32_t pk[16], rest[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float a = s[c * 32 + 2 * e], b = s[c * 32 + 2 * e + 1];
          const float u = pt_exp2(CAP ? a - m_use : fmaf(a, p.scale_log2e, -m_use)), v = pt_exp2(CAP ? b - m_use : fmaf(b, p.scale_log2e, -m_use));
          ps[e & 3] += u + v;
          pk[e] = pack_bf16x2(u, v);
          if (SPLIT) rest[e] = pack_bf16x2(u - bf16lo(pk[e]), v - bf16hi(pk[e]));
        }
        tmem_st16(at + (uint32_t)(half * (HK / 2) + c * 16), pk);
        if (SPLIT) tmem_st16(at + (uint32_t)(HK + half * (HK / 2) + c * 16), rest);
      }
      tmem_wait_st();
      tcgen05_fence_before();
      mbar_arrive(p_ready);
      l_run += (ps[0] + ps[1]) + (ps[2] + ps[3]);
    }
    limited_wait(o_full, 0, lim);
    limited_wait(v_fixed, (min(lead, tail) + used - tail - 1) & 1, lim);  // (long there; for `stray`)
    __syncwarp();
    tcgen05_fence_after();
    const int turn = (used & 1) * 256;
    mine[turn] = l_run;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l_run = half ? other[turn] + l_run : l_run + other[turn];
    float inv;
    if (p.sink) {
      const float sv = p.sink[h] * 1.4426950408889634f, M = fmaxf(m_run, sv), e = exp2f(m_run - M);
      inv = e / (l_run * e + exp2f(sv - M));
    } else {
      inv = 1.f / l_run;
    }
    if (*lim.lost) inv = __int_as_float(0x7fffffff);
    const bool live = i < n;
    const bf16* g = p.gate ? p.gate + (size_t)(sp[0] + (live ? i : 0)) * p.gate_stride : nullptr;
    if (g && !p.gate_each) inv *= sigmoidf_(to_f(g[h]));
    if (g) g += (size_t)h * V + half * (V / 2);
    const bool wide = p.gate_each && ((uintptr_t)p.gate & 15) == 0 && p.gate_stride % 8 == 0;
    bf16* dst = p.out + ((size_t)(sp[0] + i) * p.H + h) * V + half * (V / 2);
    const bool add = *stray && live;
#pragma unroll 1
    for (int c = 0; c < V / 2; c += 16) {
      uint32_t ov[16];
      tmem_ld16(o_at + (uint32_t)c, ov);
      tmem_wait_ld();
      if (add) {  // what was taken out of V, from the keys that this row sees: an infinity stays one whatever its weight
#pragma unroll 1
        for (int j = max(low(i), 0); j <= off + i; ++j) {
          if (j >= kb + lead * KEYS && j < kb + tail * KEYS) j = kb + tail * KEYS;
          const bf16* v = p.kv + (size_t)(sp[2] + j) * p.kv_stride + p.G * DK + hk * V + half * (V / 2) + c;
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float x = to_f(v[e]);
            if (!isfinite(x)) ov[e] = __float_as_uint(__uint_as_float(ov[e]) + x);
          }
        }
      }
      if (live)
#pragma unroll
        for (int v = 0; v < 16; v += 8) {
          float f[8], gv[8];
          if (p.gate_each) {
            if (wide) load8(g + c + v, gv);
            else
#pragma unroll
              for (int e = 0; e < 8; ++e) gv[e] = to_f(g[c + v + e]);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            f[e] = __uint_as_float(ov[v + e]) * inv;
            if (p.gate_each) f[e] *= sigmoidf_(gv[e]);
          }
          store8(dst + c + v, f);
        }
      __syncwarp();
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *lim.lost && p.status) atomicExch(p.status, 1);
  if (warp == 8) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
  }
}

template <int DK, int V, bool SPLIT, bool CAP, bool CHUNK>
static int run_prompt_tc(const PromptTcParams& p, int nseq, int longest, cudaStream_t st) {
  constexpr size_t smem = 1024 + (size_t)(DK / 64) * PT_ROWS * 128 + (size_t)(DK / 64 + V / 64) * pt_keys(DK, SPLIT) * 128 + 96 + 2048;
  const cudaError_t e = allow_smem<prompt_attn_tc_kernel<DK, V, SPLIT, CAP, CHUNK>>((int)smem);
  if (e != cudaSuccess) return (int)e;
  prompt_attn_tc_kernel<DK, V, SPLIT, CAP, CHUNK><<<dim3(p.H, (longest + PT_ROWS - 1) / PT_ROWS, nseq), PT_THREADS, smem, st>>>(p);
  return (int)cudaGetLastError();
}
template <int DK, int V>
static int run_prompt_tc(const PromptTcParams& p, bool split, bool cap, bool chunk, int nseq, int longest, cudaStream_t st) {
  if (split) {
    if (cap) return chunk ? run_prompt_tc<DK, V, true, true, true>(p, nseq, longest, st) : run_prompt_tc<DK, V, true, true, false>(p, nseq, longest, st);
    return chunk ? run_prompt_tc<DK, V, true, false, true>(p, nseq, longest, st) : run_prompt_tc<DK, V, true, false, false>(p, nseq, longest, st);
  }
  if (cap) return chunk ? run_prompt_tc<DK, V, false, true, true>(p, nseq, longest, st) : run_prompt_tc<DK, V, false, true, false>(p, nseq, longest, st);
  return chunk ? run_prompt_tc<DK, V, false, false, true>(p, nseq, longest, st) : run_prompt_tc<DK, V, false, false, false>(p, nseq, longest, st);
}

// 2-D bf16 rows, box of 64 columns, 128-byte swizzle; rows may be wider than `cols`
static int make_rows_map(CUtensorMap* map, const void* ptr, long long rows, long long cols, long long stride, int box_rows) {
  PFN_encodeTiled enc = get_encode_fn();
  if (!enc) return -5;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)stride * 2};
  cuuint32_t box[2] = {64u, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -6;
}

}  // namespace hyb

using namespace hyb;

// hyb_prompt_attn_mma's arguments, and how many rows q and kv have.  -3: sizes that this form does not take.
extern "C" int hyb_prompt_attn_tc(const void* q, long long q_stride, long long q_rows, const void* kv, long long kv_stride, long long kv_rows, void* out,
                                  const int* spans, int nseq, int longest, int H, int G, int DK, int V, int window, float scale, int split,
                                  const float* sink, const void* gate, long long gate_stride, int gate_each, float cap, int chunk, int* status, cudaStream_t st) {
  if (nseq == 0 || longest == 0) return 0;
  if (G < 1 || H % G || !(cap >= 0.f) || (chunk && window < 1) || (gate_each && !gate)) return -2;
  if (scale <= 0.f || (DK != 64 && DK != 128 && DK != 192) || (V != 64 && V != 128) || nseq > 65535 || H > 65535 || (longest + 127) / 128 > 65535) return -3;
  if (q_stride < (long long)H * DK || kv_stride < (long long)G * (DK + V)) return -3;  // a tensor map's rows do not overlap
  if (q_stride % 8 || kv_stride % 8 || (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)out) & 15) || q_rows > 0x7fffffff || kv_rows > 0x7fffffff) return -3;
  PromptTcParams p;
  int rc = make_rows_map(&p.map_q, q, q_rows, (long long)H * DK, q_stride, PT_ROWS);
  if (rc) return rc;
  rc = make_rows_map(&p.map_kv, kv, kv_rows, (long long)G * (DK + V), kv_stride, pt_keys(DK, split != 0));
  if (rc) return rc;
  p.kv = (const bf16*)kv; p.kv_stride = kv_stride;
  p.out = (bf16*)out; p.spans = spans; p.sink = sink; p.gate = (const bf16*)gate; p.status = status; p.gate_stride = gate_stride; p.gate_each = gate_each;
  p.H = H; p.G = G; p.window = window;
  p.scale_log2e = cap > 0.f ? scale / cap : scale * 1.4426950408889634f;
  p.cap_log2e = cap * 1.4426950408889634f;
  const bool c = cap > 0.f;
  if (DK == 64) return V == 64 ? run_prompt_tc<64, 64>(p, split, c, chunk, nseq, longest, st) : run_prompt_tc<64, 128>(p, split, c, chunk, nseq, longest, st);
  if (DK == 128) return V == 64 ? run_prompt_tc<128, 64>(p, split, c, chunk, nseq, longest, st) : run_prompt_tc<128, 128>(p, split, c, chunk, nseq, longest, st);
  return V == 64 ? run_prompt_tc<192, 64>(p, split, c, chunk, nseq, longest, st) : run_prompt_tc<192, 128>(p, split, c, chunk, nseq, longest, st);
}
