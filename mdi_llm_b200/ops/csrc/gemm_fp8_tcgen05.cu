// Block-scaled fp8 (e4m3) GEMM on the 5th-generation tensor cores: tcgen05.mma kind::f8f6f4, sm_100a.
//
//   C[M, N] = sum_kb  a_s[m, kb] * w_s[n, kb] * ( A8[m, kb*128 : +128] . W8[n, kb*128 : +128] )   (+bias, +residual)
//
// Weights are e4m3 with one fp32 scale per 128 consecutive K elements of every output row (what the decode kernels stream),
// activations are quantised the same way per token.  Scales change every 128 K elements, so the tensor core cannot accumulate the
// whole K range in one go: every K block (= one 128-byte shared-memory slab = 4 MMAs of K = 32) is accumulated into a FRESH partial
// accumulator in TMEM, and "promotion" warps fold it into fp32 register accumulators with the block's scales while the tensor core
// already works on the next blocks in the other TMEM buffers:
//
//   warp 0      TMA producer: A8 / W8 tiles (rows x 128 B, SWIZZLE_128B) into a ring of stages
//   warp 1      MMA issuer: per K block 4 x tcgen05.mma.kind::f8f6f4 into one of the partial buffers,
//               tcgen05.commit -> "stage free" and "partial full"
//   warp 2      block scales into a ring of their own
//   warp 3      TMEM allocation
//   warps 4-11  promotion + epilogue: acc += partial * (a_s[row] * w_s[col]); after the last K block bias / residual / activation and
//               bf16 stores (optionally straight into the next stage's memory: the fused prefill hop)
//
// Gated MLPs (SwiGLU / GeGLU) in one pass: the tile's first 64 columns are rows of fc_1, the others the SAME rows of fc_2, and
// a thread holds the same columns of both.  Few tiles share their K blocks in clusters (SHARED, fp8_shares).
//
// What bounds it: the promotion, a serial chain of TMEM loads and FMAs per K block (0.38 us; its MMAs take 0.14 at the nominal rate).
// us, with a column and a shared-memory exchange per thread and with two columns: 1024 x 2 x 14336 x 4096 gated 313 and 170, 1024 x 4096 x 14336
// 90 and 84, 448 x 4096 x 4096 16.7 and 16.4, 448 x 1024 x 1024 6.9 and 7.0 (8.0 while the epilogue's branches stood inside its unrolled loops).
#include <cuda_fp8.h>

#include "tcgen05.cuh"

namespace mdi {

constexpr int F8_BM = 128, F8_BK = 128;  // BK in elements == bytes
constexpr int F8_STAGES = 6;
constexpr int F8_SLOTS = 8;      // scales of a K block outlive its tiles: the promotion reads them after the MMAs have freed the stage
constexpr int F8_BN = 128, F8_PBUF = 4;  // columns of a tile; partial accumulators in TMEM (4 x 128 columns = all 512)
constexpr int F8_PROMO = 8;              // promotion warps: four per half of the tile's columns, one for each quarter of TMEM's lanes
constexpr int F8_THREADS = 128 + 32 * F8_PROMO;  // three warpgroups: the first gives registers up to the promotion (see setmaxnreg below)

// packed fp32 pair arithmetic (sm_100: FFMA2 / FMUL2 — two lanes per issue slot)
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ unsigned long long pack2(uint32_t lo, uint32_t hi) { return (unsigned long long)lo | ((unsigned long long)hi << 32); }
__device__ __forceinline__ float lo32(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi32(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// explicit shared-space loads: the pointers below derive from the re-aligned dynamic-smem base, which the compiler
// only knows as a generic address (it emitted 64-bit generic LD.E for them)
__device__ __forceinline__ unsigned long long lds_b64(uint32_t saddr) {
  unsigned long long v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(saddr));
  return v;
}
__device__ __forceinline__ float lds_f32(uint32_t saddr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(saddr));
  return v;
}

struct Fp8GemmParams {
  CUtensorMap tma_a;   // A8  [M, K] uint8, box 128 x 128
  CUtensorMap tma_b;   // W8  [N, K] uint8, box (rows one CTA loads) x 128
  CUtensorMap tma_b2;  // gated: second weight matrix, same box
  const float* a_scale_t;   // [K/128, ld_as]  (transposed: a warp reads neighbouring rows' scales)
  const float* w_scale_t;   // [K/128, N]      (transposed copy of the decode kernels' [N, K/128])
  const float* w2_scale_t;  // gated
  long long ld_as;
  bf16* C;
  const bf16* bias;
  const bf16* bias2;
  const bf16* residual;
  int M, N, K;  // N = output columns (gated: the intermediate size)
  int act;      // gated: ACT_*_GATE; 0 = plain
  int shares;   // CTAs of a cluster that share a tile's K blocks (1: no cluster)
  HopSignal signal;
  const int* ctx;
};

__device__ __forceinline__ void tcgen05_mma_f8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// cute::UMMA::InstrDescriptor for kind::f8f6f4: D = f32 (bits 4-5 = 1), A = B = E4M3 (format 0), both K-major
__device__ __forceinline__ constexpr uint32_t umma_idesc_e4m3(int m, int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// 16 lanes x 32 columns of fp32: thread t gets, of every eight columns i, columns 2 (t % 4) and the next one of lane t / 4 in
// r[4 i], r[4 i + 1] and of lane t / 4 + 8 in r[4 i + 2], r[4 i + 3]
__device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// waits for this thread's loads; the registers pass through so that no use of them moves in front of the wait
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}
// 4 x 4 transpose over the four threads that share a row: thread q ends with the q-th value of each of them
__device__ __forceinline__ void quad_transpose(uint32_t (&v)[4], int q) {
#pragma unroll
  for (int b = 0; b < 4; b += 2) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, (q & 1) ? v[b] : v[b + 1], 1);
    if (q & 1) v[b] = y; else v[b + 1] = y;
  }
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, (q & 2) ? v[b] : v[b + 2], 2);
    if (q & 2) v[b] = y; else v[b + 2] = y;
  }
}

template <bool GATED, bool SHARED>
__global__ void __launch_bounds__(F8_THREADS, 1) gemm_fp8_kernel(const __grid_constant__ Fp8GemmParams p) {
  extern __shared__ __align__(1024) unsigned char f8_smem[];
  constexpr int BN = F8_BN, PBUF = F8_PBUF;
  constexpr int A_BYTES = F8_BM * F8_BK, B_BYTES = BN * F8_BK;
  constexpr int OUT_N = GATED ? BN / 2 : BN;   // output columns per tile
  constexpr int WC = 4 * BN / F8_PROMO;        // columns of a promotion warp
  constexpr int CW = 32, NCH = WC / CW;        // ... that it reads at a time, and how many times
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(f8_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* smem_a = base;
  unsigned char* smem_b = base + F8_STAGES * A_BYTES;
  float* sc_a = reinterpret_cast<float*>(smem_b + F8_STAGES * B_BYTES);  // [F8_SLOTS][128] scales of the tile's rows
  float* sc_w = sc_a + F8_SLOTS * 128;                                   // [F8_SLOTS][BN] scales of the tile's columns
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sc_w + F8_SLOTS * BN);
  uint64_t* empty_bar = full_bar + F8_STAGES;
  uint64_t* pfull_bar = empty_bar + F8_STAGES;  // [PBUF] partial accumulator complete
  uint64_t* pempty_bar = pfull_bar + PBUF;      // [PBUF] partial accumulator drained
  uint64_t* sfull_bar = pempty_bar + PBUF;      // [F8_SLOTS] scales have landed
  uint64_t* sempty_bar = sfull_bar + F8_SLOTS;  // [F8_SLOTS] scales have been read
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(sempty_bar + F8_SLOTS);
  int* lost = reinterpret_cast<int*>(tmem_ptr_smem + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles_m = (p.M + F8_BM - 1) / F8_BM, tiles_n = (p.N + OUT_N - 1) / OUT_N, n_tiles = tiles_m * tiles_n;
  const int S = SHARED ? p.shares : 1, rank = SHARED ? (int)cluster_ctarank() : 0;
  const int kb0 = SHARED ? rank * (p.K / F8_BK) / S : 0, nkb = SHARED ? (rank + 1) * (p.K / F8_BK) / S - kb0 : p.K / F8_BK;  // this CTA's K blocks
  const WaitLimit lim{lost, const_cast<int*>(p.signal.status)};

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_b) : "memory");
    if (GATED) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_b2) : "memory");
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int s = 0; s < F8_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
      for (int b = 0; b < PBUF; ++b) { mbar_init(&pfull_bar[b], 1); mbar_init(&pempty_bar[b], F8_PROMO); }
      for (int s = 0; s < F8_SLOTS; ++s) { mbar_init(&sfull_bar[s], 1); mbar_init(&sempty_bar[s], F8_PROMO); }
      mbar_fence_init();
      *lost = 0;
    }
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_ptr_smem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);

  // 384 threads start with 168 registers each (64512 in all): 256 x 208 + 128 x 88 is the same sum
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
  if (warp == 0) {
    // ===== TMA producer =====
    if (elect_one()) {
      int it = 0;
      for (int tile = SHARED ? blockIdx.x / S : blockIdx.x; tile < n_tiles; tile += SHARED ? gridDim.x / S : gridDim.x) {
        const int m0 = (tile % tiles_m) * F8_BM, n0 = (tile / tiles_m) * OUT_N;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % F8_STAGES;
          limited_wait(&empty_bar[s], ((it / F8_STAGES) & 1) ^ 1, lim);
          mbar_expect_tx(&full_bar[s], A_BYTES + B_BYTES);
          tma_load_2d(smem_a + s * A_BYTES, &p.tma_a, &full_bar[s], (kb0 + kb) * F8_BK, m0);
          tma_load_2d(smem_b + s * B_BYTES, &p.tma_b, &full_bar[s], (kb0 + kb) * F8_BK, n0);
          if (GATED) tma_load_2d(smem_b + s * B_BYTES + B_BYTES / 2, &p.tma_b2, &full_bar[s], (kb0 + kb) * F8_BK, n0);
        }
      }
    }
  } else if (warp == 2) {
    // ===== block scales =====
    if (elect_one()) {
      int it = 0;
      for (int tile = SHARED ? blockIdx.x / S : blockIdx.x; tile < n_tiles; tile += SHARED ? gridDim.x / S : gridDim.x) {
        const int m0 = (tile % tiles_m) * F8_BM, n0 = (tile / tiles_m) * OUT_N;
        const int wn = min(OUT_N, p.N - n0);                              // N % 4 == 0: 16-byte copies
        const int an = max(0, (int)min(p.ld_as - m0, (long long)F8_BM));  // rows the scale table has
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int sl = it % F8_SLOTS;
          limited_wait(&sempty_bar[sl], ((it / F8_SLOTS) & 1) ^ 1, lim);
          mbar_expect_tx(&sfull_bar[sl], (uint32_t)((an + (GATED ? 2 : 1) * wn) * 4));
          if (an > 0) bulk_g2s(sc_a + sl * 128, p.a_scale_t + (size_t)(kb0 + kb) * p.ld_as + m0, (uint32_t)(an * 4), &sfull_bar[sl]);
          bulk_g2s(sc_w + sl * BN, p.w_scale_t + (size_t)(kb0 + kb) * p.N + n0, (uint32_t)(wn * 4), &sfull_bar[sl]);
          if (GATED) bulk_g2s(sc_w + sl * BN + OUT_N, p.w2_scale_t + (size_t)(kb0 + kb) * p.N + n0, (uint32_t)(wn * 4), &sfull_bar[sl]);
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer: one fresh partial accumulator per K block =====
    const uint32_t idesc = umma_idesc_e4m3(F8_BM, BN);
    int it = 0;
    for (int tile = SHARED ? blockIdx.x / S : blockIdx.x; tile < n_tiles; tile += SHARED ? gridDim.x / S : gridDim.x) {
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = it % F8_STAGES, pb = it % PBUF;
        limited_wait(&full_bar[s], (it / F8_STAGES) & 1, lim);
        limited_wait(&pempty_bar[pb], ((it / PBUF) & 1) ^ 1, lim);  // promotion warps are done with this buffer
        tcgen05_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = smem_u32(smem_a + s * A_BYTES), b_addr = smem_u32(smem_b + s * B_BYTES);
#pragma unroll
          for (int k = 0; k < F8_BK / 32; ++k)  // K = 32 elements = 32 bytes per MMA inside the 128-byte swizzle atom
            tcgen05_mma_f8(tmem_base + (uint32_t)(pb * BN), umma_desc_sw128(a_addr + k * 32), umma_desc_sw128(b_addr + k * 32), idesc, k ? 1u : 0u);
          tcgen05_commit(&pfull_bar[pb]);
          tcgen05_commit(&empty_bar[s]);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if constexpr (SHARED) { cluster_sync_all(); cluster_sync_all(); }
  } else {
    // ===== promotion + epilogue: a warp has TMEM lanes [32 lg, +32) and half of the tile's columns =====
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int lg = warp & 3, hf = (warp - 4) >> 2, q = lane & 3, r0 = lg * 32 + (lane >> 2);
    // first column of this warp's piece c.  Gated: fc_1 in the first pieces, the same columns of fc_2 in the others
    auto col_of = [&](int c) { return GATED ? (c < NCH / 2 ? hf * (WC / 2) + CW * c : BN / 2 + hf * (WC / 2) + CW * (c - NCH / 2)) : hf * WC + CW * c; };
    int it = 0;
    for (int tile = SHARED ? blockIdx.x / S : blockIdx.x; tile < n_tiles; tile += SHARED ? gridDim.x / S : gridDim.x) {
      const int m0 = (tile % tiles_m) * F8_BM, n0 = (tile / tiles_m) * OUT_N;
      unsigned long long acc[NCH][2][CW / 8][2];  // [piece][16 lanes][8 columns][lane or lane + 8]: two neighbouring columns
#pragma unroll
      for (int c = 0; c < NCH; ++c)
#pragma unroll
        for (int i = 0; i < CW / 2; ++i) acc[c][i / (CW / 4)][(i >> 1) % (CW / 8)][i & 1] = 0ull;
      constexpr int STEPS = 2 * NCH;  // pieces of this warp in both halves of its 32 lanes
      auto part = [&](int i) { return tmem_base + (uint32_t)((i % PBUF) * BN) + ((uint32_t)(lg * 32) << 16); };
      const uint32_t as_base = smem_u32(sc_a + r0), ws_base = smem_u32(sc_w + 2 * q);
      auto a_at = [&](int i) { return as_base + (uint32_t)(i % F8_SLOTS) * 512u; };
      auto w_at = [&](int i) { return ws_base + (uint32_t)(i % F8_SLOTS) * (4u * BN); };
      // The loop runs one step ahead of itself: while a step's partials are multiplied, the next step's are on their way from TMEM
      // (the next K block's too, whose barriers are asked one step earlier) and the weights' scales are replaced as they are spent.
      uint32_t t[2][CW / 2];
      unsigned long long w2[CW / 8];
      float a[4];
      limited_wait(&pfull_bar[it % PBUF], (it / PBUF) & 1, lim);
      limited_wait(&sfull_bar[it % F8_SLOTS], (it / F8_SLOTS) & 1, lim);
      __syncwarp();
      tcgen05_fence_after();
      tmem_ld_16x256b(part(it) + (uint32_t)col_of(0), t[0]);
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = lds_f32(a_at(it) + 32 * i);
#pragma unroll
      for (int i = 0; i < CW / 8; ++i) w2[i] = lds_b64(w_at(it) + 4 * col_of(0) + 32 * i);
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int nx = it + 1;
        const bool more = kb + 1 < nkb;
        const uint32_t taddr = part(it), w_cur = w_at(it), w_next = w_at(it + 1);
        unsigned long long a2[2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) a2[i >> 1][i & 1] = pack2(a[i], a[i]);
        bool p_there = false, s_there = false;
#pragma unroll
        for (int j = 0; j < STEPS; ++j) {
          const int c = j >> 1, h = j & 1;
          tmem_wait_ld(t[h]);
          if (j + 1 < STEPS) {
            tmem_ld_16x256b(taddr + (uint32_t)col_of((j + 1) >> 1) + (uint32_t)(h ? 0 : (16 << 16)), t[h ^ 1]);
          } else {  // everything of this K block is in registers
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&pempty_bar[it % PBUF]);
              mbar_arrive(&sempty_bar[it % F8_SLOTS]);
            }
            if (more) {
              if (!p_there) limited_wait(&pfull_bar[nx % PBUF], (nx / PBUF) & 1, lim);
              if (!s_there) limited_wait(&sfull_bar[(it + 1) % F8_SLOTS], ((it + 1) / F8_SLOTS) & 1, lim);
              __syncwarp();
              tcgen05_fence_after();
              tmem_ld_16x256b(part(nx) + (uint32_t)col_of(0), t[0]);
#pragma unroll
              for (int i = 0; i < 4; ++i) a[i] = lds_f32(a_at(it + 1) + 32 * i);
            }
          }
          if (j + 2 == STEPS && more) {
            p_there = mbar_try(smem_u32(&pfull_bar[nx % PBUF]), (nx / PBUF) & 1);
            s_there = mbar_try(smem_u32(&sfull_bar[(it + 1) % F8_SLOTS]), ((it + 1) / F8_SLOTS) & 1);
          }
#pragma unroll
          for (int i = 0; i < CW / 8; ++i) {
            acc[c][h][i][0] = fma2(pack2(t[h][4 * i], t[h][4 * i + 1]), mul2(w2[i], a2[h][0]), acc[c][h][i][0]);
            acc[c][h][i][1] = fma2(pack2(t[h][4 * i + 2], t[h][4 * i + 3]), mul2(w2[i], a2[h][1]), acc[c][h][i][1]);
          }
#pragma unroll
          for (int i = 0; i < CW / 8; ++i) {
            if (h == 1 && j + 1 < STEPS) w2[i] = lds_b64(w_cur + 4 * col_of(c + 1) + 32 * i);
            if (j + 1 == STEPS && more) w2[i] = lds_b64(w_next + 4 * col_of(0) + 32 * i);
          }
        }
      }
      const bool bad = *lim.lost != 0;
      // ---- shared K range: every CTA of the cluster finishes the column groups that are its own, with the others' sums of them ----
      if constexpr (SHARED) {
        constexpr int OG = OUT_N / 8;  // groups of eight output columns
        auto owner = [&](int og) { return og * S / OG; };
        const uint32_t place = smem_u32(smem_a);  // [S - 1 senders][own groups (gated: of fc_1, of fc_2)][128 rows][8 columns], over the stages
        const int most = (OG + S - 1) / S;  // groups of a CTA, at most
        auto at = [&](int from, int to, int og, int second, int row) {
          const int lo = (to * OG + S - 1) / S, slot = from < to ? from : from - 1;
          return place + (uint32_t)((((slot * (GATED ? 2 : 1) + second) * most + (og - lo)) * 128 + row) * 32 + 8 * q);
        };
        cluster_sync_all();  // everybody's products are done: the stages are free
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
          for (int i = 0; i < CW / 8; ++i) {
            const int second = GATED && c >= NCH / 2, og = col_of(second ? c - NCH / 2 : c) / 8 + i, to = owner(og);
            if (to != rank)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const unsigned long long v = bad ? ~0ull : acc[c][e >> 1][i][e & 1];  // (all ones: NaN)
                st_cluster(cluster_addr(at(rank, to, og, second, r0 + 8 * e), to), lo32(v), hi32(v));
              }
          }
        cluster_sync_all();
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
          for (int i = 0; i < CW / 8; ++i) {
            const int second = GATED && c >= NCH / 2, og = col_of(second ? c - NCH / 2 : c) / 8 + i;
            if (owner(og) == rank)
              for (int from = 0; from < S; ++from)
                if (from != rank)
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const unsigned long long v = lds_b64(at(from, rank, og, second, r0 + 8 * e)), a0 = acc[c][e >> 1][i][e & 1];
                    acc[c][e >> 1][i][e & 1] = pack2(lo32(a0) + lo32(v), hi32(a0) + hi32(v));
                  }
          }
      }
      // ---- epilogue: bf16 pairs, transposed over the four threads of a row so that each stores eight columns ----
      // A tile runs through it once, so fetching its code is what it takes: what most products leave out stands behind branches of its own
      // (bias, activation, columns that are not eights), not inside the unrolled loops.
      constexpr int G = CW / 8, PIECES = GATED ? NCH / 2 : NCH;  // groups of eight columns in a piece, one for each of the four threads of a row
      if (p.bias || (GATED && p.bias2)) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const bf16* bias = c < PIECES ? p.bias : p.bias2;
          const int col0 = n0 + col_of(c) - (c < PIECES ? 0 : BN / 2) + 2 * q;
#pragma unroll
          for (int i = 0; i < G; ++i)
            if (bias && col0 + 8 * i < p.N) {
              const float lo = __bfloat162float(bias[col0 + 8 * i]), hi = __bfloat162float(bias[col0 + 8 * i + 1]);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                unsigned long long& v = acc[c][e >> 1][i][e & 1];
                v = pack2(lo32(v) + lo, hi32(v) + hi);
              }
            }
        }
      }
      if constexpr (GATED) {
        auto gate = [&](auto act) {
#pragma unroll
          for (int c = 0; c < PIECES; ++c)
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                unsigned long long& g = acc[c][e >> 1][i][e & 1];
                const unsigned long long u = acc[c + NCH / 2][e >> 1][i][e & 1];
                g = pack2(round_bf16(apply_act(round_bf16(lo32(g)), act())) * round_bf16(lo32(u)),
                          round_bf16(apply_act(round_bf16(hi32(g)), act())) * round_bf16(hi32(u)));
              }
        };
        if (p.act == ACT_SILU_GATE) gate([] { return ACT_SILU_GATE; });
        else if (p.act == ACT_GELU_TANH_GATE) gate([] { return ACT_GELU_TANH_GATE; });
        else gate([] { return ACT_GELU_ERF_GATE; });
      }
      // the thread's eight columns of one of its four rows in piece c
      auto row_of = [&](int c, int e, uint32_t (&o)[G], int& row, int& col) {
#pragma unroll
        for (int i = 0; i < G; ++i) o[i] = bad ? 0x7fff7fffu : pack_bf16x2(lo32(acc[c][e >> 1][i][e & 1]), hi32(acc[c][e >> 1][i][e & 1]));
        quad_transpose(o, q);
        row = m0 + r0 + 8 * e;
        col = n0 + col_of(c) + 8 * q;
        return row < p.M && col < p.N && (!SHARED || (col - n0) / 8 * S / (OUT_N / 8) == rank);
      };
      if (p.N % 8 == 0) {
#pragma unroll
        for (int c = 0; c < PIECES; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint32_t o[G];
            int row, col;
            if (!row_of(c, e, o, row, col)) continue;
            if (p.residual) {  // eager semantics: linear output rounded to bf16, then added to the bf16 residual
              const uint4 r4 = *reinterpret_cast<const uint4*>(p.residual + (size_t)row * p.N + col);
              const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(bf16lo(o[j]) + bf16lo(rw[j]), bf16hi(o[j]) + bf16hi(rw[j]));
            }
            *reinterpret_cast<uint4*>(p.C + (size_t)row * p.N + col) = make_uint4(o[0], o[1], o[2], o[3]);
          }
      } else {  // N % 4 == 0: four columns or eight
#pragma unroll
        for (int c = 0; c < PIECES; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint32_t o[G];
            int row, col;
            if (!row_of(c, e, o, row, col)) continue;
            bf16* crow = p.C + (size_t)row * p.N + col;
            const bf16* rrow = p.residual ? p.residual + (size_t)row * p.N + col : nullptr;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + 2 * j < p.N) {
                float lo = bf16lo(o[j]), hi = bf16hi(o[j]);
                if (rrow) { lo += __bfloat162float(rrow[2 * j]); hi += __bfloat162float(rrow[2 * j + 1]); }
                crow[2 * j] = __float2bfloat16_rn(lo);
                crow[2 * j + 1] = __float2bfloat16_rn(hi);
              }
          }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 3) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
  hop_signal(p.signal, p.ctx);
}

template <bool GATED, bool SHARED>
static int launch_fp8(const Fp8GemmParams& p, int tiles, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)F8_STAGES * (F8_BM + F8_BN) * F8_BK + (size_t)F8_SLOTS * (F8_BM + F8_BN) * 4 + 512;
  cudaError_t e = cudaFuncSetAttribute(gemm_fp8_kernel<GATED, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  if constexpr (!SHARED) {
    gemm_fp8_kernel<GATED, false><<<dim3(min(tiles, device_sm_count())), F8_THREADS, smem, stream>>>(p);
    return (int)cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.shares);
  cfg.blockDim = dim3(F8_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.shares;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, gemm_fp8_kernel<GATED, SHARED>, p);
}

// ---- activation quantiser: bf16 rows -> e4m3 + one fp32 scale per 128 K elements (stored transposed) -----------
// A half warp per K block: 8 elements per lane in one 16-byte load, two blocks in flight per half warp, amax by shuffle, scale =
// amax / 448.  Bound by memory latency: 5.8 us a launch over prompts of 1024 rows (6.0 with one block in flight per warp).  Rows from
// M to ld_s get scale zero here, so that the table needs no fill of its own (a launch of 1.6 us and its gap before every
// matrix product: two layers at 1024 rows went from 1248 to 1214 us).
__device__ __forceinline__ void quantize_block(const uint4& raw, unsigned char* q, float* scale_t, bool first) {
  const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
  float v[8], amax = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = bf16lo(r[j]);
    v[2 * j + 1] = bf16hi(r[j]);
    amax = fmaxf(amax, fmaxf(fabsf(v[2 * j]), fabsf(v[2 * j + 1])));
  }
#pragma unroll
  for (int o = 8; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = amax > 0.f ? amax * (1.f / 448.f) : 1.f;
  const float inv = 1.f / scale;
  uint32_t packed[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const __nv_fp8_storage_t b = __nv_cvt_float_to_fp8(v[j] * inv, __NV_SATFINITE, __NV_E4M3);
    packed[j >> 2] |= (uint32_t)b << (8 * (j & 3));
  }
  *reinterpret_cast<uint2*>(q) = make_uint2(packed[0], packed[1]);
  if (first) *scale_t = scale;
}
__global__ void __launch_bounds__(256) quantize_rows_fp8_kernel(const bf16* __restrict__ x, unsigned char* __restrict__ q,
                                                                float* __restrict__ scale_t, int M, int K, long long ld_s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 15;
  const int row = blockIdx.x;
  const int nkb = K / 128;
  if (row >= M) {
    for (int kb = threadIdx.x; kb < nkb; kb += 256) scale_t[(size_t)kb * ld_s + row] = 0.f;
    return;
  }
  const bf16* xr = x + (size_t)row * K + sub * 8;
  unsigned char* qr = q + (size_t)row * K + sub * 8;
  float* sr = scale_t + row;
  const bool wide = ((uintptr_t)x & 15) == 0;  // a view may start on 8 bytes only
  auto load = [&](int kb) {
    const bf16* p = xr + (size_t)kb * 128;
    if (wide) return *reinterpret_cast<const uint4*>(p);
    const uint2 lo = *reinterpret_cast<const uint2*>(p), hi = *reinterpret_cast<const uint2*>(p + 4);
    return make_uint4(lo.x, lo.y, hi.x, hi.y);
  };
  // a warp takes blocks b, b + 1 (one per half) and b + 16, b + 17; the exchange is by whole warps, so behind an odd last block the
  // upper half repeats it (the same values to the same place)
  for (int b = warp * 2; b < nkb; b += 32) {
    const int half = lane >> 4, k0 = min(b + half, nkb - 1), k1 = min(b + 16 + half, nkb - 1);
    const bool two = b + 16 < nkb;
    const uint4 r0 = load(k0);
    uint4 r1 = r0;
    if (two) r1 = load(k1);
    quantize_block(r0, qr + (size_t)k0 * 128, sr + (size_t)k0 * ld_s, sub == 0);
    if (two) quantize_block(r1, qr + (size_t)k1 * 128, sr + (size_t)k1 * ld_s, sub == 0);
  }
}

// 2-D uint8 row-major [rows, cols] tensor, box = [box_rows, 128 bytes], 128-byte swizzle
static inline int make_map_u8(CUtensorMap* map, const void* ptr, long long rows, int cols, int box_rows) {
  PFN_encodeTiled enc = get_encode_fn();
  if (!enc) return -5;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols};
  cuuint32_t box[2] = {128u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -6;
}

static int fp8_tiles(int M, int N, bool gated) {
  const int out_n = gated ? F8_BN / 2 : F8_BN;
  return ((M + F8_BM - 1) / F8_BM) * ((N + out_n - 1) / out_n);
}
// Tiles that would leave most SMs idle share their K blocks, each of which is a step of a serial chain: four CTAs to a tile up to 32
// tiles, two up to 64 (clusters of other sizes and more of them do not all fit at once: 16 tiles by eight 25 us, by four 14, K = 5632).
// us alone and shared: 4096 x 14336 with up to 128 rows 43 and 23, to 256 rows 44 and 31; 2048 x 5632 20 and 14; of 4096 columns 16.3 and 15.2; with
// 2048 columns, and by two with 4096, the exchange costs what it saves.
static int fp8_shares(int tiles, int blocks) {
  const int room = device_sm_count() - 20;
  return 4 * tiles <= room && blocks >= 32 ? 4 : 2 * tiles <= room && blocks >= 40 ? 2 : 1;
}

}  // namespace mdi

using namespace mdi;

// C[M,N] (bf16) = blockscaled(A8, a_scale_t) x blockscaled(W8, w_scale_t)^T (+bias)(+residual); with W2: gated MLP.
// K must be a multiple of 128.  signal_flag != null: fused prefill hop (epilogue stores go to peer memory).
extern "C" int mdi_gemm_fp8(const void* A8, const float* a_scale_t, long long ld_as, const void* W8, const float* w_scale_t,
                            const void* W2_8, const float* w2_scale_t, void* C, const void* bias, const void* bias2,
                            const void* residual, int M, int N, int K, int act, int* signal_flag, unsigned int* done_ctr,
                            const int* ctx, const int* status, cudaStream_t stream) {
  if (K % 128 != 0 || M <= 0 || N <= 0) return -2;
  const bool gated = W2_8 != nullptr;
  if (gated && residual) return -2;
  if (signal_flag && (!done_ctr || !ctx)) return -2;
  if (N % 4 != 0 || ld_as % 4 != 0 || ld_as < M) return -2;  // scale rows are fetched with 16-byte bulk copies
  Fp8GemmParams p;
  p.a_scale_t = a_scale_t; p.w_scale_t = w_scale_t; p.w2_scale_t = w2_scale_t; p.ld_as = ld_as;
  p.C = (bf16*)C; p.bias = (const bf16*)bias; p.bias2 = (const bf16*)bias2; p.residual = (const bf16*)residual;
  p.M = M; p.N = N; p.K = K; p.act = act;
  p.signal = HopSignal{signal_flag, done_ctr, status}; p.ctx = ctx;
  int rc = make_map_u8(&p.tma_a, A8, M, K, F8_BM);
  if (rc) return rc;
  rc = make_map_u8(&p.tma_b, W8, N, K, gated ? F8_BN / 2 : F8_BN);
  if (rc) return rc;
  rc = make_map_u8(&p.tma_b2, gated ? W2_8 : W8, N, K, gated ? F8_BN / 2 : F8_BN);
  if (rc) return rc;
  const int tiles = fp8_tiles(M, N, gated);
  p.shares = fp8_shares(tiles, K / F8_BK);
  if (p.shares > 1) return gated ? launch_fp8<true, true>(p, tiles, stream) : launch_fp8<false, true>(p, tiles, stream);
  return gated ? launch_fp8<true, false>(p, tiles, stream) : launch_fp8<false, false>(p, tiles, stream);
}

// How many CTAs share the K blocks of a tile of this product.
extern "C" int mdi_gemm_fp8_shares(int M, int N, int K, int gated) { return fp8_shares(fp8_tiles(M, N, gated != 0), K / F8_BK); }

// x [M, K] bf16 -> q [M, K] e4m3 + scale_t [K/128, ld_s] fp32 (ld_s >= M; every entry is written)
extern "C" int mdi_quantize_rows_fp8(const void* x, void* q, float* scale_t, int M, int K, long long ld_s, cudaStream_t stream) {
  if (K % 128 != 0 || M <= 0 || ld_s < M) return -2;
  quantize_rows_fp8_kernel<<<(unsigned)ld_s, 256, 0, stream>>>((const bf16*)x, (unsigned char*)q, scale_t, M, K, ld_s);
  return (int)cudaGetLastError();
}
