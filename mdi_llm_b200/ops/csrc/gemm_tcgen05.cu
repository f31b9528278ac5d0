// bf16 GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), hand-written for sm_100a.
//
//   C[M, N] = A[M, K] · W[N, K]^T  (+ bias[N]) (+ residual[M, N])        bf16 in, fp32 accumulate
//
// This is the prefill path (T = prompt length rows through every linear of a stage), where the work is
// GEMM-shaped; decode (T = 1) is bandwidth-bound and uses the weight-streaming kernels in decode_linear.cu instead.
//
// Structure (one 128 x BLOCK_N output tile per CTA, warp-specialised, a ring of 4 to 8 TMA stages):
//   warp 0      : TMA producer — cp.async.bulk.tensor loads of the A and W tiles (64-element = 128 B
//                 K slabs, SWIZZLE_128B) into shared memory, completion on "full" mbarriers;
//   warp 1      : MMA issuer — one elected thread issues tcgen05.mma (M=128, N=BLOCK_N, K=16) from
//                 shared-memory descriptors into a TMEM accumulator; tcgen05.commit releases the
//                 stage ("empty" mbarrier) and finally signals the epilogue;
//   warp 2      : TMEM allocator / deallocator;
//   warps 4..7  : epilogue — tcgen05.ld (32 lanes x 32 columns per warp), bias/residual, bf16 store.
//
// Both operands are K-major (row-major with K contiguous), i.e. activations [T, C] and nn.Linear
// weights [out, in] are consumed as stored; out-of-range rows of the last M/N tile are zero-filled
// by TMA on load and masked on store.
#include <type_traits>

#include "tcgen05.cuh"

namespace mdi {

constexpr int GEMM_BLOCK_M = 128;
constexpr int GEMM_BLOCK_K = 64;  // 64 bf16 = 128 bytes = one swizzle atom row
constexpr int GEMM_THREADS = 256;
constexpr int UMMA_K = 16;

struct GemmParams {
  CUtensorMap tma_a;
  CUtensorMap tma_b;
  CUtensorMap tma_b2;         // gated mode: second weight matrix (same shape as B)
  bf16* C;                     // may be peer-mapped memory: the epilogue's stores ARE the prefill hop
  const bf16* bias;
  const bf16* bias2;
  const bf16* residual;
  int M, N, K;
  int act;                     // gated mode (ACT_*): C = act(A W^T + bias) * (A W2^T + bias2)
  int shares;                  // CTAs of a cluster that share a tile's K range (1: no cluster)
  // fused hop: after its stores every CTA takes a ticket; the last one publishes flag[slot] = signal
  // (values from ctx, like the decode kernels) with a system-scope release.
  HopSignal signal;
  const int* ctx;
  // descriptor knobs (kept as parameters so a bring-up test can sweep them; defaults are the
  // canonical K-major SWIZZLE_128B encoding)
  unsigned int desc_sbo;      // stride-byte-offset >> 4 (8 rows x 128 B = 1024 B -> 64)
  unsigned int desc_lbo;      // leading-byte-offset >> 4 (ignored for swizzled K-major; 1)
  unsigned int desc_hi_bits;  // bits [46..63] >> 32 shifted: version (bit 46) | layout type (bits 61-63)
  unsigned int k_step_bytes;  // start-address advance per UMMA_K (16 bf16 = 32 B)
};

// shared-memory matrix descriptor without its start address (bits [0,14)): K-major, SWIZZLE_128B (cute::UMMA::SmemDescriptor bit layout)
__device__ __forceinline__ uint64_t smem_desc_encoding(const GemmParams& p) {
  uint64_t d = (uint64_t)(p.desc_lbo & 0x3FFF) << 16;    // leading byte offset, bits [16,30)
  d |= (uint64_t)(p.desc_sbo & 0x3FFF) << 32;             // stride byte offset, bits [32,46)
  d |= (uint64_t)p.desc_hi_bits << 46;                    // version (bit 46) ... layout type (bits 61-63)
  return d;
}

// GATED: two B operands share the A tile; accumulators live side by side in TMEM (columns [0,BLOCK_N)
// and [BLOCK_N, 2*BLOCK_N)) and the epilogue writes act(acc0) * acc1 — SwiGLU / GeGLU in one pass.
//
// Persistent: one CTA per SM walks the tile list (m fastest, so the CTAs that run together share B tiles
// through L2).  The accumulator is double-buffered in TMEM: while the epilogue warps drain tile i
// (tcgen05.ld -> bias/act/residual -> 16-byte stores), the MMA warp is already accumulating tile i+1 in
// the other buffer and the TMA warp keeps the shared-memory ring full across tile boundaries.
//
// SHARED: the CTAs of a cluster share the K range of one tile.  When their products are done, every CTA takes the column groups that are
// its own, adds the others' sums of them (sent to its shared memory, over the stages) and finishes them.
//
// ROWS: 64 where A has no more.  The MMA reads 128 either way, the upper half of them whatever lies behind (the next stage, or W's tiles:
// sums of rows that do not exist and are not read), so a stage is 8 KB smaller and there are more of them: a product of few tiles waits for its
// loads, 3000 to 3700 cycles for as many K blocks as there are stages.  us, 4 stages of 128 rows and the exchange
// below it as it was, and now, 62 rows: 4096 x 14336 47 and 37, 4096 x 4096 24.6 and 19.5, 2048 x 2048 18.5 and 14.4, 2 x 5632 x 2048 25.7 and 21.5 (without the gap of two
// events); 200 rows 4096 x 14336 59 and 51.
template <int BLOCK_N, bool GATED, int ROWS>
struct GemmTile {
  static constexpr int A_BYTES = ROWS * GEMM_BLOCK_K * 2, B_BYTES = (GATED ? 2 : 1) * BLOCK_N * GEMM_BLOCK_K * 2;
  static constexpr int STAGES = 200 * 1024 / (A_BYTES + B_BYTES) < 8 ? 200 * 1024 / (A_BYTES + B_BYTES) : 8;
  static constexpr size_t SMEM = 1024 + (size_t)STAGES * (A_BYTES + B_BYTES) + 256;
  static_assert(STAGES * B_BYTES >= GEMM_BLOCK_M * GEMM_BLOCK_K * 2, "the last stage of A reads past its own rows");
};
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&f)[8]) {  // 32 lanes x 8 columns
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void lds8(uint32_t addr, float (&f)[8]) {  // two halves of 128 rows x 16 bytes
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(addr) : "memory");
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "r"(addr + 2048) : "memory");
}

template <int BLOCK_N, bool GATED, bool SHARED, int ROWS>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_bf16_tcgen05_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) unsigned char gemm_smem[];
  using Tile = GemmTile<BLOCK_N, GATED, ROWS>;
  constexpr int A_BYTES = Tile::A_BYTES, B_BYTES = Tile::B_BYTES, GEMM_STAGES = Tile::STAGES;
  constexpr int ACC_COLS = (GATED ? 2 : 1) * BLOCK_N;  // TMEM columns of one accumulator buffer
  constexpr int TMEM_COLS = 2 * ACC_COLS;              // two buffers (power of two, <= 512)
  static_assert(TMEM_COLS <= 512, "accumulators exceed TMEM");
  // carve: [A stages][B stages][barriers][tmem ptr]
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* smem_a = base;
  unsigned char* smem_b = base + GEMM_STAGES * A_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_b + GEMM_STAGES * B_BYTES);
  uint64_t* empty_bar = full_bar + GEMM_STAGES;
  uint64_t* tmem_full_bar = empty_bar + GEMM_STAGES;  // [2]
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;        // [2]
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles_m = (p.M + GEMM_BLOCK_M - 1) / GEMM_BLOCK_M;
  const int tiles_n = (p.N + BLOCK_N - 1) / BLOCK_N;
  const int n_tiles = tiles_m * tiles_n;
  const int S = SHARED ? p.shares : 1, rank = SHARED ? (int)cluster_ctarank() : 0, all_k_blocks = (p.K + GEMM_BLOCK_K - 1) / GEMM_BLOCK_K;
  const int kb0 = SHARED ? rank * all_k_blocks / S : 0, num_k_blocks = SHARED ? (rank + 1) * all_k_blocks / S - kb0 : all_k_blocks;

  auto load = [&](int s, int kb, int m0, int n0) {
    mbar_expect_tx(&full_bar[s], A_BYTES + B_BYTES);
    tma_load_2d(smem_a + s * A_BYTES, &p.tma_a, &full_bar[s], (kb0 + kb) * GEMM_BLOCK_K, m0);
    tma_load_2d(smem_b + s * B_BYTES, &p.tma_b, &full_bar[s], (kb0 + kb) * GEMM_BLOCK_K, n0);
    if (GATED) tma_load_2d(smem_b + s * B_BYTES + B_BYTES / 2, &p.tma_b2, &full_bar[s], (kb0 + kb) * GEMM_BLOCK_K, n0);
  };
  const int first_tile = SHARED ? blockIdx.x / S : blockIdx.x, step = SHARED ? gridDim.x / S : gridDim.x;
  const int early = first_tile < n_tiles ? min(GEMM_STAGES, num_k_blocks) : 0;
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < GEMM_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full_bar[b], 1); mbar_init(&tmem_empty_bar[b], 4); }
    mbar_fence_init();
    fence_proxy_async_smem();
    // the first loads do not wait for the allocation of TMEM (1000 cycles)
    for (int kb = 0; kb < early; ++kb) load(kb, kb, (first_tile % tiles_m) * GEMM_BLOCK_M, (first_tile / tiles_m) * BLOCK_N);
  }
  if (warp == 2) {  // whole warp: allocate both accumulator buffers
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);

  if (warp == 0) {
    // ===== TMA producer: the ring runs straight through tile boundaries =====
    if (lane == 0) {
      int it = 0;
      for (int tile = first_tile; tile < n_tiles; tile += step) {
        const int m0 = (tile % tiles_m) * GEMM_BLOCK_M, n0 = (tile / tiles_m) * BLOCK_N;
        for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
          if (it < early) continue;
          mbar_wait(&empty_bar[it % GEMM_STAGES], ((it / GEMM_STAGES) & 1) ^ 1);
          load(it % GEMM_STAGES, kb, m0, n0);
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer =====
    // instruction descriptor (cute::UMMA::InstrDescriptor): fp32 accumulate, bf16 x bf16, both K-major
    const uint64_t encoding = smem_desc_encoding(p);
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BLOCK_N >> 3) << 17) | ((uint32_t)(GEMM_BLOCK_M >> 4) << 24);
    int it = 0, lt = 0;
    for (int tile = first_tile; tile < n_tiles; tile += step, ++lt) {
      const int acc = lt & 1;
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * ACC_COLS);
      mbar_wait(&tmem_empty_bar[acc], ((lt >> 1) & 1) ^ 1);  // the epilogue has drained this buffer
      tcgen05_fence_after();
      for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
        const int s = it % GEMM_STAGES;
        const uint32_t phase = (it / GEMM_STAGES) & 1;
        mbar_wait(&full_bar[s], phase);
        tcgen05_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = smem_u32(smem_a + s * A_BYTES), b_addr = smem_u32(smem_b + s * B_BYTES);
          auto desc = [&](uint32_t addr) { return encoding | (uint64_t)((addr >> 4) & 0x3FFF); };
#pragma unroll
          for (int k = 0; k < GEMM_BLOCK_K / UMMA_K; ++k) {
            const uint64_t da = desc(a_addr + k * p.k_step_bytes), db = desc(b_addr + k * p.k_step_bytes);
            tcgen05_mma_f16(tmem_acc, da, db, idesc, (kb | k) ? 1u : 0u);
            if (GATED) tcgen05_mma_f16(tmem_acc + BLOCK_N, da, desc(b_addr + B_BYTES / 2 + k * p.k_step_bytes), idesc, (kb | k) ? 1u : 0u);
          }
          tcgen05_commit(&empty_bar[s]);                            // stage reusable once these MMAs retire
          if (kb == num_k_blocks - 1) tcgen05_commit(&tmem_full_bar[acc]);  // accumulator complete
        }
        __syncwarp();
      }
    }
  } else if (warp >= 4) {
    // ===== epilogue: TMEM -> registers -> bf16 global =====
    const int ew = warp - 4;  // TMEM lanes [32*ew, 32*ew + 32) belong to this warp
    const bool vec_ok = (p.N % 8 == 0);
    int lt = 0;
    for (int tile = first_tile; tile < n_tiles; tile += step, ++lt) {
      const int m0 = (tile % tiles_m) * GEMM_BLOCK_M, n0 = (tile / tiles_m) * BLOCK_N;
      const int acc = lt & 1;
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * ACC_COLS) + ((uint32_t)(ew * 32) << 16);
      mbar_wait(&tmem_full_bar[acc], (lt >> 1) & 1);
      if constexpr (SHARED) break;
      tcgen05_fence_after();
      const int row = m0 + ew * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < BLOCK_N; c0 += 32) {
        uint32_t acc_r[32];
        tmem_ld_32x32(tmem_acc + (uint32_t)c0, acc_r);
        const int col0 = n0 + c0;
        if (GATED) {
          uint32_t acc2[32];
          tmem_ld_32x32(tmem_acc + (uint32_t)(BLOCK_N + c0), acc2);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float g = __uint_as_float(acc_r[j]), u = __uint_as_float(acc2[j]);
            if (col0 + j < p.N) {
              if (p.bias) g += __bfloat162float(p.bias[col0 + j]);
              if (p.bias2) u += __bfloat162float(p.bias2[col0 + j]);
            }
            // eager semantics: both projections are rounded to bf16 before the activation and the product
            g = round_bf16(g); u = round_bf16(u);
            acc_r[j] = __float_as_uint(round_bf16(apply_act(g, p.act)) * u);
          }
        }
        if (row < p.M && col0 < p.N) {
          bf16* crow = p.C + (size_t)row * p.N + col0;
          const bf16* rrow = p.residual ? p.residual + (size_t)row * p.N + col0 : nullptr;
          if (vec_ok && col0 + 32 <= p.N) {
            // 4 x 16-byte stores per thread (64 contiguous bytes of one output row): full sectors on the
            // wire when C is peer memory
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                f[j] = __uint_as_float(acc_r[v * 8 + j]);
                if (!GATED && p.bias) f[j] += __bfloat162float(p.bias[col0 + v * 8 + j]);
              }
              if (rrow) {  // eager semantics: linear output rounded to bf16, then added to the bf16 residual
                const uint4 r4 = *reinterpret_cast<const uint4*>(rrow + v * 8);
                const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  f[2 * j] = round_bf16(f[2 * j]) + bf16lo(rw[j]);
                  f[2 * j + 1] = round_bf16(f[2 * j + 1]) + bf16hi(rw[j]);
                }
              }
              uint4 o;
              o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
              o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
              *reinterpret_cast<uint4*>(crow + v * 8) = o;
            }
          } else {
#pragma unroll 1
            for (int j = 0; j < 32 && col0 + j < p.N; ++j) {
              float v0 = __uint_as_float(acc_r[j]);
              if (!GATED && p.bias) v0 += __bfloat162float(p.bias[col0 + j]);
              if (rrow) v0 = round_bf16(v0) + __bfloat162float(rrow[j]);
              crow[j] = __float2bfloat16_rn(v0);
            }
          }
        }
      }
      // this warp is done reading the buffer: hand it back to the MMA warp (4 arrivals = 4 epilogue warps)
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar[acc]);
    }
  }
  if constexpr (SHARED) {
    constexpr int OG = BLOCK_N / 8, OPS = GATED ? 2 : 1;  // groups of eight output columns; accumulators of each
    const int most = (OG + S - 1) / S, tile = blockIdx.x / S, n0 = (tile / tiles_m) * BLOCK_N, r = (warp & 3) * 32 + lane;
    const int row = (tile % tiles_m) * GEMM_BLOCK_M + r;
    const uint32_t place = smem_u32(smem_a), at_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    // (the other tiles store fewer than 32 columns one by one, so rows may start anywhere then)
    const bool wide = p.N % 8 == 0 && (((uintptr_t)p.C | (uintptr_t)p.residual) & 15) == 0;
    auto at = [&](int from, int to, int og, int op) {  // [S - 1 senders][accumulator][own groups][2][128 rows][4 columns]
      const int slot = from < to ? from : from - 1;
      return place + (uint32_t)(((slot * OPS + op) * most + og - (to * OG + S - 1) / S) * 4096 + r * 16);
    };
    // Two halves of 16 bytes a row, a warp's rows one behind the other: with the 32 bytes of a row together the sends took 7500 cycles of 128
    // CTAs' 35,000 (62 rows, 4096 x 4096).  Warps without rows send nothing.  A thread's own groups lie side by side, whole sectors of C.
    const bool any = row - lane < p.M;
    const int own = OG / S, og0 = rank * own + (warp >> 2) * (own / 2);
    static_assert(OG == 16, "own groups of two or four CTAs");
    __syncwarp();
    tcgen05_fence_before();
    cluster_sync_all();  // everybody's products are done: the stages are free
    tcgen05_fence_after();
    for (int og = warp >> 2; og < OG; og += 2) {
      const int to = og * S / OG;
      if (to == rank || !any) continue;
#pragma unroll
      for (int op = 0; op < OPS; ++op) {
        float f[8];
        tmem_ld8(at_row + (uint32_t)(op * BLOCK_N + og * 8), f);
        const uint32_t d = cluster_addr(at(rank, to, og, op), to);
        st_cluster(d, f[0], f[1], f[2], f[3]);
        st_cluster(d + 2048, f[4], f[5], f[6], f[7]);
      }
    }
    const bool here = row < p.M;
    uint4 res[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (!GATED && p.residual && wide && here && i < own / 2 && n0 + (og0 + i) * 8 + 8 <= p.N)
        res[i] = *reinterpret_cast<const uint4*>(p.residual + (size_t)row * p.N + n0 + (og0 + i) * 8);
    cluster_sync_all();
    // (gated: four copies of the code of every activation took 10 us more than one, 100 rows of 2 x 5632 x 2048)
#pragma unroll (GATED ? 1 : 4)
    for (int i = 0; i < 4; ++i) {
      const int og = og0 + i;
      if (i >= own / 2 || !any) continue;
      __syncwarp();  // (rows behind the last one leave an iteration early)
      float f[OPS][8];
#pragma unroll
      for (int op = 0; op < OPS; ++op) {
        tmem_ld8(at_row + (uint32_t)(op * BLOCK_N + og * 8), f[op]);
        for (int from = 0; from < S; ++from)
          if (from != rank) {
            float v[8];
            lds8(at(from, rank, og, op), v);
#pragma unroll
            for (int j = 0; j < 8; ++j) f[op][j] += v[j];
          }
      }
      const int col0 = n0 + og * 8;
      if (row >= p.M) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (col0 + j >= p.N) continue;
        if (p.bias) f[0][j] += __bfloat162float(p.bias[col0 + j]);
        if (GATED) {
          if (p.bias2) f[OPS - 1][j] += __bfloat162float(p.bias2[col0 + j]);
          f[0][j] = round_bf16(apply_act(round_bf16(f[0][j]), p.act)) * round_bf16(f[OPS - 1][j]);
        }
      }
      bf16* crow = p.C + (size_t)row * p.N + col0;
      const bf16* rrow = p.residual ? p.residual + (size_t)row * p.N + col0 : nullptr;
      if (wide && col0 + 8 <= p.N) {
        if (!GATED && rrow) {  // eager semantics: linear output rounded to bf16, then added to the bf16 residual
          const uint32_t rw[4] = {res[i].x, res[i].y, res[i].z, res[i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f[0][2 * j] = round_bf16(f[0][2 * j]) + bf16lo(rw[j]);
            f[0][2 * j + 1] = round_bf16(f[0][2 * j + 1]) + bf16hi(rw[j]);
          }
        }
        *reinterpret_cast<uint4*>(crow) = make_uint4(pack_bf16x2(f[0][0], f[0][1]), pack_bf16x2(f[0][2], f[0][3]),
                                                     pack_bf16x2(f[0][4], f[0][5]), pack_bf16x2(f[0][6], f[0][7]));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (col0 + j < p.N) crow[j] = __float2bfloat16_rn(rrow ? round_bf16(f[0][j]) + __bfloat162float(rrow[j]) : f[0][j]);
      }
    }
    __syncwarp();
    tcgen05_fence_before();
  }
  __syncthreads();
  if (warp == 2) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
  hop_signal(p.signal, p.ctx);  // the __syncthreads above ordered every epilogue store before the ticket
}

// ---- CTA-pair variant: tcgen05.mma.cta_group::2 -----------------------------------------------------------------
// Two CTAs of a cluster (same TPC) work on ONE 256 x BLOCK_N output tile: rank r owns rows [128 r, 128 r + 128) and loads
// its own A rows plus HALF of the B tile (BLOCK_N / 2 weight rows); the leader CTA issues M = 256 MMAs that read both
// CTAs' shared memory, every CTA's TMEM receives the accumulators of its own 128 rows.  Per CTA and K block that is
// 16 KB (A) + 16 KB (B half) for a 128 x 256 share of the output instead of 16 + 32 KB: a third less shared-memory
// fill and L2 traffic per FLOP, and the tensor core is fed M = 256.
//   * "full" barriers live in the leader; both CTAs' TMA loads complete on them (cp.async.bulk.tensor ... cta_group::2)
//   * "empty" / "accumulator full" barriers exist in both CTAs; the leader's tcgen05.commit multicasts to the pair
//   * "accumulator drained" lives in the leader; rank 1's epilogue warps arrive remotely (mapa + shared::cluster)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint64_t* leader_bar, int x, int y) {
  // executed by both CTAs; clearing the peer bit makes the transaction bytes land on CTA 0's barrier
  const uint32_t bar = smem_u32(leader_bar) & 0xFEFFFFFFu;
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tcgen05_mma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                     uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tcgen05_commit_pair(uint64_t* bar) {  // arrives on the same barrier in BOTH CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cta(uint64_t* bar, uint32_t cta) {  // arrive on `bar` of CTA `cta` of the cluster
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}"
      ::"r"(smem_u32(bar)), "r"(cta) : "memory");
}

// GATED: the 256-column MMA tile is [fc_1 rows n0 .. n0+128 | fc_2 rows n0 .. n0+128] — rank 0 loads the fc_1 half of
// the B tile, rank 1 the fc_2 half — and the epilogue writes act(g) * u for 128 output columns.
constexpr int PAIR_STAGES = 6;  // 6 x (16 KB A + 16 KB B half) = 192 KB of the 227 KB
template <int BLOCK_N, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1) gemm_bf16_tcgen05_pair_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) unsigned char gemm_smem[];
  constexpr int A_BYTES = GEMM_BLOCK_M * GEMM_BLOCK_K * 2;      // this CTA's 128 rows of A
  constexpr int B_BYTES = (BLOCK_N / 2) * GEMM_BLOCK_K * 2;     // this CTA's half of the B tile
  constexpr int TMEM_COLS = BLOCK_N > 128 ? 512 : 256;          // two accumulator buffers (a power of two)
  static_assert(TMEM_COLS <= 512 && BLOCK_N % 32 == 0, "accumulators exceed TMEM");
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* smem_a = base;
  unsigned char* smem_b = base + PAIR_STAGES * A_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_b + PAIR_STAGES * B_BYTES);  // used in the leader
  uint64_t* empty_bar = full_bar + PAIR_STAGES;                                       // both CTAs (multicast commit)
  uint64_t* tmem_full_bar = empty_bar + PAIR_STAGES;                                  // [2] both CTAs
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;                                       // [2] leader: 8 epilogue warps of the pair
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  constexpr int OUT_N = GATED ? BLOCK_N / 2 : BLOCK_N;  // output columns per tile
  const int tiles_m = (p.M + 2 * GEMM_BLOCK_M - 1) / (2 * GEMM_BLOCK_M);
  const int tiles_n = (p.N + OUT_N - 1) / OUT_N;
  const int n_tiles = tiles_m * tiles_n;
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int num_k_blocks = (p.K + GEMM_BLOCK_K - 1) / GEMM_BLOCK_K;

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_b) : "memory");
    if (GATED) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.tma_b2) : "memory");
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full_bar[b], 1); mbar_init(&tmem_empty_bar[b], 8); }
    mbar_fence_init();
  }
  if (warp == 2) {  // same warp in both CTAs: the allocation is collective over the pair
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  cluster_sync_all();  // barriers of BOTH CTAs are initialised before any remote arrive / multicast commit
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);

  if (warp == 0) {
    // ===== TMA producer (both CTAs): own A rows + own half of B, completing on the leader's barrier =====
    if (lane == 0) {
      int it = 0;
      for (int tile = pair; tile < n_tiles; tile += n_pairs) {
        const int m0 = (tile % tiles_m) * 2 * GEMM_BLOCK_M + (int)rank * GEMM_BLOCK_M, nt = tile / tiles_m;
        const int n0 = GATED ? nt * OUT_N : nt * BLOCK_N + (int)rank * (BLOCK_N / 2);
        const CUtensorMap* map_b = (GATED && rank == 1) ? &p.tma_b2 : &p.tma_b;
        for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
          const int s = it % PAIR_STAGES;
          mbar_wait(&empty_bar[s], ((it / PAIR_STAGES) & 1) ^ 1);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * (A_BYTES + B_BYTES));  // bytes of the whole pair
          tma_load_2d_pair(smem_a + s * A_BYTES, &p.tma_a, &full_bar[s], kb * GEMM_BLOCK_K, m0);
          tma_load_2d_pair(smem_b + s * B_BYTES, map_b, &full_bar[s], kb * GEMM_BLOCK_K, n0);
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ===== MMA issuer (leader only): M = 256 over the pair =====
    const uint32_t idesc = umma_idesc_bf16(2 * GEMM_BLOCK_M, BLOCK_N);
    int it = 0, lt = 0;
    for (int tile = pair; tile < n_tiles; tile += n_pairs, ++lt) {
      const int acc = lt & 1;
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * BLOCK_N);
      mbar_wait(&tmem_empty_bar[acc], ((lt >> 1) & 1) ^ 1);  // both CTAs' epilogues have drained this buffer
      tcgen05_fence_after();
      for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
        const int s = it % PAIR_STAGES;
        mbar_wait(&full_bar[s], (it / PAIR_STAGES) & 1);
        tcgen05_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = smem_u32(smem_a + s * A_BYTES), b_addr = smem_u32(smem_b + s * B_BYTES);
#pragma unroll
          for (int k = 0; k < GEMM_BLOCK_K / UMMA_K; ++k)
            tcgen05_mma_f16_pair(tmem_acc, umma_desc_sw128(a_addr + k * 32), umma_desc_sw128(b_addr + k * 32), idesc, (kb | k) ? 1u : 0u);
          tcgen05_commit_pair(&empty_bar[s]);
          if (kb == num_k_blocks - 1) tcgen05_commit_pair(&tmem_full_bar[acc]);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 4) {
    // ===== epilogue (both CTAs): own 128 rows =====
    const int ew = warp - 4;
    const bool vec_ok = (p.N % 8 == 0);
    int lt = 0;
    for (int tile = pair; tile < n_tiles; tile += n_pairs, ++lt) {
      const int m0 = (tile % tiles_m) * 2 * GEMM_BLOCK_M + (int)rank * GEMM_BLOCK_M, n0 = tile / tiles_m * OUT_N;
      const int acc = lt & 1;
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * BLOCK_N) + ((uint32_t)(ew * 32) << 16);
      mbar_wait(&tmem_full_bar[acc], (lt >> 1) & 1);
      tcgen05_fence_after();
      const int row = m0 + ew * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < OUT_N; c0 += 32) {
        uint32_t acc_r[32];
        tmem_ld_32x32(tmem_acc + (uint32_t)c0, acc_r);
        const int col0 = n0 + c0;
        if (GATED) {
          uint32_t acc2[32];
          tmem_ld_32x32(tmem_acc + (uint32_t)(OUT_N + c0), acc2);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float g = __uint_as_float(acc_r[j]), u = __uint_as_float(acc2[j]);
            if (col0 + j < p.N) {
              if (p.bias) g += __bfloat162float(p.bias[col0 + j]);
              if (p.bias2) u += __bfloat162float(p.bias2[col0 + j]);
            }
            g = round_bf16(g); u = round_bf16(u);
            acc_r[j] = __float_as_uint(round_bf16(apply_act(g, p.act)) * u);
          }
        }
        if (row < p.M && col0 < p.N) {
          bf16* crow = p.C + (size_t)row * p.N + col0;
          const bf16* rrow = p.residual ? p.residual + (size_t)row * p.N + col0 : nullptr;
          if (vec_ok && col0 + 32 <= p.N) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                f[j] = __uint_as_float(acc_r[v * 8 + j]);
                if (!GATED && p.bias) f[j] += __bfloat162float(p.bias[col0 + v * 8 + j]);
              }
              if (rrow) {
                const uint4 r4 = *reinterpret_cast<const uint4*>(rrow + v * 8);
                const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  f[2 * j] = round_bf16(f[2 * j]) + bf16lo(rw[j]);
                  f[2 * j + 1] = round_bf16(f[2 * j + 1]) + bf16hi(rw[j]);
                }
              }
              uint4 o;
              o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
              o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
              *reinterpret_cast<uint4*>(crow + v * 8) = o;
            }
          } else {
#pragma unroll 1
            for (int j = 0; j < 32 && col0 + j < p.N; ++j) {
              float v0 = __uint_as_float(acc_r[j]);
              if (!GATED && p.bias) v0 += __bfloat162float(p.bias[col0 + j]);
              if (rrow) v0 = round_bf16(v0) + __bfloat162float(rrow[j]);
              crow[j] = __float2bfloat16_rn(v0);
            }
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(&tmem_empty_bar[acc], 0);  // the leader's MMA warp waits for all 8 warps of the pair
    }
  }
  tcgen05_fence_before();
  cluster_sync_all();  // nobody leaves while the peer may still touch its barriers / shared memory
  if (warp == 2) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
  hop_signal(p.signal, p.ctx);
}

// ---- a product per group of rows (the experts of a mixture) ---------------------------------------------------------
// The rows of A are sorted by group and group e multiplies them with its own weight; one launch walks the tiles of all groups.  Group sizes
// are read on the device, so the host does not wait for them.
//
// The 256 rows of an MMA are rows of the WEIGHT (rank r holds 128 of them; gated: 64 of W and the same 64 of W2), the rows of A are its columns:
// M is 256 whatever a group holds, N follows it in steps of 32.  With A's rows as M every group cost a multiple of 256 rows, and of ~250 rows
// an expert about every third one took a second tile; now the rows of a group are cut evenly, 262 into two tiles of 160 columns.  us, gate and up +
// down projection of eight experts (14336 x 4096), A's rows as M and now, in turns on one GPU: 38 rows each 488 + 210 and 330 + 165, 96 513 + 226 and
// 347 + 169, 150 445 + 193 and 352 + 169, 224 534 + 232 and 397 + 198, 249 469 + 192 and 394 + 202, 270 928 + 409 and 539 + 282, unequal ones of 997
// tokens (229 to 271) 536 + 220 and 418 + 214.  A launch per expert took 822 + 586 us for 997 tokens.
// What bounds it: from some 200 rows a group the tensor core at the clock that the power limit leaves (1.1 GHz), below that reading the weights (25 a
// group: 322 + 158 us, 5.9 TB/s).  The thread that loads is near the limit too: with a box and a choice between boxes at a time, of 16 or 64 rows, 249 rows
// took 371 + 189 as with one box of 128, but 96 447 + 218, 224 508 + 249 and 270 699 + 345; so rows come in one box or two, with a loop for each width.
// A second tile of 32 columns behind one of 256 instead of two of 160 took 15 % longer at 270 rows a group.  Wide tiles first and the waves over the
// pairs alternately from the left and from the right: a pair that got a wide tile gets a narrow one next.
// Accumulator lanes are output columns: a store writes 32 of one row, 64 bytes.  Gated, lanes 0-63 hold W's sums and 64-127 W2's: of every 32
// columns two of the four warps hand theirs, rounded to bf16 as the eager module does anyway, to the other two through shared memory, in turns.
constexpr int GROUPS = 8;  // weights per launch (their tensor maps are kernel arguments); more groups take more launches
constexpr int GROUP_ROWS = 256;
struct GroupedParams {
  CUtensorMap a[4];  // boxes of 16, 32, 64 and 128 rows
  CUtensorMap b[GROUPS], b2[GROUPS];
  bf16* C;
  const int* counts;  // rows per group, from the first group of the call
  int first, groups;  // this launch's groups
  int M, N, K, act;
};
struct GroupTiles {  // in the order of the tiles: group, first row, rows, width of its tiles, tiles before
  int e[GROUPS], row[GROUPS], rows[GROUPS], width[GROUPS], tile[GROUPS + 1];
};

template <bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1) gemm_grouped_tcgen05_kernel(const __grid_constant__ GroupedParams p) {
  extern __shared__ __align__(1024) unsigned char gemm_smem[];
  constexpr int W_BYTES = GEMM_BLOCK_M * GEMM_BLOCK_K * 2;  // this CTA's 128 rows of the weights
  constexpr int R_BYTES = GROUP_ROWS / 2 * GEMM_BLOCK_K * 2;  // this CTA's half of the rows of A, at most
  constexpr int OUT_N = GATED ? 128 : 256, OWN = OUT_N / 2;  // output columns of a tile and of this CTA
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~uintptr_t(1023));
  unsigned char* smem_w = base;
  unsigned char* smem_r = base + PAIR_STAGES * W_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_r + PAIR_STAGES * R_BYTES);  // used in the leader
  uint64_t* empty_bar = full_bar + PAIR_STAGES;                                       // both CTAs (multicast commit)
  uint64_t* tmem_full_bar = empty_bar + PAIR_STAGES;                                  // [2] both CTAs
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;                                       // [2] leader: 8 epilogue warps of the pair
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  __shared__ GroupTiles gt;
  __shared__ bf16 handed[GATED ? 2 : 1][32][64];  // [chunk & 1][row of A][output column]

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int num_k_blocks = (p.K + GEMM_BLOCK_K - 1) / GEMM_BLOCK_K;

  if (warp == 0 && lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&p.a[2]) : "memory");
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full_bar[b], 1); mbar_init(&tmem_empty_bar[b], 8); }
    mbar_fence_init();
  }
  if (warp == 2) {  // same warp in both CTAs: the allocation is collective over the pair
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr_smem)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == 3) {  // the tiles: a lane a group, the wider ones first
    int before = 0;
    for (int i = lane; i < p.first; i += 32) before += p.counts[i];
    before = __reduce_add_sync(0xffffffffu, before);
    const int n = lane < p.groups ? p.counts[p.first + lane] : 0;
    const int t = (n + GROUP_ROWS - 1) / GROUP_ROWS, w = t ? ((n + t - 1) / t + 31) & ~31 : 0;
    int slot = 0, row = before;
    for (int i = 0; i < GROUPS; ++i) {
      const int wi = __shfl_sync(0xffffffffu, w, i), ni = __shfl_sync(0xffffffffu, n, i);
      slot += wi > w || (wi == w && i < lane);
      row += i < lane ? ni : 0;
    }
    if (lane < GROUPS) { gt.e[slot] = lane; gt.row[slot] = row; gt.rows[slot] = n; gt.width[slot] = w; gt.tile[slot + 1] = t; }
    __syncwarp();
    if (lane == 0) {
      gt.tile[0] = 0;
      for (int i = 0; i < GROUPS; ++i) gt.tile[i + 1] = gt.tile[i] + gt.tile[i + 1] * ((p.N + OUT_N - 1) / OUT_N);
    }
  }
  tcgen05_fence_before();
  cluster_sync_all();  // barriers of BOTH CTAs are initialised before any remote arrive / multicast commit
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_smem, 0);
  const int n_tiles = gt.tile[GROUPS];

  // each(slot, first row, rows, width, output column of this CTA) over this pair's tiles
  auto walk = [&](auto&& each) {
    for (int wave = 0; wave * n_pairs < n_tiles; ++wave) {
      const int tile = wave * n_pairs + (wave & 1 ? n_pairs - 1 - pair : pair);
      if (tile >= n_tiles) continue;
      int g = 0;
      while (tile >= gt.tile[g + 1]) ++g;
      const int w = gt.width[g], t = (gt.rows[g] + GROUP_ROWS - 1) / GROUP_ROWS, i = tile - gt.tile[g], at = i % t * w;
      each(g, gt.row[g] + at, min(w, gt.rows[g] - at), w, i / t * OUT_N + (int)rank * OWN);
    }
  };

  if (warp == 0) {
    // ===== TMA producer (both CTAs): own rows of the weights + own half of A's rows, completing on the leader's barrier =====
    if (lane == 0) {
      int it = 0;
      walk([&](int g, int row0, int, int w, int n0) {
        const CUtensorMap* map_b = &p.b[gt.e[g]];
        const CUtensorMap* map_b2 = &p.b2[gt.e[g]];
        const int first = row0 + (int)rank * (w / 2);
        // BOX, BOX2: of A's rows, 16 << BOX and behind them 16 << BOX2, or none
        auto load = [&](auto box, auto box2) {
          constexpr int BOX = decltype(box)::value, BOX2 = decltype(box2)::value, TALL = 16 << BOX, ROWS = TALL + (BOX2 < 0 ? 0 : 16 << (BOX2 < 0 ? 0 : BOX2));
          for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
            const int s = it % PAIR_STAGES;
            mbar_wait(&empty_bar[s], ((it / PAIR_STAGES) & 1) ^ 1);
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * W_BYTES + 2 * ROWS * GEMM_BLOCK_K * 2);  // bytes of the whole pair
            tma_load_2d_pair(smem_w + s * W_BYTES, map_b, &full_bar[s], kb * GEMM_BLOCK_K, n0);
            if (GATED) tma_load_2d_pair(smem_w + s * W_BYTES + W_BYTES / 2, map_b2, &full_bar[s], kb * GEMM_BLOCK_K, n0);
            tma_load_2d_pair(smem_r + s * R_BYTES, &p.a[BOX], &full_bar[s], kb * GEMM_BLOCK_K, first);
            if (BOX2 >= 0) tma_load_2d_pair(smem_r + s * R_BYTES + TALL * GEMM_BLOCK_K * 2, &p.a[BOX2 < 0 ? 0 : BOX2], &full_bar[s], kb * GEMM_BLOCK_K, first + TALL);
          }
        };
        using std::integral_constant;
        constexpr integral_constant<int, -1> none;
        constexpr integral_constant<int, 0> b16;
        constexpr integral_constant<int, 1> b32;
        constexpr integral_constant<int, 2> b64;
        constexpr integral_constant<int, 3> b128;
        switch (w / 32) {
          case 1: load(b16, none); break;
          case 2: load(b32, none); break;
          case 3: load(b32, b16); break;
          case 4: load(b64, none); break;
          case 5: load(b64, b16); break;
          case 6: load(b64, b32); break;
          default: load(b128, none);  // (224: 16 rows more than are multiplied)
        }
      });
    }
  } else if (warp == 1 && rank == 0) {
    // ===== MMA issuer (leader only): M = 256 over the pair =====
    int it = 0, lt = 0;
    walk([&](int, int, int, int w, int) {
      const uint32_t idesc = umma_idesc_bf16(2 * GEMM_BLOCK_M, w);
      const int acc = lt & 1;
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * GROUP_ROWS);
      mbar_wait(&tmem_empty_bar[acc], ((lt >> 1) & 1) ^ 1);  // both CTAs' epilogues have drained this buffer
      tcgen05_fence_after();
      for (int kb = 0; kb < num_k_blocks; ++kb, ++it) {
        const int s = it % PAIR_STAGES;
        mbar_wait(&full_bar[s], (it / PAIR_STAGES) & 1);
        tcgen05_fence_after();
        if (elect_one()) {
          const uint32_t w_addr = smem_u32(smem_w + s * W_BYTES), r_addr = smem_u32(smem_r + s * R_BYTES);
#pragma unroll
          for (int k = 0; k < GEMM_BLOCK_K / UMMA_K; ++k)
            tcgen05_mma_f16_pair(tmem_acc, umma_desc_sw128(w_addr + k * 32), umma_desc_sw128(r_addr + k * 32), idesc, (kb | k) ? 1u : 0u);
          tcgen05_commit_pair(&empty_bar[s]);
          if (kb == num_k_blocks - 1) tcgen05_commit_pair(&tmem_full_bar[acc]);
        }
        __syncwarp();
      }
      ++lt;
    });
  } else if (warp >= 4) {
    // ===== epilogue (both CTAs): a lane per row of the weights =====
    const int ew = warp - 4, lane_row = ew * 32 + lane;
    int lt = 0, chunk = 0;
    walk([&](int, int row0, int rows, int, int n0) {
      const int acc = lt & 1, col = n0 + (GATED ? lane_row & 63 : lane_row);
      const uint32_t tmem_acc = tmem_base + (uint32_t)(acc * GROUP_ROWS) + ((uint32_t)(ew * 32) << 16);
      mbar_wait(&tmem_full_bar[acc], (lt >> 1) & 1);
      tcgen05_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < rows; c0 += 32, ++chunk) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_acc + (uint32_t)c0, r);
        if constexpr (GATED) {
          const bool hands = (chunk & 1) == (ew >> 1);
          if (hands) {
#pragma unroll
            for (int j = 0; j < 32; ++j) handed[chunk & 1][j][lane_row & 63] = __float2bfloat16_rn(__uint_as_float(r[j]));
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");  // (what is read here is written again behind the next one)
          if (hands) continue;
          // Which activation, and whose sums the gate's are, is asked once a chunk: asked for each value, the code of all three in 32 copies took
          // longer than the tile's products (eight groups of 249 rows, 14336 x 4096: 453 us and 371, and 526 and 386 where the power limit holds the clock).
          auto gate = [&](auto act) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float mine = round_bf16(__uint_as_float(r[j])), other = __bfloat162float(handed[chunk & 1][j][lane_row & 63]);
              const float g = ew < 2 ? mine : other, u = ew < 2 ? other : mine;
              r[j] = __float_as_uint(round_bf16(apply_act(g, act())) * u);
            }
          };
          if (p.act == ACT_SILU_GATE) gate([] { return ACT_SILU_GATE; });
          else if (p.act == ACT_GELU_TANH_GATE) gate([] { return ACT_GELU_TANH_GATE; });
          else gate([] { return ACT_GELU_ERF_GATE; });
        }
        if (col < p.N) {
          bf16* c = p.C + (size_t)(row0 + c0) * p.N + col;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c0 + j < rows) c[(size_t)j * p.N] = __float2bfloat16_rn(__uint_as_float(r[j]));
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(&tmem_empty_bar[acc], 0);  // the leader's MMA warp waits for all 8 warps of the pair
      ++lt;
    });
  }
  tcgen05_fence_before();
  cluster_sync_all();  // nobody leaves while the peer may still touch its barriers / shared memory
  if (warp == 2) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(512) : "memory");
  }
}

// ---- host side ------------------------------------------------------------------------------------
template <int BN, bool GATED>
static int launch_pair(const GemmParams& p, int tiles, cudaStream_t stream) {
  const size_t smem = 1024 + (size_t)PAIR_STAGES * (GEMM_BLOCK_M + BN / 2) * GEMM_BLOCK_K * 2 + 256;
  cudaError_t e = cudaFuncSetAttribute(gemm_bf16_tcgen05_pair_kernel<BN, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  gemm_bf16_tcgen05_pair_kernel<BN, GATED><<<dim3(2 * min(tiles, device_sm_count() / 2)), GEMM_THREADS, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

template <bool GATED, int ROWS>
static int launch_shared(const GemmParams& p, int tiles, cudaStream_t stream) {
  auto kernel = gemm_bf16_tcgen05_kernel<128, GATED, true, ROWS>;
  const size_t smem = GemmTile<128, GATED, ROWS>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.shares);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.shares;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, p);
}
// persistent: one CTA per SM walks the tile list
template <int BN, bool GATED, int ROWS>
static int launch_tiles(const GemmParams& p, cudaStream_t stream) {
  auto kernel = gemm_bf16_tcgen05_kernel<BN, GATED, false, ROWS>;
  const size_t smem = GemmTile<BN, GATED, ROWS>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int n_tiles = ((p.M + GEMM_BLOCK_M - 1) / GEMM_BLOCK_M) * ((p.N + BN - 1) / BN);
  kernel<<<dim3(min(n_tiles, device_sm_count())), GEMM_THREADS, smem, stream>>>(p);
  return (int)cudaGetLastError();
}

// CTAs that share the K range of a 128 x 128 tile: tiles that leave most SMs idle wait for their loads one K block after the other, so up to
// 32 of them get four CTAs, up to 64 two, as many as fit beside one another in clusters.  What that saves is the others' part of the range,
// what it costs is the exchange, 5 to 8 thousand cycles with its two cluster barriers: worth it from 1536 columns saved on against tiles of 128
// rows (gated ones load two weights to a column: 1024) and from 2048 against tiles shared by pairs, where less than that gives 1 to 2 us or
// nothing.  us with the gap of two events, the best other tile and shared: up to 128 rows 4096 x 14336 75 and 37, 2048 x 2048 14.4 and 14.4,
// 2 x 5632 x 2048 38 and 30; 200 to 512 rows 4096 x 14336 60 and 51, 2 x 768 x 3072 30.7 and 24.  Below the line: up to 128 rows 1024 x 1024 11
// and 12.3, 2048 x 1536 13 and 14.4, 8192 x 2048 17.3 and 19.4; 200 to 512 rows 3072 x 1024 14.4 and 16.4, 2560 x 2048 17.5 and 17; 900 rows
// 2 x 768 x 3072 30.8 and 31.8.
static int k_shares(int M, int N, int K, bool gated, int block_n) {
  const long long room = device_sm_count() - 20, tiles = (long long)((M + GEMM_BLOCK_M - 1) / GEMM_BLOCK_M) * ((N + 127) / 128);
  const int shares = 4 * tiles <= room ? 4 : 2 * tiles <= room ? 2 : 1;
  const int worth = M > GEMM_BLOCK_M ? 2048 : gated ? 1024 : 1536;
  return block_n != 64 && K - K / shares >= worth ? shares : 1;
}
// Width of the MMA tile: the one whose waves over the pairs take the least time.  A wave of narrower tiles costs its width plus
// what does not shrink with it (the A rows of every K block, the ramp): about 24 columns' worth.  448 rows (two row tiles):
// N = 4096 has 32 tiles of 256 for 74 pairs, 64 of 128; an 8B layer's four products take 222 us, 283 with 256 columns only.
static int pair_columns(int M, int N, bool gated) {
  const int pairs = device_sm_count() / 2, tm = (M + 2 * GEMM_BLOCK_M - 1) / (2 * GEMM_BLOCK_M);
  int best = 256;
  long long cost = -1;
  for (int bn : {256, 192, 128}) {
    const int out_n = gated ? bn / 2 : bn;
    const long long tiles = (long long)tm * ((N + out_n - 1) / out_n), c = (tiles + pairs - 1) / pairs * (bn + 24);
    if (cost < 0 || c < cost) { cost = c; best = bn; }
  }
  return best;
}
}  // namespace mdi

using namespace mdi;

// C[M,N] = A[M,K] W[N,K]^T (+bias) (+residual); with W2: C = act(A W^T + bias) * (A W2^T + bias2).
// K must be a multiple of 8 (16-byte rows for TMA).  signal_flag != null: fused hop (see GemmParams).
// knobs: sbo/lbo/hi_bits/k_step <= 0 select the canonical encoding.
extern "C" int mdi_gemm_bf16_ex(const void* A, const void* W, const void* W2, void* C, const void* bias,
                                const void* bias2, const void* residual, int M, int N, int K, int act, int block_n,
                                int* signal_flag, unsigned int* done_ctr, const int* ctx, const int* status, int sbo,
                                int lbo, int hi_bits, int k_step, cudaStream_t stream) {
  if (K % 8 != 0 || M <= 0 || N <= 0) return -2;
  if (W2 && residual) return -2;
  if (signal_flag && (!done_ctr || !ctx)) return -2;
  GemmParams p;
  p.C = (bf16*)C; p.bias = (const bf16*)bias; p.bias2 = (const bf16*)bias2; p.residual = (const bf16*)residual;
  p.M = M; p.N = N; p.K = K; p.act = act;
  p.signal = HopSignal{signal_flag, done_ctr, status}; p.ctx = ctx;
  p.desc_sbo = sbo > 0 ? (unsigned)sbo : 64u;
  p.desc_lbo = lbo > 0 ? (unsigned)lbo : 1u;
  p.desc_hi_bits = hi_bits > 0 ? (unsigned)hi_bits : (1u | (2u << 15));  // version = 1 (bit 46), SWIZZLE_128B = 2 (bits 61-63)
  p.k_step_bytes = k_step > 0 ? (unsigned)k_step : 32u;
  const bool gated = W2 != nullptr;
  p.shares = k_shares(M, N, K, gated, block_n);
  if (p.shares > 1 && sbo <= 0 && lbo <= 0 && hi_bits <= 0 && k_step <= 0) {
    int rc = make_map(&p.tma_a, A, M, K, M <= 64 ? 64 : GEMM_BLOCK_M);
    if (rc) return rc;
    rc = make_map(&p.tma_b, W, N, K, 128);
    if (rc) return rc;
    rc = make_map(&p.tma_b2, gated ? W2 : W, N, K, 128);
    if (rc) return rc;
    const int tiles = ((M + GEMM_BLOCK_M - 1) / GEMM_BLOCK_M) * ((N + 127) / 128);
    if (M <= 64) return gated ? launch_shared<true, 64>(p, tiles, stream) : launch_shared<false, 64>(p, tiles, stream);
    return gated ? launch_shared<true, 128>(p, tiles, stream) : launch_shared<false, 128>(p, tiles, stream);
  }
  if (block_n == 512) {  // CTA-pair kernel (cta_group::2): 256 x 256 MMA tiles shared by two CTAs of a cluster
    int rc2 = make_map(&p.tma_a, A, M, K, GEMM_BLOCK_M);
    if (rc2) return rc2;
    const int bn = pair_columns(M, N, gated);
    rc2 = make_map(&p.tma_b, W, N, K, bn / 2);  // each CTA loads half of the B tile's rows
    if (rc2) return rc2;
    rc2 = make_map(&p.tma_b2, gated ? W2 : W, N, K, bn / 2);
    if (rc2) return rc2;
    const int out_n = gated ? bn / 2 : bn, tiles = ((M + 255) / 256) * ((N + out_n - 1) / out_n);
    if (bn == 256) return gated ? launch_pair<256, true>(p, tiles, stream) : launch_pair<256, false>(p, tiles, stream);
    if (bn == 192) return gated ? launch_pair<192, true>(p, tiles, stream) : launch_pair<192, false>(p, tiles, stream);
    return gated ? launch_pair<128, true>(p, tiles, stream) : launch_pair<128, false>(p, tiles, stream);
  }
  if (block_n != 64 && block_n != 128 && block_n != 256) block_n = 128;
  if (gated && block_n == 256) block_n = 128;  // 2 buffers x 2 accumulators x BLOCK_N <= 512 TMEM columns
  const int rows = M <= 64 && block_n == 128 ? 64 : GEMM_BLOCK_M;
  int rc = make_map(&p.tma_a, A, M, K, rows);
  if (rc) return rc;
  rc = make_map(&p.tma_b, W, N, K, block_n);
  if (rc) return rc;
  rc = make_map(&p.tma_b2, gated ? W2 : W, N, K, block_n);
  if (rc) return rc;
  if (block_n == 64) return gated ? launch_tiles<64, true, 128>(p, stream) : launch_tiles<64, false, 128>(p, stream);
  if (block_n == 256) return launch_tiles<256, false, 128>(p, stream);
  if (rows == 64) return gated ? launch_tiles<128, true, 64>(p, stream) : launch_tiles<128, false, 64>(p, stream);
  return gated ? launch_tiles<128, true, 128>(p, stream) : launch_tiles<128, false, 128>(p, stream);
}

// How many CTAs share the K range of a tile of this product: more than one takes the shared form whatever `block_n` (other than 64) asks for.
extern "C" int mdi_gemm_k_shares(int M, int N, int K, int gated, int block_n) { return k_shares(M, N, K, gated != 0, block_n); }

extern "C" int mdi_gemm_bf16(const void* A, const void* W, void* C, const void* bias, const void* residual, int M,
                             int N, int K, int block_n, int sbo, int lbo, int hi_bits, int k_step,
                             cudaStream_t stream) {
  return mdi_gemm_bf16_ex(A, W, nullptr, C, bias, nullptr, residual, M, N, K, 0, block_n, nullptr, nullptr, nullptr,
                          nullptr, sbo, lbo, hi_bits, k_step, stream);
}

// C[rows of group e] = A[rows of group e] W_e^T, or with W2 act(A W_e^T) * (A W2_e^T): rows sorted by group, counts[e] rows of
// group e on the device (their sum is M), weights through host arrays of device pointers.
extern "C" int mdi_gemm_grouped(const void* A, const void* const* W, const void* const* W2, void* C, const int* counts, int groups, int M,
                                int N, int K, int act, cudaStream_t stream) {
  if (K % 8 != 0 || M <= 0 || N <= 0 || groups <= 0 || groups > 4096) return -2;
  const bool gated = W2 != nullptr;
  auto kernel = gated ? gemm_grouped_tcgen05_kernel<true> : gemm_grouped_tcgen05_kernel<false>;
  const size_t smem = 1024 + (size_t)PAIR_STAGES * (GEMM_BLOCK_M + GROUP_ROWS / 2) * GEMM_BLOCK_K * 2 + 256;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  GroupedParams p;
  p.C = (bf16*)C;
  p.counts = counts;
  p.M = M; p.N = N; p.K = K; p.act = act;
  int rc = 0;
  for (int i = 0; i < 4 && !rc; ++i) rc = make_map(&p.a[i], A, M, K, 16 << i);
  if (rc) return rc;
  for (int first = 0; first < groups; first += GROUPS) {
    p.first = first;
    p.groups = min(GROUPS, groups - first);
    for (int i = 0; i < GROUPS; ++i) {
      const int g = first + min(i, p.groups - 1);
      rc = make_map(&p.b[i], W[g], N, K, gated ? 64 : 128);
      if (rc) return rc;
      rc = make_map(&p.b2[i], gated ? W2[g] : W[g], N, K, gated ? 64 : 128);
      if (rc) return rc;
    }
    kernel<<<dim3(2 * (device_sm_count() / 2)), GEMM_THREADS, smem, stream>>>(p);
  }
  return (int)cudaGetLastError();
}
