// Prompt form of the gated recurrences (gated linear attention, gated delta rule) in chunks of 64 tokens.
//
// Token by token the recurrence is a chain of n steps, each a few hundred cycles of shuffles and one barrier on the few blocks
// that a prompt's heads fill: 1.1 us a token and more, whatever the GPU could do beside it.  In a chunk everything except its use
// of the state at the chunk's start is a small matrix product, so the chain shrinks to n / 64 steps.  With a_i the decay of token i
// (per key channel), S the state before the chunk and D(i, j) = a_(j+1) ... a_i:
//
//   u_i = v_i                                                         gated linear attention
//   u_i = b_i (v_i - sum_(j<i) [sum_d k_i k_j D(i, j)] u_j - (k_i D(i, -1))^T S)     delta rule: a triangular system of 64 rows,
//         solved once for both right-hand sides, u = Wv - Wk S
//   o_i = (q_i D(i, -1))^T S + sum_(j<=i) [sum_d q_i k_j D(i, j)] u_j
//   S'  = D(63, -1) S + sum_j (k_j D(63, j)) u_j^T
//
// Decays only ever enter as products of the a's themselves, which are at most one: nothing overflows, what underflows is
// zero in the token-by-token form too, and no difference of two long sums of logarithms is taken.  A chunk is cut into four
// sub-blocks of 16 tokens: rows carry the product from their sub-block's start, columns the product up to the row's sub-block,
// and the 16 x 16 blocks on the diagonal walk each row's columns backwards with a running product.  All sums are fp32.
//
//   gated_chunk_prep   a block per (chunk, head): norms, decays, both score triangles, the triangular solve
//   gated_chunk_chain  a block per (sequence, head, 16 value columns): the state through the sequence's chunks
//   gated_chunk_out    a block per (chunk, head): read-out, RMS norm, gate, cast
#include "hybrid_common.cuh"

namespace hyb {

constexpr int CH = 64, SB = 16;  // tokens of a chunk, of a sub-block

// Work space: per (chunk, head) the rows below, all fp32.  Rows of D are stored with their 16-byte groups permuted (swz), the
// way shared memory holds them.
struct ChunkWork {
  float *wk, *kend, *qt;  // [64][D]: k D(i,-1) through the solve; k D(63,j); q D(i,-1)
  float *aqk;             // [64][64]: scores of the read-out, zero above the diagonal
  float *u;               // [64][V]: Wv, then u
  float *dec;             // [D]: D(63,-1)
  float* s0;              // [D][V]: the state before the chunk
  int2* rows;             // per chunk: first row, number of rows (written by the preparation, read by the read-out)
  int h0, nh, nchunks;    // the heads of this turn, all chunks
};

// Place of 16-byte group c of row r: eight rows at the same group fall on different banks.
__device__ __forceinline__ int swz(int r, int c, int D) { return r * D + ((c ^ (r & 7)) << 2); }
__device__ __forceinline__ int swz1(int r, int d, int D) { return swz(r, d >> 2, D) + (d & 3); }

// Four values of a row; `vec`: the row's groups of four may be read at once.
__device__ __forceinline__ void load4(const float* p, bool vec, float* f) {
  if (vec) {
    float4 t = *reinterpret_cast<const float4*>(p);
    f[0] = t.x; f[1] = t.y; f[2] = t.z; f[3] = t.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = p[e];
  }
}
__device__ __forceinline__ void load4(const bf16* p, bool vec, float* f) {
  if (vec) {
    uint2 t = *reinterpret_cast<const uint2*>(p);
    f[0] = __uint_as_float(t.x << 16); f[1] = __uint_as_float(t.x & 0xffff0000u);
    f[2] = __uint_as_float(t.y << 16); f[3] = __uint_as_float(t.y & 0xffff0000u);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = to_f(p[e]);
  }
}
template <typename T> __device__ __forceinline__ bool by_four(const T* p, long long stride) {
  return ((uintptr_t)p % (4 * sizeof(T))) == 0 && stride % 4 == 0;
}

// What bounds it: latency and issue at two blocks per SM (some 1.2 M multiply-adds for a chunk and head of 128 x 128).  Loops
// stay rolled around bodies of 16 rows: with every loop over 64 rows unrolled the solve spent twice its time on fetching
// instructions (67 k against 26 k cycles of a block pair).  Three tiles of [64][D] and the triangle fit twice into an SM; a tile
// is reused as soon as its first contents are spent (decays become the rows k D(i, .), k the columns, q and k the solved rows).
template <typename T, int D, bool DELTA>
__global__ void __launch_bounds__(256, 2) gated_chunk_prep_kernel(RecArgs a, ChunkWork wk) {
  extern __shared__ __align__(128) float sm[];
  float* sA = sm;
  float* sL = sA + CH * D;        // [64][64]: sL[j][i] = b_i * (score of i against j < i)
  float* sB = sL + CH * CH;       // [64]: b
  float* sQ = sB + CH;
  float* sK = sQ + CH * D;
  float* sX = sQ;                 // [64][D + V]: solved rows, over q and k
  constexpr int NC = D / 4;       // 16-byte groups in a row
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y;
  Piece piece = find_piece(a, CH, blockIdx.x);
  int start = piece.row, n = piece.n;
  if (blockIdx.y == 0 && tid == 0) wk.rows[blockIdx.x] = make_int2(start, n);
  size_t ch = (size_t)blockIdx.x * wk.nh + blockIdx.y;
  int kvh = h / (a.H / a.G);
  float* aqk = wk.aqk + ch * (CH * CH);
  for (int i = tid; i < CH * CH / 4; i += 256) reinterpret_cast<float4*>(aqk)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  {  // a warp per token, the loads of four tokens at a time
    const T *q = (const T*)a.q + kvh * D, *k = (const T*)a.k + kvh * D, *z = (const T*)a.z + h * D;
    bool vq = by_four(q, a.q_stride), vk = by_four(k, a.k_stride), vz = by_four(z, a.z_stride);
    float rate = DELTA ? expf(to_f(((const T*)a.a_log)[h])) : 0.f;
    float ds = 1.f / sqrtf((float)D);
    bool on = lane < NC;
    float zb[4] = {0.f, 0.f, 0.f, 0.f};
    if (on && a.zb)
#pragma unroll
      for (int e = 0; e < 4; ++e) zb[e] = to_f(((const T*)a.zb)[h * D + 4 * lane + e]);
#pragma unroll 1
    for (int t0 = warp; t0 < CH; t0 += 32) {
      float qv[4][4] = {}, kv[4][4] = {}, zv[4][4] = {}, b[4] = {};
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        size_t row = (size_t)start + t0 + 8 * m;
        if (t0 + 8 * m < n) {
          if (on) {
            load4(q + row * a.q_stride + 4 * lane, vq, qv[m]);
            load4(k + row * a.k_stride + 4 * lane, vk, kv[m]);
            load4(z + row * a.z_stride + 4 * lane, vz, zv[m]);
          }
          if (DELTA) b[m] = to_f(((const T*)a.beta)[row * a.beta_stride + h]);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        int t = t0 + 8 * m;
        float qs = ds, ks = 1.f;
        if (DELTA) {
          float pq = warp_sum(qv[m][0] * qv[m][0] + qv[m][1] * qv[m][1] + qv[m][2] * qv[m][2] + qv[m][3] * qv[m][3]);
          float pk = warp_sum(kv[m][0] * kv[m][0] + kv[m][1] * kv[m][1] + kv[m][2] * kv[m][2] + kv[m][3] * kv[m][3]);
          qs = ds / sqrtf(pq + 1e-6f);
          ks = 1.f / sqrtf(pk + 1e-6f);
        }
        if (on) {
          int at = swz(t, lane, D);
          *reinterpret_cast<float4*>(sQ + at) = make_float4(qv[m][0] * qs, qv[m][1] * qs, qv[m][2] * qs, qv[m][3] * qs);
          *reinterpret_cast<float4*>(sK + at) = make_float4(kv[m][0] * ks, kv[m][1] * ks, kv[m][2] * ks, kv[m][3] * ks);
          float av[4] = {1.f, 1.f, 1.f, 1.f};  // a row behind the sequence's end changes nothing
          if (t < n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float zz = zv[m][e] + zb[e];
              av[e] = DELTA ? expf(-rate * softplusf_(zz)) : expf(-softplusf_(-zz) / a.tau);
            }
          *reinterpret_cast<float4*>(sA + at) = make_float4(av[0], av[1], av[2], av[3]);
        }
        if (DELTA && lane == 0) sB[t] = t < n ? sigmoidf_(b[m]) : 0.f;
      }
    }
  }
  __syncthreads();
  // ---- the 16 x 16 blocks on the diagonal: 16 lanes share the channels of a row and keep its 16 partial scores, which meet in
  // one exchange that leaves each lane with one score; a warp has rows 2p and 2p + 1 of every sub-block, p mirrored in every
  // other one so that each warp walks 36 columns
  {
    constexpr int GC = (NC + 15) / 16;  // groups per lane
    int hl = lane & 15;
#pragma unroll 1
    for (int s = 0; s < CH / SB; ++s) {
      int il = 2 * ((s & 1) ? 7 - warp : warp) + (lane >> 4), top = il | 1, i = s * SB + il;
      float4 qc[GC], kc[GC];
      float x[SB], y[SB];
#pragma unroll
      for (int c = 0; c < GC; ++c) {
        bool on = hl + 16 * c < NC;
        int at = swz(i, on ? hl + 16 * c : 0, D);
        qc[c] = *reinterpret_cast<const float4*>(sQ + at);
        kc[c] = *reinterpret_cast<const float4*>(sK + at);
        if (!on) qc[c] = kc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int j = SB - 1; j >= 0; --j) {
        x[j] = y[j] = 0.f;
        if (j <= top) {  // the same for the whole warp
          bool live = j <= il;
#pragma unroll
          for (int c = 0; c < GC; ++c) {
            int at = swz(s * SB + j, hl + 16 * c < NC ? hl + 16 * c : 0, D);
            float4 kj = *reinterpret_cast<const float4*>(sK + at), aj = *reinterpret_cast<const float4*>(sA + at);
            x[j] += qc[c].x * kj.x + qc[c].y * kj.y + qc[c].z * kj.z + qc[c].w * kj.w;
            if (DELTA) y[j] += kc[c].x * kj.x + kc[c].y * kj.y + kc[c].z * kj.z + kc[c].w * kj.w;
            if (!live) aj = make_float4(1.f, 1.f, 1.f, 1.f);
            qc[c].x *= aj.x; qc[c].y *= aj.y; qc[c].z *= aj.z; qc[c].w *= aj.w;
            if (DELTA) { kc[c].x *= aj.x; kc[c].y *= aj.y; kc[c].z *= aj.z; kc[c].w *= aj.w; }
          }
        }
      }
      // lane l of 16 ends with the sum of column l: halve the columns, each half goes to the lanes that have its bit
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        bool up = hl & o;
#pragma unroll
        for (int j = 0; j < o; ++j) {
          float keep = up ? x[j + o] : x[j], give = up ? x[j] : x[j + o];
          x[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          if (DELTA) {
            keep = up ? y[j + o] : y[j];
            give = up ? y[j] : y[j + o];
            y[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        }
      }
      if (hl <= il) {
        aqk[i * CH + s * SB + hl] = x[0];
        if (DELTA && hl < il) sL[(s * SB + hl) * CH + i] = sB[i] * y[0];
      }
    }
  }
  __syncthreads();
  // ---- rows (threads below D) and columns (the next D threads) of one sub-block after the other, a channel per thread
  bool isrow = tid < D, iscol = tid >= D && tid < 2 * D;
  int d = isrow ? tid : tid - D;
  float run = 1.f;  // this channel's product over the sub-blocks so far
#pragma unroll 1
  for (int s = 0; s < CH / SB; ++s) {
    float m1[SB], m2[SB], end = 1.f;  // rows: q and k times the product from the sub-block's start; columns: k times the product after it
    if (isrow) {
#pragma unroll
      for (int i = 0; i < SB; ++i) {
        int at = swz1(s * SB + i, d, D);
        end *= sA[at];
        m1[i] = sQ[at] * end;
        if (DELTA) m2[i] = sK[at] * end;
      }
    } else if (iscol) {
#pragma unroll
      for (int i = SB - 1; i >= 0; --i) {
        int at = swz1(s * SB + i, d, D);
        m1[i] = sK[at] * end;
        end *= sA[at];
      }
    }
    __syncthreads();
    if (isrow) {  // sA takes the k rows
#pragma unroll
      for (int i = 0; i < SB; ++i) {
        int at = swz1(s * SB + i, d, D);
        sQ[at] = m1[i];
        if (DELTA) sA[at] = m2[i];
      }
    }
    __syncthreads();
    if (s > 0) {  // scores of the 16 rows against all earlier columns: a warp has two tokens, a lane a column or two
      int r0 = s * SB + 2 * warp, ncol = s * SB;
      float acc[2][2][2] = {};  // [q or k][row][column]
      int c1 = lane + 32;
      bool on0 = lane < ncol, on1 = c1 < ncol;
#pragma unroll 2
      for (int c = 0; c < NC; ++c) {
        float4 f[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          f[0][r] = *reinterpret_cast<const float4*>(sQ + swz(r0 + r, c, D));
          if (DELTA) f[1][r] = *reinterpret_cast<const float4*>(sA + swz(r0 + r, c, D));
        }
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          if (cc == 0 ? on0 : on1) {
            float4 kj = *reinterpret_cast<const float4*>(sK + swz(cc ? c1 : lane, c, D));
#pragma unroll
            for (int m = 0; m < (DELTA ? 2 : 1); ++m)
#pragma unroll
              for (int r = 0; r < 2; ++r)
                acc[m][r][cc] += f[m][r].x * kj.x + f[m][r].y * kj.y + f[m][r].z * kj.z + f[m][r].w * kj.w;
          }
        }
      }
#pragma unroll
      for (int cc = 0; cc < 2; ++cc)
        if (cc == 0 ? on0 : on1)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            int j = cc ? c1 : lane, i = r0 + r;
            aqk[i * CH + j] = acc[0][r][cc];
            if (DELTA) sL[j * CH + i] = sB[i] * acc[1][r][cc];
          }
      __syncthreads();
      if (isrow) {  // rows reach back to the chunk's start
#pragma unroll
        for (int i = 0; i < SB; ++i) {
          int at = swz1(s * SB + i, d, D);
          sQ[at] = m1[i] * run;
          if (DELTA) sA[at] = m2[i] * run;
        }
      }
    }
    if (iscol) {  // earlier columns reach to the next sub-block
#pragma unroll 8
      for (int j = 0; j < s * SB; ++j) sK[swz1(j, d, D)] *= end;
#pragma unroll
      for (int i = 0; i < SB; ++i) sK[swz1(s * SB + i, d, D)] = m1[i];
    }
    run *= end;
  }
  if (isrow) wk.dec[ch * D + d] = run;
  __syncthreads();
  {
    float4* ke = reinterpret_cast<float4*>(wk.kend + ch * (CH * D));
    float4* qt = reinterpret_cast<float4*>(wk.qt + ch * (CH * D));
    for (int i = tid; i < CH * NC; i += 256) {
      ke[i] = reinterpret_cast<const float4*>(sK)[i];
      qt[i] = reinterpret_cast<const float4*>(sQ)[i];
    }
  }
  int V = a.V;
  float* u = wk.u + ch * ((size_t)CH * V);
  const T* v = (const T*)a.v + h * V;
  if (!DELTA) {
    bool vv = by_four(v, a.v_stride);
    for (int i = tid; i < CH * V / 4; i += 256) {
      int t = i / (V / 4), j = 4 * (i - t * (V / 4));
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (t < n) load4(v + ((size_t)start + t) * a.v_stride + j, vv, f);
      reinterpret_cast<float4*>(u)[i] = make_float4(f[0], f[1], f[2], f[3]);
    }
    return;
  }
  // ---- the triangular solve, a column of [b K | b V] per thread, 16 rows at a time: first everything that earlier sub-blocks
  // solved (from shared memory, the thread's own column), then the sub-block itself in registers
  float* wko = wk.wk + ch * (CH * D);
  int W = D + V, col = tid;
  __syncthreads();
  if (col >= W) return;
#pragma unroll 1
  for (int s = 0; s < CH / SB; ++s) {
    float x[SB];
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      int t = s * SB + i;
      float r = col < D ? sA[swz1(t, col, D)] : t < n ? to_f(v[((size_t)start + t) * a.v_stride + (col - D)]) : 0.f;
      x[i] = sB[t] * r;
    }
#pragma unroll 4
    for (int j = 0; j < s * SB; ++j) {
      float xj = sX[j * W + col];
#pragma unroll
      for (int g = 0; g < SB / 4; ++g) {
        float4 l = *reinterpret_cast<const float4*>(sL + j * CH + s * SB + 4 * g);
        x[4 * g] -= l.x * xj;
        x[4 * g + 1] -= l.y * xj;
        x[4 * g + 2] -= l.z * xj;
        x[4 * g + 3] -= l.w * xj;
      }
    }
#pragma unroll
    for (int j = 0; j < SB - 1; ++j)
#pragma unroll
      for (int i = j + 1; i < SB; ++i) x[i] -= sL[(s * SB + j) * CH + s * SB + i] * x[j];
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      int t = s * SB + i;
      sX[t * W + col] = x[i];
      if (col < D) wko[swz1(t, col, D)] = x[i];
      else u[t * V + (col - D)] = x[i];
    }
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
// One bulk copy of `bytes` (a multiple of 16; both places 16-byte aligned) that completes on `b`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(b)) : "memory");
}
// Waits for the copy of this thread block's own that phase `parity` of `b` belongs to.  A copy from this GPU's memory ends, the
// limit on the tries only keeps a broken caller from hanging; false when it ran out.
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
  uint32_t done = 0;
  for (int i = 0; i < (1 << 22) && !done; ++i)
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done) : "r"(smem_addr(b)), "r"(parity) : "memory");
  return done;
}

// The chain.  A warp owns 16 key channels, a block 16 value columns (D / 16 warps; 128 blocks for 16 heads of 128 columns, one
// to an SM).  Per chunk: each warp's share of Wk S (its own channels, from its own copy of S), the shares added up, then the
// warp's part of the state from registers.  The two [64][D] tiles of a chunk arrive as bulk copies while the chunk before is
// worked on.  When a wait for one runs out, the step's status word is set, no more copies are started, and the state and the
// outputs that depend on it become NaN: nothing that was computed from a tile that is not there passes for a result.
template <int D, bool DELTA>
__global__ void __launch_bounds__(2 * D, DELTA ? 1 : 3) gated_chunk_chain_kernel(RecArgs a, ChunkWork wk) {
  constexpr int NW = D / 16, TH = 2 * D, TILE = CH * D;
  extern __shared__ __align__(128) float sm[];
  float* sWk = sm;                                   // [2][64][D] (delta)
  float* sKe = sWk + (DELTA ? 2 * TILE : 0);         // [2][64][D]
  float* sP = sKe + 2 * TILE;                        // [NW][64][16] (delta)
  float* sU = sP + (DELTA ? NW * CH * 16 : 0);       // [2][64][16]
  float* sS = sU + 2 * CH * 16;                      // [16][D + 4]: the state, columns first (delta)
  __shared__ __align__(8) uint64_t bar[4];
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y, V = a.V, j0 = blockIdx.z * 16;
  int count = pieces_of(a, a.meta[4 * blockIdx.x + 1], CH);
  if (count == 0) return;
  int first = pieces_before(a, CH, blockIdx.x);
  count = min(count, wk.nchunks - first);  // (lengths that are not those the work space was laid out for)
  float* gS = a.state + ((size_t)a.meta[4 * blockIdx.x + 2] * a.H + h) * D * V + j0;
  // this lane's part of the state: channels d0 .. d0 + 3, columns c0, c0 + 1
  int dg = lane & 3, d0 = warp * 16 + 4 * dg, c0 = 2 * (lane >> 2);
  float s[4][2];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float2 t = *reinterpret_cast<const float2*>(gS + (size_t)(d0 + e) * V + c0);
    s[e][0] = t.x;
    s[e][1] = t.y;
  }
  auto tile = [&](const float* p, int c) { return p + ((size_t)(first + c) * wk.nh + blockIdx.y) * TILE; };
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) bar_init(bar + i);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (count > 0) {
      if (DELTA) bulk_load(sWk, tile(wk.wk, 0), TILE * 4, bar);
      bulk_load(sKe, tile(wk.kend, 0), TILE * 4, bar + 2);
      if (DELTA && count > 1) bulk_load(sWk + TILE, tile(wk.wk, 1), TILE * 4, bar + 1);
    }
  }
  __syncthreads();
  constexpr int UP = (CH * 4 + TH - 1) / TH;  // 16-byte groups of the [64][16] tile of u per thread
  float4 wv[UP];
  float4 dec;
  auto fetch = [&](int c) {
    size_t ch = (size_t)(first + c) * wk.nh + blockIdx.y;
#pragma unroll
    for (int i = 0; i < UP; ++i) {
      int o = tid + i * TH;
      if (o < CH * 4) wv[i] = *reinterpret_cast<const float4*>(wk.u + (ch * CH + (o >> 2)) * V + j0 + 4 * (o & 3));
    }
    dec = *reinterpret_cast<const float4*>(wk.dec + ch * D + d0);
  };
  if (count > 0) fetch(0);
  const float nan = __int_as_float(0x7fffffff);
  bool lost = false;
  auto lose = [&]() {
    lost = true;
    if (a.status) atomicExch(a.status, 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e][0] = s[e][1] = nan;
  };
  for (int c = 0; c < count; ++c) {
    int b = c & 1;
    uint32_t parity = (c >> 1) & 1;
    size_t ch = (size_t)(first + c) * wk.nh + blockIdx.y;
    {  // the state before the chunk, for the read-out
      float* g = wk.s0 + ch * ((size_t)D * V) + j0;
#pragma unroll
      for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(g + (size_t)(d0 + e) * V + c0) = make_float2(s[e][0], s[e][1]);
    }
    float* su = sU + b * (CH * 16);
    if (DELTA) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float4*>(sS + (c0 + e) * (D + 4) + d0) = make_float4(s[0][e], s[1][e], s[2][e], s[3][e]);
      __syncwarp();
      if (!lost && !bar_wait(bar + b, parity)) lose();
      const float* w = sWk + b * TILE;
      int rg = lane >> 2, cg = lane & 3;  // rows rg + 8 r, columns 4 cg + i
      float acc[8][4] = {};
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        float4 sv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sv[i] = *reinterpret_cast<const float4*>(sS + (4 * cg + i) * (D + 4) + warp * 16 + 4 * g);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          float4 f = *reinterpret_cast<const float4*>(w + swz(rg + 8 * r, warp * 4 + g, D));
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[r][i] += f.x * sv[i].x + f.y * sv[i].y + f.z * sv[i].z + f.w * sv[i].w;
        }
      }
      if (lost)
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = nan;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        *reinterpret_cast<float4*>(sP + (warp * CH + rg + 8 * r) * 16 + 4 * cg) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    }
    __syncthreads();  // the shares are there; nobody reads this chunk's Wk or the chunk before's Kend any more
    if (tid == 0 && !lost) {
      if (DELTA && c + 2 < count) bulk_load(sWk + b * TILE, tile(wk.wk, c + 2), TILE * 4, bar + b);
      if (c + 1 < count) bulk_load(sKe + (b ^ 1) * TILE, tile(wk.kend, c + 1), TILE * 4, bar + 2 + (b ^ 1));
    }
#pragma unroll
    for (int i = 0; i < UP; ++i) {
      int o = tid + i * TH;
      if (o >= CH * 4) break;
      int t = o >> 2, g = o & 3;
      float4 x = wv[i];
      if (DELTA) {
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < NW; ++p) {
          float4 f = *reinterpret_cast<const float4*>(sP + (p * CH + t) * 16 + 4 * g);
          y.x += f.x; y.y += f.y; y.z += f.z; y.w += f.w;
        }
        x.x -= y.x; x.y -= y.y; x.z -= y.z; x.w -= y.w;
        *reinterpret_cast<float4*>(wk.u + (ch * CH + t) * V + j0 + 4 * g) = x;
      }
      *reinterpret_cast<float4*>(su + t * 16 + 4 * g) = x;
    }
    float4 dc = dec;
    if (c + 1 < count) fetch(c + 1);
    __syncthreads();
    if (!lost && !bar_wait(bar + 2 + b, parity)) lose();
    const float* ke = sKe + b * TILE;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      s[0][e] *= dc.x; s[1][e] *= dc.y; s[2][e] *= dc.z; s[3][e] *= dc.w;
    }
#pragma unroll 8
    for (int t = 0; t < CH; ++t) {
      float4 k = *reinterpret_cast<const float4*>(ke + swz(t, warp * 4 + dg, D));
      float2 uu = *reinterpret_cast<const float2*>(su + t * 16 + c0);
      s[0][0] += k.x * uu.x; s[1][0] += k.y * uu.x; s[2][0] += k.z * uu.x; s[3][0] += k.w * uu.x;
      s[0][1] += k.x * uu.y; s[1][1] += k.y * uu.y; s[2][1] += k.z * uu.y; s[3][1] += k.w * uu.y;
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(gS + (size_t)(d0 + e) * V + c0) = make_float2(s[e][0], s[e][1]);
}

// The read-out: [64][D + 64] times [D + 64][V] in steps of 32, two stages of shared memory filled with cp.async; a warp has
// eight whole rows (a lane four columns), so the RMS norm needs no more than a warp's sum.  Bound by fp32 issue.
// Three blocks per SM: with four the diagonal's triangle spills (three kernels of delta, 2048 tokens, 16 heads of 128: 351 against 342 us).
template <int N>
__device__ __forceinline__ void cp_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

template <typename T, int D, bool DELTA>
__global__ void __launch_bounds__(256, 3) gated_chunk_out_kernel(RecArgs a, ChunkWork wk) {
  constexpr int KT = 32, STEPS = (D + CH) / KT;
  extern __shared__ __align__(128) float sm[];
  int V = a.V, stage = CH * KT + KT * V;
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y;
  int start = wk.rows[blockIdx.x].x, n = wk.rows[blockIdx.x].y;
  size_t ch = (size_t)blockIdx.x * wk.nh + blockIdx.y;
  auto load = [&](int st) {
    float* sA = sm + (st & 1) * stage;
    float* sB = sA + CH * KT;
    bool head = st < D / KT;
    int k0 = head ? st * KT : st * KT - D;
    const float* A = head ? wk.qt + ch * (CH * D) : wk.aqk + ch * (CH * CH);
    for (int i = tid; i < CH * KT / 4; i += 256) {
      int r = i >> 3, g = i & 7;
      cp16(sA + r * KT + 4 * g, head ? A + swz(r, k0 / 4 + g, D) : A + r * CH + k0 + 4 * g);
    }
    const float* B = head ? wk.s0 + ch * ((size_t)D * V) + (size_t)k0 * V : wk.u + ch * ((size_t)CH * V) + (size_t)k0 * V;
    for (int i = tid; i < KT * V / 4; i += 256) cp16(sB + 4 * i, B + 4 * i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  bool on = 4 * lane < V;
  float acc[8][4] = {};
#pragma unroll 1
  for (int st = 0; st < STEPS; ++st) {
    if (st + 1 < STEPS) {
      load(st + 1);
      cp_wait_group<1>();
    } else {
      cp_wait_group<0>();
    }
    __syncthreads();
    const float* sA = sm + (st & 1) * stage;
    const float* sB = sA + CH * KT;
    // scores above the diagonal are left out, not multiplied by their zeros: an infinite or undefined value of a later token
    // stays out of the rows before it.  Groups of four columns: all rows see the first `full` of them, the next two hold the
    // warp's own diagonal
    int k0 = st * KT - D, full = st < D / KT ? KT / 4 : min(KT / 4, max(0, (8 * warp - k0) / 4));
    if (on) {
#pragma unroll 2
      for (int g = 0; g < full; ++g) {
        float4 b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = *reinterpret_cast<const float4*>(sB + (4 * g + e) * V + 4 * lane);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          float4 f = *reinterpret_cast<const float4*>(sA + (8 * warp + r) * KT + 4 * g);
          acc[r][0] += f.x * b[0].x + f.y * b[1].x + f.z * b[2].x + f.w * b[3].x;
          acc[r][1] += f.x * b[0].y + f.y * b[1].y + f.z * b[2].y + f.w * b[3].y;
          acc[r][2] += f.x * b[0].z + f.y * b[1].z + f.z * b[2].z + f.w * b[3].z;
          acc[r][3] += f.x * b[0].w + f.y * b[1].w + f.z * b[2].w + f.w * b[3].w;
        }
      }
      if (k0 >= 0 && full < KT / 4 && k0 <= 8 * warp) {
        const float *dA = sA + 8 * warp * KT + 4 * full, *dB = sB + 4 * full * V + 4 * lane;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float4 b[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) b[e] = *reinterpret_cast<const float4*>(dB + (4 * g + e) * V);
#pragma unroll
          for (int r = 4 * g; r < 8; ++r) {
            float4 t = *reinterpret_cast<const float4*>(dA + r * KT + 4 * g);
            float f[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (4 * g + e <= r) {
                acc[r][0] += f[e] * b[e].x;
                acc[r][1] += f[e] * b[e].y;
                acc[r][2] += f[e] * b[e].z;
                acc[r][3] += f[e] * b[e].w;
              }
          }
        }
      }
    }
    __syncthreads();
  }
  const T *gate = (const T*)a.g + h * V, *w = (const T*)a.w;
  T* out = (T*)a.out + h * V;
  float wv[4] = {0.f, 0.f, 0.f, 0.f};
  if (on)
#pragma unroll
    for (int e = 0; e < 4; ++e) wv[e] = to_f(w[4 * lane + e]);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    int t = 8 * warp + r;
    float ss = warp_sum(acc[r][0] * acc[r][0] + acc[r][1] * acc[r][1] + acc[r][2] * acc[r][2] + acc[r][3] * acc[r][3]);
    if (t < n && on) {
      size_t row = (size_t)start + t;
      float inv = 1.f / sqrtf(ss / V + a.eps);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float gv = to_f(gate[row * a.g_stride + 4 * lane + e]);
        out[row * a.out_stride + 4 * lane + e] = from_f<T>(acc[r][e] * inv * wv[e] * (DELTA ? sigmoidf_(gv) : siluf_(gv)));
      }
    }
  }
}

template <typename T, int D, bool DELTA>
static int run_gated_chunks(const RecArgs& a, const ChunkWork& w, int nchunks, cudaStream_t st) {
  constexpr int V1 = 128;  // the widest
  constexpr int sp = (CH * D + CH * CH + CH + CH * (DELTA && V1 > D ? D + V1 : 2 * D)) * sizeof(float);
  constexpr int sc = ((DELTA ? 4 : 2) * CH * D + (DELTA ? D / 16 * CH * 16 : 0) + 2 * CH * 16 + (DELTA ? 16 * (D + 4) : 0)) * sizeof(float);
  constexpr int so = 2 * (CH * 32 + 32 * V1) * sizeof(float);
  cudaError_t e = allow_smem<gated_chunk_prep_kernel<T, D, DELTA>>(sp);
  if (e == cudaSuccess) e = allow_smem<gated_chunk_chain_kernel<D, DELTA>>(sc);
  if (e == cudaSuccess) e = allow_smem<gated_chunk_out_kernel<T, D, DELTA>>(so);
  if (e != cudaSuccess) return (int)e;
  size_t sp_v = (CH * D + CH * CH + CH + CH * (DELTA && a.V > D ? D + a.V : 2 * D)) * sizeof(float);
  gated_chunk_prep_kernel<T, D, DELTA><<<dim3(nchunks, w.nh), 256, sp_v, st>>>(a, w);
  gated_chunk_chain_kernel<D, DELTA><<<dim3(a.nseq, w.nh, a.V / 16), 2 * D, sc, st>>>(a, w);
  gated_chunk_out_kernel<T, D, DELTA><<<dim3(nchunks, w.nh), 256, 2 * (CH * 32 + 32 * a.V) * sizeof(float), st>>>(a, w);
  return (int)cudaGetLastError();
}

template <typename T, int D>
static int run_gated_chunks(const RecArgs& a, const ChunkWork& w, int nchunks, cudaStream_t st) {
  return a.mode == 1 ? run_gated_chunks<T, D, true>(a, w, nchunks, st) : run_gated_chunks<T, D, false>(a, w, nchunks, st);
}

}  // namespace hyb

using namespace hyb;

extern "C" {

// fp32 values of work space per (chunk, head); 0: the sizes have no chunked form (key channels of 32, 64 or 128, values a
// multiple of 16 up to 128: the tiles are laid out for these, anything else keeps the token scan).
long long hyb_gated_chunk_floats(int D, int V, int mode) {
  if ((D != 32 && D != 64 && D != 128) || V % 16 || V < 16 || V > 128) return 0;
  return (long long)(mode == 1 ? 3 : 2) * CH * D + CH * CH + (long long)CH * V + D + (long long)D * V;
}

// The sequences that take part (RecArgs) in `nchunks` chunks of 64 tokens.  work: space of nchunks * heads * hyb_gated_chunk_floats
// and 2 * nchunks, rounded up to 32; `heads` heads run at a time.
int hyb_gated_chunks(const RecArgs* args, int nchunks, float* work, int heads, int dt, cudaStream_t st) {
  if (args->nseq == 0 || nchunks == 0) return 0;
  RecArgs a = *args;
  if (a.G < 1 || a.H % a.G || heads < 1 || hyb_gated_chunk_floats(a.D, a.V, a.mode) == 0 || ((uintptr_t)work & 127)) return -3;
  ChunkWork w;
  w.nchunks = nchunks;
  for (w.h0 = 0; w.h0 < a.H; w.h0 += heads) {
    w.nh = a.H - w.h0 < heads ? a.H - w.h0 : heads;
    size_t n = (size_t)nchunks * w.nh;
    w.rows = (int2*)work;
    w.kend = work + (2 * (size_t)nchunks + 31) / 32 * 32;
    w.qt = w.kend + n * CH * a.D;
    w.aqk = w.qt + n * CH * a.D;
    w.u = w.aqk + n * CH * CH;
    w.s0 = w.u + n * CH * a.V;
    w.dec = w.s0 + n * a.D * a.V;
    w.wk = w.dec + n * a.D;
    int rc;
    if (dt == 0) rc = a.D == 32 ? run_gated_chunks<bf16, 32>(a, w, nchunks, st) : a.D == 64 ? run_gated_chunks<bf16, 64>(a, w, nchunks, st)
                                                                                         : run_gated_chunks<bf16, 128>(a, w, nchunks, st);
    else rc = a.D == 32 ? run_gated_chunks<float, 32>(a, w, nchunks, st) : a.D == 64 ? run_gated_chunks<float, 64>(a, w, nchunks, st)
                                                                                : run_gated_chunks<float, 128>(a, w, nchunks, st);
    if (rc) return rc;
  }
  return 0;
}

}  // extern "C"
