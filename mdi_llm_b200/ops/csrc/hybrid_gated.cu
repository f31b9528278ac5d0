// Prompt form of the gated recurrences (gated linear attention, gated delta rule) in chunks of 64 tokens.
//
// Token by token the recurrence is a chain of n steps, each a few hundred cycles of shuffles and one barrier on the few blocks
// that a prompt's heads fill: 1.1 us a token and more, whatever the GPU could do beside it.  In a chunk everything except its use
// of the state at the chunk's start is a small matrix product, so the chain shrinks to n / 64 steps.  With a_i the decay of token i
// (per key channel), S the state before the chunk and D(i, j) = a_(j+1) ... a_i:
//
//   u_i = v_i                                                         gated linear attention
//   u_i = b_i (v_i - sum_(j<i) [sum_d k_i k_j D(i, j)] u_j - (k_i D(i, -1))^T S)     delta rule: a triangular system of 64 rows,
//         solved for both right-hand sides by the inverse of the triangle, u = Wv - Wk S
//   o_i = (q_i D(i, -1))^T S + sum_(j<=i) [sum_d q_i k_j D(i, j)] u_j
//   S'  = D(63, -1) S + sum_j (k_j D(63, j)) u_j^T
//
// Decays only ever enter as products of the a's themselves, which are at most one: nothing overflows, what underflows is
// zero in the token-by-token form too, and no difference of two long sums of logarithms is taken.  A chunk is cut into eights of
// tokens: rows carry the product from the start of their eight, columns the product to the end of theirs, a table has the eights in between,
// and the 8 x 8 blocks on the diagonal walk down each column with a running product.  All values and sums are fp32; products of
// matrices run on the tensor cores with each value in three bf16 pieces (see split3).
//
//   gated_chunk_prep   a block per (chunk, head): norms, decays, both score triangles, the triangular solve
//   gated_chunk_chain  a block per (sequence, head, 16 value columns): the state through the sequence's chunks
//   gated_chunk_out    a block per (chunk, head): read-out, RMS norm, gate, cast
#include "hybrid_math.cuh"
#include "hybrid_mma.cuh"

namespace hyb {

constexpr int CH = 64, SB = 16;  // tokens of a chunk, of a sub-block

// Work space: per (chunk, head) the rows below, fp32 but for the first two, whose values are kept as the three bf16 pieces that the
// chain multiplies (split3: 24 bits, nothing is lost), in the order that shared
// memory holds them in (wk_at, piece_at).
struct ChunkWork {
  bf16 *wk, *kend;  // [D / 16][3][16][64]: k D(i,-1) through the solve; [D / 16][3][64][16]: k D(63,j)
  float* qt;        // [64][D]: q D(i,-1)
  float* aqk;       // [64][64]: scores of the read-out in the 16-column blocks up to the diagonal's, zero above the diagonal there
  float* u;         // Wv, [V][64]; then u (from the start without the delta rule), [V / 16][64 / 8] tiles in the same place
  float* dec;       // [D]: D(63,-1)
  float* s0;        // [V / 16][D / 8] tiles: the state before the chunk
  int2* rows;       // per chunk: first row, number of rows (written by the preparation, read by the read-out)
  int h0, nh, nchunks;  // the heads of this turn, all chunks
};
// Channel d (of 16) of a token's row of pieces: the two halves of a row change places every four rows, so that the eight rows of a matrix
// load fall on different banks.
__device__ __forceinline__ int piece_at(int piece, int tok, int d) { return (piece * CH + tok) * 16 + ((((d >> 3) ^ (tok >> 2)) & 1) << 3) + (d & 7); }
// Token of a channel's row of pieces: the row's groups of eight change places with the channel, for the same reason.
__device__ __forceinline__ int wk_at(int piece, int d, int tok) { return (piece * 16 + d) * CH + (((tok >> 3) ^ (d & 7)) << 3) + (tok & 7); }
constexpr int SLICE = 3 * CH * 16;  // of 16 channels
// Tiles of 16 value columns by 8 tokens or channels, a product's sums as the lanes hold them: a warp reads and writes 512 bytes in a row.
constexpr int TILE16 = 128;
__device__ __forceinline__ int in_tile(int v, int x) { return (((v & 7) << 2) + ((x & 7) >> 1)) * 4 + ((v & 8) >> 2) + (x & 1); }
__device__ __forceinline__ int u_at(int v, int tok) { return ((v >> 4) * (CH / 8) + (tok >> 3)) * TILE16 + in_tile(v, tok); }

// Place of 16-byte group c of row r in rows of D floats.  Fragments are read as 16-byte groups 4k .. 4k + 3 of two neighbouring rows,
// or as half groups of four rows two apart: the permutation sends both to different banks.
__device__ __forceinline__ int swz(int r, int c, int D) { return r * D + ((c ^ ((r & 6) ^ ((r & 1) << 2))) << 2); }
__device__ __forceinline__ int swz1(int r, int d, int D) { return swz(r, d >> 2, D) + (d & 3); }

// Products on the tensor cores with fp32 operands: x = h + m + l in bf16 pieces, exactly (8 significant bits each), and the six products
// of pieces down to 2^-16 of the first, smallest first.  What is left out (m l, l m, l l) is below 2^-24 of the product.  The products of
// 16 terms start from zero and are added to the running sum in fp32 (the tensor core cuts its sums off, an addition rounds).
// Six products of m16n8k16 take a multiprocessor 12 cycles for 2048 multiply-adds, a third less than the fp32 pipe, and their operands
// come from shared memory once for 8 or 16 uses instead of once for two to four.
struct Piece3A { uint32_t h[4], m[4], l[4]; };
struct Piece3B { uint32_t h[2], m[2], l[2]; };
__device__ __forceinline__ uint32_t pack_bf(float x, float y) {
  __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<uint32_t*>(&t);
}
// (x, y) - (u, v), the two at once
__device__ __forceinline__ void sub2(float& x, float& y, float u, float v) {
  asm("{ .reg .b64 p, q, r; mov.b64 p, {%0, %1}; mov.b64 q, {%2, %3}; mov.b64 r, {%4, %4}; fma.rn.f32x2 p, q, r, p; mov.b64 {%0, %1}, p; }"
      : "+f"(x), "+f"(y) : "f"(u), "f"(v), "f"(-1.f));
}
__device__ __forceinline__ void add2(float& x, float& y, float u, float v) {
  asm("{ .reg .b64 p, q; mov.b64 p, {%0, %1}; mov.b64 q, {%2, %3}; add.rn.f32x2 p, p, q; mov.b64 {%0, %1}, p; }"
      : "+f"(x), "+f"(y) : "f"(u), "f"(v));
}
__device__ __forceinline__ void split3(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf(x, y);
  sub2(x, y, low_bf(h), high_bf(h));
  m = pack_bf(x, y);
  sub2(x, y, low_bf(m), high_bf(m));
  l = pack_bf(x, y);
}
__device__ __forceinline__ void mma16(float* c, const uint32_t* a, const uint32_t* b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma16_from_zero(float* c, const uint32_t* a, const uint32_t* b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
// t[i] = a[i * STEP] b[i] for N tiles of eight columns
template <int N, int STEP = 1>
__device__ __forceinline__ void products(float (*t)[4], const Piece3A* a, const Piece3B* b) {
#pragma unroll
  for (int i = 0; i < N; ++i) mma16_from_zero(t[i], a[i * STEP].l, b[i].h);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i * STEP].h, b[i].l);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i * STEP].m, b[i].m);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i * STEP].m, b[i].h);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i * STEP].h, b[i].m);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i * STEP].h, b[i].h);
}
// The same where B (A) holds bf16 numbers, its other pieces zero: three of the six products, the others would add zeros.
template <int N>
__device__ __forceinline__ void products_whole_b(float (*t)[4], const Piece3A& a, const Piece3B* b) {
#pragma unroll
  for (int i = 0; i < N; ++i) mma16_from_zero(t[i], a.l, b[i].h);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a.m, b[i].h);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a.h, b[i].h);
}
template <int N>
__device__ __forceinline__ void products_whole_a(float (*t)[4], const Piece3A* a, const Piece3B* b) {
#pragma unroll
  for (int i = 0; i < N; ++i) mma16_from_zero(t[i], a[i].h, b[i].l);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i].h, b[i].m);
#pragma unroll
  for (int i = 0; i < N; ++i) mma16(t[i], a[i].h, b[i].h);
}
template <int N>
__device__ __forceinline__ void product(float (*t)[4], const Piece3A& a, const Piece3B* b) { products<N, 0>(t, &a, b); }
// c[i] += a b[i]
template <int N>
__device__ __forceinline__ void add_product(float (*c)[4], const Piece3A& a, const Piece3B* b) {
  float t[N][4];
  product<N>(t, a, b);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    add2(c[i][0], c[i][1], t[i][0], t[i][1]);
    add2(c[i][2], c[i][3], t[i][2], t[i][3]);
  }
}
// The pieces of a 16 x 16 tile of A from the 16-byte groups that this lane holds of rows g and g + 8 (the group's four columns are the
// lane's four places in k; B's rows are read the same way), and of a 16 x 8 tile of B.
__device__ __forceinline__ void split_a(const float4& r0, const float4& r1, Piece3A& p) {
  split3(r0.x, r0.y, p.h[0], p.m[0], p.l[0]);
  split3(r1.x, r1.y, p.h[1], p.m[1], p.l[1]);
  split3(r0.z, r0.w, p.h[2], p.m[2], p.l[2]);
  split3(r1.z, r1.w, p.h[3], p.m[3], p.l[3]);
}
__device__ __forceinline__ void split_b(float x, float y, float z, float w, Piece3B& p) {
  split3(x, y, p.h[0], p.m[0], p.l[0]);
  split3(z, w, p.h[1], p.m[1], p.l[1]);
}
// Two tiles of sums, side by side, are the operand A of the next product as they are.
__device__ __forceinline__ void split_sums(const float* c0, const float* c1, Piece3A& p) {
  split3(c0[0], c0[1], p.h[0], p.m[0], p.l[0]);
  split3(c0[2], c0[3], p.h[1], p.m[1], p.l[1]);
  split3(c1[0], c1[1], p.h[2], p.m[2], p.l[2]);
  split3(c1[2], c1[3], p.h[3], p.m[3], p.l[3]);
}
// Two neighbouring tiles of B from their pieces, `next` apart: a lane names one row of eight of the four 8 x 8 matrices
template <bool TRANS>
__device__ __forceinline__ void load_b(Piece3B* b, const bf16* p, int next) {
  uint32_t f[3][4];
#pragma unroll
  for (int e = 0; e < 3; ++e) TRANS ? ldm4t(f[e], p + e * next) : ldm4(f[e], p + e * next);
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      b[j].h[e] = f[0][2 * j + e];
      b[j].m[e] = f[1][2 * j + e];
      b[j].l[e] = f[2][2 * j + e];
    }
}
__device__ __forceinline__ void load_a(Piece3A& a, const bf16* p, int next) {
  ldm4(a.h, p);
  ldm4(a.m, p + next);
  ldm4(a.l, p + 2 * next);
}

template <int N, typename T> __device__ __forceinline__ void load_n(const T* p, bool vec, float* f) {
  Row<T, N> r;
  r.load(p, vec);
  r.to(f);
}
template <int N, typename T> __device__ __forceinline__ bool by_n(const T* p, long long stride) {
  return ((uintptr_t)p % (N * sizeof(T))) == 0 && stride % N == 0;
}
// N neighbouring floats of shared or global memory, N * 4 bytes aligned
template <int N> __device__ __forceinline__ void get_n(const float* p, float* f) { load_n<N>(p, true, f); }
template <int N> __device__ __forceinline__ void put_n(float* p, const float* f) {
  if (N == 4) *reinterpret_cast<float4*>(p) = make_float4(f[0], f[N > 1 ? 1 : 0], f[N > 2 ? 2 : 0], f[N > 3 ? 3 : 0]);
  else if (N == 2) *reinterpret_cast<float2*>(p) = make_float2(f[0], f[N > 1 ? 1 : 0]);
  else p[0] = f[0];
}

// Shared memory of the preparation, in floats.
template <int D, bool DELTA> struct PrepLayout {
  static constexpr int TD = 20, PD = CH + 8;  // row lengths of the triangle's 16 x 16 blocks, of the pieces (rows four banks apart)
  static constexpr int pieces = 3 * CH * PD / 2, inv = pieces + CH * TD;
  static constexpr int q = 0, k = DELTA && inv > CH * D ? inv : CH * D;  // the inverse lies over q once the scores are there,
  static constexpr int s = k + CH * D;                                   // the triangle over the columns of the scores
  static constexpr int mid = s + (DELTA && pieces > CH * D ? pieces : CH * D), t8 = mid + 12 * D, dg = t8 + 8 * D, b = dg + 2 * CH * 8, total = b + CH;
};

// Scores of 16 rows (first: r0; of shared memory `rows`, decayed from the start of their eight) against the eights of columns b0 .. b0 + N - 1
// of `cols` (decayed to the end of their eight); the eights in between are in `mid`.
template <int D, int N>
__device__ __forceinline__ void score_tiles(float (*c)[4], const float* rows, const float* cols, const float* t8, const float* mid, int s, int b0) {
  int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll 2
  for (int kp = 0; kp < D / 16; ++kp) {
    int d = 16 * kp + 4 * t;
    float4 r0 = *reinterpret_cast<const float4*>(rows + swz(16 * s + g, 4 * kp + t, D));
    float4 r1 = *reinterpret_cast<const float4*>(rows + swz(16 * s + 8 + g, 4 * kp + t, D));
    float4 f = *reinterpret_cast<const float4*>(t8 + 2 * s * D + d);  // the second eight rows reach back over the first
    r1.x *= f.x; r1.y *= f.y; r1.z *= f.z; r1.w *= f.w;
    Piece3A a;
    split_a(r0, r1, a);
    Piece3B b[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      float4 x = *reinterpret_cast<const float4*>(cols + swz(8 * (b0 + i) + g, 4 * kp + t, D));
      float4 m = *reinterpret_cast<const float4*>(mid + (s * (s - 1) + b0 + i) * D + d);
      split_b(x.x * m.x, x.y * m.y, x.z * m.z, x.w * m.w, b[i]);
    }
    add_product<N>(c, a, b);
  }
}
// Scores of the second eight rows of sub-block s against its first eight columns: rows of q on top, of k below.  Two products side by side.
template <int D, bool DELTA>
__device__ __forceinline__ void score_corner(float* c, const float* q, const float* k, const float* cols, int s) {
  int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3, r = 16 * s + 8 + g;
#pragma unroll 1
  for (int kp = 0; kp < D / 16; kp += 2) {
    Piece3A a[2];
    Piece3B b[2];
    float y[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      int at = 4 * (kp + i) + t;
      float4 r0 = *reinterpret_cast<const float4*>(q + swz(r, at, D)), r1 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (DELTA) r1 = *reinterpret_cast<const float4*>(k + swz(r, at, D));
      float4 x = *reinterpret_cast<const float4*>(cols + swz(r - 8, at, D));
      split_a(r0, r1, a[i]);
      split_b(x.x, x.y, x.z, x.w, b[i]);
    }
    products<2>(y, a, b);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      add2(c[0], c[1], y[i][0], y[i][1]);
      add2(c[2], c[3], y[i][2], y[i][3]);
    }
  }
}

// What bounds it: the latency of each warp's own chain of instructions, at two blocks per SM by shared memory and registers (a block takes
// as long beside another as alone).  So everything is written to run side by side: a warp has eight tokens, a lane D / 32 channels of them,
// all their loads are out before the first is used, the exponentials and roots have no branches, and norms, decays, the running
// products within the eight and the 8 x 8 scores on its diagonal stay in registers.  All other scores are 16 x 8 tiles on the tensor
// cores.  The triangular system goes through the inverse of 1 + L: its 16 x 16 blocks on the diagonal by substitution, three warps for the
// blocks below, and then every warp multiplies 16 columns of b K and of b V by it, transposed: what a lane holds is what it stores.
// Delta, 2048 tokens, 16 heads of 128 x 128: 86 us (158 with sums and solve on the fp32 pipe, a column per thread, and loads that waited
// for one another).
template <typename T, int D, bool DELTA>
__global__ void __launch_bounds__(256, 2) gated_chunk_prep_kernel(RecArgs a, ChunkWork wk) {
  using L = PrepLayout<D, DELTA>;
  extern __shared__ __align__(128) float sm[];
  float *sQ = sm + L::q, *sK = sm + L::k, *sS = sm + L::s, *sMid = sm + L::mid, *sT8 = sm + L::t8, *sDg = sm + L::dg, *sB = sm + L::b;
  // The triangle L (b times the scores against earlier k), negated: pieces of its blocks below the diagonal, [3][64][72], and the blocks on
  // the diagonal, [4][16][20]; the inverse of 1 + L, transposed, in pieces, [3][64][72].
  bf16 *sC = reinterpret_cast<bf16*>(sm + L::s), *sT = reinterpret_cast<bf16*>(sm + L::q);
  float* nL = sm + L::q + L::pieces;
  constexpr int EC = D / 32;
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y;
  int g = lane >> 2, t4 = lane & 3;
  Piece piece = find_piece(a, CH, blockIdx.x);
  int start = piece.row, n = piece.n;
  if (blockIdx.y == 0 && tid == 0) wk.rows[blockIdx.x] = make_int2(start, n);
  size_t ch = (size_t)blockIdx.x * wk.nh + blockIdx.y;
  int kvh = h / (a.H / a.G), V = a.V;
  float* aqk = wk.aqk + ch * (CH * CH);
  float* u = wk.u + ch * ((size_t)CH * V);
  const T* v = (const T*)a.v + h * V;
  const int e0 = EC * lane;
  // ---- norms and decays of the warp's eight tokens, the loads of four at a time
  {
    const T *q = (const T*)a.q + kvh * D, *k = (const T*)a.k + kvh * D, *z = (const T*)a.z + h * D;
    bool vq = by_n<EC>(q, a.q_stride), vk = by_n<EC>(k, a.k_stride), vz = by_n<EC>(z, a.z_stride);
    float rate = DELTA ? expf(to_f(((const T*)a.a_log)[h])) : 0.f;
    float ds = 1.f / sqrtf((float)D), tau_inv = DELTA ? 0.f : 1.f / a.tau;
    bool vec = vq && vk && vz;
    float zb[EC];
#pragma unroll
    for (int e = 0; e < EC; ++e) zb[e] = a.zb ? to_f(((const T*)a.zb)[h * D + e0 + e]) : 0.f;
    constexpr int AT_ONCE = sizeof(T) == 2 ? 8 : 4;
#pragma unroll 1
    for (int t0 = 8 * warp; t0 < 8 * warp + 8; t0 += AT_ONCE) {
      Row<T, EC> qr[AT_ONCE], kr[AT_ONCE], zr[AT_ONCE];
      Row<T, 1> br[AT_ONCE];
      auto ask = [&](int m, bool x, bool y, bool w) {
        if (t0 + m >= n) return;
        size_t row = (size_t)start + t0 + m;
        qr[m].load(q + row * a.q_stride + e0, x);
        kr[m].load(k + row * a.k_stride + e0, y);
        zr[m].load(z + row * a.z_stride + e0, w);
        if (DELTA) br[m].load((const T*)a.beta + row * a.beta_stride + h, false);
      };
      if (vec) {
#pragma unroll
        for (int m = 0; m < AT_ONCE; ++m) ask(m, true, true, true);
      } else {
#pragma unroll
        for (int m = 0; m < AT_ONCE; ++m) ask(m, vq, vk, vz);
      }
#pragma unroll
      for (int m = 0; m < AT_ONCE; ++m) {
        int t = t0 + m;
        float qs = ds, ks = 1.f, qv[EC], kv[EC], zv[EC];
        qr[m].to(qv);
        kr[m].to(kv);
        zr[m].to(zv);
        if (DELTA) {
          float pq = 0.f, pk = 0.f;
#pragma unroll
          for (int e = 0; e < EC; ++e) {
            pq += qv[e] * qv[e];
            pk += kv[e] * kv[e];
          }
          qs = ds * inverse_root(warp_sum(pq) + 1e-6f);
          ks = inverse_root(warp_sum(pk) + 1e-6f);
        }
        float av[EC];
#pragma unroll
        for (int e = 0; e < EC; ++e) {
          qv[e] *= qs;
          kv[e] *= ks;
          float zz = zv[e] + zb[e], y = DELTA ? expf(-rate * softplus_flat(zz)) : expf(divided(-softplus_flat(-zz), a.tau, tau_inv));
          av[e] = t < n ? y : 1.f;  // a row behind the sequence's end changes nothing
        }
        int at = swz1(t, e0, D);
        put_n<EC>(sQ + at, qv);
        put_n<EC>(sK + at, kv);
        put_n<EC>(sS + at, av);
        if (DELTA) {
          float b;
          br[m].to(&b);
          b = sigmoid_flat(b);
          if (lane == 0) sB[t] = t < n ? b : 0.f;
        }
      }
    }
    for (int i = lane; i < 128; i += 32) sDg[(i >> 6) * (CH * 8) + 64 * warp + (i & 63)] = 0.f;
    __syncwarp();
  }
  // ---- the 8 x 8 scores on the diagonal and the products within the eight
  {
    float kk[8][EC], aa[8][EC];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int at = swz1(8 * warp + i, e0, D);
      get_n<EC>(sK + at, kk[i]);
      get_n<EC>(sS + at, aa[i]);
    }
    // columns p and 7 - p at a time: 16 sums over the channels, which meet in one exchange that leaves each lane with one
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = 0.f;
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int j = w ? 7 - p : p, base = w ? 15 - 2 * p : 0;
        float kd[EC];
#pragma unroll
        for (int e = 0; e < EC; ++e) kd[e] = kk[j][e];
#pragma unroll
        for (int i = j; i < 8; ++i) {
          float qi[EC];
          get_n<EC>(sQ + swz1(8 * warp + i, e0, D), qi);
#pragma unroll
          for (int e = 0; e < EC; ++e) {
            if (i > j) kd[e] *= aa[i][e];
            x[base + i - j] += qi[e] * kd[e];
            if (DELTA && i > j) x[base + 8 - j + i - j - 1] += kk[i][e] * kd[e];
          }
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
          float keep = up ? x[i + o] : x[i], give = up ? x[i] : x[i + o];
          x[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], 16);
      if (lane < 16) {
        int second = lane >= 15 - 2 * p, j = second ? 7 - p : p, at = second ? lane - (15 - 2 * p) : lane;
        int low = at >= 8 - j, i = low ? j + 1 + at - (8 - j) : j + at;
        sDg[low * (CH * 8) + (8 * warp + i) * 8 + j] = x[0];
      }
    }
    float run[EC];
#pragma unroll
    for (int e = 0; e < EC; ++e) run[e] = 1.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int at = swz1(8 * warp + i, e0, D);
      float qi[EC], ki[EC];
      get_n<EC>(sQ + at, qi);
#pragma unroll
      for (int e = 0; e < EC; ++e) {
        run[e] *= aa[i][e];
        qi[e] *= run[e];
        ki[e] = kk[i][e] * run[e];
      }
      put_n<EC>(sQ + at, qi);
      if (DELTA) put_n<EC>(sK + at, ki);
    }
    put_n<EC>(sT8 + warp * D + e0, run);
#pragma unroll
    for (int e = 0; e < EC; ++e) run[e] = 1.f;
#pragma unroll
    for (int j = 7; j >= 0; --j) {
      float ki[EC];
#pragma unroll
      for (int e = 0; e < EC; ++e) {
        ki[e] = kk[j][e] * run[e];
        run[e] *= aa[j][e];
      }
      put_n<EC>(sS + swz1(8 * warp + j, e0, D), ki);
    }
  }
  __syncthreads();
  // ---- products over whole eights: rows back to the chunk's start, columns to its end, the eights in between for the scores
  float front[EC];
  {
    float back[EC];
#pragma unroll
    for (int e = 0; e < EC; ++e) front[e] = back[e] = 1.f;
    for (int m = 0; m < 8; ++m) {
      float f[EC];
      get_n<EC>(sT8 + m * D + e0, f);
#pragma unroll
      for (int e = 0; e < EC; ++e) {
        if (m < warp) front[e] *= f[e];
        if (m > warp) back[e] *= f[e];
      }
    }
    float* qt = wk.qt + ch * (CH * D);
    bf16* ke = wk.kend + ch * (D / 16 * SLICE) + (e0 >> 4) * SLICE;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int t = 8 * warp + i, at = swz1(t, e0, D);
      float x[EC], y[EC];
      get_n<EC>(sQ + at, x);
      get_n<EC>(sS + at, y);
#pragma unroll
      for (int e = 0; e < EC; ++e) {
        x[e] *= front[e];
        y[e] *= back[e];
      }
      put_n<EC>(qt + t * D + e0, x);
      if (EC == 1) {  // (a lane's pair is its own and its neighbour's)
        float z = __shfl_down_sync(0xffffffffu, y[0], 1);
        uint32_t p[3];
        split3(y[0], z, p[0], p[1], p[2]);
        if (!(lane & 1))
#pragma unroll
          for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(ke + piece_at(e, t, e0 & 15)) = p[e];
      } else {
        uint32_t p[3][2];
#pragma unroll
        for (int e = 0; e + 1 < EC; e += 2) split3(y[e], y[e + 1 < EC ? e + 1 : 0], p[0][e / 2], p[1][e / 2], p[2][e / 2]);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          bf16* o = ke + piece_at(e, t, e0 & 15);
          if (EC == 4) *reinterpret_cast<uint2*>(o) = make_uint2(p[e][0], p[e][1]);
          else *reinterpret_cast<uint32_t*>(o) = p[e][0];
        }
      }
    }
    if (warp == 7) {
      float f[EC];
      get_n<EC>(sT8 + 7 * D + e0, f);
#pragma unroll
      for (int e = 0; e < EC; ++e) f[e] *= front[e];
      put_n<EC>(wk.dec + ch * D + e0, f);
    }
    for (int m = warp; m < 12; m += 8) {
      int s = m >= 6 ? 3 : m >= 2 ? 2 : 1, b = m - s * (s - 1);
      float f[EC];
#pragma unroll
      for (int e = 0; e < EC; ++e) f[e] = 1.f;
      for (int i = b + 1; i < 2 * s; ++i) {
        float x[EC];
        get_n<EC>(sT8 + i * D + e0, x);
#pragma unroll
        for (int e = 0; e < EC; ++e) f[e] *= x[e];
      }
      put_n<EC>(sMid + m * D + e0, f);
    }
    if (!DELTA) {  // u is v: a lane has a token, so that its stores are a row's
      bool vv = by_n<4>(v, a.v_stride);
      int t = (warp & 1) * 32 + lane;
      Row<T, 4> r[8];
      auto ask = [&](bool vec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          int j = 4 * (warp >> 1) + 16 * i;
          if (t < n && j < V) r[i].load(v + ((size_t)start + t) * a.v_stride + j, vec);
        }
      };
      if (vv) ask(true);
      else ask(false);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        int j = 4 * (warp >> 1) + 16 * i;
        float f[4];
        r[i].to(f);
        if (j < V)
#pragma unroll
          for (int e = 0; e < 4; ++e) u[u_at(j + e, t)] = f[e];
      }
    }
  }
  __syncthreads();
  // ---- scores: the tiles below the diagonal's eights, by warps (of 12 tiles for q and 12 for k three each, or 12 by two), and the four corners
  float c[3][4] = {}, c2[2][4] = {};
  constexpr int NB = DELTA ? 3 : 2;
  int mat = DELTA ? warp >> 2 : 0, role = DELTA ? warp & 3 : warp;
  int s1 = DELTA ? (role < 2 ? 3 : role == 2 ? 2 : 1) : role < 3 ? 3 : role < 5 ? 2 : 1;
  int b1 = DELTA ? (role == 1 ? 3 : 0) : role < 3 ? 2 * role : role < 5 ? 2 * role - 6 : 0;
  const float* rows = mat ? sK : sQ;
  bool tiles = DELTA || role < 6, extra = DELTA && role == 3;  // the fourth tile of the third sub-block goes with the two of the second
  int n1 = DELTA && role < 3 ? 3 : 2;
  if (DELTA && role < 3) score_tiles<D, NB>(c, rows, sS, sT8, sMid, s1, b1);
  else if (tiles) score_tiles<D, 2>(c, rows, sS, sT8, sMid, s1, b1);
  if (extra) score_tiles<D, 1>(c + 2, rows, sS, sT8, sMid, 2, 3);
  int nc = DELTA ? ((warp & 1) ? 0 : 1) : warp >= 6 ? 2 : 0, corner = DELTA ? warp >> 1 : 2 * (warp - 6);
#pragma unroll
  for (int i = 0; i < (DELTA ? 1 : 2); ++i)
    if (i < nc) score_corner<D, DELTA>(c2[i], sQ, sK, sS, corner + i);
  auto place = [&](int i, int& row, int& col) {  // of tile i: the first row, the first column
    row = extra && i == 2 ? 32 : 16 * s1;
    col = 8 * (extra && i == 2 ? 3 : b1 + i);
  };
  int nt = !tiles ? 0 : extra ? 3 : n1;
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (mat == 0 && i < nt) {
      int r, j;
      place(i, r, j);
      *reinterpret_cast<float2*>(aqk + (r + g) * CH + j + 2 * t4) = make_float2(c[i][0], c[i][1]);
      *reinterpret_cast<float2*>(aqk + (r + 8 + g) * CH + j + 2 * t4) = make_float2(c[i][2], c[i][3]);
    }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (i < nc)
      *reinterpret_cast<float2*>(aqk + (16 * (corner + i) + 8 + g) * CH + 16 * (corner + i) + 2 * t4) = make_float2(c2[i][0], c2[i][1]);
  {  // the diagonal's eights, and zeros in the rest of its 16 x 16 blocks
    int r = tid >> 2, q4 = tid & 3;
    bool odd = (r >> 3) & 1;
    if (odd ? q4 >= 2 : true) {
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (odd || q4 < 2) f = *reinterpret_cast<const float4*>(sDg + r * 8 + 4 * (q4 & 1));
      *reinterpret_cast<float4*>(aqk + r * CH + (r & ~15) + 4 * q4) = f;
    }
  }
  if (!DELTA) return;
  __syncthreads();
  // ---- the triangle, negated, and b k D(i, -1) in place of k.  Within a 16 x 16 block of pieces token 4 q + 2 j + e stands in place
  // 8 j + 2 q + e, so that the four tokens that a lane has of two tiles are neighbours.
  auto spot = [](int t) { return (t & ~15) + ((t & 2) << 2) + ((t & 12) >> 1) + (t & 1); };
  auto put_pieces = [&](int row, int col, float x, float y) {
    uint32_t p[3];
    split3(x, y, p[0], p[1], p[2]);
#pragma unroll
    for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(sC + (e * CH + spot(row)) * L::PD + spot(col)) = p[e];
  };
#pragma unroll
  for (int i = 0; i < NB; ++i)
    if (mat == 1 && i < nt) {
      int r, j;
      place(i, r, j);
      float b0 = -sB[r + g], b8 = -sB[r + 8 + g];
      put_pieces(r + g, j + 2 * t4, b0 * c[i][0], b0 * c[i][1]);
      put_pieces(r + 8 + g, j + 2 * t4, b8 * c[i][2], b8 * c[i][3]);
    }
  if (nc) {
    int r = 16 * corner + 8 + g;
    float b = -sB[r];
    *reinterpret_cast<float2*>(nL + r * L::TD + 2 * t4) = make_float2(b * c2[0][2], b * c2[0][3]);
  }
  {
    int r = tid >> 2, j = 2 * (tid & 3);
    float b = -sB[r];
    const float* f = sDg + CH * 8 + r * 8 + j;
    *reinterpret_cast<float2*>(nL + r * L::TD + (r & 8) + j) = make_float2(b * f[0], b * f[1]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int t = 8 * warp + i, at = swz1(t, e0, D);
    float x[EC], b = sB[t];
    get_n<EC>(sK + at, x);
#pragma unroll
    for (int e = 0; e < EC; ++e) x[e] *= b * front[e];
    put_n<EC>(sK + at, x);
  }
  __syncthreads();
  // places of this lane's row in the matrix loads of two tiles of B, from rows of the second index (sC) and of the first (sT), and of A
  const int cat = ((lane & 7) + ((lane >> 4) << 3)) * L::PD + (lane & 8), tat = (lane & 15) * L::PD + ((lane >> 4) << 3);
  // a warp solves for 16 columns of K, of V or of both; V's rows are asked for here, together
  const int vt = warp < D / 16 ? warp + 8 - D / 16 : warp - D / 16;  // the warp's tile of V
  Row<T, 2> vr[16];
  {
    bool v2 = by_n<2>(v, a.v_stride);
    auto ask = [&](bool vec) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        int t = SB * (i >> 2) + 4 * t4 + (i & 3);
        if (t < n) vr[i].load(v + ((size_t)start + t) * a.v_stride + 16 * vt + 2 * g, vec);
      }
    };
    if (16 * vt < V) {
      if (v2) ask(true);
      else ask(false);
    }
  }
  if (tid < 4 * SB) {  // the inverted blocks on the diagonal, a column per thread, four rows finished at a time
    int s = tid >> 4, col = tid & 15;
    float x[SB];
#pragma unroll
    for (int i = 0; i < SB; ++i) x[i] = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < SB; j0 += 4)
#pragma unroll
      for (int i = j0; i < SB; ++i) {
        float4 l = *reinterpret_cast<const float4*>(nL + (SB * s + i) * L::TD + j0);
        const float f[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j0 + e < i) x[i] += f[e] * x[j0 + e];
        if (i < j0 + 4) x[i] = i < col ? 0.f : i == col ? 1.f : x[i];
      }
    bf16* o = sT + spot(SB * s + col) * L::PD + SB * s;
#pragma unroll
    for (int i = 0; i < SB; i += 2) {
      uint32_t p[3];
      split3(x[i], x[i + 1], p[0], p[1], p[2]);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint32_t*>(o + e * CH * L::PD + spot(i)) = p[e];
    }
  }
  __syncthreads();
  // A value that is not finite must reach the rows from its own on and no others, and a zero of an inverted block would carry it to the
  // rows before: it enters a product as zero, and from its row on the column is undefined.  x: tiles of sums or values of 16 tokens; lost0,
  // lost1: the first such token of a lane's two columns.
  auto keep_out = [&](float* x0, float* x1, int s, int& lost0, int& lost1) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float& x = j ? x1[e] : x0[e];
        if (!finite(x)) {
          int t = SB * s + 4 * t4 + 2 * j + (e & 1);
          if (e < 2) lost0 = min(lost0, t);
          else lost1 = min(lost1, t);
          x = 0.f;
        }
      }
  };
  auto meet = [](int& lost0, int& lost1) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      lost0 = min(lost0, __shfl_xor_sync(0xffffffffu, lost0, o));
      lost1 = min(lost1, __shfl_xor_sync(0xffffffffu, lost1, o));
    }
  };
  auto undefined_from = [&](float* x0, float* x1, int s, int lost0, int lost1) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (SB * s + 4 * t4 + 2 * j + (e & 1) >= (e < 2 ? lost0 : lost1)) (j ? x1[e] : x0[e]) = __int_as_float(0x7fffffff);
  };
  auto all_finite = [](const float* x0, const float* x1) {  // (any other value times zero is no number)
    float y = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) y = fmaf(x0[e], 0.f, fmaf(x1[e], 0.f, y));
    return y == 0.f;
  };
  // ---- the blocks of the inverse below the diagonal: a warp per 16 columns, 16 rows after the other
  if (warp < 3) {
    Piece3A solved[3];
    load_a(solved[0], sT + 16 * warp * (L::PD + 1) + tat, CH * L::PD);
    int lost0 = CH, lost1 = CH;
#pragma unroll
    for (int s = 1; s < 4; ++s) {  // counted from the warp's block on the diagonal
      if (warp + s > 3) break;
      int row = 16 * (warp + s);
      float x[2][4] = {};
#pragma unroll
      for (int r = 0; r < s; ++r) {
        Piece3B b[2];
        load_b<false>(b, sC + row * L::PD + 16 * (warp + r) + cat, CH * L::PD);
        add_product<2>(x, solved[r], b);
      }
      if (__any_sync(0xffffffffu, !all_finite(x[0], x[1]))) {
        keep_out(x[0], x[1], warp + s, lost0, lost1);
        meet(lost0, lost1);
      }
      Piece3A p;
      Piece3B b[2];
      split_sums(x[0], x[1], p);
      load_b<true>(b, sT + row * (L::PD + 1) + tat, CH * L::PD);
      product<2>(x, p, b);
      undefined_from(x[0], x[1], warp + s, lost0, lost1);
      split_sums(x[0], x[1], p);
      bf16* o = sT + (16 * warp + g) * L::PD + row + 2 * t4;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int at = (e & 1) * 8 * L::PD + (e >> 1) * 8;
        *reinterpret_cast<uint32_t*>(o + at) = p.h[e];
        *reinterpret_cast<uint32_t*>(o + CH * L::PD + at) = p.m[e];
        *reinterpret_cast<uint32_t*>(o + 2 * CH * L::PD + at) = p.l[e];
      }
      if (s < 3) solved[s < 3 ? s : 0] = p;
    }
  }
  // ---- the solve: the inverse times [b K | b V], 16 columns at a time, lane: columns 2 g and 2 g + 1 (rows g and g + 8 of the transposed tile)
  bf16* wko = wk.wk + ch * (D / 16 * SLICE);
  bool waited = false;
#pragma unroll 1
  for (int turn = warp < D / 16 ? 0 : 1; turn < 2; ++turn) {
    bool kpart = turn == 0;
    if (!kpart && 16 * vt >= V) break;
    int col = 16 * (kpart ? warp : vt) + 2 * g;
    Piece3A rhs[4];
    int lost0 = CH, lost1 = CH;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      float x[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        int t = SB * s + 4 * t4 + i;
        float f[2];
        if (kpart) get_n<2>(sK + swz1(t, col, D), f);
        else {
          float b = sB[t];
          vr[4 * s + i].to(f);
          f[0] *= b;
          f[1] *= b;
        }
        x[i >> 1][i & 1] = f[0];
        x[i >> 1][2 + (i & 1)] = f[1];
      }
      if (!all_finite(x[0], x[1])) keep_out(x[0], x[1], s, lost0, lost1);
      split_sums(x[0], x[1], rhs[s]);
    }
    bool any = __any_sync(0xffffffffu, lost0 < CH || lost1 < CH);
    if (any) meet(lost0, lost1);
    if (!waited) __syncthreads();  // the inverse is there
    waited = true;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      float x[2][4] = {};
#pragma unroll
      for (int r = 0; r <= s; r += 2) {  // two blocks of rows side by side
        Piece3A p[4];
        Piece3B b[4];
        float y[4][4];
        const int both = r < s ? 4 : 2;
#pragma unroll
        for (int i = 0; i < both; i += 2) {
          load_b<true>(b + i, sT + 16 * (r + i / 2) * L::PD + 16 * s + tat, CH * L::PD);
          p[i] = p[i + 1] = rhs[r + i / 2 < 4 ? r + i / 2 : 0];
        }
        if (r < s) products<4>(y, p, b);
        else products<2>(y, p, b);
#pragma unroll
        for (int i = 0; i < both; ++i) {
          add2(x[i & 1][0], x[i & 1][1], y[i][0], y[i][1]);
          add2(x[i & 1][2], x[i & 1][3], y[i][2], y[i][3]);
        }
      }
      if (any) undefined_from(x[0], x[1], s, lost0, lost1);
      int t = SB * s + 4 * t4;
      if (kpart) {
        Piece3A p;
        split_sums(x[0], x[1], p);
        bf16* o = wko + warp * SLICE;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          *reinterpret_cast<uint2*>(o + wk_at(0, 2 * g + e, t)) = make_uint2(p.h[e], p.h[2 + e]);
          *reinterpret_cast<uint2*>(o + wk_at(1, 2 * g + e, t)) = make_uint2(p.m[e], p.m[2 + e]);
          *reinterpret_cast<uint2*>(o + wk_at(2, 2 * g + e, t)) = make_uint2(p.l[e], p.l[2 + e]);
        }
      } else {
        *reinterpret_cast<float4*>(u + col * CH + t) = make_float4(x[0][0], x[0][1], x[1][0], x[1][1]);
        *reinterpret_cast<float4*>(u + (col + 1) * CH + t) = make_float4(x[0][2], x[0][3], x[1][2], x[1][3]);
      }
    }
  }
  if (!waited) __syncthreads();
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

// Shared memory of the chain, in bytes.
template <int D, bool DELTA> struct ChainLayout {
  static constexpr int KS = DELTA ? 2 : 3;  // tiles of Kend in flight or in use: without the delta rule a chunk is too short to hide one copy
  static constexpr int tile = D / 16 * SLICE * 2, UP = CH + 8;  // rows of the pieces of u: four banks apart
  static constexpr int wk = 0, ke = wk + (DELTA ? 2 * tile : 0), u = ke + KS * tile, total = u + 2 * 3 * 16 * UP * 2;
};

// The chain, transposed: a block has 16 value columns, which are the rows of its tiles, a warp 16 key channels (D / 16 warps, and one more
// that asks for the copies; 128 blocks for 16 heads of 128 columns, one to an SM).  A warp's part of the state is two tiles of sums in
// registers.  Per chunk: the warps' shares of Wk S (each its own channels; the sums are operand A as they lie; a share takes the place of
// the warp's slice of Wk), then a warp adds up the shares of 8 tokens (64 / D of 128 / D), whose u = Wv - Wk S goes to shared memory in
// pieces, then its part of the state.  Wk and Kend arrive as bulk copies, in pieces (eight blocks read each: cutting them up here was half of
// the instructions), while the chunk before is worked on.  Bound by the tensor cores' products (96 a warp and chunk: 1536 of 4200
// cycles) and what lies between them and the barriers; with the state's pieces in shared memory for all warps, each with its own
// tokens, it was 4400: three times the operands from shared memory.
// Delta, 2048 tokens, 16 heads of 128 x 128: 71 us (104 on the fp32 pipe, six wavefronts of shared memory for eight multiply-adds).
// When a wait for a copy runs out, the step's status word is set, no more copies are started, and the state and the outputs that depend
// on it become NaN: nothing that was computed from a tile that is not there passes for a result.
template <int D, bool DELTA, bool WHOLE>  // WHOLE: u is v, in bf16
__global__ void __launch_bounds__(2 * D + 32, DELTA ? 1 : 2) gated_chunk_chain_kernel(RecArgs a, ChunkWork wk) {
  using L = ChainLayout<D, DELTA>;
  constexpr int NW = D / 16, TILE = NW * SLICE, KS = L::KS, NT = 8 / NW;  // NT: tiles of eight tokens for a warp
  extern __shared__ __align__(128) unsigned char smb[];
  bf16* sWk = reinterpret_cast<bf16*>(smb + L::wk);  // [2][NW][3][16][64] (delta)
  bf16* sKe = reinterpret_cast<bf16*>(smb + L::ke);  // [KS][NW][3][64][16]
  bf16* sU = reinterpret_cast<bf16*>(smb + L::u);    // [2][3][16][72]
  __shared__ __align__(8) uint64_t bar[5];           // Wk, Kend
  __shared__ int stop;
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y, V = a.V, j0 = blockIdx.z * 16;
  int g = lane >> 2, t4 = lane & 3;
  int count = pieces_of(a, a.meta[4 * blockIdx.x + 1], CH);
  if (count == 0) return;
  int first = pieces_before(a, CH, blockIdx.x);
  count = min(count, wk.nchunks - first);  // (lengths that are not those the work space was laid out for)
  auto tile = [&](const bf16* p, int c) { return p + ((size_t)(first + c) * wk.nh + blockIdx.y) * TILE; };
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 5; ++i) bar_init(bar + i);
    stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (warp == NW) {  // the copies; the barriers are those of the other warps' loop
    auto wk_copy = [&](int c) {
      if (DELTA && lane == 0 && c < count) bulk_load(sWk + (c & 1) * TILE, tile(wk.wk, c), TILE * 2, bar + (c & 1));
    };
    auto ke_copy = [&](int c) {
      if (lane == 0 && c < count) bulk_load(sKe + c % KS * TILE, tile(wk.kend, c), TILE * 2, bar + 2 + c % KS);
    };
    wk_copy(0);
    ke_copy(0);
    wk_copy(1);
    if (!DELTA) ke_copy(1);
    for (int c = 0; c < count; ++c) {
      if (DELTA) __syncthreads();
      if (DELTA && !*(volatile int*)&stop) ke_copy(c + 1);  // over the one that the chunk before has used
      __syncthreads();
      if (*(volatile int*)&stop) continue;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // behind the shares
      DELTA ? wk_copy(c + 2) : ke_copy(c + 2);
    }
    return;
  }
  // this lane's part of the state: value columns g and g + 8, channels d0, d0 + 1 and d0 + 8, d0 + 9
  int d0 = warp * 16 + 2 * t4;
  float* gS = a.state + ((size_t)a.meta[4 * blockIdx.x + 2] * a.H + h) * D * V + (size_t)d0 * V + j0 + g;
  float s[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[i][e] = gS[(size_t)(8 * i + (e & 1)) * V + 8 * (e >> 1)];
  // the chunk's decay of this lane's channels, and its part of Wv (or v): the same columns, two neighbouring tokens of each tile
  float dec[2][2] = {}, wv[NT][4] = {};
  auto utile = [&](int c) { return wk.u + ((size_t)(first + c) * wk.nh + blockIdx.y) * ((size_t)CH * V) + j0 * CH; };
  auto fetch = [&](int c) {
    const float* p = wk.dec + ((size_t)(first + c) * wk.nh + blockIdx.y) * D + d0;
    get_n<2>(p, dec[0]);
    get_n<2>(p + 8, dec[1]);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float* q = utile(c);
      if (DELTA) {
        q += g * CH + 8 * (warp + NW * i) + 2 * t4;
        get_n<2>(q, wv[i]);
        get_n<2>(q + 8 * CH, wv[i] + 2);
      } else {
        get_n<4>(q + (warp + NW * i) * TILE16 + 4 * lane, wv[i]);
      }
    }
  };
  if (count > 0) fetch(0);
  const float nan = __int_as_float(0x7fffffff);
  bool lost = false;
  auto lose = [&]() {
    lost = true;
    *(volatile int*)&stop = 1;
    if (a.status) atomicExch(a.status, 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) s[0][e] = s[1][e] = nan;
  };
  // places of this lane's row in the matrix loads: of Wk 16 channels by two tiles of eight tokens (the tiles' number by exclusive or), of
  // Kend 16 tokens by two tiles of eight channels
  const int wat = warp * SLICE + (lane & 15) * CH, wx = (lane >> 4) ^ (lane & 7), kat = warp * SLICE + piece_at(0, lane & 15, (lane >> 4) << 3);
  for (int c = 0; c < count; ++c) {
    int b = c & 1;
    if (DELTA) {
      Piece3A p;
      split_sums(s[0], s[1], p);
      if (!lost && !bar_wait(bar + b, (c >> 1) & 1)) lose();
      const bf16* w = sWk + b * TILE + wat;
      float r[8][4];
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        Piece3B q[4];
        load_b<true>(q, w + ((wx ^ i) << 3), 16 * CH);
        load_b<true>(q + 2, w + ((wx ^ (i + 2)) << 3), 16 * CH);
        product<4>(r + i, p, q);
      }
      if (lost)
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i][0] = r[i][1] = r[i][2] = r[i][3] = nan;
      __syncwarp();  // the slice has been read
      float4* o = reinterpret_cast<float4*>(sWk + b * TILE + warp * SLICE) + lane;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[32 * i] = make_float4(r[i][0], r[i][1], r[i][2], r[i][3]);
      __syncthreads();  // the shares are there; nobody reads the chunk before's Kend any more
    }
    bf16* uc = sU + b * (3 * 16 * L::UP);
    float x[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i][e] = wv[i][e];
      if (DELTA) {
        const float4* f0 = reinterpret_cast<const float4*>(sWk + b * TILE) + 32 * (warp + NW * i) + lane;
        float y[4] = {};
#pragma unroll
        for (int p = 0; p < NW; ++p) {
          float4 f = f0[p * (SLICE / 8)];
          add2(y[0], y[1], f.x, f.y);
          add2(y[2], y[3], f.z, f.w);
        }
        sub2(x[i][0], x[i][1], y[0], y[1]);
        sub2(x[i][2], x[i][3], y[2], y[3]);
        if (lost) x[i][0] = x[i][1] = x[i][2] = x[i][3] = nan;
      }
      bf16* o = uc + g * L::UP + 8 * (warp + NW * i) + 2 * t4;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        uint32_t f[3];
        split3(x[i][2 * e], x[i][2 * e + 1], f[0], f[1], f[2]);
#pragma unroll
        for (int k = 0; k < (WHOLE ? 1 : 3); ++k) *reinterpret_cast<uint32_t*>(o + (k * 16 + 8 * e) * L::UP) = f[k];
      }
    }
    if (!lost && !bar_wait(bar + 2 + c % KS, (c / KS) & 1)) lose();
    const bf16 *ke = sKe + c % KS * TILE + kat, *at = uc + (lane & 15) * L::UP + 8 * (lane >> 4);
    Piece3B q[4][2];
    load_b<true>(q[0], ke, CH * 16);
    load_b<true>(q[1], ke + 16 * 16, CH * 16);
    __syncthreads();  // u's pieces are there; nobody reads the shares any more
    load_b<true>(q[2], ke + 2 * (16 * 16), CH * 16);
    load_b<true>(q[3], ke + 3 * (16 * 16), CH * 16);
    {  // the state before the chunk, for the read-out
      float* o = wk.s0 + ((size_t)(first + c) * wk.nh + blockIdx.y) * ((size_t)D * V) + (blockIdx.z * (D / 8) + 2 * warp) * TILE16 + 4 * lane;
      put_n<4>(o, s[0]);
      put_n<4>(o + TILE16, s[1]);
    }
    if (DELTA)
#pragma unroll
      for (int i = 0; i < NT; ++i) put_n<4>(utile(c) + (warp + NW * i) * TILE16 + 4 * lane, x[i]);  // (every warp has its part of Wv)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[i][e] *= dec[i][e & 1];
    fetch(min(c + 1, count - 1));  // (without a branch: values that two paths bring are moved, and the move waits for them)
#pragma unroll
    for (int kp = 0; kp < CH / 16; kp += 2) {  // two products of 16 tokens side by side
      Piece3A p[4];
      Piece3B f[4];
      float t[4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (WHOLE) ldm4(p[2 * i].h, at + 16 * (kp + i));
        else load_a(p[2 * i], at + 16 * (kp + i), 16 * L::UP);
        p[2 * i + 1] = p[2 * i];
        f[2 * i] = q[kp + i][0];
        f[2 * i + 1] = q[kp + i][1];
      }
      if (WHOLE) products_whole_a<4>(t, p, f);
      else products<4>(t, p, f);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          add2(s[j][0], s[j][1], t[2 * i + j][0], t[2 * i + j][1]);
          add2(s[j][2], s[j][3], t[2 * i + j][2], t[2 * i + j][3]);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) gS[(size_t)(8 * i + (e & 1)) * V + 8 * (e >> 1)] = s[i][e];
}

// The read-out: [64][D + 64] times [V][D + 64] transposed in steps of 32 columns.  The block cuts each step's values into pieces once, into
// one of two places in shared memory, while the next step's are on their way to its registers; a warp has 32 rows and 32 value columns.
// Bound by the tensor cores' products (four to five hundred a warp, two blocks to an SM) beside the cutting up.
// Delta, 2048 tokens, 16 heads of 128 x 128: 46 us (65 on the fp32 pipe).
template <int V1> struct OutLayout {
  static constexpr int KT = 32, group = (CH + V1) * 8 + 16, piece = KT / 8 * group, stage = 3 * piece;  // in bf16: eight columns of all rows
};

template <typename T, int D, bool DELTA>
__global__ void __launch_bounds__(256, 2) gated_chunk_out_kernel(RecArgs a, ChunkWork wk) {
  constexpr int KT = 32, STEPS = (D + CH) / KT;
  constexpr bool WHOLE = !DELTA && sizeof(T) == 2;  // u is v, in bf16: half of its products
  using L = OutLayout<128>;
  extern __shared__ __align__(128) bf16 sp[];  // [2][3][4][64 + V][8]: the rows of A, then of B; groups of eight columns 32 bytes further apart
  __shared__ __align__(16) float sSum[CH][4];
  int V = a.V;
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = wk.h0 + blockIdx.y;
  int g = lane >> 2, t4 = lane & 3, r0 = 32 * (warp & 1), v0 = 32 * (warp >> 1);
  int start = wk.rows[blockIdx.x].x, n = wk.rows[blockIdx.x].y;
  size_t ch = (size_t)blockIdx.x * wk.nh + blockIdx.y;
  const float *u = wk.u + ch * ((size_t)CH * V), *qt = wk.qt + ch * (CH * D), *aqk = wk.aqk + ch * (CH * CH), *s0 = wk.s0 + ch * ((size_t)D * V);
  // a thread has four columns of A's rows tr and tr + 32, and of up to four of B's tiles (32 columns are four tiles of each 16 value
  // columns) two columns of two rows
  int tr = tid >> 3, tc = 4 * (tid & 7), tile = tid >> 5;
  float4 f[6];
  auto fetch = [&](int st) {
    bool head = st < D / KT;
    int c0 = (head ? st * KT : st * KT - D);
    const float *A = (head ? qt : aqk) + c0 + tc, *B = (head ? s0 : u) + c0 * 16 + ((tile & 3) * TILE16) + 4 * lane;
    int ld = head ? D : CH;
#pragma unroll
    for (int i = 0; i < 2; ++i) f[i] = *reinterpret_cast<const float4*>(A + (tr + 32 * i) * ld);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (tile + 8 * i < V / 4) f[2 + i] = *reinterpret_cast<const float4*>(B + ((tile >> 2) + 2 * i) * (16 * ld));
  };
  int bad = 0;
  fetch(0);
  float acc[2][4][4] = {};
#pragma unroll 1
  for (int st = 0; st < STEPS; ++st) {
    bool head = st < D / KT;
    bf16* stage = sp + (st & 1) * L::stage;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint2 p[3];
      split3(f[i].x, f[i].y, p[0].x, p[1].x, p[2].x);
      split3(f[i].z, f[i].w, p[0].y, p[1].y, p[2].y);
      bf16* o = stage + (tc >> 3) * L::group + (tr + 32 * i) * 8 + (tc & 4);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<uint2*>(o + e * L::piece) = p[e];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (tile + 8 * i >= V / 4) continue;
      float4 x = f[2 + i];
      if (!head && !(finite(x.x) && finite(x.y) && finite(x.z) && finite(x.w))) {  // kept out of the product, see below
        bad = 1;
        x.x = finite(x.x) ? x.x : 0.f; x.y = finite(x.y) ? x.y : 0.f; x.z = finite(x.z) ? x.z : 0.f; x.w = finite(x.w) ? x.w : 0.f;
      }
      uint32_t p[3], q[3];
      split3(x.x, x.y, p[0], p[1], p[2]);
      split3(x.z, x.w, q[0], q[1], q[2]);
      bf16* o = stage + (tile & 3) * L::group + (CH + 16 * ((tile >> 2) + 2 * i) + g) * 8 + 2 * t4;
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        *reinterpret_cast<uint32_t*>(o + e * L::piece) = p[e];
        *reinterpret_cast<uint32_t*>(o + e * L::piece + 64) = q[e];
      }
    }
    if (st + 1 < STEPS) fetch(st + 1);
    __syncthreads();  // the step's pieces are there, and the other place has been read
    if (v0 < V) {
#pragma unroll
      for (int kp = 0; kp < KT / 16; ++kp) {
        int k0 = st * KT - D + 16 * kp;  // first token of these columns, behind the head
        if (!head && k0 >= r0 + 32) continue;
        const bf16* base = stage + 2 * kp * L::group;
        Piece3A p[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) load_a(p[m], base + (lane >> 4) * L::group + (r0 + 16 * m + (lane & 15)) * 8, L::piece);
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          if (v0 + 8 * i >= V) continue;
          Piece3B b[2];
          load_b<false>(b, base + ((lane >> 3) & 1) * L::group + (CH + v0 + 8 * i + (lane & 7) + ((lane >> 4) << 3)) * 8, L::piece);
          if (WHOLE && !head) {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (m == 0 && k0 >= r0 + 16) continue;
              float t[2][4];
              products_whole_b<2>(t, p[m], b);
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                add2(acc[m][i + j][0], acc[m][i + j][1], t[j][0], t[j][1]);
                add2(acc[m][i + j][2], acc[m][i + j][3], t[j][2], t[j][3]);
              }
            }
            continue;
          }
          if (head || k0 < r0 + 16) add_product<2>(acc[0] + i, p[0], b);
          add_product<2>(acc[1] + i, p[1], b);
        }
      }
    }
  }
  // A value of u that is not finite reaches the rows that see its token, and no row before it: in the products above its weight there
  // is a zero, which would not have kept it out.
  if (__syncthreads_or(bad)) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        int col = v0 + 8 * i + 2 * t4 + e, seen = CH;
        if (v0 + 8 * i < V)
          for (int j = CH - 1; j >= 0; --j)
            if (!finite(u[u_at(col, j)])) seen = j;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int r = 0; r < 2; ++r)
            if (r0 + 16 * m + 8 * r + g >= seen) acc[m][i][2 * r + e] = __int_as_float(0x7fffffff);
      }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) ss += acc[m][i][2 * r] * acc[m][i][2 * r] + acc[m][i][2 * r + 1] * acc[m][i][2 * r + 1];
      ss += __shfl_xor_sync(0xffffffffu, ss, 1);
      ss += __shfl_xor_sync(0xffffffffu, ss, 2);
      if (t4 == 0) sSum[r0 + 16 * m + 8 * r + g][warp >> 1] = ss;  // zero from the warps behind the last column
    }
  __syncthreads();
  const T *gate = (const T*)a.g + h * V, *w = (const T*)a.w;
  T* out = (T*)a.out + h * V;
  bool g2 = by_n<2>(gate, a.g_stride), w2 = by_n<2>(w, 0), o2 = by_n<2>(out, a.out_stride);
  Row<T, 2> gr[4][4], wr[4];  // the gates' rows, asked for together
  auto ask = [&](bool vec) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int col = v0 + 8 * i + 2 * t4;
      if (v0 + 8 * i >= V) continue;
      wr[i].load(w + col, vec);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        int t = r0 + 8 * m + g;
        if (t < n) gr[m][i].load(gate + ((size_t)start + t) * a.g_stride + col, vec);
      }
    }
  };
  if (g2 && w2) ask(true);
  else ask(false);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    int t = r0 + 8 * m + g;
    float4 f = *reinterpret_cast<const float4*>(sSum[t]);
    float inv = inverse_root(((f.x + f.y) + (f.z + f.w)) / V + a.eps);
    T* o = out + ((size_t)start + t) * a.out_stride + v0 + 2 * t4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float gv[2], wv[2], y[2];
      gr[m][i].to(gv);
      wr[i].to(wv);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float sg = sigmoid_flat(gv[e]);
        y[e] = acc[m >> 1][i][2 * (m & 1) + e] * inv * wv[e] * (DELTA ? sg : gv[e] * sg);
      }
      struct alignas(2 * sizeof(T)) Pair { T v[2]; };
      if (t >= n || v0 + 8 * i >= V) continue;
      if (o2) *reinterpret_cast<Pair*>(o + 8 * i) = Pair{from_f<T>(y[0]), from_f<T>(y[1])};
      else {
        o[8 * i] = from_f<T>(y[0]);
        o[8 * i + 1] = from_f<T>(y[1]);
      }
    }
  }
}

template <typename T, int D, bool DELTA>
static int run_gated_chunks(const RecArgs& a, const ChunkWork& w, int nchunks, cudaStream_t st) {
  constexpr int sp = PrepLayout<D, DELTA>::total * sizeof(float), sc = ChainLayout<D, DELTA>::total;
  constexpr int so = 2 * OutLayout<128>::stage * sizeof(bf16);  // of the widest V
  cudaError_t e = allow_smem<gated_chunk_prep_kernel<T, D, DELTA>>(sp);
  if (e == cudaSuccess) e = allow_smem<gated_chunk_chain_kernel<D, DELTA, !DELTA && sizeof(T) == 2>>(sc);
  if (e == cudaSuccess) e = allow_smem<gated_chunk_out_kernel<T, D, DELTA>>(so);
  if (e != cudaSuccess) return (int)e;
  gated_chunk_prep_kernel<T, D, DELTA><<<dim3(nchunks, w.nh), 256, sp, st>>>(a, w);
  gated_chunk_chain_kernel<D, DELTA, !DELTA && sizeof(T) == 2><<<dim3(a.nseq, w.nh, a.V / 16), 2 * D + 32, sc, st>>>(a, w);
  gated_chunk_out_kernel<T, D, DELTA><<<dim3(nchunks, w.nh), 256, so, st>>>(a, w);
  return (int)cudaGetLastError();
}

template <typename T, int D>
static int run_gated_chunks(const RecArgs& a, const ChunkWork& w, int nchunks, cudaStream_t st) {
  return a.mode == 1 ? run_gated_chunks<T, D, true>(a, w, nchunks, st) : run_gated_chunks<T, D, false>(a, w, nchunks, st);
}

__global__ void flat_math_kernel(int which, const float* __restrict__ x, float by, float* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float v = x[i];
  out[i] = which == 0 ? inverse(v) : which == 1 ? inverse_root(v) : which == 2 ? divided(v, by, 1.f / by) : which == 3 ? softplus_flat(v)
           : which == 4 ? sigmoid_flat(v) : small_tanh(v);
}

}  // namespace hyb

using namespace hyb;

extern "C" {

// The functions of hybrid_math.cuh, value by value: inverse, inverse_root, divided (by `by`), softplus_flat, sigmoid_flat, small_tanh.
int hyb_flat_math(int which, const float* x, float by, float* out, int n, cudaStream_t st) {
  if (which < 0 || which > 5 || n < 0) return -2;
  if (n == 0) return 0;
  flat_math_kernel<<<(n + 255) / 256, 256, 0, st>>>(which, x, by, out, n);
  return (int)cudaGetLastError();
}

// fp32 values (4 bytes) of work space per (chunk, head); 0: the sizes have no chunked form (key channels of 32, 64 or 128, values a
// multiple of 16 up to 128: the tiles are laid out for these, anything else keeps the token scan).
long long hyb_gated_chunk_floats(int D, int V, int mode) {
  if ((D != 32 && D != 64 && D != 128) || V % 16 || V < 16 || V > 128) return 0;
  return (long long)(mode == 1 ? 8 : 5) * CH * D / 2 + CH * CH + (long long)CH * V + D + (long long)D * V;
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
    w.qt = work + (2 * (size_t)nchunks + 31) / 32 * 32;
    w.aqk = w.qt + n * CH * a.D;
    w.u = w.aqk + n * CH * CH;
    w.s0 = w.u + n * CH * a.V;
    w.dec = w.s0 + n * a.D * a.V;
    w.kend = (bf16*)(w.dec + n * a.D);
    w.wk = w.kend + n * CH * a.D * 3;
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
