// Shared device helpers of the hybrid model family's kernels: conversions, 8-wide loads and stores, warp and block
// reductions, activations.  The files that include it are compiled WITHOUT fast-math: exponentials, divisions and
// square roots are the IEEE ones.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

namespace hyb {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ void load8(const float* p, float* f) {
  float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void load8(const bf16* p, float* f) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ void store8(float* p, const float* f) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void store8(bf16* p, const float* f) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    w[i] = *reinterpret_cast<uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float low_bf(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high_bf(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
// N values of a row as they lie in memory; `vec`: groups of N may be read at once.  Taken apart only by `to`: a value that is unpacked
// where it is loaded makes the next load wait for it.
template <typename T, int N> struct Row {
  static constexpr int W = (N * sizeof(T) + 3) / 4;
  uint32_t w[W];
  __device__ __forceinline__ Row() {
#pragma unroll
    for (int e = 0; e < W; ++e) w[e] = 0;
  }
  __device__ __forceinline__ void load(const T* p, bool vec) {
    if constexpr (N * sizeof(T) == 32) {
      if (vec) {
        uint4 t = reinterpret_cast<const uint4*>(p)[0], u = reinterpret_cast<const uint4*>(p)[1];
        w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w; w[4] = u.x; w[5] = u.y; w[6] = u.z; w[7] = u.w;
        return;
      }
    } else if constexpr (N * sizeof(T) == 16) {
      if (vec) {
        uint4 t = *reinterpret_cast<const uint4*>(p);
        w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
        return;
      }
    } else if constexpr (N * sizeof(T) == 8) {
      if (vec) {
        uint2 t = *reinterpret_cast<const uint2*>(p);
        w[0] = t.x; w[1] = t.y;
        return;
      }
    } else if constexpr (N * sizeof(T) == 4) {
      if (vec) {
        w[0] = *reinterpret_cast<const uint32_t*>(p);
        return;
      }
    }
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int e = 0; e < N; ++e) w[e] = reinterpret_cast<const uint32_t*>(p)[e];
    } else {
      const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
      for (int e = 0; e < N; e += 2) w[e / 2] = h[e] | (e + 1 < N ? (uint32_t)h[e + 1 < N ? e + 1 : e] << 16 : 0u);
    }
  }
  __device__ __forceinline__ void to(float* f) const {
#pragma unroll
    for (int e = 0; e < N; ++e) f[e] = sizeof(T) == 4 ? __uint_as_float(w[e]) : e & 1 ? high_bf(w[e / 2]) : low_bf(w[e / 2]);
  }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum over the block; every thread gets the result.  `red` holds 33 floats.  Safe to call back to back.
__device__ __forceinline__ float block_sum(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}
// The same sum (bit for bit) with one barrier: `red` holds 32 floats that nobody else writes until every thread has passed another barrier.
__device__ __forceinline__ float block_sum_once(float v, float* red) {
  int lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.f);
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float siluf_(float x) { return x / (1.f + expf(-x)); }
// SiLU for results that are rounded to T: with a 16-bit T the approximate exponential and division (a few ulp of fp32) do
template <typename T> __device__ __forceinline__ float silu_as(float x) { return siluf_(x); }
template <> __device__ __forceinline__ float silu_as<bf16>(float x) { return __fdividef(x, 1.f + __expf(-x)); }
__device__ __forceinline__ float gelu_erff_(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }

// Arguments of the gated recurrences (hybrid_mixers.cu: token by token; hybrid_gated.cu: in chunks).
struct RecArgs {
  const void *q, *k, *v, *z, *g, *beta, *zb, *a_log, *w;
  void* out;
  float* state;
  const int* meta;
  long long q_stride, k_stride, v_stride, z_stride, g_stride, beta_stride, out_stride;
  int H, G, D, V, mode;
  float tau, eps;
  int* status;       // set to 1 when a wait ran out (may be null)
  int nseq, lo, hi;  // sequences of the step; those with lo <= tokens < hi take part
};

// The tokens of the sequences that take part, cut into pieces of up to `len` and numbered one after the other: piece `i` (a whole
// warp asks; all lanes get it).  Launches are laid out by the number of pieces, so nothing has to be tabulated before them.
struct Piece { int row, n; };
__device__ __forceinline__ int pieces_of(const RecArgs& a, int tokens, int len) {
  return tokens >= a.lo && tokens < a.hi ? (tokens + len - 1) / len : 0;
}
__device__ __forceinline__ bool takes_all(const RecArgs& a) { return a.lo <= 1 && a.hi == 0x7fffffff; }
__device__ __forceinline__ Piece find_piece(const RecArgs& a, int len, int i) {
  int lane = threadIdx.x & 31, before = 0;
  for (int s0 = 0; s0 < a.nseq; s0 += 32) {
    int row = 0, n = 0;
    if (s0 + lane < a.nseq) {
      row = a.meta[4 * (s0 + lane)];
      n = a.meta[4 * (s0 + lane) + 1];
    }
    int mine = pieces_of(a, n, len), end = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int x = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += x;
    }
    unsigned hit = __ballot_sync(0xffffffffu, before + end > i);
    if (hit) {
      int l = __ffs(hit) - 1, at = (i - before - __shfl_sync(0xffffffffu, end - mine, l)) * len;
      row = __shfl_sync(0xffffffffu, row, l);
      n = __shfl_sync(0xffffffffu, n, l);
      return {row + at, min(len, n - at)};
    }
    before += __shfl_sync(0xffffffffu, end, 31);
  }
  return {0, 0};
}
// Number of the first piece of sequence `seq`.
__device__ __forceinline__ int pieces_before(const RecArgs& a, int len, int seq) {
  int k = 0;
  for (int s = threadIdx.x & 31; s < seq; s += 32) k += pieces_of(a, a.meta[4 * s + 1], len);
  return __reduce_add_sync(0xffffffffu, k);
}

// Lets KERNEL use `bytes` (always the same) of shared memory: asked for once per device, the call costs a microsecond.
template <auto KERNEL>
static cudaError_t allow_smem(int bytes) {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

}  // namespace hyb
