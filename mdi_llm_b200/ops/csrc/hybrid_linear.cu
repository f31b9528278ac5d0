// Products of few rows: y[N][O] = x[N][K] w[O][K]^T (+ b), N up to 8 (a step that brings one token for each of a few sequences), bf16
// in and out, fp32 sums.
//
// What bounds it: every weight is read once, so the HBM rate; the matrices are 8 to 130 MB, a few microseconds each, and what is
// lost is lost in ramps.  A block therefore asks for a whole tile of 16 weight rows at once where K allows it (eight warps share the
// columns, sixteen 16-byte loads in flight per lane, 64 KB per block), two blocks to an SM.  A warp reads 128 contiguous bytes of
// each of its 16 rows as the A operand of m16n8k16 straight into registers: a lane's 16 bytes are eight neighbouring columns, which
// is not the order that the instruction numbers its k in, but x is read the same way and a sum has no order.  The warps' partial
// sums meet in shared memory.  us for 8 rows, library and this, cold weights in a graph: 4160 x 2048 7.9 and 5.1, 3072 x 1536 6.8 and 4.2,
// 2048 x 2048 7.1 and 3.8, 8192 x 2048 8.0 and 8.0, 2048 x 8192 21 and 8.5, 32000 x 2048 25.9 and 22.1, 2048 x 16 2.2 and 1.9.
// With 9 to 16 rows (two groups of eight) it was slower than the library at 8192 x 2048 and 6224 x 2048: left to the library.
#include "hybrid_mma.cuh"

namespace hyb {

constexpr int FR_WARPS = 8, FR_UNROLL = 4;  // warps of a block; chunks of 64 columns that a warp asks for at a time

__device__ __forceinline__ uint4 ld_stream(const bf16* p) {  // weights: read once, not kept in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// K a multiple of 8, rows of x and w on 16-byte boundaries.  SPLIT: CTAs of a cluster that share the columns of a tile (one tile to a
// cluster); the first adds the others' sums to its own.
template <int SPLIT>
__global__ void __launch_bounds__(FR_WARPS * 32, 2)
few_rows_linear_kernel(const bf16* __restrict__ x, long long x_stride, const bf16* __restrict__ w, long long w_stride,
                       const bf16* __restrict__ b, bf16* __restrict__ y, long long y_stride, int N, int K, int O) {
  __shared__ float part[SPLIT > 1 ? 1 : 2][SPLIT * FR_WARPS][8][17];
  // Nothing is stored to the first CTA before it is known to run: everybody says so here and asks behind the products, which cover it.
  if (SPLIT > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int chunks = (K + 63) / 64, tiles = (O + 15) / 16, rank = SPLIT > 1 ? blockIdx.x % SPLIT : 0;
  const bf16* xg = x + (size_t)min(g, N - 1) * x_stride + 8 * t;  // rows from N on are computed and not stored
  int turn = 0;
  for (int tile = blockIdx.x / SPLIT; tile < tiles; tile += gridDim.x / SPLIT, turn ^= 1) {
    const bf16* w0 = w + (size_t)min(tile * 16 + g, O - 1) * w_stride + 8 * t;
    const bf16* w1 = w + (size_t)min(tile * 16 + g + 8, O - 1) * w_stride + 8 * t;
    float acc[4] = {};
    for (int c0 = rank * FR_WARPS + warp; c0 < chunks; c0 += SPLIT * FR_WARPS * FR_UNROLL) {
      uint4 wa[FR_UNROLL][2][2], xa[FR_UNROLL][2];
#pragma unroll
      for (int u = 0; u < FR_UNROLL; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = (c0 + u * SPLIT * FR_WARPS) * 64 + 32 * h;
          wa[u][h][0] = wa[u][h][1] = make_uint4(0, 0, 0, 0);
          if (k + 8 * t < K) {
            wa[u][h][0] = ld_stream(w0 + k);
            wa[u][h][1] = ld_stream(w1 + k);
          }
        }
#pragma unroll
      for (int u = 0; u < FR_UNROLL; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = (c0 + u * SPLIT * FR_WARPS) * 64 + 32 * h;
          xa[u][h] = make_uint4(0, 0, 0, 0);
          if (k + 8 * t < K) xa[u][h] = *reinterpret_cast<const uint4*>(xg + k);
        }
#pragma unroll
      for (int u = 0; u < FR_UNROLL; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 p = wa[u][h][0], q = wa[u][h][1], v = xa[u][h];
          const uint32_t a0[4] = {p.x, q.x, p.y, q.y}, a1[4] = {p.z, q.z, p.w, q.w}, b0[2] = {v.x, v.y}, b1[2] = {v.z, v.w};
          mma(acc, a0, b0);
          mma(acc, a1, b1);
        }
    }
    float(*sums)[8][17] = part[turn];
    if (SPLIT > 1) {  // the same place in the first CTA of the cluster
      __syncwarp();
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      uint64_t far;
      asm("mapa.u64 %0, %1, 0;" : "=l"(far) : "l"(sums));
      sums = reinterpret_cast<float(*)[8][17]>(far);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) sums[rank * FR_WARPS + warp][2 * t + (e & 1)][g + 8 * (e >> 1)] = acc[e];
    // (the other turn's sums are read by nobody that has not passed here)
    if (SPLIT > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
    const int r = threadIdx.x & 15, n = threadIdx.x >> 4, o = tile * 16 + r;
    if (rank == 0 && n < N && o < O) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < SPLIT * FR_WARPS; ++i) s += part[turn][i][n][r];
      if (b) s += to_f(b[o]);
      y[(size_t)n * y_stride + o] = from_f<bf16>(s);
    }
    if (SPLIT > 1) break;  // a barrier's phase for each of the two waits above, so one tile
  }
}

template <int SPLIT>
static int run_few_rows(const bf16* x, long long x_stride, const bf16* w, long long w_stride, const bf16* b, bf16* y, long long y_stride,
                        int N, int K, int O, int clusters /* SPLIT > 1: as many as tiles */, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * SPLIT);
  cfg.blockDim = dim3(FR_WARPS * 32);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = SPLIT;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = SPLIT > 1 ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, few_rows_linear_kernel<SPLIT>, x, x_stride, w, w_stride, b, y, y_stride, N, K, O);
}

}  // namespace hyb

using namespace hyb;

// x [N, K] and w [O, K] by rows (16-byte aligned, strides multiples of 8), y [N, O]; b may be null.  -2: sizes or places it does not take.
extern "C" int hyb_few_rows_linear(const void* x, long long x_stride, const void* w, long long w_stride, const void* b, void* y, long long y_stride,
                                   int N, int K, int O, cudaStream_t st) {
  if (N < 1 || N > 8 || K < 8 || K % 8 || O < 1 || x_stride % 8 || w_stride % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return -2;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 148;
  const int tiles = (O + 15) / 16;
  const bf16 *xb = (const bf16*)x, *wb = (const bf16*)w, *bb = (const bf16*)b;
  // Few tiles of many columns: two CTAs to a tile (2048 x 8192 10.0 us alone, 8.5 by two; 1024 x 4096 5.3 and 4.3).  With fewer columns
  // or more tiles the cluster's barrier costs more than the second CTA brings (2048 x 2048 3.8 and 4.4, 4096 x 1024 3.8 and 5.8).
  if (tiles <= sms && K >= 4096) return run_few_rows<2>(xb, x_stride, wb, w_stride, bb, (bf16*)y, y_stride, N, K, O, tiles, st);
  return run_few_rows<1>(xb, x_stride, wb, w_stride, bb, (bf16*)y, y_stride, N, K, O, tiles < 2 * sms ? tiles : 2 * sms, st);
}
