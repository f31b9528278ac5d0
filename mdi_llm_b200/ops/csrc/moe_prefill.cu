// Routing of a whole prompt through a mixture of experts (reference: LLaMAMoE, model.py:823-853) on the device: choice and
// weights per token, rows sorted by expert, the gather in front of the grouped GEMMs (gemm_tcgen05.cu) and the weighted sum
// behind them.  Row counts stay on the device, nothing waits for the host.  All of it moves a few rows of activations and is
// bound by launches; the sorts, scatters and bf16 atomics of a general library took 200 us for 997 tokens of top 2 of 8.
#include "common.cuh"

namespace mdi {

// A warp per token: the `top` largest of the bf16 logits (the lower index first among equals), softmax over them in fp32,
// rounded to bf16 as the eager module does.
__global__ void __launch_bounds__(256) moe_rows_route_kernel(const bf16* __restrict__ logits, int T, int E, int top, int* __restrict__ sel,
                                                             bf16* __restrict__ wts) {
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  float v[8];  // E <= 256: expert lane + 32 i
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = lane + 32 * i < E ? __bfloat162float(logits[(size_t)t * E + lane + 32 * i]) : -INFINITY;
  unsigned taken = 0;
  float mx = 0.f, z = 0.f, mine = 0.f;
  for (int k = 0; k < top; ++k) {
    float b = -INFINITY;
    int bi = 1 << 20;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(taken >> i & 1) && lane + 32 * i < E && (bi == 1 << 20 || v[i] > b || v[i] != v[i])) { b = v[i]; bi = lane + 32 * i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, b, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      const bool nan = b != b, onan = ob != ob;  // a NaN counts as the largest, as in torch.topk
      const bool other = oi != (1 << 20) && (bi == (1 << 20) || (nan != onan ? onan : (!nan && ob != b ? ob > b : oi < bi)));
      if (other) { b = ob; bi = oi; }
    }
    if ((bi & 31) == lane) taken |= 1u << (bi >> 5);
    if (k == 0) mx = b;
    const float e = expf(b - mx);
    z += e;
    if (lane == k) { mine = e; sel[(size_t)t * top + k] = bi; }
  }
  if (lane < top) wts[(size_t)t * top + lane] = __float2bfloat16_rn(mine / z);
}

// Stable order by expert: counts[e], the token of every sorted row, and the sorted place of every (token, choice).  A warp walks
// its part of the pairs (of few experts each has several warps) once to count its expert and once to place it, eight loads at a time: one
// after the other their latencies were all of it (1994 pairs of 8 experts 17.9 us, and 9.6).
__global__ void __launch_bounds__(1024, 1) moe_rows_sort_kernel(const int* __restrict__ sel, int pairs, int E, int top, int* __restrict__ counts,
                                                             int* __restrict__ token, int* __restrict__ where) {
  __shared__ int cnt[256], base[257];  // per expert and part
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int parts = E <= 16 && pairs > 256 ? 32 / E : 1, units = E * parts, part = ((pairs + parts - 1) / parts + 31) & ~31;
  auto walk = [&](int u, auto&& each) {
    const int e = parts == 1 ? u : u / parts, lo = (u - e * parts) * part, hi = min(pairs, lo + part);
    int i0 = lo;
    for (; i0 + 256 <= hi; i0 += 256) {
      int v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = sel[i0 + 32 * k + lane];
#pragma unroll
      for (int k = 0; k < 8; ++k) each(i0 + 32 * k + lane, v[k] == e);
    }
    if (i0 >= hi) return;
    int v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = i0 + 32 * k + lane < hi ? sel[i0 + 32 * k + lane] : -1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (i0 + 32 * k >= hi) break;
      each(i0 + 32 * k + lane, v[k] == e);
    }
  };
  for (int u = warp; u < units; u += 32) {
    int n = 0;
    walk(u, [&](int, bool is) { n += is; });
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) cnt[u] = n;
  }
  __syncthreads();
  if (warp == 0) {  // what comes before each unit, up to eight of them a lane (by one thread, one after the other, 7 us of 128 experts)
    const int per = (units + 31) / 32;
    int sum = 0;
    for (int k = per * lane; k < min(units, per * (lane + 1)); ++k) sum += cnt[k];
    int before = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += x;
    }
    before -= sum;
    for (int k = per * lane; k < min(units, per * (lane + 1)); ++k) {
      base[k] = before;
      before += cnt[k];
    }
    if (lane == 31) base[units] = before;
  }
  __syncthreads();
  if (threadIdx.x < E) counts[threadIdx.x] = base[(threadIdx.x + 1) * parts] - base[threadIdx.x * parts];
  for (int u = warp; u < units; u += 32) {
    int at = base[u];
    walk(u, [&](int i, bool is) {
      const unsigned m = __ballot_sync(0xffffffffu, is);
      if (is) {
        const int r = at + __popc(m & ((1u << lane) - 1u));
        token[r] = i / top;
        where[i] = r;
      }
      at += __popc(m);
    });
  }
}

__global__ void __launch_bounds__(256) moe_rows_gather_kernel(const uint4* __restrict__ h, const int* __restrict__ token, uint4* __restrict__ out, int n8) {
  const uint4* src = h + (size_t)token[blockIdx.x] * n8;
  uint4* dst = out + (size_t)blockIdx.x * n8;
  for (int i = threadIdx.x; i < n8; i += 256) dst[i] = src[i];
}

// y = bf16(x + s), s = the token's outputs times their bf16 weights, each product and each partial sum rounded to bf16 in the
// order of the choices (the eager module's rounding points).
__global__ void __launch_bounds__(256) moe_rows_combine_kernel(const bf16* __restrict__ x, const bf16* __restrict__ y, const int* __restrict__ where,
                                                               const bf16* __restrict__ wts, bf16* __restrict__ out, int top, int C) {
  const int t = blockIdx.x;
  for (int i = threadIdx.x * 8; i < C; i += 256 * 8) {
    float s[8] = {};
    for (int k = 0; k < top; ++k) {
      const uint4 v = *reinterpret_cast<const uint4*>(y + (size_t)where[(size_t)t * top + k] * C + i);
      const float w = __bfloat162float(wts[(size_t)t * top + k]);
      const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[2 * j] = round_bf16(s[2 * j] + round_bf16(bf16lo(vw[j]) * w));
        s[2 * j + 1] = round_bf16(s[2 * j + 1] + round_bf16(bf16hi(vw[j]) * w));
      }
    }
    const uint4 xv = *reinterpret_cast<const uint4*>(x + (size_t)t * C + i);
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(bf16lo(xw[j]) + s[2 * j], bf16hi(xw[j]) + s[2 * j + 1]);
    *reinterpret_cast<uint4*>(out + (size_t)t * C + i) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace mdi

using namespace mdi;

// logits [T, E] bf16 -> sel / wts [T, top], counts [E], token [T * top], where [T, top]; rows [T * top, C] = h[token]
extern "C" int mdi_moe_rows_sort(const void* logits, const void* h, int T, int E, int top, int C, int* sel, void* wts, int* counts, int* token,
                                 int* where, void* rows, cudaStream_t stream) {
  if (T <= 0 || E < 1 || E > 256 || top < 1 || top > E || top > 8 || C % 8) return -2;
  if (((uintptr_t)h | (uintptr_t)rows) & 15) return -2;
  moe_rows_route_kernel<<<(T + 7) / 8, 256, 0, stream>>>((const bf16*)logits, T, E, top, sel, (bf16*)wts);
  moe_rows_sort_kernel<<<1, 1024, 0, stream>>>(sel, T * top, E, top, counts, token, where);
  moe_rows_gather_kernel<<<T * top, 256, 0, stream>>>((const uint4*)h, token, (uint4*)rows, C / 8);
  return (int)cudaGetLastError();
}

extern "C" int mdi_moe_rows_combine(const void* x, const void* y, const int* where, const void* wts, void* out, int T, int top, int C,
                                    cudaStream_t stream) {
  if (T <= 0 || top < 1 || C % 8 || (((uintptr_t)x | (uintptr_t)y | (uintptr_t)out) & 15)) return -2;
  moe_rows_combine_kernel<<<T, 256, 0, stream>>>((const bf16*)x, (const bf16*)y, where, (const bf16*)wts, (bf16*)out, top, C);
  return (int)cudaGetLastError();
}
