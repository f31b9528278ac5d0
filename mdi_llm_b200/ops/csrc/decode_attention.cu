// Split-KV ("flash-decoding") attention for single-token decode over the slot KV pool, sm_100a.
//
// Reference behaviour being replaced: F.scaled_dot_product_attention over ALL S
// cache slots through a [1,1,1,S] boolean mask row, with K/V already expanded to n_head heads
// (model.py:704-751).  Here the cache holds the G group heads only, a CTA serves all q_per_kv
// query heads of one group from a single pass over that group's K/V (GQA packing: 4x fewer
// bytes for Llama-3) and only the live prefix [0, pos] is scanned.
//
// One kernel, grid (G, n_split), 8 warps per CTA, a warp owns 16-position tiles:
//   * the context is cut into spans of >= 128 positions, so short contexts use few CTAs and
//     the others exit at once (the grid is fixed at graph-capture time, the length is not);
//   * ALL K and V loads of a tile are issued together before anything is consumed, the next tile's as soon as a
//     tile's registers are free — decode attention is a latency chain (ctx -> q -> K -> softmax -> V -> merge), not a
//     bandwidth problem; small tiles over many warps keep the serial instruction count per warp low;
//   * scores are m16n8k16 products of bf16 K (16 positions) and bf16 q (up to eight heads are the columns), straight from the
//     registers that the loads fill: a lane's 16 bytes are eight neighbouring channels, K and q alike.  The softmax
//     of all heads runs side by side on the products' sums; weights stay fp32 and meet V on the fp32 pipe.  With scores
//     as multiply-adds on q from shared memory (four-way conflicts, one head after the other) a tile of 4 x 128 took
//     7700 cycles, now 3000; four 8B layers of fp8 weights at 2048 positions 271 us a step, now 259;
//   * the last CTA of a group to finish merges the spans (atomic ticket) and writes bf16
//     y[H*hs] directly: no separate combine launch;
//   * K / V of OLD positions do not depend on this step's QKV projection: every warp requests its first tile
//     BEFORE the programmatic-dependency wait (the kernel is resident while the QKV kernel still streams its
//     weights), so after the wait only q — and the tile that holds the newest position — remain to be fetched.
#include "common.cuh"

namespace mdi {

constexpr int ATT_WARPS = 8;
constexpr int ATT_THREADS = ATT_WARPS * 32;
constexpr int ATT_TILE = 16;

struct AttnArgs {
  const bf16* q;   // [H * hs] (already roped)
  const bf16* kv;  // this layer's pool [n_slots, 2, G, S, hs]
  bf16* y;         // [H * hs]
  float* part;     // [H, n_split, hs + 2]
  unsigned int* tickets;  // [G] zero-initialised, self-resetting
  const int* ctx;
  int n_head, n_groups, max_seq, n_split;
  float scale_log2;  // (1/sqrt(hs)) * log2(e)
  unsigned long long* trace;
  DepWait dep_wait;      // flag dependency on the QKV kernel (else griddepcontrol.wait)
  DepSignal dep_signal;  // flag for the out-projection
  int cl_iters;  // tiles per warp up to which the spans of a group are kept to one cluster
};

// CLUSTER: the spans of a KV group are launched as thread-block clusters of ATT_CL CTAs along y.  While the live
// context fits into one cluster (n_active <= ATT_CL spans: up to 1024 positions at 128 per span, longer ones by cluster_tiles) the spans are
// merged through DISTRIBUTED SHARED MEMORY: every CTA writes its (max, sum, partial output) into rank 0's shared
// memory (st.shared::cluster), one cluster barrier, rank 0 folds them and writes y — no partial buffer in global
// memory, no fence + ticket, no second round of L2 reads (measured: the global merge was 3.8 us of the kernel's 11).
// Longer contexts fall back to the ticket merge below.
constexpr int ATT_CL = 8;

__device__ __forceinline__ uint32_t att_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(const float* local_smem, uint32_t cta, float v) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(local_smem)), "r"(cta));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}

// Loads that stay where they are written: the compiler may move a read-only load (__ldg) over the dependency wait, where this step's
// newest row is not there yet.
__device__ __forceinline__ uint4 ld_here(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ld_here(const bf16* p, uint32_t (&v)[1]) { asm volatile("ld.global.u32 %0, [%1];" : "=r"(v[0]) : "l"(p) : "memory"); }
__device__ __forceinline__ void ld_here(const bf16* p, uint32_t (&v)[2]) {
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void ld_here(const bf16* p, uint32_t (&v)[4]) {
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int HS, int QPK, bool CLUSTER>
__global__ void __launch_bounds__(ATT_THREADS) attn_decode_kernel(const AttnArgs a) {
  constexpr int DPL = HS / 32;   // output dims per lane in the PV phase
  constexpr int KJ = HS / 32;    // 16-byte loads of K per lane and position: four lanes share 32 channels
  __shared__ __align__(16) float p_s[ATT_WARPS][ATT_TILE][QPK], corr_s[ATT_WARPS][QPK];
  __shared__ float mrg_m[ATT_WARPS][QPK], mrg_l[ATT_WARPS][QPK];
  __shared__ float mrg_acc[ATT_WARPS][QPK][HS];
  __shared__ int sh_last;
  __shared__ float cl_part[CLUSTER ? ATT_CL : 1][CLUSTER ? QPK : 1][CLUSTER ? HS + 2 : 1];  // rank 0: the cluster's partials

  const int g = blockIdx.x, split = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  trace_mark(a.trace, 0, true);
  // ctx was written at the start of the step (advance_step / the host's descriptor copy), at least two launches ago:
  // readable before the dependency wait
  const int slot = a.ctx[MDI_CTX_SLOT], L = a.ctx[MDI_CTX_POS] + 1;
  // spans of whole tiles, at least ATT_WARPS tiles (128 positions) each
  const int tiles = (L + ATT_TILE - 1) / ATT_TILE;
  int tiles_per_split = (tiles + a.n_split - 1) / a.n_split;
  if (tiles_per_split < ATT_WARPS) tiles_per_split = ATT_WARPS;
  // up to cl_iters tiles per warp the group's spans stay in one cluster (see cluster_tiles)
  if (CLUSTER && tiles > ATT_CL * ATT_WARPS && tiles <= ATT_CL * ATT_WARPS * a.cl_iters) tiles_per_split = (tiles + ATT_CL - 1) / ATT_CL;
  const int n_active = (tiles + tiles_per_split - 1) / tiles_per_split;
  const bool active = split < n_active;
  // merge through distributed shared memory: every live span sits in the group's first cluster.  Rank 0 must be known to run before it is
  // written to: the cluster's CTAs say so here and ask behind their tiles, which cover it.
  const bool cl_merge = CLUSTER && n_active > 1 && n_active <= ATT_CL;
  if (cl_merge && split < ATT_CL) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int t_lo = split * tiles_per_split, t_hi = min(tiles, t_lo + tiles_per_split);
  const bf16* kbase = a.kv + (((size_t)slot * 2 + 0) * a.n_groups + g) * (size_t)a.max_seq * HS;
  const bf16* vbase = a.kv + (((size_t)slot * 2 + 1) * a.n_groups + g) * (size_t)a.max_seq * HS;

  // K / V registers of one tile: all of it is requested together, so the warp's first tile can be requested before the
  // wait when it only holds positions older than this step's
  uint4 kk[2][KJ];
  uint32_t vv[ATT_TILE][DPL / 2];
  auto load_k = [&](int p0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int pos = min(p0 + 8 * r + (lane >> 2), L - 1);  // clamp: masked below
      const uint4* kr = reinterpret_cast<const uint4*>(kbase + (size_t)pos * HS + (lane & 3) * 8);
#pragma unroll
      for (int j = 0; j < KJ; ++j) kk[r][j] = ld_here(kr + 4 * j);
    }
  };
  auto load_v = [&](int p0) {
#pragma unroll
    for (int r = 0; r < ATT_TILE; ++r) {
      const int pos = min(p0 + r, L - 1);  // masked rows have p == 0
      ld_here(vbase + (size_t)pos * HS + lane * DPL, vv[r]);
    }
  };
  const int t_first = t_lo + warp;
  bool pre = false;
  if (active && t_first < t_hi && (t_first + 1) * ATT_TILE <= L - 1) {  // no row of this tile is written by this step
    load_k(t_first * ATT_TILE);
    load_v(t_first * ATT_TILE);
    pre = true;
  }
  if (a.dep_wait.flag) dep_wait(a.dep_wait, a.ctx); else pdl_wait_prior();
  trace_mark(a.trace, 1, true);
  pdl_launch_dependents();
  if (!active) {  // idle span: only its ticket (and, inside the merging cluster, its barrier arrivals)
    if (cl_merge && split < ATT_CL) {
      __syncwarp();
      asm volatile("barrier.cluster.wait.aligned;\n\tbarrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    dep_signal(a.dep_signal, a.ctx);
    return;
  }
  trace_mark(a.trace, 2, false);

  // q as operand B: column lane / 4 is a head, the channels as K's
  uint4 qf[KJ];
#pragma unroll
  for (int j = 0; j < KJ; ++j)
    qf[j] = make_uint4(0u, 0u, 0u, 0u);
  if ((lane >> 2) < QPK) {
    const bf16* qr = a.q + (size_t)(g * QPK + (lane >> 2)) * HS + (lane & 3) * 8;
    if (((uintptr_t)a.q & 15) == 0) {
#pragma unroll
      for (int j = 0; j < KJ; ++j) qf[j] = *reinterpret_cast<const uint4*>(qr + 32 * j);
    } else {
      const unsigned short* h = reinterpret_cast<const unsigned short*>(qr);
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        auto two = [&](int i) { return h[32 * j + i] | (uint32_t)h[32 * j + i + 1] << 16; };
        qf[j] = make_uint4(two(0), two(2), two(4), two(6));
      }
    }
  }
  if (!pre && t_first < t_hi) {
    load_k(t_first * ATT_TILE);
    load_v(t_first * ATT_TILE);
  }

  float m[2], l[2], acc[QPK][DPL];  // m, l: of heads 2 (lane % 4) and the next
#pragma unroll
  for (int e = 0; e < 2; ++e) { m[e] = -INFINITY; l[e] = 0.f; }
#pragma unroll
  for (int h = 0; h < QPK; ++h)
#pragma unroll
    for (int d = 0; d < DPL; ++d) acc[h][d] = 0.f;

  for (int t = t_first; t < t_hi; t += ATT_WARPS) {
    const int p0 = t * ATT_TILE, p_next = p0 + ATT_WARPS * ATT_TILE;
    const bool more = t + ATT_WARPS < t_hi;
    float c[2][4] = {};
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      const uint4 x = kk[0][j], y = kk[1][j], b = qf[j];
      mma_bf16(c[0], x.x, y.x, x.y, y.y, b.x, b.y);
      mma_bf16(c[1], x.z, y.z, x.w, y.w, b.z, b.w);
    }
    if (more) load_k(p_next);
    // ---- online softmax: sums e and e + 2 are head e's of this lane at positions lane / 4 and 8 later ----
    float s[4], corr[2];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = p0 + 8 * (e >> 1) + (lane >> 2) < L ? (c[0][e] + c[1][e]) * a.scale_log2 : -INFINITY;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float mx = fmaxf(s[e], s[e + 2]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m[e], mx);
#pragma unroll
      for (int i = e; i < 4; i += 2) s[i] = (s[i] == -INFINITY) ? 0.f : exp2f(s[i] - m_new);
      corr[e] = (m[e] == -INFINITY) ? 0.f : exp2f(m[e] - m_new);
      float sum = s[e] + s[e + 2];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[e] = l[e] * corr[e] + sum;
      m[e] = m_new;
      const int h = 2 * (lane & 3) + e;
      if (h < QPK) {
        p_s[warp][lane >> 2][h] = s[e];
        p_s[warp][8 + (lane >> 2)][h] = s[e + 2];
        if (lane < 4) corr_s[warp][h] = corr[e];
      }
    }
    __syncwarp();
    // ---- PV: lane owns DPL consecutive output dims ---------------------------------------------------
    float w[QPK];
    auto heads = [&](const float* from) {
      if constexpr (QPK % 4 == 0) {
#pragma unroll
        for (int h = 0; h < QPK; h += 4) {
          const float4 f = *reinterpret_cast<const float4*>(from + h);
          w[h] = f.x; w[h + 1] = f.y; w[h + 2] = f.z; w[h + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int h = 0; h < QPK; ++h) w[h] = from[h];
      }
    };
    heads(corr_s[warp]);
#pragma unroll
    for (int h = 0; h < QPK; ++h)
#pragma unroll
      for (int d = 0; d < DPL; ++d) acc[h][d] *= w[h];
#pragma unroll
    for (int r = 0; r < ATT_TILE; ++r) {
      heads(p_s[warp][r]);
#pragma unroll
      for (int h = 0; h < QPK; ++h)
#pragma unroll
        for (int d = 0; d < DPL / 2; ++d) {
          acc[h][2 * d] = fmaf(w[h], bf16lo(vv[r][d]), acc[h][2 * d]);
          acc[h][2 * d + 1] = fmaf(w[h], bf16hi(vv[r][d]), acc[h][2 * d + 1]);
        }
    }
    if (more) load_v(p_next);
    __syncwarp();
  }

  __syncthreads();
  trace_phase(a.trace, 6);  // all tiles done
  // ---- merge the CTA's warps ------------------------------------------------------------------
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (lane < 4 && 2 * lane + e < QPK) { mrg_m[warp][2 * lane + e] = m[e]; mrg_l[warp][2 * lane + e] = l[e]; }
#pragma unroll
  for (int h = 0; h < QPK; ++h) {
#pragma unroll
    for (int d = 0; d < DPL; ++d) mrg_acc[warp][h][lane * DPL + d] = acc[h][d];
  }
  __syncthreads();
  if (cl_merge) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  for (int i = threadIdx.x; i < QPK * HS; i += ATT_THREADS) {
    const int h = i / HS, d = i % HS;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, mrg_m[w][h]);
    float o = 0.f, ll = 0.f;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
      const float sc = (mrg_m[w][h] == -INFINITY) ? 0.f : exp2f(mrg_m[w][h] - mm);
      o = fmaf(sc, mrg_acc[w][h][d], o);
      ll = fmaf(sc, mrg_l[w][h], ll);
    }
    if (n_active == 1) {  // single span: final answer, no round trip through the partial buffer
      a.y[(size_t)(g * QPK + h) * HS + d] = __float2bfloat16_rn(ll > 0.f ? o / ll : 0.f);
    } else if (cl_merge) {  // into rank 0's shared memory (my slot = my span index)
      st_cluster_f32(&cl_part[split][h][2 + d], 0, o);
      if (d == 0) { st_cluster_f32(&cl_part[split][h][0], 0, mm); st_cluster_f32(&cl_part[split][h][1], 0, ll); }
    } else {
      float* dst = a.part + ((size_t)(g * QPK + h) * a.n_split + split) * (HS + 2);
      dst[2 + d] = o;
      if (d == 0) { dst[0] = mm; dst[1] = ll; }
    }
  }
  if (n_active == 1) { dep_signal(a.dep_signal, a.ctx); trace_mark(a.trace, 3, true); trace_mark(a.trace, 4, false); return; }

  if (CLUSTER && cl_merge) {
    // ---- rank 0 folds the cluster's partials out of its own shared memory ------------------------------
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (split != 0) { dep_signal(a.dep_signal, a.ctx); trace_mark(a.trace, 3, true); trace_mark(a.trace, 4, false); return; }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int i = threadIdx.x; i < QPK * HS; i += ATT_THREADS) {
      const int h = i / HS, d = i % HS;
      float mm = -INFINITY;
      for (int sp = 0; sp < n_active; ++sp) mm = fmaxf(mm, cl_part[sp][h][0]);
      float o = 0.f, ll = 0.f;
      for (int sp = 0; sp < n_active; ++sp) {
        const float pm = cl_part[sp][h][0];
        const float sc = (pm == -INFINITY) ? 0.f : exp2f(pm - mm);
        o = fmaf(sc, cl_part[sp][h][2 + d], o);
        ll = fmaf(sc, cl_part[sp][h][1], ll);
      }
      a.y[(size_t)(g * QPK + h) * HS + d] = __float2bfloat16_rn(ll > 0.f ? o / ll : 0.f);
    }
    dep_signal(a.dep_signal, a.ctx);
    trace_mark(a.trace, 3, true);
    trace_mark(a.trace, 4, false);
    return;
  }

  // ---- the group's last CTA merges the spans ------------------------------------------------------
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int prev = atomicAdd(a.tickets + g, 1u);
    sh_last = (prev == (unsigned)n_active - 1);
    if (sh_last) a.tickets[g] = 0;
  }
  __syncthreads();
  if (!sh_last) { dep_signal(a.dep_signal, a.ctx); trace_mark(a.trace, 3, true); trace_mark(a.trace, 4, false); return; }
  __threadfence();
  for (int i = threadIdx.x; i < QPK * HS; i += ATT_THREADS) {
    const int h = i / HS, d = i % HS;
    const float* base = a.part + (size_t)(g * QPK + h) * a.n_split * (HS + 2);
    float mm = -INFINITY;
    for (int s = 0; s < n_active; ++s) mm = fmaxf(mm, __ldcg(base + (size_t)s * (HS + 2)));
    float o = 0.f, ll = 0.f;
#pragma unroll 4
    for (int s = 0; s < n_active; ++s) {
      const float* p = base + (size_t)s * (HS + 2);
      const float pm = __ldcg(p), pl = __ldcg(p + 1), po = __ldcg(p + 2 + d);
      const float sc = (pm == -INFINITY) ? 0.f : exp2f(pm - mm);
      o = fmaf(sc, po, o);
      ll = fmaf(sc, pl, ll);
    }
    a.y[(size_t)(g * QPK + h) * HS + d] = __float2bfloat16_rn(ll > 0.f ? o / ll : 0.f);
  }
  dep_signal(a.dep_signal, a.ctx);
  trace_mark(a.trace, 3, true);
  trace_mark(a.trace, 4, false);
}

static int g_attn_cluster = 8;  // mdi_set_attn_cluster: 0 = always merge through global memory, n = through the cluster up to n tiles per warp at most

// Up to how many tiles per warp (1024 positions each) the spans of a group stay in one cluster.  Its loop gets longer, but the merge
// through global memory (fence, ticket, a second round of loads by the last CTA, some 5 us) goes.  About twelve clusters of eight CTAs run at
// a time.  Split against cluster, us a launch with cold keys (q heads per group x head size, groups, positions):
//   4 x 128, 8 groups   2048: 13.3  8.5   4096: 19.8 12.3   8000: 31.6 19.4
//   4 x 64, 8 groups    2048:  8.9  6.3   8000: 20.9 14.2                      8 x 64, 1 group    2048: 11.0  6.3   8000: 20.4 13.6
//   4 x 128, 1 group    3000: 12.7  8.9   4096: 16.0 10.8   8000: 21.5 17.8    2 x 128, 1 group   2048:  7.8  5.8   4096:  9.8  8.7
//   1 x 256, 4 groups   2048:  9.4  7.9   8000: 22.9 18.2                      2 x 256, 8 groups  2048: 17.4  9.7   8000: 39.8 23.1
//   4 x 128, 16 groups  4096: 26.3 15.2   8000: 39.7 24.6                      1 x 256, 16 groups 2048: 19.2 15.3   8000: 49.8 39.0
// By these figures the cluster form is the faster one throughout, 1.05 to 1.8 times, beyond the limits below too: those under eight tiles were set for
// a kernel whose tiles took two and a half times as long (few groups: what a position costs decided; many: two rounds of clusters), and
// have not been moved since.
static int cluster_tiles(int head_size, int qpk, int groups) {
  if (head_size > 128) return groups >= 8 && groups < 16 ? 8 : 1;
  if (head_size < 128 || qpk == 1) return 8;
  if (groups <= 3) return qpk == 2 ? 2 : 3;
  return qpk == 4 && groups >= 16 ? 4 : 8;
}

template <int HS, int QPK>
static int launch_attn(const AttnArgs& a, int use_pdl, cudaStream_t stream) {
  // the cluster's partials and the kernel's other static arrays (mrg_acc, p_s, corr_s, mrg_m, mrg_l) must fit the 48 KB static shared-memory window
  constexpr size_t CL_FLOATS = (size_t)ATT_CL * QPK * (HS + 2) + (size_t)ATT_WARPS * QPK * (HS + ATT_TILE + 3);
  constexpr bool CL_FITS = CL_FLOATS * 4 + 256 <= 48 * 1024;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(a.n_groups, a.n_split);
  cfg.blockDim = dim3(ATT_THREADS);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl ? 1 : 0;
  if (CL_FITS && g_attn_cluster && a.n_split % ATT_CL == 0) {
    if (!use_pdl) { attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = ATT_CL; attr[0].val.clusterDim.z = 1; }
    else { attr[1].id = cudaLaunchAttributeClusterDimension; attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = ATT_CL; attr[1].val.clusterDim.z = 1; }
    cfg.numAttrs += 1;
    return (int)cudaLaunchKernelEx(&cfg, attn_decode_kernel<HS, QPK, CL_FITS>, a);
  }
  return (int)cudaLaunchKernelEx(&cfg, attn_decode_kernel<HS, QPK, false>, a);
}

}  // namespace mdi

using namespace mdi;

extern "C" void mdi_set_attn_cluster(int on) { g_attn_cluster = on; }
extern "C" int mdi_attn_cluster_tiles(int head_size, int q_per_kv, int n_groups) { return cluster_tiles(head_size, q_per_kv, n_groups); }

// part: fp32 [H, n_split, hs + 2]; tickets: uint32 [G], zeroed once at allocation.
extern "C" int mdi_attn_decode(const void* q, const void* kv, void* y, float* part, unsigned int* tickets,
                               const int* ctx, int n_head, int n_groups, int head_size, int max_seq, int n_split,
                               int use_pdl, unsigned long long* trace, const int* dep_wait_flag, int* dep_signal_flag,
                               unsigned int* dep_ctr, int* status, long long wait_max_cycles, cudaStream_t stream) {
  AttnArgs a;
  a.trace = trace;
  a.dep_wait = DepWait{dep_wait_flag, status, wait_max_cycles}; a.dep_signal = DepSignal{dep_signal_flag, dep_ctr};
  a.q = (const bf16*)q; a.kv = (const bf16*)kv; a.y = (bf16*)y; a.part = part; a.tickets = tickets; a.ctx = ctx;
  a.n_head = n_head; a.n_groups = n_groups; a.max_seq = max_seq; a.n_split = n_split;
  a.scale_log2 = 1.4426950408889634f / sqrtf((float)head_size);
  const int qpk = n_head / n_groups;
  a.cl_iters = min(g_attn_cluster, cluster_tiles(head_size, qpk, n_groups));
#define MDI_ATT_CASE(HS_, QPK_) \
  if (head_size == HS_ && qpk == QPK_) return launch_attn<HS_, QPK_>(a, use_pdl, stream);
  MDI_ATT_CASE(128, 1) MDI_ATT_CASE(128, 2) MDI_ATT_CASE(128, 4) MDI_ATT_CASE(128, 8)
  MDI_ATT_CASE(64, 1) MDI_ATT_CASE(64, 2) MDI_ATT_CASE(64, 4) MDI_ATT_CASE(64, 8)
  MDI_ATT_CASE(256, 1) MDI_ATT_CASE(256, 2)  // Gemma-7b / Pythia-1b class heads (static shared memory <= 48 KB)
#undef MDI_ATT_CASE
  return -3;  // unsupported (head_size, q_per_kv): caller falls back to the eager path
}
