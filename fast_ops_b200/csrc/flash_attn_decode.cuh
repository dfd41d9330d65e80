// Attention forward for a single query row per head (decoding one token against stored keys and
// values): softmax(scale q K^T) V with Sq = 1, no mask, bias or dropout.
//
// Bound by memory: every key and value is used by one query row (or, when the heads share one K/V
// head, by one row of each), so the 128-row tensor-core tiles of the other kernels would do 1/128
// useful work, and one CTA per head leaves most SMs idle.  Here the keys of a
// head (or of kHeads heads that share K and V) are split over the CTAs of a cluster and, inside a
// CTA, over its warps:
//   - a key's row is held by kLanes lanes, 16 bytes (8 elements) each; a warp takes kBatch rows
//     per lane group and step, all of them in flight together (K of the next step is requested
//     while V of this one is consumed);
//   - q . k sums are reduced and scattered in one butterfly (kBatch - 1 exchanges for kBatch rows),
//     after which the lanes hold one key's score each and take one exponential each;
//   - everything is fp32 (probabilities too: unlike the tensor-core kernels nothing is rounded to
//     16 bits before the result);
//   - warps combine through shared memory, CTAs of the cluster through distributed shared memory,
//     so no workspace and no second launch.
// Measured (one B200, us per launch, kernel alone; before = one 128-row tile per head):
//   B4 H32 Sk4096 D128 bf16 52 -> 42 (41.6 at the measured copy rate); B1 H8 Sk32768 D128 354 -> 36;
//   B32 H40 Sk2000 D64, one shared K/V head, 143 -> 53; B16 H40 Sk1000 D128, shared, 50 -> 37.
#pragma once

#include <cooperative_groups.h>

#include <atomic>

#include "flash_attn_common.cuh"
#include "fo_host.h"

namespace fo {

struct DecodeParams {
  const uint16_t *q, *k, *v;
  uint16_t* o;
  float* lse;  // (B, H, 1), may be null
  int64_t q_stride_b, q_stride_h;
  int64_t k_stride_b, k_stride_h, k_stride_s;  // head stride 0 when the heads share K and V
  int64_t v_stride_b, v_stride_h, v_stride_s;
  int64_t o_stride_b, o_stride_h;
  int H, Sk, d_real;
  int chunk;  // keys per CTA
  float scale_log2;
  const int* device_status;
};

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// grid = (cluster size * head groups, B); a head group is kHeads heads (1 when K and V are per head).
// Blocks of kWarps warps that one SM holds: 16 warps of the per-head form, 8 of the shared-head form.
template <int kHeads, int kWarps>
constexpr int kDecodePerSm = (kHeads == 1 ? 16 : 8) / kWarps;

template <int D, bool kBf16, int kHeads, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, kDecodePerSm<kHeads, kWarps>)
attn_decode_kernel(const DecodeParams prm) {
  namespace cg = cooperative_groups;
  constexpr int kLanes = D / 8;        // lanes per key row
  constexpr int kGroups = 32 / kLanes; // rows a warp loads per instruction
  constexpr int kBatch = 8;            // rows per lane group and step
  constexpr int kStep = kGroups * kBatch;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int n_ranks = static_cast<int>(cluster.num_blocks());
  const int b = blockIdx.y;
  const int h0 = (blockIdx.x / n_ranks) * kHeads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = lane / kLanes, sub = lane % kLanes;
  const int d0 = sub * 8;
  const bool d_ok = d0 < prm.d_real;  // d_real is a multiple of 8; missing columns are zeros

  // One row per (warp or CTA) partial result: D values of the unnormalised output, maximum, sum.
  __shared__ __align__(16) float s_part[kWarps][kHeads][D];
  __shared__ float s_ml[kWarps][kHeads][2];
  __shared__ __align__(16) float s_cta[kHeads][D];        // this CTA's partial, read by the cluster's rank 0
  __shared__ float s_cta_ml[kHeads][2];

  float2 q[kHeads][4];
#pragma unroll
  for (int r = 0; r < kHeads; ++r) {
    const int h = min(h0 + r, prm.H - 1);  // a ragged last group repeats the last head and does not store it
    uint4 w = make_uint4(0, 0, 0, 0);
    if (d_ok) w = __ldg(reinterpret_cast<const uint4*>(prm.q + b * prm.q_stride_b + h * prm.q_stride_h + d0));
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpack2<kBf16>(ww[i]);
      q[r][i] = make_float2(f.x * prm.scale_log2, f.y * prm.scale_log2);
    }
  }
  const uint16_t* const kp = prm.k + b * prm.k_stride_b + h0 * prm.k_stride_h + d0;
  const uint16_t* const vp = prm.v + b * prm.v_stride_b + h0 * prm.v_stride_h + d0;
  const int begin = min(rank * prm.chunk, prm.Sk);
  const int end = min(begin + prm.chunk, prm.Sk);

  float2 acc[kHeads][4];
  float m[kHeads], l[kHeads];
#pragma unroll
  for (int r = 0; r < kHeads; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[r][i] = make_float2(0.f, 0.f);
  }

  // Rows of a step: lane group g holds rows base + g * kBatch + i.  Rows past the end are zeros.
  auto load_rows = [&](uint4 (&w)[kBatch], const uint16_t* p, int64_t stride, int base) {
    const int row0 = base + group * kBatch;
    const uint16_t* rp = p + row0 * stride;
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      w[i] = make_uint4(0, 0, 0, 0);
      if (d_ok && row0 + i < end) w[i] = ldg_stream(rp + i * stride);
    }
  };
  // After the butterfly lane `sub` holds the score of row `own` of its group.
  constexpr int kScatter = kBatch;  // rows scattered over kScatter lane classes; kLanes / kBatch lanes share a class
  const int own = (kLanes == 8) ? sub : (sub >> 1);
  const bool counts = (kLanes == 8) || (sub & 1) == 0;  // one lane per row adds it to the sum

  uint4 kw[kBatch], vw[kBatch];
  int base = begin + warp * kStep;
  if (base < end) load_rows(kw, kp, prm.k_stride_s, base);
  for (; base < end; base += kWarps * kStep) {
    load_rows(vw, vp, prm.v_stride_s, base);
    float s[kHeads];
#pragma unroll
    for (int r = 0; r < kHeads; ++r) {
      float t[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const uint32_t ww[4] = {kw[i].x, kw[i].y, kw[i].z, kw[i].w};
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int x = 0; x < 4; ++x) a = __ffma2_rn(unpack2<kBf16>(ww[x]), q[r][x], a);
        t[i] = a.x + a.y;
      }
      // reduce and scatter: at each exchange a lane keeps the half of the rows its lane bit names
      int off = kLanes / 2;
#pragma unroll
      for (int n = kScatter / 2; n >= 1; n >>= 1, off >>= 1) {
        const bool hi = (sub & off) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const float send = hi ? t[i] : t[i + n];
          const float keep = hi ? t[i + n] : t[i];
          t[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
      if constexpr (kLanes > kScatter) t[0] += __shfl_xor_sync(0xffffffffu, t[0], 1);
      s[r] = (base + group * kBatch + own < end) ? t[0] : -INFINITY;
    }
    // K of the next step: its registers are free now
    if (base + kWarps * kStep < end) load_rows(kw, kp, prm.k_stride_s, base + kWarps * kStep);
    float p[kHeads];
#pragma unroll
    for (int r = 0; r < kHeads; ++r) {
      float mx = s[r];
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m[r], mx);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float corr = fast_exp2(m[r] - m_use);
      m[r] = m_new;
      p[r] = fast_exp2(s[r] - m_use);
      l[r] = l[r] * corr + (counts ? p[r] : 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[r][i] = __fmul2_rn(acc[r][i], make_float2(corr, corr));
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const uint32_t ww[4] = {vw[i].x, vw[i].y, vw[i].z, vw[i].w};
      float2 f[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) f[x] = unpack2<kBf16>(ww[x]);
#pragma unroll
      for (int r = 0; r < kHeads; ++r) {
        const float pi = __shfl_sync(0xffffffffu, p[r], (kLanes == 8) ? i : 2 * i, kLanes);
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[r][x] = __ffma2_rn(make_float2(pi, pi), f[x], acc[r][x]);
      }
    }
  }

  // ---- warp: lane groups together (they share m), sums over all lanes ----
#pragma unroll
  for (int r = 0; r < kHeads; ++r) {
#pragma unroll
    for (int off = kLanes; off < 32; off <<= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[r][i].x += __shfl_xor_sync(0xffffffffu, acc[r][i].x, off);
        acc[r][i].y += __shfl_xor_sync(0xffffffffu, acc[r][i].y, off);
      }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], off);
    if (group == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(&s_part[warp][r][d0 + 2 * i]) = acc[r][i];
    }
    if (lane == 0) {
      s_ml[warp][r][0] = m[r];
      s_ml[warp][r][1] = l[r];
    }
  }
  __syncthreads();
  // ---- CTA ----
  for (int x = tid; x < kHeads * D; x += kWarps * 32) {
    const int r = x / D, d = x % D;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, s_ml[w][r][0]);
    const float m_use = mx == -INFINITY ? 0.f : mx;
    float a = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = fast_exp2(s_ml[w][r][0] - m_use);
      a = fmaf(f, s_part[w][r][d], a);
      sum = fmaf(f, s_ml[w][r][1], sum);
    }
    s_cta[r][d] = a;
    if (d == 0) {
      s_cta_ml[r][0] = mx;
      s_cta_ml[r][1] = sum;
    }
  }
  cluster.sync();
  // ---- cluster: rank 0 reads every CTA's partial through distributed shared memory ----
  // (nothing is stored while the device's status word says that an earlier launch gave up)
  if (rank == 0 && *reinterpret_cast<const volatile int*>(prm.device_status) == 0) {
    for (int x = tid; x < kHeads * (D / 2); x += kWarps * 32) {
      const int r = x / (D / 2), d = (x % (D / 2)) * 2;
      const int h = h0 + r;
      if (h >= prm.H) continue;
      float mx = -INFINITY;
      for (int c = 0; c < n_ranks; ++c) mx = fmaxf(mx, cluster.map_shared_rank(&s_cta_ml[r][0], c)[0]);
      const float m_use = mx == -INFINITY ? 0.f : mx;
      float a0 = 0.f, a1 = 0.f, sum = 0.f;
      for (int c = 0; c < n_ranks; ++c) {
        const float* const ml = cluster.map_shared_rank(&s_cta_ml[r][0], c);
        const float2 part = *reinterpret_cast<const float2*>(cluster.map_shared_rank(&s_cta[r][d], c));
        const float f = fast_exp2(ml[0] - m_use);
        sum = fmaf(f, ml[1], sum);
        a0 = fmaf(f, part.x, a0);
        a1 = fmaf(f, part.y, a1);
      }
      const float inv = sum > 0.f ? 1.f / sum : 0.f;
      if (d < prm.d_real)
        *reinterpret_cast<uint32_t*>(prm.o + b * prm.o_stride_b + h * prm.o_stride_h + d) = pack2<kBf16>(a0 * inv, a1 * inv);
      if (d == 0 && prm.lse != nullptr)
        prm.lse[static_cast<int64_t>(b) * prm.H + h] = sum > 0.f ? (m_use + log2f(sum)) * 0.6931471805599453f : -INFINITY;
    }
  }
  cluster.sync();  // no CTA leaves while its shared memory is being read
}

// CTAs of this kernel that can be resident together in clusters of 16 (asked once per device; the
// largest cluster must find all its SMs inside one GPC, so the chip holds fewer of them).
template <auto kKernel, int kThreads>
inline int resident_ctas_in_clusters_of_16(int device) {
  static std::atomic<int> known[64];  // CTAs + 1, 0 = not asked yet
  if (device < 0 || device >= 64) return 0;
  int n = known[device].load(std::memory_order_acquire);
  if (n == 0) {
    int clusters = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kThreads);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kKernel, &cfg) != cudaSuccess) {
      cudaGetLastError();  // not an error of the call: clusters of 16 are not used
      clusters = 0;
    }
    n = clusters * 16 + 1;
    known[device].store(n, std::memory_order_release);
  }
  return n - 1;
}

// How the keys are divided: heads per CTA, warps per CTA, CTAs per head (0: launch_decode decides).
struct DecodeShape {
  int heads, warps, split;
};

// Up to 1024 keys the work of a CTA is a few steps, and what counts is how many rounds of CTAs the chip
// takes, not how many warps share a head.  The shape with the least cost = rounds * (steps of a warp + 4),
// in steps of eight rows per lane group, a step of the four-head form counting 1.3; a later candidate (four
// heads, fewer warps, more CTAs) has to be 5 % ahead.  The constants are a fit to measured times: over
// 64 to 4096 heads, one to 1000 keys, head_dim 64 and 128, it is within 2 % of the best shape on average
// and 15 % at most.  Against eight warps throughout (us, head_dim 128, keys per head): 640 heads, 300:
// 32.2 -> 21.1; 384, 300: 17.4 -> 10.6; 4096, 300: 128 -> 105; 4096, 64: 59.5 -> 30.7; one K/V head
// shared by 32 query heads, 64 keys: 5.4 -> 4.2.  Beyond 1024 keys the bandwidth evens the shapes out and
// the rule of launch_decode is the better one (640 heads, 1500 keys: 93 by this rule, 89 by that one).
inline DecodeShape decode_shape(int B, int H, int Sk, int D, bool shared_kv, int num_sms) {
  if (Sk > 1024) return {shared_kv ? 4 : 1, 8, 0};
  const int rows = D <= 64 ? 32 : 16;  // rows of a warp's step
  DecodeShape best = {1, 8, 1};
  double best_cost = 0;
  for (int heads = 1; heads <= (shared_kv ? 4 : 1); heads += 3)
    for (int warps = 8; warps >= 2; warps /= 2)
      for (int split = 1; split <= 8 && (split == 1 || Sk / split >= 64); split *= 2) {
        const int64_t ctas = static_cast<int64_t>((H + heads - 1) / heads) * B * split;
        const int slots = num_sms * ((heads == 1 ? 16 : 8) / warps);
        const int steps = (Sk + split * rows * warps - 1) / (split * rows * warps);
        const double cost = static_cast<double>((ctas + slots - 1) / slots) * (steps * (heads == 1 ? 1.0 : 1.3) + 4);
        if (best_cost == 0 || cost < 0.95 * best_cost) {
          best_cost = cost;
          best = {heads, warps, split};
        }
      }
  return best;
}

// `split`: CTAs that share a head's keys, or 0: the power of two up to 16 that takes the fewest rounds of
// resident CTAs (two per SM, one in the shared-head form) per unit of split, the smaller unless
// the larger saves 15 % of that (each doubling costs a little: more partial results, shorter
// CTAs), while a CTA keeps at least 128 keys.  Measured at splits 1 / 2 / 4 / 8 / 16 (us):
// B4 H32 Sk4096 D128 57 / 43 / 46 / 52 / 79 (takes 2); B1 H8 Sk32768 D128 389 / 197 / 101 / 54 / 36
// (16); B8 H40 Sk3000 D96 92 / 82 / 80 / 96 (4).
template <int D, bool kBf16, int kHeads, int kWarps>
int launch_decode(const DecodeParams& base, int B, int split, int num_sms, int device, cudaStream_t stream) {
  constexpr auto kernel = attn_decode_kernel<D, kBf16, kHeads, kWarps>;
  const int64_t groups = static_cast<int64_t>((base.H + kHeads - 1) / kHeads) * B;
  if (split == 0) {
    const int resident = num_sms * kDecodePerSm<kHeads, kWarps>;
    double best = 0;
    for (int s = 1; s <= 16 && (s == 1 || base.Sk / s >= 128); s *= 2) {
      const int slots = s == 16 ? resident_ctas_in_clusters_of_16<kernel, kWarps * 32>(device) : resident;
      if (slots < s) break;
      const double cost = static_cast<double>((groups * s + slots - 1) / slots) / s;
      if (s == 1 || cost < 0.85 * best) {
        best = cost;
        split = s;
      }
    }
  }
  DecodeParams prm = base;
  prm.chunk = ((base.Sk + split - 1) / split + 15) / 16 * 16;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(groups / B * split), B);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FO_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, prm));
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return FO_OK;
}

}  // namespace fo
