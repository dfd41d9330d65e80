// Attention backward for sm_100a: dQ, dK, dV from dO, Q, K, V and the forward's LSE.
//
// The reference's CUDA path has no backward (fast_ops/flash_attention/flash_attention.py:41-45
// raises); the semantics follow its complete implementation
// (fast_ops/flash_attention/flash_attention_triton.py:273-315 for delta = rowsum(O o dO),
// :322-638 for the main loop): one CTA owns a 128-key tile, keeps dK and dV for it in tensor
// memory, walks the query tiles that see those keys, and adds its share of dQ into an fp32
// buffer (the reference uses scalar atomics, :610; here each tile goes through shared memory and
// tiled bulk reduce-adds, cp.reduce.async.bulk.tensor).
//
// The scores are held transposed (key rows in the tensor-memory lanes, query columns).  With
// query rows in the lanes, P and dS would both have to go through shared memory to be transposed
// for dV += P^T dO and dK += dS^T Q, and the shared-memory port (128 bytes per clock for
// tensor-core operands, thread stores and bulk copies together) would carry about 576 KB per query
// tile at head_dim 128: 4600 cycles against 2560 of arithmetic.  Per query tile, five tcgen05
// MMAs (all fp32 accumulation in tensor memory):
//   S^T  = K Q^T          (K, Q K-major from shared memory; key rows in the lanes)
//   dP^T = V dO^T         (V, dO K-major)
//   -- threads: P^T = exp2(S^T*scale - LSE[query]), written over S^T in tensor memory as 16-bit;
//      dS^T = P^T o (dP^T - delta[query]) * scale, written over dP^T in tensor memory as 16-bit
//      and to shared memory as a [key row][query] tile --
//   dV += P^T dO          (P^T read from tensor memory, dO as the N-major B operand)
//   dK += dS^T Q          (dS^T read from tensor memory, Q N-major)
//   dQ  = dS K            (dS^T tile of shared memory as the M-major A operand, K N-major)
// so P never touches shared memory and two of the five matmuls read one operand from tensor memory.
// dQ is written over dP^T / dS^T (not over S^T), and Q has two shared-memory slots, so the S^T
// matmul of the next query tile is issued right behind this tile's dV matmul: the exponentials of
// tile i+1 run while the tensor core does dK and dQ of tile i, and only dP^T of tile i+1 waits for
// dQ of tile i to leave tensor memory.  Matmuls that overwrite tensor-memory columns an earlier
// matmul reads (S^T of the next tile over P^T, dQ over dS^T) rely on the tensor core executing one
// thread's tcgen05.mma in issue order.
//
// Warps 0-7: two threads per key row, each taking 64 of the tile's 128 query columns; in the
// epilogue one thread per key row for dK (warps 0-3) and dV (warps 4-7).  Warps 8-11: one thread
// per query row takes dQ out of tensor memory (all of it at once, so the columns are free again
// after one load), then stages it 64 columns at a time in a 32 KB area of its own and adds it into
// the fp32 buffer with tiled bulk reductions (cp.reduce.async.bulk.tensor).  Warp 12 issues the
// MMAs, warp 13 the TMA loads, warp 14 brings LSE and delta of the next query tile into shared
// memory (they vary along the columns, so every thread needs all 128 of them).
// The wide form (BwdConfig::kWide) has sixteen compute warps, four threads per key row with 32 query
// columns each (in the epilogue two for dK, two for dV), and the other roles in warps 16 to 22.
#pragma once

#include "flash_attn_common.cuh"
#include "fo_host.h"

namespace fo {

struct AttnBwdParams {
  const float* lse;    // (B, H, Sq) natural-log LSE of the forward
  const float* delta;  // (B, H, Sq) rowsum(O o dO)
  float* dq_accum;     // (B, H, Sq, D) fp32, zeroed before the launch
  void* dk;
  void* dv;
  int64_t dk_stride_b, dk_stride_h, dk_stride_s;
  int64_t dv_stride_b, dv_stride_h, dv_stride_s;
  int B, H, Sq, Sk;
  int d_real;  // head_dim of the tensors (<= the kernel's D; the missing columns are zero-filled by TMA)
  int causal;
  float scale;       // softmax scale
  float scale_log2;  // scale * log2(e)
  int* device_status;
  unsigned long long* trace;  // optional timeline of CTA (0,0) (debug), or null
  int device;  // device index of the launch (host side only)
  AttnExtras ex;  // bias / dropout of the forward; read only by the kernel variants built for them
};

__device__ __forceinline__ void bwd_trace(const AttnBwdParams& prm, int role, int it, int ev) {
#if FO_ATTN_TRACE
  if (prm.trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && (threadIdx.x & 31) == 0 && it < kTraceIters)
    prm.trace[(role * kTraceIters + it) * kTraceEvents + ev] = clock64();
#else
  (void)prm; (void)role; (void)it; (void)ev;
#endif
}

// Writes 8 consecutive 16-bit values (one 16-byte unit) of row `r`, unit `u` (0..15 over 128
// columns) of a [128 x 128] tile stored as two [128 x 64] boxes with the 128-byte swizzle.
__device__ __forceinline__ void store_swizzled_unit(uint8_t* tile, int r, int u, uint4 v) {
  const int box = u >> 3;
  const int slot = (u & 7) ^ (r & 7);
  *reinterpret_cast<uint4*>(tile + box * kBoxBytes + r * 128 + slot * 16) = v;
}


// kExt, the variants compiled: bit 0 a bias that is the same for every query row ("vector"), bit 1
// dropout, bit 2 a bias with a row stride ("matrix").
constexpr int kBwdVecBias = 1, kBwdDropout = 2, kBwdMatBias = 4;

template <int D, int kExt>
struct BwdConfig {
  // head_dim 64 with dropout or a matrix bias: sixteen compute warps (four threads per key row, 32
  // query columns each) instead of eight.  Hashing and fetching bias values are long chains per
  // thread, and eight warps do not cover their latency.  us, whole backward, B2 H16 S2048 / B8 H12 S1024
  // causal / B32 H12 S128, before this form and with it: dropout 300 and 234 / 181 and 138 / 43 and 36;
  // vector bias with dropout 317 and 235 / 188 and 139 / 44 and 37.  (A matrix bias also got its values
  // 32 at a time: 2048 and 264 / 582 and 132 / 75 and 34, with dropout 2160 and 392 / 636 and 190 / 81 and
  // 41.)  The compiler spills 24 to 84 bytes in all four.  Without dropout or a matrix bias eight warps are
  // the faster form (B8 H12 S1024 D64 causal 81 against 84 us), and at head_dim 128 the registers do not
  // reach.
  static constexpr bool kWide = D == 64 && (kExt & (kBwdDropout | kBwdMatBias)) != 0;
  static constexpr int kComputeWarps = kWide ? 16 : 8;
  static constexpr int kThreads = kComputeWarps * 32 + 256;
  static constexpr int kCols = 128 * 4 / kComputeWarps;  // query columns of one compute thread
  static constexpr int kPieces = kCols / 32;
  // Register budgets (setmaxnreg): they add up to what the block is launched with,
  // 512 x 128 = 256 x 152 + 128 x 152 + 128 x 56 and 768 x 80 = 512 x 88 + 128 x 64 + 128 x 64.
  static constexpr int kRegsCompute = kWide ? 88 : 152;
  static constexpr int kRegsDQ = kWide ? 64 : 152;
  static constexpr int kRegsRest = kWide ? 64 : 56;
  // The wide form's dQ warps cannot hold a whole dQ row, but at head_dim 64 tensor memory has 128
  // columns and shared memory 48 KB to spare: dQ gets two column ranges of its own, dS^T two tiles
  // and dO two slots, so that dP^T of the next query tile follows dK without waiting for dQ to be
  // computed or read out.
  static constexpr bool kSepDQ = kWide;
  static constexpr int kSlots = kSepDQ ? 2 : 1;  // dO slots, dS^T tiles, dQ column ranges
  // Barrier of query tile t among a [kSlots] set, and its phase there: with two slots a waiter two
  // tiles behind cannot mistake one phase for another.
  __device__ static __forceinline__ int par(int t) { return t & (kSlots - 1); }
  __device__ static __forceinline__ int phase(int t) { return (t >> (kSlots - 1)) & 1; }
  static constexpr int kTileBytes = kBlockM * D * 2;      // Q, dO, K, V tiles
  static constexpr int kDSBytes = kBlockN * kBlockM * 2;  // dS^T: [128 key rows][128 queries] 16-bit
  static constexpr int kStageBytes = kBlockM * 64 * 4;    // dQ, 64 columns at a time: two swizzled boxes of [128 rows][32 floats]
  static constexpr int kOffK = 0;
  static constexpr int kOffV = kTileBytes;
  static constexpr int kOffQ = 2 * kTileBytes;  // two slots
  static constexpr int kOffDO = 4 * kTileBytes;
  static constexpr int kOffDS = kOffDO + kSlots * kTileBytes;
  static constexpr int kOffStage = kOffDS + kSlots * kDSBytes;
  static constexpr int kOffBars = kOffStage + kStageBytes;
  static constexpr int kNumBars = 24;
  static constexpr int kOffMisc = kOffBars + kNumBars * 8;
  // [kSlots][128] float each: -LSE*log2(e) and -delta*scale of the query tile; read as float4
  static constexpr int kOffNegLse = (kOffMisc + 64 + 15) & ~15;
  static constexpr int kOffNegDelta = kOffNegLse + kSlots * 128 * 4;
  static constexpr int kSmemBytes = kOffNegDelta + kSlots * 128 * 4 + 1024;
  static constexpr uint32_t kTmemCols = 512;
  // dK | dV | S^T | dP^T, dQ over dP^T; wide form: dK | dV | dQ | dQ | S^T | dP^T
  static constexpr uint32_t kColDK = 0, kColDV = D, kColS = 256, kColDP = 384;
  static constexpr uint32_t kColDQ = kSepDQ ? 128 : kColDP;
  static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
};

__device__ __forceinline__ void tmem_st_packed(uint32_t taddr, const uint32_t (&r)[16]) { tmem_st16(taddr, r); }
__device__ __forceinline__ void tmem_st_packed(uint32_t taddr, const uint32_t (&r)[32]) { tmem_st32(taddr, r); }

// 32 bias values (log2(e) * value) of one key and consecutive query rows: consecutive lanes hold
// consecutive keys, so each load of a warp is one contiguous segment; all 32 are in flight
// together (one load per element inside the exponential loop was waited for one by one: this
// kernel took 2160 us at B2 H16 S2048 D64 with dropout, against 392).  `p` points at (first row, key)
// with the key clamped into the row; rows past Sq (`rows_left` of them remain) are not loaded and give
// 0: their -LSE is -inf, which makes P zero.
template <bool kBf16>
__device__ __forceinline__ void load_bias_rows32(const AttnExtras& ex, const uint8_t* p, int rows_left,
                                                 float (&out)[32]) {
  constexpr float kLog2e = 1.4426950408889634f;
  const bool full = rows_left >= 32;
  if (ex.bias_f32) {
    const float* f = reinterpret_cast<const float*>(p);
    const int64_t step = ex.bias_stride_q;
#pragma unroll
    for (int x = 0; x < 32; ++x)
      out[x] = full || x < rows_left ? __ldg(f + x * step) : 0.f;
#pragma unroll
    for (int x = 0; x < 32; ++x) out[x] *= kLog2e;
  } else {
    const uint16_t* f = reinterpret_cast<const uint16_t*>(p);
    const int64_t step = ex.bias_stride_q;
    uint16_t raw[32];
#pragma unroll
    for (int x = 0; x < 32; ++x)
      raw[x] = full || x < rows_left ? __ldg(f + x * step) : static_cast<uint16_t>(0);
#pragma unroll
    for (int x = 0; x < 32; ++x) {
      if constexpr (kBf16) out[x] = __uint_as_float(static_cast<uint32_t>(raw[x]) << 16) * kLog2e;
      else out[x] = __half2float(__ushort_as_half(raw[x])) * kLog2e;
    }
  }
}

// grid = (key tiles, B*H); block = BwdConfig<D, kExt>::kThreads.
// kMma is the head_dim that the matmuls compute, D the width of the tiles: the zero columns between
// them are left out of the K Q^T and V dO^T steps and of the width of dV, dK and dQ.
template <int D, bool kBf16, int kExt, int kMma = D>
__global__ void __launch_bounds__(BwdConfig<D, kExt>::kThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                  const __grid_constant__ CUtensorMap tm_dq, const AttnBwdParams prm) {
  using Cfg = BwdConfig<D, kExt>;
  constexpr int kTileBytes = Cfg::kTileBytes;
  constexpr int kBoxes = D / kBoxCols;
  constexpr int kHalves = D / 64;  // dQ is staged in pieces of 64 columns (two boxes of 32 floats)
  constexpr int kCW = Cfg::kComputeWarps;
  constexpr bool kSepDQ = Cfg::kSepDQ;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sK = smem + Cfg::kOffK;
  uint8_t* sV = smem + Cfg::kOffV;
  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sDO = smem + Cfg::kOffDO;
  uint8_t* sDS = smem + Cfg::kOffDS;
  uint8_t* sStage = smem + Cfg::kOffStage;
  float* sNegLse = reinterpret_cast<float*>(smem + Cfg::kOffNegLse);
  float* sNegDelta = reinterpret_cast<float*>(smem + Cfg::kOffNegDelta);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  // Every thread arrives for itself: one arrival per warp behind a __syncwarp measured 1 % slower.
  uint64_t* bar_kv = bars + 0;           // TMA -> MMA: K and V of this CTA are in shared memory
  uint64_t* bar_q_full = bars + 1;       // [2] TMA -> MMA: Q_i loaded into slot i % 2
  uint64_t* bar_q_empty = bars + 3;      // [2] MMA -> TMA: the matmuls reading that slot (S^T, dK) have completed
  uint64_t* bar_do_full = bars + 5;      // [kSlots] TMA -> MMA: dO_i loaded
  uint64_t* bar_do_empty = bars + 7;     // [kSlots] MMA -> TMA: the matmuls reading dO_i (dP^T, dV) have completed
  uint64_t* bar_s_full = bars + 9;       // MMA -> threads: S^T is in tensor memory
  uint64_t* bar_dp_full = bars + 10;     // MMA -> threads: dP^T is in tensor memory
  uint64_t* bar_p_full = bars + 11;      // [kSlots] threads -> MMA, row loader: P^T is in tensor memory
  uint64_t* bar_ds_full = bars + 13;     // [kSlots] threads -> MMA, row loader: dS^T is in tensor and shared memory
  uint64_t* bar_dq_full = bars + 15;     // [kSlots] MMA -> dQ warps: dQ tile complete
  uint64_t* bar_dq_free = bars + 17;     // [kSlots] dQ warps -> MMA: dQ read, its columns are reusable
  uint64_t* bar_lse_full = bars + 19;    // [kSlots] row loader -> threads: -LSE of the query tile's rows is in shared memory
  uint64_t* bar_delta_full = bars + 21;  // [kSlots] row loader -> threads: -delta of the query tile's rows is in shared memory
  uint64_t* bar_done = bars + 23;        // MMA -> threads: every matmul has completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffMisc);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* skip = cta_abort + 1;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int j = blockIdx.x;  // key tile
  const int bh = blockIdx.y;
  const int b = bh / prm.H;
  const int h = bh - b * prm.H;
  const int k0 = j * kBlockN;
  const int n_q_tiles = (prm.Sq + kBlockM - 1) / kBlockM;
  // query tiles that see this key tile: all of them, or with a causal mask those whose last
  // row is not above the tile's first key
  const int i0 = prm.causal ? min(j, n_q_tiles) : 0;
  const int n_iter = n_q_tiles - i0;
  int* const dstat = prm.device_status;

  if (tid == 0) {
    *cta_abort = 0;
    *skip = *reinterpret_cast<volatile int*>(prm.device_status);
    mbar_init(bar_kv, 1);
    for (int x = 0; x < 2; ++x) {
      mbar_init(bar_q_full + x, 1);
      mbar_init(bar_q_empty + x, 1);
      mbar_init(bar_do_full + x, 1);
      mbar_init(bar_do_empty + x, 1);
      mbar_init(bar_p_full + x, kCW * 32);
      mbar_init(bar_ds_full + x, kCW * 32);
      mbar_init(bar_dq_full + x, 1);
      mbar_init(bar_dq_free + x, 128);
      mbar_init(bar_lse_full + x, 1);
      mbar_init(bar_delta_full + x, 1);
    }
    mbar_init(bar_s_full, 1);
    mbar_init(bar_dp_full, 1);
    mbar_init(bar_done, 1);
    fence_mbar_init();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_do);
    prefetch_tensormap(&tm_dq);
  }
  __syncthreads();
  if (*skip) return;
  auto load_q = [&](int t) {
    mbar_arrive_expect_tx(bar_q_full + (t & 1), kTileBytes);
    for (int c = 0; c < kBoxes; ++c)
      tma_load_4d(sQ + (t & 1) * kTileBytes + c * kBoxBytes, &tm_q, bar_q_full + (t & 1), c * kBoxCols, (i0 + t) * kBlockM, h, b);
  };
  auto load_do = [&](int t) {
    const int slot = t & (Cfg::kSlots - 1);
    mbar_arrive_expect_tx(bar_do_full + slot, kTileBytes);
    for (int c = 0; c < kBoxes; ++c)
      tma_load_4d(sDO + slot * kTileBytes + c * kBoxBytes, &tm_do, bar_do_full + slot, c * kBoxCols, (i0 + t) * kBlockM, h, b);
  };
  // K, V and the first Q / dO need only the barriers: requested here, under the tensor-memory allocation
  if (warp == kCW + 5 && lane == 0) {
    mbar_arrive_expect_tx(bar_kv, 2 * kTileBytes);
    for (int c = 0; c < kBoxes; ++c) tma_load_4d(sK + c * kBoxBytes, &tm_k, bar_kv, c * kBoxCols, k0, h, b);
    for (int c = 0; c < kBoxes; ++c) tma_load_4d(sV + c * kBoxBytes, &tm_v, bar_kv, c * kBoxCols, k0, h, b);
    for (int t = 0; t < min(n_iter, 2); ++t) load_q(t);
    for (int t = 0; t < min(n_iter, Cfg::kSlots); ++t) load_do(t);
  }
  if (warp == kCW + 4) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish_alloc_permit();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < kCW) {
    // ================================ compute threads ================================
    reg_alloc<Cfg::kRegsCompute>();
    constexpr int kCols = Cfg::kCols;
    constexpr int kPieces = Cfg::kPieces;
    const int r = (warp & 3) * 32 + lane;  // key row of the tile (tensor-memory lane)
    const int part = warp >> 2;            // which kCols query columns this thread takes
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // this thread's fp32 columns of S^T / dP^T; its 16-bit results go over the first half of them
    const uint32_t tS = tmem_base + Cfg::kColS + lane_base + part * kCols;
    const uint32_t tDP = tmem_base + Cfg::kColDP + lane_base + part * kCols;
    constexpr bool vec_bias = (kExt & kBwdVecBias) != 0;
    constexpr bool mat_bias = (kExt & kBwdMatBias) != 0;
    constexpr bool has_drop = (kExt & kBwdDropout) != 0;
    // with dropout dP arrives without the 1 / (1 - p) factor of the kept elements
    const float dp_scale = kExt ? prm.scale * prm.ex.drop_rescale : prm.scale;
    const int key = k0 + r;
    const bool key_ok = key < prm.Sk;
    // A bias that is the same for every query row depends only on this thread's key: one register.
    float bias_key = 0.f;
    const uint8_t* bias_col = nullptr;  // (row 0, this thread's key) of a matrix bias
    if constexpr (vec_bias || mat_bias) {
      const int esize = prm.ex.bias_f32 ? 4 : 2;
      bias_col = static_cast<const uint8_t*>(prm.ex.bias) +
                 (b * prm.ex.bias_stride_b + h * prm.ex.bias_stride_h + min(key, prm.Sk - 1)) * esize;
      if (vec_bias && key_ok) bias_key = load_bias1<kBf16>(prm.ex, bias_col, 0);
    }
    for (int it = 0; it < n_iter; ++it) {
      const int i = i0 + it;
      const int q0 = i * kBlockM;
      const int qc0 = q0 + part * kCols;  // first query of this thread's columns
      // masks are rare (diagonal tiles, a ragged last key tile); rows past Sq have -LSE = -inf
      const bool need_mask = !key_ok || (prm.causal && k0 + kBlockN - 1 > q0);
      // What does not depend on S^T comes first: the keep decisions and the first bias values.
      uint32_t keep[kPieces];  // dropout: bit x of keep[cc] = element kept
      if constexpr (has_drop) {
        const uint32_t base = prm.ex.drop_base + static_cast<uint32_t>(bh) * static_cast<uint32_t>(prm.Sq) * static_cast<uint32_t>(prm.Sk) +
                              static_cast<uint32_t>(key);
#pragma unroll
        for (int cc = 0; cc < kPieces; ++cc) {
          uint32_t kb = 0;
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            const uint32_t idx = base + static_cast<uint32_t>(qc0 + cc * 32 + x) * static_cast<uint32_t>(prm.Sk);
            if (dropout_hash(idx, prm.ex.drop_seed) > prm.ex.drop_threshold) kb |= 1u << x;
          }
          keep[cc] = kb;
        }
      }
      float bias_v[32];
      auto load_bias_piece = [&](int cc) {
        const int q = qc0 + cc * 32;
        load_bias_rows32<kBf16>(prm.ex, bias_col + static_cast<int64_t>(q) * prm.ex.bias_stride_q * (prm.ex.bias_f32 ? 4 : 2),
                                prm.Sq - q, bias_v);
      };
      if constexpr (mat_bias) load_bias_piece(0);
      mbar_wait(bar_lse_full + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      mbar_wait(bar_s_full, it & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
      tcgen05_fence_after_sync();
      if (warp == 0) bwd_trace(prm, 0, it, 0);
      // ---- P^T = exp2(S^T * scale - LSE) of this thread's columns, fp32 in registers; the dP^T matmul runs meanwhile ----
      uint32_t sr[kPieces][32];
#pragma unroll
      for (int cc = 0; cc < kPieces; ++cc) tmem_ld32(tS + cc * 32, sr[cc]);
#pragma unroll
      for (int cc = 0; cc < kPieces; ++cc) {
        const float* nl = sNegLse + (it & (Cfg::kSlots - 1)) * 128 + part * kCols + cc * 32;
        tmem_ld_wait(sr[cc]);
        if constexpr (mat_bias) {
          if (cc > 0) load_bias_piece(cc);
        }
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const float4 t = *reinterpret_cast<const float4*>(nl + x);  // broadcast read
          const float nlv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            const float sv = __uint_as_float(sr[cc][x + y]);
            float e;
            if constexpr (mat_bias) e = fmaf(sv, prm.scale_log2, bias_v[x + y]) + nlv[y];
            else if constexpr (vec_bias) e = fmaf(sv, prm.scale_log2, bias_key) + nlv[y];
            else e = fmaf(sv, prm.scale_log2, nlv[y]);
            sr[cc][x + y] = __float_as_uint(fast_exp2(e));
          }
        }
        if (need_mask) {
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            const int q = qc0 + cc * 32 + x;
            if (!key_ok || (prm.causal && key > q)) sr[cc][x] = 0u;
          }
        }
      }
      if (warp == 0) bwd_trace(prm, 0, it, 4);
      // ---- P^T (zero where the forward dropped the element), 16-bit, over the first half of this thread's S^T columns ----
      uint32_t pp[kPieces * 16];
#pragma unroll
      for (int cc = 0; cc < kPieces; ++cc) {
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          float z0 = __uint_as_float(sr[cc][x]), z1 = __uint_as_float(sr[cc][x + 1]);
          if constexpr (has_drop) {
            if (!((keep[cc] >> x) & 1u)) z0 = 0.f;
            if (!((keep[cc] >> (x + 1)) & 1u)) z1 = 0.f;
          }
          pp[cc * 16 + (x >> 1)] = pack2<kBf16>(z0, z1);
        }
      }
      tmem_st_packed(tS, pp);
      tcgen05_wait_st();
      tcgen05_fence_before_sync();
      mbar_arrive(bar_p_full + Cfg::par(it));  // the dV matmul may start
      if (warp == 0) bwd_trace(prm, 0, it, 5);

      // ---- dS^T = P^T o (dP^T - delta) * scale, dP = 0 for a dropped element ----
      mbar_wait(bar_delta_full + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      mbar_wait(bar_dp_full, it & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
      tcgen05_fence_after_sync();
      {
        // The dS^T tile written here was last read by the dQ matmul of the query tile before (one
        // tile) or two before (two tiles), which was issued ahead of, and so completed before, this
        // query tile's dP^T matmul.
        uint8_t* const ds_tile = sDS + (it & (Cfg::kSlots - 1)) * Cfg::kDSBytes;
        uint32_t dd[kPieces * 16];
#pragma unroll
        for (int cc = 0; cc < kPieces; ++cc) {
          const float* nd = sNegDelta + (it & (Cfg::kSlots - 1)) * 128 + part * kCols + cc * 32;
          uint32_t dpr[32];
          tmem_ld32(tDP + cc * 32, dpr);
          tmem_ld_wait(dpr);
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            const float4 t = *reinterpret_cast<const float4*>(nd + x);  // broadcast read
            const float ndv[4] = {t.x, t.y, t.z, t.w};
            float dsv[4];
#pragma unroll
            for (int y = 0; y < 4; ++y) {
              float g = __uint_as_float(dpr[x + y]);
              if constexpr (has_drop) {
                if (!((keep[cc] >> (x + y)) & 1u)) g = 0.f;
              }
              dsv[y] = __uint_as_float(sr[cc][x + y]) * fmaf(g, dp_scale, ndv[y]);
            }
            dd[cc * 16 + (x >> 1)] = pack2<kBf16>(dsv[0], dsv[1]);
            dd[cc * 16 + (x >> 1) + 1] = pack2<kBf16>(dsv[2], dsv[3]);
          }
        }
        tmem_st_packed(tDP, dd);
#pragma unroll
        for (int u = 0; u < kPieces * 4; ++u)
          store_swizzled_unit(ds_tile, r, part * kPieces * 4 + u, make_uint4(dd[4 * u], dd[4 * u + 1], dd[4 * u + 2], dd[4 * u + 3]));
      }
      tcgen05_wait_st();
      fence_proxy_async_smem();  // shared-memory writes of these threads must be visible to the tensor core's reads
      tcgen05_fence_before_sync();
      mbar_arrive(bar_ds_full + Cfg::par(it));
      if (warp == 0) bwd_trace(prm, 0, it, 1);
    }

    // ---- epilogue: key row (k0 + r); the first half of the warps write dK, the second dV ----
    constexpr int kWarpsPerRow = kCW / 4;                 // threads that share a key row
    constexpr int kOutCols = 2 * D / kWarpsPerRow;        // columns of dK or dV of one thread
    const int which = part / (kWarpsPerRow / 2);          // 0: dK, 1: dV
    const int col0 = (part % (kWarpsPerRow / 2)) * kOutCols;
    uint16_t* out_row = which ? static_cast<uint16_t*>(prm.dv) + b * prm.dv_stride_b + h * prm.dv_stride_h + static_cast<int64_t>(key) * prm.dv_stride_s
                              : static_cast<uint16_t*>(prm.dk) + b * prm.dk_stride_b + h * prm.dk_stride_h + static_cast<int64_t>(key) * prm.dk_stride_s;
    if (n_iter > 0) {
      mbar_wait(bar_done, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
      tcgen05_fence_after_sync();
    }
    {
      const uint32_t tAcc = tmem_base + (which ? Cfg::kColDV : Cfg::kColDK) + lane_base + col0;
      // dV was accumulated from the kept P without the dropout factor
      const float out_scale = (kExt && which) ? prm.ex.drop_rescale : 1.f;
#pragma unroll
      for (int c = 0; c < kOutCols / 32; ++c) {
        uint32_t ar[32];
        if (n_iter > 0) {
          tmem_ld32(tAcc + c * 32, ar);
          tmem_ld_wait(ar);
        } else {
#pragma unroll
          for (int x = 0; x < 32; ++x) ar[x] = 0;  // no query tile sees these keys
        }
        if (key_ok) {
#pragma unroll
          for (int x = 0; x < 32; x += 8) {
            uint4 v;
            if constexpr (kExt != 0) {
#pragma unroll
              for (int y = 0; y < 8; ++y) ar[x + y] = __float_as_uint(__uint_as_float(ar[x + y]) * out_scale);
            }
            v.x = pack2<kBf16>(__uint_as_float(ar[x + 0]), __uint_as_float(ar[x + 1]));
            v.y = pack2<kBf16>(__uint_as_float(ar[x + 2]), __uint_as_float(ar[x + 3]));
            v.z = pack2<kBf16>(__uint_as_float(ar[x + 4]), __uint_as_float(ar[x + 5]));
            v.w = pack2<kBf16>(__uint_as_float(ar[x + 6]), __uint_as_float(ar[x + 7]));
            const int col = col0 + c * 32 + x;
            if (col < prm.d_real) *reinterpret_cast<uint4*>(out_row + col) = v;
          }
        }
      }
    }
  } else if (warp < kCW + 4) {
    // ================================ dQ warps ================================
    // Query row r of the tile: dQ out of tensor memory (at D = 128 all of it at once, which frees
    // the columns for the next tile's dP^T), 64 columns at a time through the staging area (two
    // swizzled boxes of [128 rows x 32 floats]) into the fp32 accumulation buffer with tiled bulk
    // reductions (rows past Sq are dropped by the hardware).  One thread issues every reduction, so
    // the bulk groups it waits for are its own.
    if constexpr (Cfg::kRegsDQ > 80) reg_alloc<Cfg::kRegsDQ>();
    else reg_dealloc<Cfg::kRegsDQ>();
    const int r = (warp & 3) * 32 + lane;
    const uint32_t tQ = tmem_base + Cfg::kColDQ + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const bool issuer = tid == kCW * 32;
    auto stage32 = [&](int cc, const uint32_t (&v)[32]) {  // 32 columns into box cc of the staging area
      uint8_t* box = sStage + cc * kBoxBytes;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(box + r * 128 + ((u ^ (r & 7)) * 16)) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
    };
    auto reduce64 = [&](int hh, int q0) {  // issuer: adds the staged 64 columns hh into the fp32 buffer
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const int c = hh * 2 + cc;
        if (c * 32 < prm.d_real) tma_reduce_add_3d(&tm_dq, sStage + cc * kBoxBytes, c * 32, q0, bh);
      }
      tma_store_commit();
    };
    for (int it = 0; it < n_iter; ++it) {
      const int q0 = (i0 + it) * kBlockM;
      if constexpr (kSepDQ) {
        // the reduction that last read the staging area must have finished reading
        if (issuer) tma_store_wait_read();
        named_barrier_sync(1, 128);
      }
      mbar_wait(bar_dq_full + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
      tcgen05_fence_after_sync();
      if (warp == kCW) bwd_trace(prm, 1, it, 0);
      if constexpr (kSepDQ) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t qr[32];
          tmem_ld32(tQ + (it & 1) * 64 + cc * 32, qr);
          tmem_ld_wait(qr);
          if (cc == 1) {
            tcgen05_fence_before_sync();
            mbar_arrive(bar_dq_free + Cfg::par(it));
          }
          stage32(cc, qr);
        }
        fence_proxy_async_smem();
        named_barrier_sync(1, 128);
        if (issuer) reduce64(0, q0);
      } else {
        uint32_t qr[D / 32][32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld32(tQ + c * 32, qr[c]);
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld_wait(qr[c]);
        tcgen05_fence_before_sync();
        mbar_arrive(bar_dq_free + Cfg::par(it));  // the next query tile's dP^T may be written
        if (warp == kCW) bwd_trace(prm, 1, it, 1);
#pragma unroll
        for (int hh = 0; hh < kHalves; ++hh) {
          if (issuer) tma_store_wait_read();
          named_barrier_sync(1, 128);
          stage32(0, qr[hh * 2]);
          stage32(1, qr[hh * 2 + 1]);
          fence_proxy_async_smem();
          named_barrier_sync(1, 128);
          if (issuer) reduce64(hh, q0);
        }
      }
      if (warp == kCW) bwd_trace(prm, 1, it, 2);
    }
    if (issuer) tma_store_wait_all();  // the reductions must have landed before the CTA ends
  } else {
    reg_dealloc<Cfg::kRegsRest>();
    if (warp == kCW + 4) {
      // ================================ MMA issuer ================================
      constexpr uint32_t idesc_s = make_idesc(kBf16, kBlockN, kBlockM, 0, 0);  // S^T, dP^T: both K-major
      constexpr uint32_t idesc_a = make_idesc(kBf16, kBlockN, kMma, 0, 1);     // dV, dK: A from tensor memory, B N-major
      constexpr uint32_t idesc_q = make_idesc(kBf16, kBlockM, kMma, 1, 1);     // dQ: A M-major, B N-major
      constexpr uint32_t kBoxStep = kBoxBytes >> 4;
      // 16 queries per step; a thread's 16-bit results sit in the first half of its kCols columns
      // (kCols = 64: columns 0-31 and 64-95; kCols = 32: 0-15, 32-47, 64-79, 96-111).  Four steps go out
      // per election: one election per matmul step made the whole backward 1 to 1.5 % slower
      // (B2 H32 S4096 D128 causal 749 against 739 us), a branch per step 10 %.
      constexpr int kA1 = 8, kA2 = Cfg::kCols == 64 ? 16 : 32, kA3 = kA2 + 8;
      const uint32_t q_k = desc_lo(smem_u32(sQ), 16), do_k = desc_lo(smem_u32(sDO), 16);
      const uint32_t k_k = desc_lo(smem_u32(sK), 16), v_k = desc_lo(smem_u32(sV), 16);
      const uint32_t q_n = desc_lo(smem_u32(sQ), kBoxBytes), do_n = desc_lo(smem_u32(sDO), kBoxBytes);
      const uint32_t k_n = desc_lo(smem_u32(sK), kBoxBytes);
      const uint32_t ds_m = desc_lo(smem_u32(sDS), kBoxBytes);
      const uint32_t tDK = tmem_base + Cfg::kColDK, tDV = tmem_base + Cfg::kColDV;
      const uint32_t tS = tmem_base + Cfg::kColS, tDP = tmem_base + Cfg::kColDP, tDQ = tmem_base + Cfg::kColDQ;
      constexpr int kSlotMask = Cfg::kSlots - 1, kSlotShift = Cfg::kSlots - 1;  // slot of tile t, and its phase (t >> shift) & 1

      auto issue_head_dim = [&](uint32_t d, uint32_t a, uint32_t b) {  // d = A B^T over the kMma columns
#pragma unroll
        for (int x = 0; x < kMma / 64; ++x)  // a 64-column box is four 16-column slices, 32 bytes apart
          umma_ss4_elect<2, 2>(d, a + x * kBoxStep, b + x * kBoxStep, idesc_s, x > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = kMma / 64 * 4; kk < kMma / 16; ++kk)
          umma_ss_lo_elect(d, a + (kk >> 2) * kBoxStep + (kk & 3) * 2, b + (kk >> 2) * kBoxStep + (kk & 3) * 2, idesc_s, 1u);
      };
      auto issue_st = [&](int t) {  // S^T = K Q^T of query tile t  (K = head_dim)
        mbar_wait(bar_q_full + (t & 1), (t >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
        tcgen05_fence_after_sync();
        const uint32_t qs = q_k + (t & 1) * (kTileBytes >> 4);
        issue_head_dim(tS, k_k, qs);
        tcgen05_commit_elect(bar_s_full);
      };
      auto issue_dpt = [&](int t) {  // dP^T = V dO^T of query tile t
        mbar_wait(bar_do_full + (t & kSlotMask), (t >> kSlotShift) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
        tcgen05_fence_after_sync();
        const uint32_t dos = do_k + (t & kSlotMask) * (kTileBytes >> 4);
        issue_head_dim(tDP, v_k, dos);
        tcgen05_commit_elect(bar_dp_full);
      };
      auto issue_dq = [&](int t) {  // dQ = dS K  (K = 16 keys per step)
        const uint32_t ds = ds_m + (t & kSlotMask) * (Cfg::kDSBytes >> 4);
        const uint32_t d = tDQ + (kSepDQ ? (t & 1) * 64 : 0);
#pragma unroll
        for (int x = 0; x < kBlockN / 64; ++x)
          umma_ss4_elect<128, 128>(d, ds + x * 512, k_n + x * 512, idesc_q, x > 0 ? 1u : 0u);
        tcgen05_commit_elect(bar_dq_full + Cfg::par(t));
      };
      mbar_wait(bar_kv, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      if (n_iter > 0) {
        issue_st(0);
        issue_dpt(0);
      }
      for (int it = 0; it < n_iter; ++it) {
        bwd_trace(prm, 2, it, 0);
        mbar_wait(bar_p_full + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        tcgen05_fence_after_sync();
        bwd_trace(prm, 2, it, 1);
        const uint32_t don = do_n + (it & kSlotMask) * (kTileBytes >> 4);
#pragma unroll
        for (int x = 0; x < 2; ++x)  // dV += P^T dO
          umma_ts4_elect<kA1, kA2, kA3, 128>(tDV, tS + x * 64, don + x * 512, idesc_a, (it > 0 || x > 0) ? 1u : 0u);
        tcgen05_commit_elect(bar_do_empty + (it & kSlotMask));  // dO_i has no reader after this point
        if (it + 1 < n_iter) issue_st(it + 1);  // over P^T, behind the matmul that reads it
        mbar_wait(bar_ds_full + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        tcgen05_fence_after_sync();
        bwd_trace(prm, 2, it, 2);
        const uint32_t qn = q_n + (it & 1) * (kTileBytes >> 4);
#pragma unroll
        for (int x = 0; x < 2; ++x)  // dK += dS^T Q
          umma_ts4_elect<kA1, kA2, kA3, 128>(tDK, tDP + x * 64, qn + x * 512, idesc_a, (it > 0 || x > 0) ? 1u : 0u);
        tcgen05_commit_elect(bar_q_empty + (it & 1));  // this Q slot has no reader after this point
        if constexpr (kSepDQ) {
          if (it + 1 < n_iter) issue_dpt(it + 1);  // over dS^T, behind the matmul that reads it
          if (it >= 2) {
            mbar_wait(bar_dq_free + Cfg::par(it), Cfg::phase(it - 2), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
            tcgen05_fence_after_sync();
          }
          issue_dq(it);
        } else {
          issue_dq(it);  // over dS^T, behind the matmul that reads it
          bwd_trace(prm, 2, it, 3);
          if (it + 1 < n_iter) {
            mbar_wait(bar_dq_free + Cfg::par(it), Cfg::phase(it), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
            tcgen05_fence_after_sync();
            issue_dpt(it + 1);
          }
        }
      }
      tcgen05_commit_elect(bar_done);
    } else if (warp == kCW + 5) {
      // ================================ TMA producer ================================
      constexpr int kSlots = Cfg::kSlots;
      for (int it = 1; it < n_iter; ++it) {  // the first tiles went out before the allocation
        if (it >= 2) {
          mbar_wait(bar_q_empty + (it & 1), ((it >> 1) - 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
          if (lane == 0) load_q(it);
        }
        if (it >= kSlots) {
          const int use = (it >> (kSlots - 1)) - 1;  // which use of the slot must have ended
          mbar_wait(bar_do_empty + (it & (kSlots - 1)), use & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
          if (lane == 0) load_do(it);
        }
        __syncwarp();
      }
      if (n_iter == 0) mbar_wait(bar_kv, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);  // drain the K/V load before exit
    } else if (warp == kCW + 6) {
      // ================================ row loader ================================
      // -LSE * log2(e) and -delta * scale of the query tile's 128 rows, four per lane.  A row past
      // the end, or one whose keys are all masked (LSE = -inf), gets -inf, so that its P and dS are 0.
      const float* const lse_bh = prm.lse + static_cast<int64_t>(bh) * prm.Sq;
      const float* const delta_bh = prm.delta + static_cast<int64_t>(bh) * prm.Sq;
      for (int it = 0; it < n_iter; ++it) {
        const int row0 = (i0 + it) * kBlockM + lane * 4;
        float nl[4], nd[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          const bool ok = row0 + y < prm.Sq;
          const float l = ok ? lse_bh[row0 + y] : -INFINITY;
          nl[y] = (l == -INFINITY) ? -INFINITY : -l * 1.4426950408889634f;
          nd[y] = ok ? -delta_bh[row0 + y] * prm.scale : 0.f;
        }
        if constexpr ((kExt & kBwdMatBias) != 0) {
          // the next query tile's block of the bias into L2, four rows per lane
          const int esize = prm.ex.bias_f32 ? 4 : 2;
          const uint8_t* const bias_bh = static_cast<const uint8_t*>(prm.ex.bias) +
                                         (b * prm.ex.bias_stride_b + h * prm.ex.bias_stride_h) * esize;
          for (int y = 0; y < 4; ++y) {
            const int q = row0 + kBlockM + y;
            if (q < prm.Sq)
              prefetch_bias(prm.ex, bias_bh + q * prm.ex.bias_stride_q * esize, k0, min(kBlockN, prm.Sk - k0));
          }
        }
        // a slot is free once P^T (-LSE) and dS^T (-delta) of the tile that used it last are complete
        const int last = it - Cfg::kSlots;
        if (last >= 0) mbar_wait(bar_p_full + Cfg::par(last), Cfg::phase(last), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        *reinterpret_cast<float4*>(sNegLse + (it & (Cfg::kSlots - 1)) * 128 + lane * 4) = make_float4(nl[0], nl[1], nl[2], nl[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_lse_full + Cfg::par(it));
        if (last >= 0) mbar_wait(bar_ds_full + Cfg::par(last), Cfg::phase(last), cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        *reinterpret_cast<float4*>(sNegDelta + (it & (Cfg::kSlots - 1)) * 128 + lane * 4) = make_float4(nd[0], nd[1], nd[2], nd[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_delta_full + Cfg::par(it));
      }
    }
  }

  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == kCW + 4) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

}  // namespace fo
