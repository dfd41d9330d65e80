// The 64-key forward kernel for attention with a bias (flash_attn_ws64.cuh has the roles, buffers and
// barriers; this is the same pipeline): a CTA takes its key tiles from the last to the first, or from
// the first to the last where the bias falls along the keys.
//
// A bias that moves against the order raises the row maxima by more than the rescaling threshold at
// almost every step, and each time the step's exponentials are taken again and O is rescaled in tensor
// memory; with the order the first tile sets the maximum.  The CTA compares the bias of its first and
// last key (read under the barrier set-up) and goes up if the first is larger by more than the
// threshold; a bias that moves less than that never needs the choice.  us at B2 H16 S3072 with linear
// biases, one order wrong and right: rising D128 causal 219 and 146, D64 284 and 179 without a mask;
// falling D128 causal 181 and 149, D64 228 and 178.  Key padding (D128 causal 160 by the ascending
// kernel of before) takes 144 either way.
// A 16-bit matrix bias with 16-byte aligned rows is fetched into registers a step ahead.  B2 H16 S2048
// against the ascending kernel: D64 170 to 129 us, with dropout 247 to 187, D128 causal 99 to 83.
// It is a kernel of its own because the plain one does not bear the generalisation: compiled from
// this source, without the bias, it took 341 us instead of 290 at B2 H32 S4096 D128 causal (the
// order in which the assembler places the exponentials around the turn-taking barriers changes).
#pragma once

#include "flash_attn_ring.h"
#include "flash_attn_ws64.cuh"

namespace fo {

// kExt: kFwdVecBias, kFwdMatBias or kFwdMatBias32, with or without kFwdDropout.
template <int D, bool kBf16, int kExt>
__global__ void __launch_bounds__(512, 1)
attn_fwd_ws64r_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const AttnParams prm) {
  using Cfg = Ws64Config<D>;
  constexpr int kTileBytes = Cfg::kTileBytes;
  constexpr int kStages = Cfg::kStages;
  constexpr int kBoxes = Cfg::kBoxes;
  // Registers of the softmax warps and of the last four: 8 x kRegsSoftmax + 4 x 80 + 4 x kRegsRest are
  // what the block was launched with, 16 x 128.  With dropout and a vector or 16-bit bias the second
  // split and the hash index of a step formed in one register (kTight) avoid spills: B2 H16 S2048, vector
  // bias D64 158 to 154 us, matrix bias D64 198 to 187, D128 225 to 203; the other forms measured slower
  // with them (vector bias D128 S3072 198 to 229 us, fp32 matrix bias with dropout 259 to 285).
  constexpr bool kTight = (kExt & kFwdDropout) != 0 && (kExt & kFwdMatBias32) == 0;
  constexpr int kRegsSoftmax = kTight ? 184 : 192, kRegsRest = kTight ? 64 : 48;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem + Cfg::kOffQ;    // two tiles
  uint8_t* sKV = smem + Cfg::kOffKV;  // kStages tiles
  float* s_alpha = reinterpret_cast<float*>(smem + Cfg::kOffAlpha);
  float* s_final = reinterpret_cast<float*>(smem + Cfg::kOffFinal);
  float* s_bias = reinterpret_cast<float*>(smem + Cfg::kOffBias);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* bar_q_full = bars;                     // TMA -> MMA
  uint64_t* bar_kv_full = bars + 1;                // [kStages] TMA -> MMA
  uint64_t* bar_kv_empty = bar_kv_full + kStages;  // [kStages] MMA -> TMA
  uint64_t* bar_s_full = bar_kv_empty + kStages;   // [2 tiles][2 buffers] MMA -> softmax
  // [2][2] softmax and correction -> MMA (256 arrivals): P of the step is in tensor memory (128
  // softmax threads) and O has been rescaled if the step needed it (128 correction threads).
  // One barrier for both, because every wait on the issuing warp's path costs about 200 cycles
  // even when the phase completed long ago.  The correction threads arrive as soon as they have
  // the step's rescale factors, unless a factor differs from 1: only then do they wait for the
  // previous P V and rescale O first.
  uint64_t* bar_p_full = bar_s_full + 4;
  uint64_t* bar_o_full = bar_p_full + 4;           // [2] MMA -> correction
  // [2][2] softmax -> correction (128 arrivals), one barrier per step parity: the softmax
  // threads can be two steps ahead of the correction warps, which a single barrier's phase
  // bit could not tell from zero steps ahead
  uint64_t* bar_corr = bar_o_full + 2;
  uint64_t* bar_final = bar_corr + 4;              // [2] softmax -> correction, once
  // [2] MMA -> epilogue, once: every P V of the tile has finished.  bar_o_full cannot serve: by
  // then nobody may have waited on it for many steps, and its phase bit alone does not say
  // whether the last P V is the one that completed.
  uint64_t* bar_o_done = bar_final + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffMisc);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* skip = cta_abort + 1;
  volatile int* ascending = cta_abort + 2;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int bh_count = prm.B * prm.H;
  const int num_pairs = (prm.num_q_tiles + 1) >> 1;
  // block -> (head group, pair, head): see flash_attn_ws.cuh
  const int group_blocks = prm.head_group * num_pairs;
  const int group = static_cast<int>(blockIdx.x) / group_blocks;
  const int in_group = static_cast<int>(blockIdx.x) - group * group_blocks;
  const int heads_here = min(prm.head_group, bh_count - group * prm.head_group);
  const int pair = num_pairs - 1 - in_group / heads_here;
  const int bh = group * prm.head_group + in_group % heads_here;
  const int b = bh / prm.H;
  const int h = bh - b * prm.H;
  const int hk = prm.kv_head_bcast ? 0 : h;  // head coordinate of K and V
  // keys visible to query tile 0 / 1 of this pair, in 64-key steps (T) and 128-key tiles (n)
  const int vis0 = prm.causal ? min(prm.Sk, (2 * pair + 1) * kBlockM) : prm.Sk;
  const int vis1 = prm.causal ? min(prm.Sk, (2 * pair + 2) * kBlockM) : prm.Sk;
  const int n0 = (vis0 + kBlockN - 1) / kBlockN;
  const int n1 = (vis1 + kBlockN - 1) / kBlockN;
  const int T0 = 2 * n0, T1 = 2 * n1;  // T1 >= T0 >= 2
  // The steps of a query tile are `first` to `end` - 1, two per key tile.  When the last key tile's upper
  // half has no visible key (`odd`), one is left out (taken, with all its scores masked, it made 64 keys
  // cost 38 us instead of 29 at B64 H12 D64, and 1088 keys 128 instead of 120 at B8 H16): going up the
  // very last one, going down step 0, whose barrier phases are then completed at the set-up, so that
  // step numbers stand for buffers and phases as ever.
  const int odd0 = (vis0 + kStepN - 1) / kStepN & 1, odd1 = (vis1 + kStepN - 1) / kStepN & 1;

  if (tid == 0) {
    *cta_abort = 0;
    // the ends of the bias over the keys that tile 0 sees (a matrix bias: in tile 1's first row); with a
    // single key tile the order does not matter
    float bias_first = 0.f, bias_last = 0.f;
    if (n1 > 1) {
      const int64_t row = min((2 * pair + 1) * kBlockM, prm.Sq - 1);
      const uint8_t* const p = static_cast<const uint8_t*>(prm.ex.bias) +
                               (b * prm.ex.bias_stride_b + h * prm.ex.bias_stride_h + row * prm.ex.bias_stride_q) *
                                   (prm.ex.bias_f32 ? 4 : 2);
      bias_first = load_bias1<kBf16>(prm.ex, p, 0);
      bias_last = load_bias1<kBf16>(prm.ex, p, vis0 - 1);
    }
    const int status = *reinterpret_cast<volatile int*>(prm.device_status);
    mbar_init(bar_q_full, 1);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bar_kv_full + i, 1);
      mbar_init(bar_kv_empty + i, 2);  // one arrival from each MMA-issuing warp
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(bar_s_full + i, 1);
      mbar_init(bar_p_full + i, 256);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_o_full + s, 1);
      mbar_init(bar_corr + 2 * s, 128);
      mbar_init(bar_corr + 2 * s + 1, 128);
      mbar_init(bar_final + s, 128);
      mbar_init(bar_o_done + s, 1);
    }
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    *skip = status;
    const bool ascend = bias_first - bias_last > kRescaleThreshold;
    *ascending = ascend;
    for (int s = 0; s < 2; ++s)
      if (!ascend && (s ? odd1 : odd0)) {  // the phases of a step 0 that is left out
        mbar_arrive(bar_s_full + 2 * s);
        mbar_arrive_n(bar_p_full + 2 * s, 256);
        mbar_arrive_n(bar_corr + 2 * s, 128);
        mbar_arrive(bar_o_full + s);
      }
    fence_mbar_init();
  }
  __syncthreads();
  if (*skip) return;  // another CTA already timed out: do nothing
  const bool up = *ascending != 0;
  const int first0 = up ? 0 : odd0, first1 = up ? 0 : odd1;
  const int end0 = up ? T0 - odd0 : T0, end1 = up ? T1 - odd1 : T1;
  // Tile 1 of the pair has up to two steps more than tile 0, those next to the diagonal: going down
  // tile 0 joins `lead0` steps late, going up it ends `tail0` steps early.
  const int extra = (end1 - first1) - (end0 - first0);
  const int lead0 = up ? 0 : extra, tail0 = up ? extra : 0;
  // First key of step t.  A key tile's lower half comes before its upper half (in the tile on the
  // diagonal more rows see it), and behind it if step 0 is left out.
  const int tile_dir = up ? kBlockN : -kBlockN;
  auto step_key = [tile_dir](int t, int first, int key0) {
    return key0 + (t >> 1) * tile_dir + ((t & 1) ^ first) * kStepN;
  };

  // The first loads (Q and the first ring fill of K and V) need only the barriers: they go out
  // here, under the tensor-memory allocation, instead of after it.
  const int first_fill = min(kStages, 2 * n1);
  auto load_kv = [&](int i) {  // ring entry i: K_{i/2} (even) or V_{i/2} (odd)
    const int st = i % kStages;
    mbar_arrive_expect_tx(bar_kv_full + st, kTileBytes);
    const CUtensorMap* map = (i & 1) ? &tm_v : &tm_k;
    for (int c = 0; c < kBoxes; ++c)
      tma_load_4d(sKV + st * kTileBytes + c * kBoxBytes, map, bar_kv_full + st, c * kBoxCols,
                  (up ? i >> 1 : n1 - 1 - (i >> 1)) * kBlockN, hk, b);
  };
  if (warp == 13 && lane == 0) {
    mbar_arrive_expect_tx(bar_q_full, 2 * kTileBytes);
    for (int s = 0; s < 2; ++s)
      for (int c = 0; c < kBoxes; ++c)
        tma_load_4d(sQ + s * kTileBytes + c * kBoxBytes, &tm_q, bar_q_full, c * kBoxCols,
                    (2 * pair + s) * kBlockM, h, b);
    for (int i = 0; i < first_fill; ++i) load_kv(i);
  }
  if (warp == 12) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish_alloc_permit();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  int* const dstat = prm.device_status;

  if (warp < 8) {
    // ================================ softmax ================================
    reg_alloc<kRegsSoftmax>();
    const int s = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const int q0 = (2 * pair + s) * kBlockM;
    const int row = q0 + r;
    const int first = s ? first1 : first0, end = s ? end1 : end0;
    const int key0 = up ? 0 : (s ? n1 - 1 : n0 - 1) * kBlockN;  // first key of the first key tile
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS_tile = tmem_base + Cfg::kColS0 + s * kBlockN + lane_base;
    float* alpha_slot = s_alpha + s * 256 + r;
    float m_run = -INFINITY, l_run = 0.f;
    constexpr bool vec_bias = (kExt & kFwdVecBias) != 0, mat_bias16 = (kExt & kFwdMatBias) != 0;
    constexpr bool mat_bias = mat_bias16 || (kExt & kFwdMatBias32) != 0;
    constexpr bool has_drop = (kExt & kFwdDropout) != 0;
    const uint8_t* bias_row = nullptr;
    if (mat_bias && row < prm.Sq)
      bias_row = static_cast<const uint8_t*>(prm.ex.bias) +
                 (b * prm.ex.bias_stride_b + h * prm.ex.bias_stride_h + static_cast<int64_t>(row) * prm.ex.bias_stride_q) *
                     (prm.ex.bias_f32 ? 4 : 2);
    const uint32_t drop_row = prm.ex.drop_base +
                              static_cast<uint32_t>(bh) * static_cast<uint32_t>(prm.Sq) * static_cast<uint32_t>(prm.Sk) +
                              static_cast<uint32_t>(row) * static_cast<uint32_t>(prm.Sk);
    // the scores are scaled when the bias is added, not in the exponent
    const float exp_scale = 1.f;
    // a row-independent bias goes through shared memory, fetched one 128-key tile ahead
    const uint8_t* bias_vec = nullptr;
    float* sb = s_bias + s * 256;
    float bias_next = 0.f;
    if constexpr (vec_bias) {
      bias_vec = static_cast<const uint8_t*>(prm.ex.bias) +
                 (b * prm.ex.bias_stride_b + h * prm.ex.bias_stride_h) * (prm.ex.bias_f32 ? 4 : 2);
      const int col = key0 + r;
      bias_next = (col < prm.Sk) ? load_bias1<kBf16>(prm.ex, bias_vec, col) : 0.f;
    }

    // S of the next step is normally complete long before it is needed: polled once while the
    // current step's exponentials are in flight, waited on only if that poll failed
    // The two tiles' softmax warps share the ex2 units.  Left alone they fall into lockstep: both
    // reduce maxima at the same time (ex2 idle), then both exponentiate (ex2 contended).  The
    // exponentials of the two tiles are therefore made to alternate with a pair of named barriers
    // (tile 0 goes first): while one tile exponentiates, the other loads S, reduces its maxima
    // and stores P.  A tile that runs out of steps keeps passing the turn on.
    constexpr int kTurn0 = 3, kTurn1 = 4, kTurnCount = 256;  // named barriers: "tile 0 may exponentiate", "tile 1 may"
    const bool ping_pong = prm.ping_pong != 0;
    if (ping_pong && s == 1) named_barrier_arrive(kTurn0, kTurnCount);
    // tile 0 takes and passes the turn for the steps that only tile 1 has
    if (ping_pong && s == 0)
      for (int t = 0; t < lead0; ++t) {
        named_barrier_sync(kTurn0, kTurnCount);
        named_barrier_arrive(kTurn1, kTurnCount);
      }

    uint32_t sr[2][32];  // scores of the current step (scaled and biased already when there is a bias)

    // Stages the row-independent bias of the key tile that step `tn` starts.
    auto stage_vec_bias = [&](int tn) {
      const int j = tn >> 1;
      sb[(j & 1) * 128 + r] = bias_next;
      const int col = key0 + (j + 1) * tile_dir + r;  // of the key tile after this one (there may be none)
      bias_next = (col >= 0 && col < prm.Sk) ? load_bias1<kBf16>(prm.ex, bias_vec, col) : 0.f;
      // a buffer is rewritten two key tiles later, behind the barrier of the tile between
      named_barrier_sync(1 + s, 128);
    };
    // Issues the tensor-memory loads of step tn's scores (S must be complete).
    auto issue_load = [&](int tn, int c) {
      const uint32_t tSn = tS_tile + (tn & 1) * kStepN;
      tmem_ld32(tSn + c * 32, sr[c]);
    };
    // A 16-bit matrix bias whose rows are 16-byte aligned is fetched into registers ahead of the
    // step that adds it (every thread reads its own row: 128 bytes per step), other forms when they
    // are added.
    uint4 bias_raw[mat_bias16 ? 8 : 1];
    bool bias_held = false;
    auto fetch_mat_bias = [&](int tn) {
      const int k0n = step_key(tn, first, key0);
      bias_held = bias_row != nullptr && prm.ex.bias_vec && k0n + kStepN <= prm.Sk;
      if (bias_held) {
        const uint4* const p = reinterpret_cast<const uint4*>(bias_row + static_cast<int64_t>(k0n) * 2);
#pragma unroll
        for (int i = 0; i < (mat_bias16 ? 8 : 1); ++i) bias_raw[i] = __ldg(p + i);
      }
    };
    auto add_bias2 = [&](int c, int i, float2 bias2) {  // scores i and i + 1 of chunk c, scaled, plus their bias
      const float2 x = __ffma2_rn(make_float2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])),
                                  make_float2(prm.scale_log2, prm.scale_log2), bias2);
      sr[c][i] = __float_as_uint(x.x);
      sr[c][i + 1] = __float_as_uint(x.y);
    };
    // Waits for those loads and applies bias and masks in place.
    auto prep_loads = [&](int tn) {
      const int k0n = step_key(tn, first, key0);
      const bool need_mask = (k0n + kStepN > prm.Sk) || (prm.causal && k0n + kStepN - 1 > q0);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        tmem_ld_wait(sr[c]);
        if ((warp & 3) == 0 && tn > 0) trace_event(prm, s, tn - 1, c == 0 ? 1 : 4);  // loads in
        if constexpr (vec_bias) {
          const float4* bv = reinterpret_cast<const float4*>(sb + ((tn >> 1) & 1) * 128 + ((tn & 1) ^ first) * kStepN + c * 32);
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 v4 = bv[i >> 2];  // the same address in every thread: a broadcast
            add_bias2(c, i, make_float2(v4.x, v4.y));
            add_bias2(c, i + 2, make_float2(v4.z, v4.w));
          }
        }
        if constexpr (mat_bias) {
          float bb[32];
          if (mat_bias16 && bias_held) {
            constexpr float kLog2e = 1.4426950408889634f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint4 v = bias_raw[mat_bias16 ? c * 4 + i : 0];
              const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int y = 0; y < 4; ++y) {
                const float2 f = __fmul2_rn(unpack2<kBf16>(w[y]), make_float2(kLog2e, kLog2e));
                bb[8 * i + 2 * y] = f.x;
                bb[8 * i + 2 * y + 1] = f.y;
              }
            }
          } else {
            load_bias32<kBf16, mat_bias16 ? kBias16 : kBias32>(prm.ex, bias_row, k0n + c * 32, prm.Sk, bb);
          }
#pragma unroll
          for (int i = 0; i < 32; i += 2) add_bias2(c, i, make_float2(bb[i], bb[i + 1]));
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int col = k0n + c * 32 + i;
            if (col >= prm.Sk || (prm.causal && col > row)) sr[c][i] = 0xff800000u;  // -inf
          }
        }
      }
    };
    // Row maximum of the scores in sr: four independent accumulators (and 3-input max) keep the
    // dependency chain short.
    auto row_max = [&]() {
      float mxa = -INFINITY, mxb = -INFINITY, mxc = -INFINITY, mxd = -INFINITY;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          mxa = max3(mxa, __uint_as_float(sr[c][i + 0]), __uint_as_float(sr[c][i + 1]));
          mxb = max3(mxb, __uint_as_float(sr[c][i + 2]), __uint_as_float(sr[c][i + 3]));
          mxc = max3(mxc, __uint_as_float(sr[c][i + 4]), __uint_as_float(sr[c][i + 5]));
          mxd = max3(mxd, __uint_as_float(sr[c][i + 6]), __uint_as_float(sr[c][i + 7]));
        }
      }
      return fmaxf(fmaxf(mxa, mxb), fmaxf(mxc, mxd));
    };

    // prologue: scores of the first step; their row maximum is the first reference maximum
    if constexpr (vec_bias) stage_vec_bias(first);
    if constexpr (mat_bias16) fetch_mat_bias(first);
    mbar_wait(bar_s_full + 2 * s + first, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
    tcgen05_fence_after_sync();
    issue_load(first, 0);
    issue_load(first, 1);
    prep_loads(first);
    m_run = row_max() * exp_scale;

    // The exponentials of a step do not wait for the step's own row maximum: they are taken
    // against the reference maximum the row already has (lazy rescaling moves it only when the
    // true maximum exceeds it by kRescaleThreshold), and the maximum is reduced alongside them,
    // its instructions filling issue slots that the ex2 unit's rate leaves empty.  Only if a row
    // of the warp turns out to need a new reference (rare after the first steps) are the step's
    // exponentials taken again.  Each iteration then fetches step t + 1 (whose S the tensor core
    // finished meanwhile) behind the P stores, so that the latencies of the loads, of the P store
    // and of the barriers overlap instead of adding up.
    for (int t = first; t < end; ++t) {
      const int u = t & 1;
      const int k0 = step_key(t, first, key0);
      const uint32_t drop_idx = drop_row + (kTight ? static_cast<uint32_t>(k0) : 0u);
      const uint32_t tS = tS_tile + u * kStepN;
      float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
      if (ping_pong) named_barrier_sync_dep(s ? kTurn1 : kTurn0, kTurnCount, neg_m);  // exponentials start after this
      if ((warp & 3) == 0) trace_event(prm, s, t, 0);  // turn taken
      const float2 sc2 = make_float2(exp_scale, exp_scale);
      float2 acc0, acc1;
      uint32_t pr[2][16];
      const bool more = t + 1 < end;
      bool s_next_ready = false;
      float mxa = -INFINITY, mxb = -INFINITY;
      // P = exp2(S * scale - reference) for the whole step; `first` is the pass that also passes
      // the turn on, polls the next S and reduces the row maximum
      auto exp_pass = [&](float neg_ref, const bool first) {
        const float2 nm2 = make_float2(neg_ref, neg_ref);
        acc0 = make_float2(0.f, 0.f);
        acc1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          // one non-blocking look at S of step t + 1 (as a rule complete by now); the answer is
          // needed only after the exponentials, so its latency is hidden
          if (first && c == 1 && more) s_next_ready = mbar_test_wait(bar_s_full + 2 * s + (u ^ 1), ((t + 1) >> 1) & 1);
          // The turn is passed on after the first half (the partial row sums depend on all of its
          // exponentials): the other tile's first half then shares the ex2 units with this tile's
          // second half, two warps per scheduler, which hides the latencies a lone warp exposes.
          float2 nm2c = nm2;
          if (first && c == 1 && ping_pong) {
            float dep = neg_ref;
            named_barrier_arrive_mid(s ? kTurn0 : kTurn1, kTurnCount, dep, acc0.x + acc0.y, acc1.x + acc1.y);
            nm2c = make_float2(dep, dep);  // the second half's arithmetic hangs on the arrive
          }
#pragma unroll
          for (int q = 0; q < 16; ++q) {  // column pair q of the chunk
            const float a = __uint_as_float(sr[c][2 * q]), b = __uint_as_float(sr[c][2 * q + 1]);
            float2 x = __ffma2_rn(make_float2(a, b), sc2, nm2c);
            x.x = fast_exp2(x.x);
            x.y = fast_exp2(x.y);
            if (q & 1) acc1 = __fadd2_rn(acc1, x); else acc0 = __fadd2_rn(acc0, x);
            if (first) {
              if (q & 1) mxb = max3(mxb, a, b); else mxa = max3(mxa, a, b);
            }
            if constexpr (has_drop) {
              // dropped elements leave the row sum untouched and enter P V as zeros; the factor
              // 1 / (1 - p) is applied once, to O, in the epilogue
              const uint32_t idx = drop_idx + static_cast<uint32_t>((kTight ? 0 : k0) + c * 32 + 2 * q);
              if (dropout_hash(idx, prm.ex.drop_seed) <= prm.ex.drop_threshold) x.x = 0.f;
              if (dropout_hash(idx + 1u, prm.ex.drop_seed) <= prm.ex.drop_threshold) x.y = 0.f;
            }
            pr[c][q] = pack2<kBf16>(x.x, x.y);
          }
        }
      };
      exp_pass(neg_m, true);
      // did a row outgrow its reference?
      const float m_cand = fmaxf(m_run, fmaxf(mxa, mxb) * exp_scale);
      const bool grow = m_cand - m_run > kRescaleThreshold;  // false when both are -inf (NaN)
      float alpha = 1.f;
      if (__any_sync(0xffffffffu, grow)) {
        // new reference for the rows that need one; the others repeat what they had
        const float m_new = grow ? m_cand : m_run;
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        alpha = grow ? fast_exp2(m_run - m_use) : 1.f;
        m_run = m_new;
        exp_pass(-m_use, false);
      }
      // hand the rescale factor to the correction warps
      alpha_slot[u * 128] = alpha;
      mbar_arrive(bar_corr + 2 * s + u);
      if ((warp & 3) == 0) trace_event(prm, s, t, 2);
      // P (two 16-bit values per column) over the first 32 columns of this step's buffer
      tmem_st16(tS, pr[0]);
      tmem_st16(tS + 16, pr[1]);
      if (more) {
        // S of step t + 1 was issued when P of step t - 1 was handed over: complete by now as a
        // rule.  Its loads go out behind the P stores; the score registers are free, everything
        // of step t is in pr.
        if (vec_bias && u == 1) stage_vec_bias(t + 1);
        if constexpr (mat_bias16) fetch_mat_bias(t + 1);
        if (mat_bias && bias_row != nullptr && t + 2 < end) {
          const int c0 = step_key(t + 2, first, key0);
          prefetch_bias(prm.ex, bias_row, c0, min(kStepN, prm.Sk - c0), up);
        }
        if (!s_next_ready)
          mbar_wait(bar_s_full + 2 * s + (u ^ 1), ((t + 1) >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
        tcgen05_fence_after_sync();
        issue_load(t + 1, 0);
        issue_load(t + 1, 1);
      }
      tcgen05_wait_st();
      tcgen05_fence_before_sync();
      mbar_arrive(bar_p_full + 2 * s + u);
      if ((warp & 3) == 0) trace_event(prm, s, t, 3);
      const float rsum = (acc0.x + acc0.y) + (acc1.x + acc1.y);
      l_run = l_run * alpha + rsum;
      if (more) prep_loads(t + 1);
      if ((warp & 3) == 0) trace_event(prm, s, t, 5);
    }
    // Tile 0 keeps taking and passing the turn for the steps that only tile 1 still has, one at a time
    // (arrivals sent ahead of the other tile's waits would complete a barrier phase on their own and
    // strand it).  Tile 1's very last arrival finds nobody waiting: the CTA ends with that barrier half
    // counted, which is harmless.
    if (ping_pong && s == 0)
      for (int t = 0; t < tail0; ++t) {
        named_barrier_sync(kTurn0, kTurnCount);
        named_barrier_arrive(kTurn1, kTurnCount);
      }
    s_final[s * 256 + r] = l_run;
    s_final[s * 256 + 128 + r] = m_run;
    mbar_arrive(bar_final + s);
  } else if (warp < 12) {
    // ================================ correction + epilogue ================================
    reg_dealloc<80>();
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // epilogue of one query tile: O / l and LSE
    auto epilogue = [&](int s) {
      mbar_wait(bar_final + s, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
      mbar_wait(bar_o_done + s, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
      tcgen05_fence_after_sync();
      const float l_run = s_final[s * 256 + r];
      const float m_run = s_final[s * 256 + 128 + r];
      const float o_scale = prm.ex.drop_rescale;
      const float inv_l = (l_run > 0.f) ? o_scale / l_run : 0.f;
      const int row = (2 * pair + s) * kBlockM + r;
      const bool row_ok = row < prm.Sq;
      uint16_t* orow = static_cast<uint16_t*>(prm.o) + b * prm.o_stride_b + h * prm.o_stride_h +
                       static_cast<int64_t>(row) * prm.o_stride_s;
      const uint32_t tO = tmem_base + Cfg::kColO0 + s * D + lane_base;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t orr[32];
        tmem_ld32(tO + c * 32, orr);
        tmem_ld_wait(orr);
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 v;
            v.x = pack2<kBf16>(__uint_as_float(orr[i + 0]) * inv_l, __uint_as_float(orr[i + 1]) * inv_l);
            v.y = pack2<kBf16>(__uint_as_float(orr[i + 2]) * inv_l, __uint_as_float(orr[i + 3]) * inv_l);
            v.z = pack2<kBf16>(__uint_as_float(orr[i + 4]) * inv_l, __uint_as_float(orr[i + 5]) * inv_l);
            v.w = pack2<kBf16>(__uint_as_float(orr[i + 6]) * inv_l, __uint_as_float(orr[i + 7]) * inv_l);
            if (c * 32 + i < prm.d_real) *reinterpret_cast<uint4*>(orow + c * 32 + i) = v;
          }
        }
      }
      if (row_ok && prm.lse != nullptr) {
        prm.lse[static_cast<int64_t>(bh) * prm.Sq + row] =
            (l_run > 0.f) ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
      }
    };
    for (int g = first1; g < end1; ++g) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int first = s ? first1 : first0;
        const int t = s ? g : g - first1 - lead0 + first0;
        if (t < first || t >= (s ? end1 : end0)) continue;
        mbar_wait(bar_corr + 2 * s + (t & 1), (t >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        const float alpha = s_alpha[s * 256 + (t & 1) * 128 + r];
        if (t > first && __any_sync(0xffffffffu, alpha != 1.f)) {
          // this step's P V is not issued before this warp arrives below; O is complete up to
          // the previous step once that step's P V has finished.  (The P V of step t - 2 is
          // known to have finished, since S of step t exists: the phase bit is unambiguous.)
          mbar_wait(bar_o_full + s, (t - 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
          tcgen05_fence_after_sync();
          {
            const uint32_t tO = tmem_base + Cfg::kColO0 + s * D + lane_base;
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t orr[32];
              tmem_ld32(tO + c * 32, orr);
              tmem_ld_wait(orr);
#pragma unroll
              for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
              tmem_st32(tO + c * 32, orr);
            }
            tcgen05_wait_st();
          }
          tcgen05_fence_before_sync();
        }
        mbar_arrive(bar_p_full + 2 * s + (t & 1));
      }
    }
    epilogue(0);
    epilogue(1);
  } else {
    reg_dealloc<kRegsRest>();
    if (warp == 12 || warp == 14) {
      // ================================ MMA issuers ================================
      // One warp per query tile (12: tile 0, 14: tile 1).  The tensor core's instruction queue
      // is short: whenever the issuing warp is not issuing (a barrier wait costs it about 200
      // cycles even on a completed phase) the pipe runs dry.  With two issuers one tile's waits
      // hide behind the other tile's instructions.  Nothing orders the two streams against each
      // other, and nothing has to: each tile owns its S / P buffers and its O accumulator, and a
      // K/V ring slot is released by both warps (bar_kv_empty counts two arrivals).
      const int s = (warp == 14) ? 1 : 0;
      const int first = s ? first1 : first0, end = s ? end1 : end0;
      constexpr uint32_t idesc_qk = make_idesc(kBf16, kBlockM, kStepN, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc(kBf16, kBlockM, D, 0, 1);
      // Everything below is warp-uniform; only the tcgen05 instructions themselves are issued by
      // one elected lane.  Descriptors are kept as 32-bit low halves: per instruction one add.
      const uint32_t q_lo = desc_lo(smem_u32(sQ) + s * kTileBytes, 16);
      const uint32_t kv_k_lo = desc_lo(smem_u32(sKV), 16);         // K tiles: K-major
      const uint32_t kv_v_lo = desc_lo(smem_u32(sKV), kBoxBytes);  // V tiles: N-major
      constexpr uint32_t kStageStep = kTileBytes >> 4;
      constexpr uint32_t kBoxStep = kBoxBytes >> 4;
      const uint32_t tS_tile = tmem_base + Cfg::kColS0 + s * kBlockN;
      const uint32_t tO = tmem_base + Cfg::kColO0 + s * D;
      // S(s, t) = Q_s K^T over the step's half of the K tile in ring slot `stage`, u = t & 1: 64 rows
      // of a K-major box are 64 * 128 bytes further on
      auto issue_s = [&](int u, int stage) {
        const uint32_t b_lo = kv_k_lo + stage * kStageStep + (u ^ first) * ((kStepN * 128) >> 4);
        const uint32_t tS = tS_tile + u * kStepN;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          // k-slice kk: box kk/4, 32 bytes per slice inside the 128-byte swizzle span
          const uint32_t off = (kk >> 2) * kBoxStep + (kk & 3) * 2;
          umma_ss_lo_elect(tS, q_lo + off, b_lo + off, idesc_qk, kk > 0 ? 1u : 0u);
        }
      };
      // O_s (+)= P(s, t) V over the step's half of the V tile in ring slot `stage`
      auto issue_pv = [&](int u, int stage, bool acc) {
        const uint32_t tP = tS_tile + u * kStepN;
        const uint32_t b_lo = kv_v_lo + stage * kStageStep + (u ^ first) * (kStepN / 16) * 128;
#pragma unroll
        for (int kk = 0; kk < kStepN / 16; ++kk) {
          // 16 key rows per slice: 2048 bytes of V, 8 packed columns of P
          umma_ts_lo_elect(tO, tP + kk * 8, b_lo + kk * 128, idesc_pv, (acc || kk > 0) ? 1u : 0u);
        }
      };

      auto wait_kv = [&](int slot, uint32_t parity) {
        mbar_wait(bar_kv_full + slot, parity, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      };
      auto kv_ready = [&](int slot, uint32_t parity) { return mbar_test_wait(bar_kv_full + slot, parity); };
      auto release_kv = [&](int slot) { tcgen05_commit_elect(bar_kv_empty + slot); };
      auto scores = [&](int t, int slot) {
        tcgen05_fence_after_sync();
        issue_s(t & 1, slot);
        tcgen05_commit_elect(bar_s_full + 2 * s + (t & 1));
      };
      // P is polled (without blocking) one step ahead and waited for only if the poll failed.
      bool p_ready = false;
      auto step = [&](int t, int v_slot, int k_slot) {
        const int u = t & 1;
        if (s == 0) trace_event(prm, 2, t, 0);
        if (!p_ready)
          mbar_wait(bar_p_full + 2 * s + u, (t >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        tcgen05_fence_after_sync();
        if (s == 0) trace_event(prm, 2, t, 1);
        issue_pv(u, v_slot, t > first);
        tcgen05_commit_elect(bar_o_full + s);
        if (t + 1 == end) tcgen05_commit_elect(bar_o_done + s);
        if (s == 0) trace_event(prm, 2, t, 2);
        // step t + 2 goes into the buffer that P(s, t) is being read from; the tensor core runs
        // one thread's instructions in order, so the read comes first
        if (t + 2 < end) {
          issue_s(u, k_slot);
          tcgen05_commit_elect(bar_s_full + 2 * s + u);
        }
        if (s == 0) trace_event(prm, 2, t, 3);
        p_ready = (t + 1 < end) && mbar_test_wait(bar_p_full + 2 * s + (u ^ 1), ((t + 1) >> 1) & 1);
      };
      mbar_wait(bar_q_full, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      struct {
        decltype(wait_kv) wait;
        decltype(kv_ready) ready;
        decltype(release_kv) release;
        decltype(scores) scores;
        decltype(step) step;
      } const ops{wait_kv, kv_ready, release_kv, scores, step};
      const int j0 = s || up ? 0 : n1 - n0;  // first of the ring's key tiles that this query tile reads
      walk_kv_ring<kStages>(j0, j0 + (s ? n1 : n0), n1, first, end, ops);
    } else if (warp == 13) {
      // ================================ TMA producer ================================
      const bool issuer = lane == 0;
      for (int i = first_fill; i < 2 * n1; ++i) {  // the rest of the ring, as slots are released
        const int st = i % kStages;
        mbar_wait(bar_kv_empty + st, ((i / kStages) & 1) ^ 1, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
        if (issuer) load_kv(i);
        __syncwarp();
      }
    }
  }

  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

template <int D, bool kBf16, int kExt>
int launch_ws64r(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& prm,
                cudaStream_t stream) {
  auto kernel = attn_fwd_ws64r_kernel<D, kBf16, kExt>;
  constexpr int smem = Ws64Config<D>::kSmemBytes;
  cudaError_t ea = ensure_dynamic_smem<attn_fwd_ws64r_kernel<D, kBf16, kExt>>(smem, prm.device);
  if (ea != cudaSuccess)
    return fail(FO_ERR_CUDA, "cudaFuncSetAttribute(shared memory %d) failed: %s", smem, cudaGetErrorString(ea));
  const int num_pairs = (prm.num_q_tiles + 1) / 2;
  const int64_t blocks = static_cast<int64_t>(num_pairs) * prm.B * prm.H;
  if (blocks > 0x7fffffffLL) return fail(FO_ERR_INVALID_ARGUMENT, "too many query tiles for one launch");
  kernel<<<static_cast<unsigned>(blocks), 512, smem, stream>>>(tq, tk, tv, prm);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FO_ERR_CUDA, "attention launch failed: %s", cudaGetErrorString(e));
  return FO_OK;
}

}  // namespace fo
