// Attention forward, warp-specialised kernel for sm_100a with 64-key softmax steps.
//
// Same roles, shared-memory ring and tensor-memory budget as the kernel in flash_attn_ws.cuh
// (one CTA = two consecutive 128-row query tiles of one (batch, head); warps 0-3 / 4-7 softmax,
// 8-11 correction and epilogue, 12 and 14 MMA issuers (one per query tile), 13 TMA producer), but
// the 128 score columns that
// a query tile owns in tensor memory are used as TWO buffers of 64 key columns:
// (the kernel in flash_attn_ws.cuh has a single MMA issuer and leaves warps 14-15 idle)
//
//   tensor memory: S0a | S0b | S1a | S1b | O0 | O1      (64 + 64 + 64 + 64 + D + D columns)
//
// A key tile of 128 rows in shared memory is consumed as two steps of 64 keys.  While the
// softmax threads of a query tile work on step t (buffer t & 1), the tensor core already holds
// or is computing S of step t + 1 in the other buffer, so the threads go from one step to the
// next without waiting for an MMA: the chain "P written -> P V -> next Q K^T -> S ready", which
// bounds the 128-column kernel, is off their critical path.  P of a step overwrites the first
// 32 columns of its own buffer and is read by the P V MMA of that step, after which the buffer
// takes the Q K^T of step t + 2.
#pragma once

#include "flash_attn_common.cuh"
#include "flash_attn_ws.cuh"
#include "fo_host.h"

namespace fo {

constexpr int kStepN = 64;  // keys per softmax step


template <int D>
struct Ws64Config : WsConfig<D> {
  // barriers: q_full, kv_full/empty per stage, then s_full[2][2], p_full[2][2], o_full[2],
  // corr[2][2], final[2], o_done[2]
  static constexpr int kNumBars = 1 + 2 * WsConfig<D>::kStages + 4 + 4 + 2 + 4 + 2 + 2;
  static constexpr int kOffMisc = WsConfig<D>::kOffBars + kNumBars * 8;
  static constexpr int kSmemBytes = kOffMisc + 64 + 1024 /* alignment slack */;
};

// kExt: 0 or kFwdDropout (with a bias flash_attn_ws64r.cuh is the kernel).
// kMma: the head_dim the matmuls compute, at most the tiles' width D (the columns between are zeros;
// B1 H48 Sq1000 Sk1531 D80: 57 to 55.7 us with 96 instead of 128 columns computed).
template <int D, bool kBf16, int kExt, int kMma = D>
__global__ void __launch_bounds__(512, 1)
attn_fwd_ws64_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const AttnParams prm) {
  static_assert(kExt == 0 || kExt == kFwdDropout, "a bias runs in attn_fwd_ws64r_kernel");
  using Cfg = Ws64Config<D>;
  constexpr int kTileBytes = Cfg::kTileBytes;
  constexpr int kStages = Cfg::kStages;
  constexpr int kBoxes = Cfg::kBoxes;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sQ = smem + Cfg::kOffQ;    // two tiles
  uint8_t* sKV = smem + Cfg::kOffKV;  // kStages tiles
  float* s_alpha = reinterpret_cast<float*>(smem + Cfg::kOffAlpha);
  float* s_final = reinterpret_cast<float*>(smem + Cfg::kOffFinal);
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
  const int T0 = (vis0 + kStepN - 1) / kStepN;  // T1 >= T0 >= 1
  const int T1 = (vis1 + kStepN - 1) / kStepN;
  const int n1 = (T1 + 1) >> 1;

  if (tid == 0) {
    *cta_abort = 0;
    *skip = *reinterpret_cast<volatile int*>(prm.device_status);
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
    fence_mbar_init();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
  }
  __syncthreads();
  if (*skip) return;  // another CTA already timed out: do nothing

  // The first loads (Q and the first ring fill of K and V) need only the barriers: they go out
  // here, under the tensor-memory allocation, instead of after it.
  const int first_fill = min(kStages, 2 * n1);
  auto load_kv = [&](int i) {  // ring entry i: K_{i/2} (even) or V_{i/2} (odd)
    const int st = i % kStages;
    mbar_arrive_expect_tx(bar_kv_full + st, kTileBytes);
    const CUtensorMap* map = (i & 1) ? &tm_v : &tm_k;
    for (int c = 0; c < kBoxes; ++c)
      tma_load_4d(sKV + st * kTileBytes + c * kBoxBytes, map, bar_kv_full + st, c * kBoxCols,
                  (i >> 1) * kBlockN, hk, b);
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
    reg_alloc<192>();
    const int s = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const int q0 = (2 * pair + s) * kBlockM;
    const int row = q0 + r;
    const int T_s = s ? T1 : T0;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS_tile = tmem_base + Cfg::kColS0 + s * kBlockN + lane_base;
    float* alpha_slot = s_alpha + s * 256 + r;
    float m_run = -INFINITY, l_run = 0.f;
    constexpr bool has_drop = kExt == kFwdDropout;
    uint32_t drop_row = 0;
    if constexpr (has_drop)
      drop_row = prm.ex.drop_base + static_cast<uint32_t>(bh) * static_cast<uint32_t>(prm.Sq) * static_cast<uint32_t>(prm.Sk) +
                 static_cast<uint32_t>(row) * static_cast<uint32_t>(prm.Sk);
    const float exp_scale = prm.scale_log2;

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

    uint32_t sr[2][32];  // scores of the current step

    // Issues the tensor-memory loads of step tn's scores (S must be complete).
    auto issue_load = [&](int tn, int c) {
      const uint32_t tSn = tS_tile + (tn & 1) * kStepN;
      tmem_ld32(tSn + c * 32, sr[c]);
    };
    // Waits for those loads and applies the masks in place.
    auto prep_loads = [&](int tn) {
      const int k0n = tn * kStepN;
      const bool need_mask = (k0n + kStepN > prm.Sk) || (prm.causal && k0n + kStepN - 1 > q0);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        tmem_ld_wait(sr[c]);
        if ((warp & 3) == 0 && tn > 0) trace_event(prm, s, tn - 1, c == 0 ? 1 : 4);  // loads in
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

    // prologue: scores of step 0; their row maximum is the first reference maximum
    mbar_wait(bar_s_full + 2 * s, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_MMA);
    tcgen05_fence_after_sync();
    issue_load(0, 0);
    issue_load(0, 1);
    prep_loads(0);
    m_run = row_max() * exp_scale;

    // The exponentials of a step do not wait for the step's own row maximum: they are taken
    // against the reference maximum the row already has (lazy rescaling moves it only when the
    // true maximum exceeds it by kRescaleThreshold), and the maximum is reduced alongside them,
    // its instructions filling issue slots that the ex2 unit's rate leaves empty.  Only if a row
    // of the warp turns out to need a new reference (rare after the first steps) are the step's
    // exponentials taken again.  Each iteration then fetches step t + 1 (whose S the tensor core
    // finished meanwhile) behind the P stores, so that the latencies of the loads, of the P store
    // and of the barriers overlap instead of adding up.
    for (int t = 0; t < T_s; ++t) {
      const int u = t & 1;
      const int k0 = t * kStepN;
      const uint32_t tS = tS_tile + u * kStepN;
      float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
      if (ping_pong) named_barrier_sync_dep(s ? kTurn1 : kTurn0, kTurnCount, neg_m);  // exponentials start after this
      if ((warp & 3) == 0) trace_event(prm, s, t, 0);  // turn taken
      const float2 sc2 = make_float2(exp_scale, exp_scale);
      float2 acc0, acc1;
      uint32_t pr[2][16];
      const bool more = t + 1 < T_s;
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
              const uint32_t idx = drop_row + static_cast<uint32_t>(k0 + c * 32 + 2 * q);
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
    s_final[s * 256 + r] = l_run;
    s_final[s * 256 + 128 + r] = m_run;
    mbar_arrive(bar_final + s);
    // Keep taking and passing the turn for the steps that only the other tile still has, one at
    // a time (arrivals sent ahead of the other tile's waits would complete a barrier phase on
    // their own and strand it).  Tile 1's very last arrival finds nobody waiting: the CTA ends
    // with that barrier half counted, which is harmless.
    if (ping_pong && s == 0)
      for (int t = T0; t < T1; ++t) {
        named_barrier_sync(kTurn0, kTurnCount);
        named_barrier_arrive(kTurn1, kTurnCount);
      }
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
      const float o_scale = (kExt != 0) ? prm.ex.drop_rescale : 1.f;
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
    for (int t = 0; t < T1; ++t) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (t >= (s ? T1 : T0)) continue;
        mbar_wait(bar_corr + 2 * s + (t & 1), (t >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
        const float alpha = s_alpha[s * 256 + (t & 1) * 128 + r];
        if (t > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
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
      // With a causal mask tile 0 has two steps fewer than tile 1: its epilogue runs here, between
      // two arrivals for tile 1, instead of at the CTA's tail.
      if (t == T0 && T0 < T1) epilogue(0);
    }
    if (T0 == T1) epilogue(0);
    epilogue(1);
  } else {
    reg_dealloc<48>();
    if (warp == 12 || warp == 14) {
      // ================================ MMA issuers ================================
      // One warp per query tile (12: tile 0, 14: tile 1).  The tensor core's instruction queue
      // is short: whenever the issuing warp is not issuing (a barrier wait costs it about 200
      // cycles even on a completed phase) the pipe runs dry.  With two issuers one tile's waits
      // hide behind the other tile's instructions.  Nothing orders the two streams against each
      // other, and nothing has to: each tile owns its S / P buffers and its O accumulator, and a
      // K/V ring slot is released by both warps (bar_kv_empty counts two arrivals).
      const int s = (warp == 14) ? 1 : 0;
      const int T_s = s ? T1 : T0;
      constexpr uint32_t idesc_qk = make_idesc(kBf16, kBlockM, kStepN, 0, 0);
      constexpr uint32_t idesc_pv = make_idesc(kBf16, kBlockM, kMma, 0, 1);
      // Everything below is warp-uniform; only the tcgen05 instructions themselves are issued by
      // one elected lane.  Descriptors are kept as 32-bit low halves: per instruction one add.
      const uint32_t q_lo = desc_lo(smem_u32(sQ) + s * kTileBytes, 16);
      const uint32_t kv_k_lo = desc_lo(smem_u32(sKV), 16);         // K tiles: K-major
      const uint32_t kv_v_lo = desc_lo(smem_u32(sKV), kBoxBytes);  // V tiles: N-major
      constexpr uint32_t kStageStep = kTileBytes >> 4;
      constexpr uint32_t kBoxStep = kBoxBytes >> 4;
      const uint32_t tS_tile = tmem_base + Cfg::kColS0 + s * kBlockN;
      const uint32_t tO = tmem_base + Cfg::kColO0 + s * D;
      // S(s, t) = Q_s K^T over keys [64 u, 64 u + 64) of the K tile in ring slot `stage`, u = t & 1:
      // 64 rows of a K-major box are 64 * 128 bytes further on
      auto issue_s = [&](int u, int stage) {
        const uint32_t b_lo = kv_k_lo + stage * kStageStep + u * ((kStepN * 128) >> 4);
        const uint32_t tS = tS_tile + u * kStepN;
#pragma unroll
        for (int kk = 0; kk < kMma / 16; ++kk) {
          // k-slice kk: box kk/4, 32 bytes per slice inside the 128-byte swizzle span
          const uint32_t off = (kk >> 2) * kBoxStep + (kk & 3) * 2;
          umma_ss_lo_elect(tS, q_lo + off, b_lo + off, idesc_qk, kk > 0 ? 1u : 0u);
        }
      };
      // O_s (+)= P(s, t) V over key rows [64 u, 64 u + 64) of the V tile in ring slot `stage`
      auto issue_pv = [&](int u, int stage, bool acc) {
        const uint32_t tP = tS_tile + u * kStepN;
        const uint32_t b_lo = kv_v_lo + stage * kStageStep + u * (kStepN / 16) * 128;
#pragma unroll
        for (int kk = 0; kk < kStepN / 16; ++kk) {
          // 16 key rows per slice: 2048 bytes of V, 8 packed columns of P
          umma_ts_lo_elect(tO, tP + kk * 8, b_lo + kk * 128, idesc_pv, (acc || kk > 0) ? 1u : 0u);
        }
      };

      mbar_wait(bar_q_full, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
      mbar_wait(bar_kv_full + 0, 0, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);  // K_0 is ring slot 0
      tcgen05_fence_after_sync();
      // prologue: the first two steps, both on K_0
      issue_s(0, 0);
      tcgen05_commit_elect(bar_s_full + 2 * s);
      if (T_s > 1) {
        issue_s(1, 0);
        tcgen05_commit_elect(bar_s_full + 2 * s + 1);
      }
      tcgen05_commit_elect(bar_kv_empty + 0);
      // Barriers are polled (without blocking) one iteration ahead and waited on only if the
      // poll failed.
      bool p_ready = false, kv_ready = false;
      for (int t = 0; t < T1; ++t) {  // both warps walk all key tiles: the ring needs both
        const int j = t >> 1, u = t & 1;
        const int iv = 2 * j + 1;  // ring index of V_j; K_{j+1} is iv + 1
        const int st_v = iv % kStages;
        const int st_k = (iv + 1) % kStages;
        const bool k_next = j + 1 < n1;  // K_{j+1} exists
        if (u == 0 && !kv_ready) {
          mbar_wait(bar_kv_full + st_v, (iv / kStages) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
          if (k_next) mbar_wait(bar_kv_full + st_k, ((iv + 1) / kStages) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_TMA);
        }
        if (s == 0) trace_event(prm, 2, t, 0);
        kv_ready = false;
        if (t < T_s) {
          if (!p_ready)
            mbar_wait(bar_p_full + 2 * s + u, (t >> 1) & 1, cta_abort, dstat, FO_STATUS_TIMEOUT_SOFTMAX);
          tcgen05_fence_after_sync();
          if (s == 0) trace_event(prm, 2, t, 1);
          issue_pv(u, st_v, t > 0);
          tcgen05_commit_elect(bar_o_full + s);
          if (t + 1 == T_s) tcgen05_commit_elect(bar_o_done + s);
          if (s == 0) trace_event(prm, 2, t, 2);
          // step t + 2 goes into the buffer that P(s, t) is being read from; the tensor core runs
          // one thread's instructions in order, so the read comes first
          if (t + 2 < T_s) {
            issue_s(u, st_k);
            tcgen05_commit_elect(bar_s_full + 2 * s + u);
          }
          if (s == 0) trace_event(prm, 2, t, 3);
          p_ready = (t + 1 < T_s) && mbar_test_wait(bar_p_full + 2 * s + (u ^ 1), ((t + 1) >> 1) & 1);
        }
        if (u == 1 || t + 1 == T1) {
          // this warp's readers of V_j (and of K_{j+1}) have all been issued
          tcgen05_commit_elect(bar_kv_empty + st_v);
          if (k_next) tcgen05_commit_elect(bar_kv_empty + st_k);
          if (t + 1 < T1) {
            const int iv2 = iv + 2;
            kv_ready = mbar_test_wait(bar_kv_full + iv2 % kStages, (iv2 / kStages) & 1) &&
                       (!(j + 2 < n1) || mbar_test_wait(bar_kv_full + (iv2 + 1) % kStages, ((iv2 + 1) / kStages) & 1));
          }
        }
      }
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

template <int D, bool kBf16, int kExt, int kMma = D>
int launch_ws64(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& prm,
                cudaStream_t stream) {
  auto kernel = attn_fwd_ws64_kernel<D, kBf16, kExt, kMma>;
  constexpr int smem = Ws64Config<D>::kSmemBytes;
  cudaError_t ea = ensure_dynamic_smem<attn_fwd_ws64_kernel<D, kBf16, kExt, kMma>>(smem, prm.device);
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
