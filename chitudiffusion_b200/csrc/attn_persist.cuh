// Attention forward of a plain call (local tensors, no exchange): attn_fwd_kernel's query blocks and softmax, as
// a persistent kernel.
//
// A CTA works on one query block (256 rows of a head) after the other.  What attn_fwd_kernel does once per
// CTA with the tensor pipe idle - launch, barrier and tensor-memory set-up, fetching Q and the first key
// tile, the epilogue's stores - costs about five key-tile steps there (216 CTAs x 36 tiles 138 us, 432 CTAs x 18
// tiles 143 us).  Here the set-up is paid once per SM and the rest overlaps: while the softmax warps write
// out one query block, the next one's Q, K and V are on their way and its first scores are being computed.
//
// Work units.  Unit u of the grid is a run of key-tile steps in the flattened order (query block, key tile):
//   u < n_whole   one whole query block,
//   otherwise     with b = u - n_whole, steps [b * bundle_steps, (b + 1) * bundle_steps) of the first cut_items query blocks.
// Query blocks that do not fill the last wave of the machine are cut into equal bundles, at most one per SM, so that
// all SMs finish together.  The bundles come last: a CTA asks for its next unit while it works on one, so whole blocks
// behind bundles would go to CTAs that have a whole block in hand as often as to those that took a bundle.  A bundle touches at most two query blocks and leaves a fragment of each in scratch
// memory, and the warp that completes the last fragment of its 32 rows merges them (nobody waits).
//
// Units are handed out by the hardware: the grid has one CTA per unit, and a running CTA takes over units that
// have not started yet (clusterlaunchcontrol), one ahead of what it is working on.  So there is no counter
// in memory to reset, and an SM that another kernel holds (a collective on a side stream) simply takes none.
//
// Tensor memory (512 columns): S | P0 | P1 | O0 | O1 with ONE set of 128 score columns for both query tiles, and
// probabilities of their own (64 columns each) instead of over their scores.  A tile's scores leave for registers
// in some 150 cycles, so the next QK^T - the other tile's - starts there while the exponentials are formed, and no
// tile waits for PV and QK^T of its own between two steps (in attn_fwd_kernel 1030 of every 2850 cycles).
//
// Warps: 0-3 / 4-7 softmax of tile 0 / 1, 8 issues QK^T of both tiles in turn, 9 TMA, 10 / 11 issue PV of tile
// 0 / 1.  With one issuing thread (its six waits per step each let the tensor pipe run dry) the same layout took
// 218 us at S = 4608, H = 24, with three 195; S and P of a tile overlaid, as in attn_fwd_kernel, 201.
//
// Between two query blocks of a CTA:
//   * Q_t is free once the last QK^T of tile t has run;
//   * O_t is overwritten by the next block's first PV, which waits for probabilities that the same
//     softmax warps form after their epilogue has read O_t.
#pragma once

#include "attn_fwd.cuh"

namespace chitu {

constexpr int kPersistStages = 4;     // K/V ring slots
constexpr int kClcStages = 4;         // answers of the work distributor
constexpr int kStoreBytes = 8 * 4096; // epilogue staging: 32 rows x 64 columns per softmax warp
constexpr int kPersistSmemBytes = (kQTiles + kPersistStages) * kTileBytes + kStoreBytes + 512 + 1024;

// Division of a 31-bit dividend by a number fixed per launch: q = x * mul >> (32 + shift), exact because
// mul = ceil(2^(32 + shift) / d) with 2^shift < d <= 2^(shift + 1) is off by less than 2^(shift + 1) in its product with d
// (Granlund and Montgomery, "Division by invariant integers using multiplication", 1994).  A division by an unknown
// costs a few hundred cycles of a warp's time, and a unit's decoding takes four.
struct FastDiv {
  uint32_t d, mul, shift;
  void set(int divisor) {
    d = static_cast<uint32_t>(divisor);
    shift = 0;
    while ((2u << shift) < d) ++shift;
    mul = d == 1 ? 0u : static_cast<uint32_t>(((1ull << (32 + shift)) + d - 1) / d);
  }
  __device__ __forceinline__ int div(int x) const {
    return mul == 0 ? x : static_cast<int>(__umulhi(static_cast<uint32_t>(x), mul) >> shift);
  }
};

struct AttnPersistParams {
  float* lse;  // [B, H, Sq] fp32 natural-log, or nullptr
  int* status;
  int B, H, Sq, Sk;
  float scale_log2;
  int n_kv;          // key tiles
  int n_qblocks;     // query blocks per head; item = (head * B + batch) * n_qblocks + block, so that CTAs which run
                     // together share heads' keys in L2
  int n_whole;       // units that are whole query blocks; the others are the
  int n_bundles;     // bundles into which the first cut_items query blocks are cut, of
  int bundle_steps;  // key-tile steps each (< n_kv)
  int cut_items;
  FastDiv by_n_kv, by_n_qblocks, by_batch, by_bundle_steps;
  // scratch (cut_items > 0): counters [cut_items][2 tiles][4 warps], zero between calls; a fragment's normalised fp32 rows
  // [bundle * 2 + k][2 tiles][32 chunks][128 rows] float4 (k = 0, 1: the bundle's first / second query block) and
  // their natural log-sum-exps [bundle * 2 + k][2 tiles][128 rows]
  int* count;
  float* part_o;
  float* part_lse;
};

// Ask for a unit that has not started (16-byte answer, completes 16 transaction bytes on bar).
__device__ __forceinline__ void clc_try_cancel(uint32_t answer, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer),
               "r"(bar)
               : "memory");
}
// The unit's index, or -1 when there is none left.
__device__ __forceinline__ int clc_unit(uint32_t answer) {
  uint32_t ok, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
      : "=r"(ok), "=r"(x)
      : "r"(answer)
      : "memory");
  return ok ? static_cast<int>(x) : -1;
}

// Position in the K/V ring.
struct Ring {
  int slot = 0, phase = 0;
  __device__ __forceinline__ void advance() {
    if (++slot == kPersistStages) {
      slot = 0;
      phase ^= 1;
    }
  }
};

// Where a softmax warp's query tile lives: tensor-memory addresses (this warp's lanes) and barriers.
struct TileRefs {
  uint32_t t_s, t_p, t_o;  // scores (both tiles share them), this tile's probabilities and accumulator
  uint32_t bar_s_empty;    // the scores are in registers (one arrival per warp)
  uint32_t bar_p;          // [2] keys [0, 64) and [64, 128) of the probabilities are stored (every thread arrives)
  uint32_t bar_pv;         // a step's PV is complete (phase = step)
};

// One softmax step of a query tile's four warps (thread = one row, 128 scores): scores in, probabilities out.
// `step` counts the tile's steps since the launch, `first` says that there is no accumulator yet, `valid` how many keys
// of the tile exist (kTileN: all).
//
// The scores go to registers at once and their tensor memory is given back before anything else, because the
// other tile's scores are computed into the same columns meanwhile.  Every exponential takes the MUFU unit: 128 of them
// are 1024 of its cycles, two warps' worth what the tensor pipe needs for a step of both tiles, and now that no
// chain holds the warps up the polynomial of attn_fwd_kernel only costs issue slots (of every 8 pairs 2 / 1 / 0
// polynomial: 203 / 195 / 195 us at S = 4608, H = 24, 4768 / 4678 / 4665 us at S = 32760, H = 12).
template <bool kFp16>
__device__ __forceinline__ void persist_softmax_step(const TileRefs& r, int step, bool first, int valid, float sl2,
                                                     float& m_used, float& l_sum, volatile int* abort_flag, int* status) {
  uint32_t s[4][32];
  float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld32(r.t_s + c * 32, s[c]);
  tmem_wait_ld();
  tc_fence_before_sync();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(r.bar_s_empty);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (valid < kTileN) {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (c * 32 + i >= valid) s[c][i] = 0xff800000u;  // -inf
    }
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      mx0 = max3(mx0, __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
      mx1 = max3(mx1, __uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3]));
    }
  }
  const float mx = fmaxf(mx0, mx1);

  if (first) {
    m_used = mx;
  } else {
    const bool need = (mx - m_used) * sl2 > kRescaleThreshold;
    if (__any_sync(0xffffffffu, need)) {
      mbar_wait(r.bar_pv, (step - 1) & 1, abort_flag, status, kDevTimeoutSoftmax);
      tc_fence_after_sync();
      const float f = need ? fast_exp2((m_used - mx) * sl2) : 1.0f;
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        uint32_t o[16];
        tmem_ld16(r.t_o + c * 16, o);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
        tmem_st16(r.t_o + c * 16, o);
      }
      l_sum *= f;
      if (need) m_used = mx;
    }
  }

  // (looked at early, so that the answer is there when the first probabilities are stored)
  const bool pv_done = step == 0 || mbar_try_wait(r.bar_pv, (step - 1) & 1);

  // p = 2^(s*scale - m*scale): packed two-wide FMA / add, one MUFU per element
  const float2 sl2_2 = make_float2(sl2, sl2);
  // (a row without a finite score so far has nothing to subtract: its probabilities are zero, not NaN)
  const float neg_m = m_used == -INFINITY ? 0.f : -m_used * sl2;
  const float2 neg_m2 = make_float2(neg_m, neg_m);
  uint32_t pk[2][32];
  float2 la = make_float2(0.f, 0.f), lb = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      float2 x0 = __ffma2_rn(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), sl2_2, neg_m2);
      float2 x1 =
          __ffma2_rn(make_float2(__uint_as_float(s[c][i + 2]), __uint_as_float(s[c][i + 3])), sl2_2, neg_m2);
      x0.x = fast_exp2(x0.x);
      x0.y = fast_exp2(x0.y);
      x1.x = fast_exp2(x1.x);
      x1.y = fast_exp2(x1.y);
      la = __fadd2_rn(la, x0);
      lb = __fadd2_rn(lb, x1);
      pk[c >> 1][(c & 1) * 16 + (i >> 1)] = pack2<kFp16>(x0.x, x0.y);
      pk[c >> 1][(c & 1) * 16 + (i >> 1) + 1] = pack2<kFp16>(x1.x, x1.y);
      if ((c & 1) == 1 && i == 28) {
        // 64 probabilities done: hand this half to the MMA warp
        if (c == 1) {
          if (!pv_done) mbar_wait(r.bar_pv, (step - 1) & 1, abort_flag, status, kDevTimeoutSoftmax);
          __syncwarp();  // (lanes may have found out on their own; the store below is the warp's)
          tc_fence_after_sync();
        }
        tmem_st32(r.t_p + (c >> 1) * 32, pk[c >> 1]);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(r.bar_p + 8 * (c >> 1));
      }
    }
  l_sum += (la.x + la.y) + (lb.x + lb.y);
}

// The steps of a unit, one run of one query block's key tiles at a time.
struct UnitWalk {
  int pos, end;
  __device__ __forceinline__ UnitWalk(const AttnPersistParams& p, int unit) {
    if (unit < p.n_whole) {
      pos = (p.cut_items + unit) * p.n_kv;
      end = pos + p.n_kv;
    } else {
      pos = (unit - p.n_whole) * p.bundle_steps;
      end = min(pos + p.bundle_steps, p.cut_items * p.n_kv);
    }
  }
  __device__ __forceinline__ bool next(const AttnPersistParams& p, int& item, int& kv0, int& n) {
    if (pos >= end) return false;
    item = p.by_n_kv.div(pos);
    kv0 = pos - item * p.n_kv;
    n = min(p.n_kv - kv0, end - pos);
    pos += n;
    return true;
  }
};

template <bool kFp16>
__global__ void __launch_bounds__(kAttnThreads, 1)
attn_persist_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_out,
                    const AttnPersistParams p) {
  constexpr int kSt = kPersistStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t q_smem = smem_base;                          // 2 tiles
  const uint32_t kv_smem = smem_base + kQTiles * kTileBytes;  // kSt tiles
  uint8_t* store_smem = smem_gen + (kQTiles + kSt) * kTileBytes;
  uint8_t* ctl_gen = store_smem + kStoreBytes;
  const uint32_t ctl = smem_u32(ctl_gen);
  const uint32_t clc_answer = ctl;                         // [kClcStages] x 16 bytes
  const uint32_t bar_clc_full = ctl + 16 * kClcStages;     // [kClcStages]
  const uint32_t bar_clc_empty = bar_clc_full + 8 * kClcStages;
  const uint32_t bar_q_full = bar_clc_empty + 8 * kClcStages;  // [2]
  const uint32_t bar_q_empty = bar_q_full + 16;                // [2]
  const uint32_t bar_kv_full = bar_q_empty + 16;               // [kSt]
  const uint32_t bar_kv_empty = bar_kv_full + 8 * kSt;         // [kSt]
  const uint32_t bar_s_full = bar_kv_empty + 8 * kSt;          // [2]
  const uint32_t bar_p_full = bar_s_full + 16;                 // [2][2]
  const uint32_t bar_pv = bar_p_full + 32;                     // [2]
  const uint32_t bar_s_empty = bar_pv + 16;
  const uint32_t bar_drain = bar_s_empty + 8;                  // [3]
  uint8_t* tail = ctl_gen + (16 + 8 + 8) * kClcStages + 32 + 16 * kSt + 16 + 32 + 16 + 8 + 24;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kClcStages; ++s) {
      mbar_init(bar_clc_full + 8 * s, 1);
      mbar_init(bar_clc_empty + 8 * s, 11);  // the three MMA warps and the eight softmax warps
    }
    for (int s = 0; s < kSt; ++s) {
      mbar_init(bar_kv_full + 8 * s, 1);
      mbar_init(bar_kv_empty + 8 * s, 1 + (s & 1));  // keys (even slots): one reader; values (odd slots): two
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(bar_q_full + 8 * t, 1);
      mbar_init(bar_q_empty + 8 * t, 1);
      mbar_init(bar_s_full + 8 * t, 1);
      mbar_init(bar_p_full + 16 * t, kTileM);
      mbar_init(bar_p_full + 16 * t + 8, kTileM);
      mbar_init(bar_pv + 8 * t, 1);
    }
    mbar_init(bar_s_empty, 4);
    for (int i = 0; i < 3; ++i) mbar_init(bar_drain + 8 * i, 1);
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  if (warp == 9 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_out);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // (query block, head, batch, query tiles) of an item
  struct Item {
    int q0, head, batch, n_qt;
  };
  auto decode = [&](int item) {
    Item it;
    const int bh = p.by_n_qblocks.div(item);
    it.q0 = (item - bh * p.n_qblocks) * (kQTiles * kTileM);
    it.head = p.by_batch.div(bh);
    it.batch = bh - it.head * p.B;
    it.n_qt = it.q0 + kTileM < p.Sq ? 2 : 1;
    return it;
  };
  // The unit after the n-th: every reader of the answer releases its slot (the reads are ordered before the
  // distributor's next write into it, which goes through the async proxy).
  auto next_unit = [&](int n, int code) {
    const int st = n & (kClcStages - 1);
    // (lanes poll on their own and may see a wait given up at different times: the warp decides as one)
    if (!__all_sync(0xffffffffu, mbar_wait(bar_clc_full + 8 * st, (n / kClcStages) & 1, abort_flag, p.status, code))) return -1;
    const int u = clc_unit(clc_answer + 16 * st);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_clc_empty + 8 * st);
    return u;
  };

  // A role has timed out.  Warps look on their own and may part here - one goes home, another takes up the next unit -
  // so nothing between here and the CTA's last barrier may wait for another warp other than by a bounded mbarrier wait.
  auto gave_up = [&] { return __any_sync(0xffffffffu, *abort_flag) != 0; };

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 9) {
      // ---------------------------------------------------------------- TMA producer; asks for the next unit
      int n_units = 0;
      Ring ring;
      int q_loads[2] = {0, 0};     // fills of each Q tile so far
      int unit = blockIdx.x;
      while (unit >= 0) {
        const int st = n_units & (kClcStages - 1);
        if (n_units >= kClcStages)
          mbar_wait(bar_clc_empty + 8 * st, (n_units / kClcStages - 1) & 1, abort_flag, p.status, kDevTimeoutLoad);
        if (lane == 0) {
          mbar_arrive_expect_tx(bar_clc_full + 8 * st, 16);
          clc_try_cancel(clc_answer + 16 * st, bar_clc_full + 8 * st);
        }
        __syncwarp();
        UnitWalk walk(p, unit);
        int item, kv0, n;
        while (walk.next(p, item, kv0, n)) {
          const Item w = decode(item);
          for (int i = 0; i < 2 * n; ++i, ring.advance()) {  // K_0, (Q,) V_0, K_1, V_1, ...
            const int slot = ring.slot;
            // (a fresh barrier counts as having completed the phase before its first: the first round does not wait)
            mbar_wait(bar_kv_empty + 8 * slot, ring.phase ^ 1, abort_flag, p.status, kDevTimeoutLoad);
            if (lane == 0) {
              const CUtensorMap* tm = (i & 1) ? &tm_v : &tm_k;
              const int row = (kv0 + (i >> 1)) * kTileN;
              const uint32_t dst = kv_smem + slot * kTileBytes;
              const uint32_t bar = bar_kv_full + 8 * slot;
              mbar_arrive_expect_tx(bar, kTileBytes);
              tma_load_4d(dst, tm, bar, 0, w.head, row, w.batch);
              tma_load_4d(dst + kHalfTileBytes, tm, bar, 64, w.head, row, w.batch);
            }
            __syncwarp();
            if (i == 0) {
              for (int t = 0; t < w.n_qt; ++t) {
                if (q_loads[t] > 0)
                  mbar_wait(bar_q_empty + 8 * t, (q_loads[t] - 1) & 1, abort_flag, p.status, kDevTimeoutLoad);
                if (lane == 0) {
                  const uint32_t dst = q_smem + t * kTileBytes;
                  mbar_arrive_expect_tx(bar_q_full + 8 * t, kTileBytes);
                  tma_load_4d(dst, &tm_q, bar_q_full + 8 * t, 0, w.head, w.q0 + t * kTileM, w.batch);
                  tma_load_4d(dst + kHalfTileBytes, &tm_q, bar_q_full + 8 * t, 64, w.head, w.q0 + t * kTileM, w.batch);
                }
                ++q_loads[t];
                __syncwarp();
              }
            }
          }
        }
        // the answer (this warp is the next to write the slot, so it needs no release)
        if (__all_sync(0xffffffffu, mbar_wait(bar_clc_full + 8 * st, (n_units / kClcStages) & 1, abort_flag, p.status, kDevTimeoutLoad))) {
          unit = clc_unit(clc_answer + 16 * st);
          fence_proxy_async_smem();
        } else {
          unit = -1;
        }
        if (gave_up()) unit = -1;
        ++n_units;
      }
      if (lane == 0) {
        // Should a role give up - even after this point - nothing of ours may still be landing in this CTA's shared
        // memory when the CTA retires (bounded polls): the last answer, the Q tiles, the last copy into every K/V slot.
        // (Where nobody gives up, the readers wait for the same copies.)
        const int last = n_units - 1;
        for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar_clc_full + 8 * (last & (kClcStages - 1)), (last / kClcStages) & 1); ++spin) {
        }
        for (int t = 0; t < 2; ++t)
          for (int spin = 0; q_loads[t] > 0 && spin < (1 << 20) && !mbar_try_wait(bar_q_full + 8 * t, (q_loads[t] - 1) & 1); ++spin) {
          }
        // (a slot that was never filled counts as complete in its phase before the first)
        for (int i = 0; i < kSt; ++i)
          for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar_kv_full + 8 * i, i < ring.slot ? ring.phase : ring.phase ^ 1); ++spin) {
          }
      }
    } else {
      // ---------------------------------------------------------------- MMA issuers
      // Warp 8 issues every QK^T, warps 10 and 11 the PV of tile 0 and 1.  An issuing thread is held up while the
      // tensor pipe works off what it has issued, and a wait costs it some 100 cycles even when there is nothing to
      // wait for: with one thread for all three kinds the pipe ran dry at each of its six waits per step.
      const bool leader = elect_one();
      const int role = warp == 8 ? 0 : warp - 9;  // 0 scores; 1, 2 PV of tile 0, 1
      int n_units = 0;
      Ring ring;  // the next K (scores) or V item to consume
      if (role > 0) ring.advance();
      auto wait_item = [&] {
        mbar_wait(bar_kv_full + 8 * ring.slot, ring.phase, abort_flag, p.status, kDevTimeoutMma);
      };
      int unit = blockIdx.x;
      if (role == 0) {
        constexpr uint32_t kIdescQK = umma_idesc(1, kFp16 ? 0 : 1, kFp16 ? 0 : 1, 0, kTileM, kTileN);
        const uint64_t q_desc0 = umma_smem_desc_sw128(q_smem, 16, 1024);
        const uint64_t k_desc0 = umma_smem_desc_sw128(kv_smem, 16, 1024);
        int q_uses[2] = {0, 0};  // Q tiles consumed so far
        int scores = 0;          // QK^T so far
        while (unit >= 0) {
          UnitWalk walk(p, unit);
          int item, kv0, n;
          while (walk.next(p, item, kv0, n)) {
            const int n_qt = decode(item).n_qt;
            for (int j = 0; j < n; ++j) {
              wait_item();
              for (int t = 0; t < n_qt; ++t) {
                if (j == 0) {
                  mbar_wait(bar_q_full + 8 * t, q_uses[t] & 1, abort_flag, p.status, kDevTimeoutMma);
                  ++q_uses[t];
                }
                // the columns of the scores are free once the softmax warps have the previous ones in registers
                if (scores > 0) mbar_wait(bar_s_empty, (scores - 1) & 1, abort_flag, p.status, kDevTimeoutMma);
                ++scores;
                tc_fence_after_sync();
                if (leader) {
                  // S = Q_t K^T : both operands K-major, 8 steps of 16 along head_dim
                  const uint64_t a0 = q_desc0 + static_cast<uint64_t>((t * kTileBytes) >> 4);
                  const uint64_t b0 = k_desc0 + static_cast<uint64_t>((ring.slot * kTileBytes) >> 4);
#pragma unroll
                  for (int k = 0; k < kHeadDim / 16; ++k) {
                    const uint64_t off = static_cast<uint64_t>(((k >> 2) * kHalfTileBytes + (k & 3) * 32) >> 4);
                    umma_ss_f16(tmem_base, a0 + off, b0 + off, kIdescQK, k > 0);
                  }
                  umma_commit(bar_s_full + 8 * t);
                  if (j + 1 == n) umma_commit(bar_q_empty + 8 * t);
                }
                __syncwarp();
              }
              if (leader) umma_commit(bar_kv_empty + 8 * ring.slot);
              __syncwarp();
              ring.advance();
              ring.advance();
            }
          }
          unit = next_unit(n_units++, kDevTimeoutMma);
          if (gave_up()) unit = -1;
        }
      } else {
        constexpr uint32_t kIdescPV = umma_idesc(1, kFp16 ? 0 : 1, kFp16 ? 0 : 1, 1, kTileM, kHeadDim);
        const int t = role - 1;
        const uint64_t v_desc0 = umma_smem_desc_sw128(kv_smem, kHalfTileBytes, 1024);
        const uint32_t t_p = tmem_base + kTileN + t * 64;
        const uint32_t t_o = tmem_base + 2 * kTileN + t * kHeadDim;
        int steps = 0;  // the tile's steps so far
        while (unit >= 0) {
          UnitWalk walk(p, unit);
          int item, kv0, n;
          while (walk.next(p, item, kv0, n)) {
            const int n_qt = decode(item).n_qt;
            for (int j = 0; j < n; ++j) {
              wait_item();
              if (t < n_qt) {
                // the PV MMAs of the first 64 keys start while the softmax warps still work on the rest
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  mbar_wait(bar_p_full + 16 * t + 8 * h, steps & 1, abort_flag, p.status, kDevTimeoutMma);
                  tc_fence_after_sync();
                  if (leader) {
                    // O_t += P_t[:, 64h .. 64h+64) V[64h .. 64h+64) : A = P from tensor memory (two 16-bit values
                    // per column), B = V tile as loaded ([key][d], d contiguous => MN-major), 4 steps of 16 keys
                    const uint64_t b0 = v_desc0 + static_cast<uint64_t>((ring.slot * kTileBytes + h * 8192) >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                      umma_ts_f16(t_o, t_p + h * 32 + k * 8, b0 + static_cast<uint64_t>((k * 2048) >> 4), kIdescPV,
                                  (h > 0 || k > 0 || j > 0) ? 1u : 0u);
                    if (h == 1) umma_commit(bar_pv + 8 * t);
                  }
                  __syncwarp();
                }
                ++steps;
              }
              if (leader) umma_commit(bar_kv_empty + 8 * ring.slot);
              __syncwarp();
              ring.advance();
              ring.advance();
            }
          }
          unit = next_unit(n_units++, kDevTimeoutMma);
          if (gave_up()) unit = -1;
        }
      }
      // One more commit and a bounded poll on it: every arrival of this warp's commits has landed, and nothing
      // writes tensor memory after it has been freed below.
      if (leader) umma_commit(bar_drain + 8 * role);
      __syncwarp();
      for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar_drain + 8 * role, 0); ++spin) {
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int t = warp >> 2;
    const int quad = warp & 3;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_o = tmem_base + lane_base + 2 * kTileN + t * kHeadDim;
    const TileRefs refs{tmem_base + lane_base, tmem_base + lane_base + kTileN + t * 64, t_o, bar_s_empty, bar_p_full + 16 * t,
                        bar_pv + 8 * t};
    uint8_t* stage = store_smem + warp * 4096;
    const float sl2 = p.scale_log2;
    const int tail_valid = p.Sk - (p.n_kv - 1) * kTileN;  // 1..128 valid keys in the last tile of K
    int n_units = 0;
    int steps = 0;  // this tile's steps so far
    constexpr int kNotAsked = -2;
    int unit = blockIdx.x;
    while (unit >= 0) {
      int following = kNotAsked;
      UnitWalk walk(p, unit);
      int item, kv0, n;
      while (walk.next(p, item, kv0, n)) {
        const Item w = decode(item);
        if (t >= w.n_qt) continue;
        float m_used = -INFINITY;
        float l_sum = 0.f;
        for (int j = 0; j < n; ++j, ++steps) {
          mbar_wait(bar_s_full + 8 * t, steps & 1, abort_flag, p.status, kDevTimeoutSoftmax);
          tc_fence_after_sync();
          persist_softmax_step<kFp16>(refs, steps, j == 0, kv0 + j == p.n_kv - 1 ? tail_valid : kTileN, sl2, m_used, l_sum,
                                     abort_flag, p.status);
        }
        // (the proxy fence behind a read answer is cheap here; with the epilogue's stores in flight it took 900 cycles)
        if (walk.pos >= walk.end) following = next_unit(n_units++, kDevTimeoutSoftmax);
        mbar_wait(bar_pv + 8 * t, (steps - 1) & 1, abort_flag, p.status, kDevTimeoutEpilogue);
        tc_fence_after_sync();
        const bool whole = n == p.n_kv;
        // no finite score at all: undefined over a whole row, no weight in a merge
        const bool empty = m_used == -INFINITY;
        if (whole && empty) l_sum = __int_as_float(0x7fffffff);
        float lse_row = 0.f;
        if (!whole || p.lse != nullptr) lse_row = (m_used * sl2 + log2f(l_sum)) * 0.6931471805599453f;
        bool write_out = true;
        const float4* parts = nullptr;  // merging: the item's first fragment of this tile, this row
        const float* lses = nullptr;
        int n_parts = 0, part0 = 0;
        float mx = 0.f, inv_w = 0.f;
        auto slot_of = [&](int bundle) {  // scratch slot of a bundle's fragment of this item
          return (bundle * 2 + item - p.by_n_kv.div(bundle * p.bundle_steps)) * 2 + t;
        };
        if (!whole) {
          // this fragment's normalised rows and log-sum-exps go to scratch memory
          const int first = p.by_bundle_steps.div(item * p.n_kv);
          const int last = min(p.by_bundle_steps.div((item + 1) * p.n_kv - 1), p.n_bundles - 1);
          const float inv_l = empty ? 0.f : 1.0f / l_sum;
          const size_t slot = slot_of(p.by_bundle_steps.div(item * p.n_kv + kv0));
          float4* mine = reinterpret_cast<float4*>(p.part_o) + slot * (32 * kTileM) + row_in_tile;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld32(t_o + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              mine[(c * 8 + (i >> 2)) * kTileM] =
                  make_float4(__uint_as_float(o[i]) * inv_l, __uint_as_float(o[i + 1]) * inv_l,
                              __uint_as_float(o[i + 2]) * inv_l, __uint_as_float(o[i + 3]) * inv_l);
          }
          p.part_lse[slot * kTileM + row_in_tile] = lse_row;
          // Every warp counts its 32 rows in by itself and merges them if they are the query block's last: no barrier
          // among the tile's warps (see gave_up).
          int done = 0;
          __syncwarp();
          if (lane == 0) {
            __threadfence();
            int* counter = p.count + (item * 2 + t) * 4 + quad;
            done = atomicAdd(counter, 1) == last - first;
            if (done) *counter = 0;
            __threadfence();
          }
          write_out = __shfl_sync(0xffffffffu, done, 0) != 0;
          __syncwarp();
          if (write_out) {
            // out = sum_i exp(lse_i - lse) * part_i, lse = log sum_i exp(lse_i), fragments in key order
            part0 = first;
            n_parts = last - first + 1;
            parts = reinterpret_cast<const float4*>(p.part_o) + row_in_tile;
            lses = p.part_lse + row_in_tile;
            mx = -INFINITY;
            for (int i = 0; i < n_parts; ++i) mx = fmaxf(mx, __ldcg(lses + static_cast<size_t>(slot_of(part0 + i)) * kTileM));
            float wsum = 0.f;
            for (int i = 0; i < n_parts; ++i)
              wsum += expf(__ldcg(lses + static_cast<size_t>(slot_of(part0 + i)) * kTileM) - mx);
            inv_w = 1.0f / wsum;
            lse_row = mx + logf(wsum);
          }
        }
        if (!write_out) continue;
        // 64 columns at a time through this warp's staging rows; the tensor copies that take them to memory run on
        // their own, so that the warp goes on to the next query block as soon as the second half is parked
        const float inv_l = 1.0f / l_sum;
        const int row0 = w.q0 + t * kTileM + quad * 32;
        uint32_t v[64];  // the row, packed
        if (whole) {
          uint32_t o[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(t_o + c * 32, o[c]);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            const uint32_t a = o[i >> 4][(2 * i) & 31], b = o[i >> 4][(2 * i + 1) & 31];
            v[i] = pack2<kFp16>(__uint_as_float(a) * inv_l, __uint_as_float(b) * inv_l);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float f[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = 0.f;
#pragma unroll 1
            for (int i = 0; i < n_parts; ++i) {
              const size_t slot = slot_of(part0 + i);
              const float wi = expf(__ldcg(lses + slot * kTileM) - mx) * inv_w;
              const float4* src = parts + slot * (32 * kTileM) + (c * 8) * kTileM;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 x = __ldcg(src + j * kTileM);
                f[4 * j] = fmaf(wi, x.x, f[4 * j]);
                f[4 * j + 1] = fmaf(wi, x.y, f[4 * j + 1]);
                f[4 * j + 2] = fmaf(wi, x.z, f[4 * j + 2]);
                f[4 * j + 3] = fmaf(wi, x.w, f[4 * j + 3]);
              }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) v[c * 16 + i] = pack2<kFp16>(f[2 * i], f[2 * i + 1]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (lane == 0) tma_store_wait_read();  // the previous copy has left the staging rows
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<uint4*>(stage + lane * 128 + ((i ^ (lane & 7)) << 4)) =
                make_uint4(v[h * 32 + 4 * i], v[h * 32 + 4 * i + 1], v[h * 32 + 4 * i + 2], v[h * 32 + 4 * i + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && row0 < p.Sq) {
            tma_store_4d(&tm_out, smem_u32(stage), h * 64, w.head, row0, w.batch);
            tma_store_commit();
          }
        }
        const int row = row0 + lane;
        if (p.lse != nullptr && row < p.Sq)
          p.lse[(static_cast<size_t>(w.batch) * p.H + w.head) * p.Sq + row] = lse_row;
      }
      unit = following == kNotAsked ? next_unit(n_units++, kDevTimeoutSoftmax) : following;
      if (gave_up()) unit = -1;
    }
    if (lane == 0) tma_store_wait();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace chitu
