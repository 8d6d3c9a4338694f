// bf16 fused causal attention forward for sm_100a, head size 64: a persistent kernel, one CTA
// per SM, that works on TWO 128-row query tiles of one (batch, head) at a time.
//
// The arithmetic is that of the reference's flash_fwd_kernel (cuda/attention.cu:17-73: online
// softmax over key tiles, lse = max + ln(sum) of the scaled scores) with bf16 operands and fp32
// accumulation. What differs is the shape of the work. At head size 64 a 128x128 score tile
// costs 640 clocks of tensor pipe but 1024 clocks of the exp2 unit and, written naively, more
// than 1200 issue slots per scheduler: the softmax, not the MMAs, is what has to be fed. So:
//   * a work item is a PAIR of adjacent query tiles (A = tile 2p, B = tile 2p + 1) of one
//     (batch, head); both use the same K/V tiles from one shared-memory ring and each has its
//     own softmax group. While group A computes exponentials the tensor pipe runs B's products
//     and vice versa;
//   * a K/V tile is worked through in two sub-steps of 64 keys, and every group has TWO score
//     buffers of 64 columns in tensor memory: while the group's threads work on the scores of
//     one sub-step, the product for the next one is already running into the other buffer, so in
//     steady state nobody waits for the tensor pipe and the tensor pipe waits for nobody;
//   * a group is 256 threads, TWO per query row: one takes key columns 0-31 of every sub-step,
//     the other columns 32-63. Each keeps its OWN running max / sum and its OWN output
//     accumulator in tensor memory (split-K inside the CTA), so the two threads of a row never
//     talk inside the loop; they are merged once per item, in the epilogue. Sixteen softmax
//     warps, four per scheduler, are what hides the tensor-memory and exp2 latencies;
//   * the probabilities never touch shared memory: a thread reads its 32 scores from tensor
//     memory once, keeps them in registers for the max and the exponentials, and writes P back
//     as packed bf16 over the first half of the same columns, from where the P V product takes
//     it as its A operand;
//   * scale-and-subtract and the row sums run as packed two-float instructions (fma.rn.f32x2,
//     add.rn.f32x2), the row max as three-input max, and one pair of exponentials in eight as a
//     cubic on the FMA pipe (us at 192 x 1024 / 48 x 4096: none 44.4 / 129, one in eight 42.8 / 124, one
//     in four 41.7 / 121, half 43.7 / 127). It is the last pair of sixteen columns: the first fourteen rows
//     of a sequence, whose probabilities are the largest, see exact ones only (with columns 2 and 3 of
//     eight and a cubic of 1.0e-4 their lse was off by 4e-5 instead of 3e-7, and results there by a unit
//     of bf16). A bf16x2 exp2 on the special-function unit was tried: no faster, and it cost a digit of
//     lse. Only the 32 x 32 block on the diagonal pays for the causal compare: the softmax is bound by
//     instruction issue and the exp2 unit alike;
//   * CTAs are persistent: barriers, tensor memory and descriptors are set up once, items are
//     dealt out heaviest first in a fixed serpentine order (no global counter to reset), the
//     next item's Q tiles and first K/V tiles are in flight while the current one finishes, and
//     its first score products are issued before the current item's epilogue.
//
//   warp 0        TMA producer (Q pair double-buffered, K/V through a 4-stage ring)
//   warp 1        MMA issuer of group A, owner of the tensor-memory allocation
//   warp 18       MMA issuer of group B (one issuing thread per group: a group's products are
//                 issued the moment its probabilities are ready, whatever the other group does)
//   warps 2-9     softmax group A (2-5: key columns 0-31 of a sub-step, 6-9: 32-63)
//   warps 10-17   softmax group B likewise
// Tensor memory: score buffer b of group X at 128 X + 64 b; O of (group X, half h) at
// 256 + 64 (2 X + h); P of half h aliases the first 16 columns of its 32 columns of the buffer.
//
// Every mbarrier wait is bounded (sm100_ptx.cuh); on expiry the CTA raises its abort flag, all
// roles fall through to the common exit, tensor memory is freed and DADATTN_E_TIMEOUT is left in
// the device status word. No cluster launch, no multicast: each CTA loads its own tiles.
#include <cuda_bf16.h>

#include <cfloat>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

using namespace ptx;

constexpr int kT = 128;               // tile edge: query rows per group, keys per K/V tile
constexpr int kHD = 64;               // head size
constexpr int kPanel = 128 * 128;     // [128 rows][64 bf16]: 16 KB, 128-byte rows, swizzled
constexpr int kKvStages = 4;
constexpr int kFwd64Threads = 19 * 32;
constexpr int kHalfThreads = 128;     // threads of one half of a softmax group
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleAt = 8.0f;    // log2 units: O is rescaled only when the max grew by 2^8

struct F64Smem {
  static constexpr int kQ = 0;                                // [2 items][A, B] panels
  static constexpr int kK = kQ + 4 * kPanel;
  static constexpr int kV = kK + kKvStages * kPanel;
  static constexpr int kStat = kV + kKvStages * kPanel;      // float2 [2 items][group][half][128]: (max, sum)
  static constexpr int kBars = kStat + 2 * 2 * 2 * 128 * 8;
  static constexpr int kBytes = kBars + 512;
  static_assert(kBytes <= 232448, "shared memory budget of one CTA exceeded");
};

struct F64Bars {
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[kKvStages], v_full[kKvStages], kv_empty[kKvStages];
  uint64_t s_full[2][2], p_full[2][2], o_done[2][2], o_free[2], stat_full[2], settled[2];   // [group][buffer]
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(F64Bars) <= 512, "barrier block");

// ---- work items --------------------------------------------------------------------------------
// Item e (0 = heaviest): query-tile pair p = n_pairs - 1 - e / BH of (batch, head) e % BH.
// Which items a CTA takes, in order, is fixed before the launch; every role computes the same
// list, nothing is shared or reset. For small launches the host deals the weight-sorted list out
// greedily (each item to the CTA with the least work so far) and passes the result as a kernel
// parameter: entry k * G + c is the k-th item of CTA c. With only a handful of items per CTA the
// closed-form deal below can leave some CTAs two K/V steps (of about 26) behind the others.
// Larger launches use the closed form: CTA c of G takes the items k * G + (k even ? c : G-1-c), a
// serpentine deal, so that a CTA that got an early (heavy) item in one row gets a late (light)
// one in the next.
constexpr int kDealEntries = 1536;
constexpr uint16_t kDealNone = 0xffffu;
struct F64Deal {
  int rows;                      // 0: closed-form deal
  uint16_t item[kDealEntries];
};
struct F64NoDeal {};   // sequences of one tile: 3 KB less to copy per launch
template <bool ONE>
using F64DealOf = std::conditional_t<ONE, F64NoDeal, F64Deal>;
struct F64Item {
  int bh, qa, n_a, n_b, n_kv;   // n_b = 0 when there is nothing for group B
  // Sequences of one tile (S <= 128): the pair is that tile of units bh and bh + 1. The units share no
  // K/V: ring tile 0 is group A's, ring tile 1 group B's (off_b). With one unit per item group B would
  // idle and there would be twice as many items (192 x 128: 8.0 us a call, now 6.5).
  int bh_b, off_b;
  bool valid;
};
__host__ __device__ inline int f64_items(int BH, int n_tiles) {
  return n_tiles == 1 ? (BH + 1) / 2 : BH * ((n_tiles + 1) / 2);
}
template <bool ONE>   // ONE: sequences of one tile
__device__ __forceinline__ F64Item f64_item(const F64DealOf<ONE>& deal, int k, int BH, int n_tiles, int n_items) {
  const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  int e = k * G + ((k & 1) ? (G - 1 - c) : c);
  if constexpr (!ONE) {
    if (deal.rows > 0) {
      const uint16_t t = k < deal.rows ? deal.item[k * G + c] : kDealNone;
      e = t == kDealNone ? n_items : t;
    }
  }
  F64Item it;
  it.valid = e < n_items;
  if constexpr (ONE) {
    it.bh = 2 * e;
    it.bh_b = it.bh + 1;
    it.qa = 0;
    it.n_a = 1;
    it.n_b = it.off_b = it.bh_b < BH ? 1 : 0;
    it.n_kv = 1 + it.n_b;
    return it;
  }
  const int row = e / BH;
  const int n_pairs = (n_tiles + 1) / 2;
  it.bh = e - row * BH;
  it.qa = 2 * (n_pairs - 1 - row);
  it.n_a = it.qa + 1;
  it.n_b = (it.qa + 1 < n_tiles) ? it.qa + 2 : 0;
  it.n_kv = it.n_b ? it.n_b : it.n_a;
  return it;
}

// DROP: 0 = no dropout, 1 = Philox drawn in the kernel, 2 = keep bits read from `mask_bits`.
// F32: the output is written as fp32 tensor of bf16 values (heads-split layout only).
template <int DROP, bool F32, bool ONE>
__global__ void __launch_bounds__(kFwd64Threads, 1)
flash_fwd64_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                   float* __restrict__ lse, int BH, int S, UnitLayout lay, float scale, float rate,
                   PhiloxKey rng, int64_t unit0, const uint4* __restrict__ mask_bits,
                   int* __restrict__ status, const __grid_constant__ F64DealOf<ONE> deal) {
  using L = F64Smem;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColO = 256;   // score buffer (X,b) at 128 X + 64 b, O_(X,h) at kColO + 64 (2 X + h)

  extern __shared__ __align__(1024) uint8_t smem[];
  F64Bars* bars = reinterpret_cast<F64Bars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;

  // the warp index through a shuffle, so that the compiler knows it is uniform across the warp
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
  const int lane = threadIdx.x % 32;
  const int n_tiles = (S + kT - 1) / kT;
  const int n_items = f64_items(BH, n_tiles);

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicExch(status, DADATTN_E_CUDA);
    return;
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->q_full[b], 1);
      mbar_init(&bars->q_empty[b], 16);             // one arrival per softmax warp
      for (int i = 0; i < 2; ++i) {
        mbar_init(&bars->s_full[b][i], 1);
        mbar_init(&bars->p_full[b][i], 2 * kHalfThreads);
      }
      mbar_init(&bars->o_done[b][0], 1);
      mbar_init(&bars->o_done[b][1], 1);
      mbar_init(&bars->o_free[b], 2 * kHalfThreads);
      mbar_init(&bars->stat_full[b], 2 * kHalfThreads);
      mbar_init(&bars->settled[b], 1);
    }
    for (int s = 0; s < kKvStages; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->kv_empty[s], 2);             // one arrival per issuer
    }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  // Set-up is done. Global memory, which the previous grid in the stream may still read or write, is
  // touched only behind pdl_wait, by the roles that touch it; the products have nothing to wait for but
  // the producer's loads.

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      prefetch_tensormap(&map_q);
      prefetch_tensormap(&map_k);
      prefetch_tensormap(&map_v);
      prefetch_tensormap(&map_out);
      int g = 0, k = 0;  // K/V tiles and Q pairs loaded so far, over all items
      bool ok = true;
      F64Item it = f64_item<ONE>(deal, 0, BH, n_tiles, n_items);
      pdl_wait();
      pdl_launch_dependents();   // once every CTA of this grid is here the next grid may start its set-up
      for (; ok && it.valid; it = f64_item<ONE>(deal, ++k, BH, n_tiles, n_items)) {
        const int qb = k & 1;
        // the Q buffer frees when the results of the item before last, which are staged in it, have left
        if (k >= 2 && !mbar_wait(&bars->q_empty[qb], ((k >> 1) - 1) & 1, abort_flag)) break;
        int ub = it.bh / lay.heads, uh = it.bh - ub * lay.heads;   // (batch, head) of the unit
        const int ub_b = ONE ? it.bh_b / lay.heads : ub, uh_b = ONE ? it.bh_b - ub_b * lay.heads : uh;
        mbar_arrive_expect_tx(&bars->q_full[qb], it.n_b ? 2 * kPanel : kPanel);
        tma_load_4d(smem + L::kQ + (qb * 2 + 0) * kPanel, &map_q, &bars->q_full[qb], 0, it.qa * kT, uh, ub);
        if (it.n_b)
          tma_load_4d(smem + L::kQ + (qb * 2 + 1) * kPanel, &map_q, &bars->q_full[qb], 0, (ONE ? 0 : it.qa + 1) * kT, uh_b, ub_b);
        for (int j = 0; j < it.n_kv; ++j, ++g) {
          const int s = g % kKvStages, use = g / kKvStages;
          if (use > 0 && !(ok = mbar_wait(&bars->kv_empty[s], (use - 1) & 1, abort_flag))) break;
          const int row0 = ONE ? 0 : j * kT;
          if (ONE && j == 1) ub = ub_b, uh = uh_b;
          mbar_arrive_expect_tx(&bars->k_full[s], kPanel);
          tma_load_4d(smem + L::kK + s * kPanel, &map_k, &bars->k_full[s], 0, row0, uh, ub);
          mbar_arrive_expect_tx(&bars->v_full[s], kPanel);
          tma_load_4d(smem + L::kV + s * kPanel, &map_v, &bars->v_full[s], 0, row0, uh, ub);
        }
      }
      settle_ring(bars->q_full, 2, k);
      settle_ring(bars->k_full, kKvStages, g);
      settle_ring(bars->v_full, kKvStages, g);
    }
  } else if (warp == 1 || warp == 18) {
    // ------------------------------ MMA issuers ------------------------------
    // One issuing thread per group. Issuer X walks the K/V ring tiles of all items in order, each
    // tile as two sub-steps of 64 keys. For sub-step (g, c) it issues O_X += P_X V(g, c) and then
    // S_X = Q_X K(g+1, c)^T, the scores two sub-steps ahead, into the buffer that P_X(g, c) has
    // just left (also across an item boundary). A ring stage is released by both issuers: each commits
    // (or, where its group has nothing to do with the tile, arrives) once.
    {   // (whole warps: mma_ss_warp)
      const uint32_t lead = elect_one(), tm = __reduce_max_sync(0xffffffffu, tmem);   // (known to be uniform, so)
      const int X = __reduce_max_sync(0xffffffffu, warp == 1 ? 0u : 1u);
      constexpr uint32_t idesc_s = make_idesc_bf16(kT, 64, 0, 0);    // Q, K: K-major; 64 keys
      constexpr uint32_t idesc_o = make_idesc_bf16(kT, kHD, 0, 1);   // P from TMEM, V MN-major
      const SmemDescBase q_desc0 = make_desc_base_sw128(smem_u32(smem + L::kQ), 0);
      const SmemDescBase k_desc0 = make_desc_base_sw128(smem_u32(smem + L::kK), 0);
      const SmemDescBase v_desc0 = make_desc_base_sw128(smem_u32(smem + L::kV), 0);
      const uint32_t tSx = tm + kColS + X * 128, tOx = tm + kColO + X * 2 * kHD;
      int n_pv = 0;      // sub-steps of this group whose P V products have been issued
      int n_done = 0;    // items finished so far in which the group took part
      bool ok = true;

      // S_X = Q_X K^T for the 64 keys of sub-step c of K/V ring tile g, item in Q buffer qb; the
      // group's sub-steps alternate between its two score buffers, and c is the buffer
      auto issue_s = [&](int qb, int g, int c) {
        const SmemDescBase qd{q_desc0.lo + (qb * 2 + X) * (kPanel >> 4), q_desc0.hi};
        const SmemDescBase kd{k_desc0.lo + (g % kKvStages) * (kPanel >> 4), k_desc0.hi};
#pragma unroll
        for (int kk = 0; kk < kHD / 16; ++kk)
          mma_ss_warp(tSx + c * 64, desc_at(qd, kk * 32), desc_at(kd, c * 8192 + kk * 32), idesc_s, kk > 0 ? 1u : 0u, lead);
        mma_commit_warp(&bars->s_full[X][c], lead);
      };
      // O_(X,h) (+)= P_(X,h) V[keys 64 c + 32 h .. + 31] of ring tile g, both halves. P of half h
      // sits in the first 16 columns of its 32 columns of buffer c, 16 keys (8 columns of packed
      // bf16 pairs) per MMA; V is MN-major, 16 keys = 2048 bytes further down.
      auto issue_pv = [&](int g, int c, bool first_of_item) -> bool {
        // the epilogue of the group's previous item must have read O_X before it is overwritten
        if (first_of_item && n_done > 0 && !warp_wait(&bars->o_free[X], (n_done - 1) & 1, abort_flag))
          return false;
        if (!warp_wait(&bars->p_full[X][c], (n_pv >> 1) & 1, abort_flag)) return false;
        tc_fence_after_sync();
        const SmemDescBase vd{v_desc0.lo + (g % kKvStages) * (kPanel >> 4), v_desc0.hi};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)
            mma_ts_warp(tOx + h * kHD, tSx + c * 64 + h * 32 + kk * 8, desc_at(vd, (c * 4 + h * 2 + kk) * 2048),
                   idesc_o, (!first_of_item || kk > 0) ? 1u : 0u, lead);
        }
        mma_commit_warp(&bars->o_done[X][n_pv & 1], lead);
        ++n_pv;
        return true;
      };
      // the group takes part in the item's ring tiles begin_of .. end_of - 1
      auto begin_of = [&](const F64Item& it) { return ONE && X ? it.off_b : 0; };
      auto end_of = [&](const F64Item& it) { return X ? (ONE ? it.off_b : 0) + it.n_b : it.n_a; };
      auto n_of = [&](const F64Item& it) { return X ? it.n_b : it.n_a; };

      F64Item cur = f64_item<ONE>(deal, 0, BH, n_tiles, n_items);
      F64Item nxt = f64_item<ONE>(deal, 1, BH, n_tiles, n_items);
      int g = 0;
      if (cur.valid) {
        ok = warp_wait(&bars->q_full[0], 0, abort_flag) && warp_wait(&bars->k_full[0], 0, abort_flag);
        if (ok) {
          tc_fence_after_sync();
          if (n_of(cur) > 0 && begin_of(cur) == 0) {
            issue_s(0, 0, 0);
            issue_s(0, 0, 1);
          }
        }
      }
      for (int k = 0; ok && cur.valid; ++k) {
        const int qb = k & 1;
        const int n_x = n_of(cur), j0 = begin_of(cur), j1 = end_of(cur);
        for (int j = 0; ok && j < cur.n_kv; ++j, ++g) {
          const int s = g % kKvStages;
          // The tile after this one in the ring: the item's next tile, or the next item's first.
          const bool last = (j + 1 == cur.n_kv);
          const bool have_next = !last || nxt.valid;
          const F64Item& ni = last ? nxt : cur;
          const int nj = last ? 0 : j + 1, nqb = last ? (qb ^ 1) : qb;
          // Every release below follows a wait on the matching "full" barrier of the same use,
          // also where this group has nothing to do with the tile: an idle issuer must not run
          // ahead and arrive twice within one phase of a release barrier.
          bool issued = false;
          ok = warp_wait(&bars->v_full[s], (g / kKvStages) & 1, abort_flag);
          // the group has scores to form in the next tile
          const bool s_next = have_next && n_of(ni) > 0 && nj >= begin_of(ni) && nj < end_of(ni);
          bool next_ready = false;
#pragma unroll
          for (int c = 0; c < 2 && ok; ++c) {
            if (j >= j0 && j < j1) {
              ok = issue_pv(g, c, j == j0 && c == 0);
              issued = ok;
            }
            if (ok && s_next) {
              if (!next_ready) {
                // An issuer does not wait for K and Q of tiles and items that its group has nothing to do with, and yet
                // cannot take an old phase for the present one: tile g is there only once the other issuer has given
                // back tile g - kKvStages, behind its own wait for K of the tile after that and for Q of the item two before
                // `ni` (an item that leaves a group idle has three tiles or more, the one between one or more).
                static_assert(kKvStages <= 4, "an idle issuer could take an old phase of q_full for the present one");
                if (nj == begin_of(ni)) ok = warp_wait(&bars->q_full[nqb], ((last ? k + 1 : k) >> 1) & 1, abort_flag);
                ok = ok && warp_wait(&bars->k_full[(g + 1) % kKvStages], ((g + 1) / kKvStages) & 1, abort_flag);
                if (ok) tc_fence_after_sync();
                next_ready = true;
              }
              if (ok) {
                issue_s(nqb, g + 1, c);
                issued = true;
              }
            }
          }
          // this issuer's share of the stage's release: after every product of its that reads it
          if (ok) {
            if (issued) mma_commit_warp(&bars->kv_empty[s], lead); else if (lead) mbar_arrive(&bars->kv_empty[s]);
          }
        }
        if (n_x > 0) ++n_done;
        cur = nxt;
        nxt = f64_item<ONE>(deal, k + 2, BH, n_tiles, n_items);
      }
      settle_products_warp(&bars->settled[X], lead);
    }
  } else {
    // ------------------------------ softmax groups ------------------------------
    const int X = (warp - 2) / 8;         // 0: group A (first tile of the pair), 1: group B (warps 2-17)
    const int half = ((warp - 2) / 4) & 1;  // which 32 key columns of every 64-key sub-step
    const int quad = warp % 4;            // TMEM lane quadrant this warp may touch
    const int row = quad * 32 + lane;     // row within the tile = TMEM lane
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t tS0 = tlane + kColS + X * 128 + half * 32;   // this thread's columns of buffer 0
    const float scale_log2 = scale * kLog2e;
    const float keep_scale = DROP ? 1.0f / (1.0f - rate) : 1.0f;
    int t = 0;        // 64-key sub-steps this group has processed so far, over all items
    int n_item = 0;   // items this group has taken part in
    int owed = -1;    // Q buffer that this warp has staged results in and not yet given back
    bool ok = true;
    // gives it back, once the store has read it (lane 0 issued that)
    auto give_back = [&]() {
      if (owed >= 0 && lane == 0) {
        bulk_wait_read<0>();
        mbar_arrive(&bars->q_empty[owed]);
      }
      owed = -1;
    };
    if (DROP == 2) pdl_wait();   // (the mask)

    for (int k = 0; ok; ++k) {
      const F64Item it = f64_item<ONE>(deal, k, BH, n_tiles, n_items);
      if (!it.valid) break;
      const int n_x = X ? it.n_b : it.n_a;
      if (n_x == 0) {                       // nothing for this group: its share of the Q buffer, once that is loaded
        give_back();
        if ((ok = mbar_wait(&bars->q_full[k & 1], (k >> 1) & 1, abort_flag)) && lane == 0) mbar_arrive(&bars->q_empty[k & 1]);
        continue;
      }
      const int qt = ONE ? 0 : it.qa + X, bh = ONE && X ? it.bh_b : it.bh;
      float m = -INFINITY;                  // running max of the scaled scores, log2 units
      float2 l2 = make_float2(0.f, 0.f);    // running sum, two interleaved partial sums
      const uint32_t* bits1 = reinterpret_cast<const uint32_t*>(mask_bits);
      uint32_t keep = ~0u, keep_next = ~0u;
      if (DROP == 2) keep_next = __ldg(bits1 + mask_bits_record(bh, qt, 0, row, n_tiles) * 4 + half);

      for (int v = 0; v < 2 * n_x; ++v, ++t) {
        const int j = v >> 1, c = v & 1;    // K/V tile and its sub-step; c is also the score buffer
        if (DROP == 2) {
          keep = keep_next;   // fetched a sub-step ahead: its latency hides behind this one's work
          if (v + 1 < 2 * n_x)
            keep_next = __ldg(bits1 + mask_bits_record(bh, qt, (v + 1) >> 1, row, n_tiles) * 4 +
                              ((v + 1) & 1) * 2 + half);
        }
        if (v == 1) give_back();   // (every item has two sub-steps; the store is long through)
        if (!(ok = mbar_wait(&bars->s_full[X][c], (t >> 1) & 1, abort_flag))) break;
        tc_fence_after_sync();
        const uint32_t tS = tS0 + c * 64;
        const bool diagonal = (j == n_x - 1);

        // ---- the thread's 32 scores: read once, kept in registers for the max and the
        // exponentials ----
        uint32_t xa[32];
        auto load_scores = [&]() {
          tmem_ld32(tS, xa);
          tmem_wait_ld();
          if (diagonal && c * 2 + half == quad) {   // the block on the diagonal; those below it see all keys
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i > lane) xa[i] = 0xff800000u;  // -inf
          }
        };
        if (diagonal && c * 64 + half * 32 > quad * 32 + 31) {   // the warp's block lies beyond the diagonal
          uint32_t zero[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) zero[i] = 0u;
          tmem_st16(tS, zero);
          tmem_wait_st();
          tc_fence_before_sync();
          mbar_arrive(&bars->p_full[X][c]);
          continue;   // (an item's first block: m stays -inf)
        }
        load_scores();
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          mx0 = fmax3(mx0, __uint_as_float(xa[i]), __uint_as_float(xa[i + 1]));
          mx1 = fmax3(mx1, __uint_as_float(xa[i + 2]), __uint_as_float(xa[i + 3]));
        }
        const float mx = fmaxf(mx0, mx1) * scale_log2;   // scale > 0 commutes with max

        // ---- lazy rescale: O and the sum move to a new max only when it grew by 2^8 ----
        if (v == 0) {
          m = mx;  // O is first written by an MMA that does not accumulate: nothing to rescale
        } else if (__any_sync(0xffffffffu, mx > m + kRescaleAt)) {
          // P V of this group's previous sub-step must have completed before O is touched
          if (!(ok = mbar_wait(&bars->o_done[X][(t - 1) & 1], ((t - 1) >> 1) & 1, abort_flag))) break;
          tc_fence_after_sync();
          const float m_new = fmaxf(m, mx);
          // m = -inf: nothing but zeros has been accumulated so far (every earlier column masked)
          const float corr = (m == -INFINITY) ? 0.f : ex2(m - m_new);
#pragma unroll 1
          for (int cc = 0; cc < kHD / 32; ++cc) {
            uint32_t o[32];
            tmem_ld32(tlane + kColO + (X * 2 + half) * kHD + cc * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
            tmem_st32(tlane + kColO + (X * 2 + half) * kHD + cc * 32, o);
          }
          tmem_wait_st();
          l2 = fmul2(l2, make_float2(corr, corr));
          m = m_new;
          // read the scores again rather than keep them alive across this rare path
          load_scores();
        }

        // ---- p = exp2(s * scale * log2e - m); P goes back to tensor memory as packed bf16
        // pairs over the first 16 of this thread's columns. A half-row with no visible key yet has
        // m = -inf: its scores are all -inf and must give p = 0, not exp2(nan). ----
        const float neg_m = (m == -INFINITY) ? 0.f : -m;
        const float2 sl = make_float2(scale_log2, scale_log2), nm = make_float2(neg_m, neg_m);
        float2 la = make_float2(0.f, 0.f), lb = la;   // this sub-step's sums, two independent chains
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 e = ffma2(make_float2(__uint_as_float(xa[i]), __uint_as_float(xa[i + 1])), sl, nm);
          float2 p;
          if ((i & 15) == 14) {   // one pair in eight on the FMA pipe
            p = ex2_poly2(e);
          } else {
            p.x = ex2(e.x);
            p.y = ex2(e.y);
          }
          if (i & 2) lb = fadd2(lb, p); else la = fadd2(la, p);
          if (DROP == 1) {
            const uint64_t idx = (static_cast<uint64_t>(unit0 + bh) * S + qt * kT + row) * S + j * kT +
                                 c * 64 + half * 32 + i;
            p.x = (p.x != 0.f && philox_keep(rng, idx, rate)) ? p.x * keep_scale : 0.f;
            p.y = (p.y != 0.f && philox_keep(rng, idx + 1, rate)) ? p.y * keep_scale : 0.f;
          } else if (DROP == 2) {
            p.x = ((keep >> i) & 1u) ? p.x * keep_scale : 0.f;
            p.y = ((keep >> (i + 1)) & 1u) ? p.y * keep_scale : 0.f;
          }
          pk[i / 2] = pack_bf16(p.x, p.y);
        }
        tmem_st16(tS, pk);          // P of this thread's 32 keys -> its first 16 columns
        l2 = fadd2(l2, fadd2(la, lb));
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(&bars->p_full[X][c]);
      }
      if (!ok) break;

      // ---- epilogue: merge the two halves of each row. out = (O_0 w_0 + O_1 w_1) / (l_0 w_0 +
      // l_1 w_1) with w_h = exp2(m_h - max(m_0, m_1)); lse in natural-log units of the scaled
      // scores. Each thread of the pair writes 32 of the row's 64 outputs. ----
      // (Two buffers: the scores of an item of one tile do not wait for the epilogue of the item before, so that a
      // half may be here again while a warp of the other has not read its row's pairs. A third time needs scores that
      // come behind products, and those the probabilities that both halves store after the first.)
      float2* stat = reinterpret_cast<float2*>(smem + L::kStat) + ((n_item & 1) * 2 + X) * 256;   // [half][128]
      const int r = qt * kT + row;          // query index
      stat[half * 128 + row] = make_float2(m, l2.x + l2.y);
      mbar_arrive(&bars->stat_full[X]);
      if (!(ok = mbar_wait(&bars->stat_full[X], n_item & 1, abort_flag))) break;
      // the group's last P V products (both halves)
      if (!(ok = mbar_wait(&bars->o_done[X][(t - 1) & 1], ((t - 1) >> 1) & 1, abort_flag))) break;
      tc_fence_after_sync();
      const float2 s0 = stat[row], s1 = stat[128 + row];
      const float m_tot = fmaxf(s0.x, s1.x);   // half 0 always sees key 0: finite
      const float w0 = ex2(s0.x - m_tot);
      const float w1 = (s1.x == -INFINITY) ? 0.f : ex2(s1.x - m_tot);
      const float l_tot = s0.y * w0 + s1.y * w1;
      const float f0 = w0 / l_tot, f1 = w1 / l_tot;
      // Through shared memory and TMA: as 16-byte stores of one row per lane, 32 lines an instruction, they took
      // 1800-2400 clocks an item and held up the loads of the next one (192 x 1024: 48.3 us, now 44.3; 48 x 4096
      // 133 and 125; 192 x 128 6.1 and 5.7, part of it the first item and the descriptors read ahead of pdl_wait).
      // A warp's 32 rows x 32 columns are its own 2 KB of the group's Q tile, whose last product is behind the last
      // scores. (fp32 rows of 32 columns would need 4 KB: 16 columns, then the others.)
      uint8_t* stage = smem + L::kQ + ((k & 1) * 2 + X) * kPanel + (half * 4 + quad) * 2048;
      auto put = [&](int chunk, uint4 w) {   // 64-byte rows, swizzled
        *reinterpret_cast<uint4*>(stage + lane * 64 + ((chunk ^ ((lane >> 1) & 3)) << 4)) = w;
      };
      auto send = [&](int column) {
        fence_proxy_async_smem();
        __syncwarp();
        const int ub = bh / lay.heads, uh = bh - ub * lay.heads, row0 = qt * kT + quad * 32;
        if (lane == 0 && row0 < S) {   // (rows beyond S are not written)
          tma_store_4d(&map_out, stage, half * 32 + column, row0, uh, ub);
          bulk_commit();
        }
      };
      if (n_item == 0) pdl_wait();
#pragma unroll
      for (int c = 0; c < 2; ++c) {   // 16 output columns at a time
        uint32_t oa[16], ob[16];
        tmem_ld16(tlane + kColO + (X * 2 + 0) * kHD + half * 32 + c * 16, oa);
        tmem_ld16(tlane + kColO + (X * 2 + 1) * kHD + half * 32 + c * 16, ob);
        tmem_wait_ld();
        if (c == 1) {
          tc_fence_before_sync();
          mbar_arrive(&bars->o_free[X]);   // O and the statistics have been read: the next item may start
        }
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 16; e += 2)
          w[e / 2] = pack_bf16(__uint_as_float(oa[e]) * f0 + __uint_as_float(ob[e]) * f1,
                               __uint_as_float(oa[e + 1]) * f0 + __uint_as_float(ob[e + 1]) * f1);
        if (F32) {   // rounded to bf16 like every operand, widened again
          if (c == 1) {
            if (lane == 0) bulk_wait_read<0>();
            __syncwarp();
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            put(e, make_uint4(w[2 * e] << 16, w[2 * e] & 0xffff0000u, w[2 * e + 1] << 16, w[2 * e + 1] & 0xffff0000u));
          send(c * 16);
        } else {
          put(2 * c, make_uint4(w[0], w[1], w[2], w[3]));
          put(2 * c + 1, make_uint4(w[4], w[5], w[6], w[7]));
          if (c == 1) send(0);
        }
      }
      owed = k & 1;
      ++n_item;
      if (half == 0 && r < S) lse[static_cast<size_t>(bh) * S + r] = (m_tot + log2f(l_tot)) * kLn2;
    }
    if (lane == 0) bulk_wait0();   // the results have landed before the CTA retires
  }

  // ------------------------------ common exit ------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (threadIdx.x == 0 && bars->abort_flag) report_timeout(status, bars->abort_flag);
}

// The greedy deal for a launch of G CTAs, or rows = 0 when the closed form serves (too many
// items for the table). An item's weight is its K/V steps plus a half for its prologue and
// epilogue. The last deal is kept: a training loop asks for the same one again and again.
const F64Deal& fwd64_deal(int BH, int n_tiles, int G) {
  struct Cached {
    int BH = -1, n_tiles = -1, G = -1;
    F64Deal deal;
  };
  static thread_local Cached cache;
  if (cache.BH == BH && cache.n_tiles == n_tiles && cache.G == G) return cache.deal;
  cache.BH = BH, cache.n_tiles = n_tiles, cache.G = G;
  F64Deal& d = cache.deal;
  d.rows = 0;
  const int n_pairs = (n_tiles + 1) / 2;
  const long long n_items = f64_items(BH, n_tiles);
  if (n_items > kDealEntries || G <= 0) return d;   // (every item takes an entry: no table could hold them)
  std::vector<int> load(G, 0), count(G, 0);
  std::vector<std::vector<uint16_t>> list(G);
  // G is at most a few hundred and the table small: a linear scan for the least loaded CTA
  for (int e = 0; e < static_cast<int>(n_items); ++e) {
    const int qa = 2 * (n_pairs - 1 - e / BH);
    const int n_kv = (qa + 1 < n_tiles) ? qa + 2 : qa + 1;
    int best = 0;
    for (int c = 1; c < G; ++c)
      if (load[c] < load[best]) best = c;
    load[best] += 2 * n_kv + 1;
    list[best].push_back(static_cast<uint16_t>(e));
  }
  size_t rows = 0;
  for (int c = 0; c < G; ++c) rows = list[c].size() > rows ? list[c].size() : rows;
  if (rows * G > kDealEntries) return d;
  for (size_t k = 0; k < rows; ++k)
    for (int c = 0; c < G; ++c) d.item[k * G + c] = k < list[c].size() ? list[c][k] : kDealNone;
  d.rows = static_cast<int>(rows);
  return d;
}

template <int DROP, bool F32 = false>
int launch_fwd64(void* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v,
                 int BH, int S, const UnitLayout& lay, float scale, float rate, uint64_t seed,
                 uint64_t offset, int64_t unit0, const uint32_t* mask_bits, cudaStream_t st) {
  CUtensorMap mq, mk, mv, mo;
  if (int rc = make_tensor_map_bf16_units(&mq, q, BH, S, kHD, kT, lay)) return rc;
  if (int rc = make_tensor_map_bf16_units(&mk, k, BH, S, kHD, kT, lay)) return rc;
  if (int rc = make_tensor_map_bf16_units(&mv, v, BH, S, kHD, kT, lay)) return rc;
  if (int rc = make_tensor_map_rows64(&mo, out, F32, BH, S, kHD, 32, lay)) return rc;
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int n_tiles = (S + kT - 1) / kT;
  if (static_cast<long long>(BH) * ((n_tiles + 1) / 2) > INT32_MAX / 2) return fail(DADATTN_E_UNSUPPORTED, "too many (query tile pair, batch x head) items");
  const int n_items = f64_items(BH, n_tiles);
  const dim3 grid(static_cast<unsigned>(n_items < sms ? n_items : sms));
  auto launch = [&](auto kern, const auto& deal) -> int {
    DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F64Smem::kBytes));
    DAD_CUDA(launch_pdl(kern, grid, dim3(kFwd64Threads), F64Smem::kBytes, st, mq, mk, mv, mo, lse, BH, S, lay, scale,
                        rate, make_philox(seed, offset), unit0, reinterpret_cast<const uint4*>(mask_bits), status, deal));
    return DADATTN_OK;
  };
  return n_tiles == 1 ? launch(flash_fwd64_kernel<DROP, F32, true>, F64NoDeal{})
                      : launch(flash_fwd64_kernel<DROP, F32, false>, fwd64_deal(BH, n_tiles, static_cast<int>(grid.x)));
}

}  // namespace

int launch_fwd_bf16_d64_f32(float* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v, int BH,
                            int S, float scale, cudaStream_t st) {
  return launch_fwd64<0, true>(out, lse, q, k, v, BH, S, unit_layout(BH, 1, S, kHD, false), scale, 0.f, 0, 0, 0,
                               nullptr, st);
}

// Forward at head size 64. mask_bits != nullptr: keep bits from dadattn_dropout_mask_bits;
// otherwise rate > 0 draws the Philox mask inside the kernel. heads > 0: q, k, v, out are the
// interleaved [B*S, heads*64] activations (BH = B * heads units); heads = 0: heads-split [BH,S,64].
int launch_fwd_bf16_d64(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v,
                        int BH, int S, float scale, float rate, uint64_t seed, uint64_t offset,
                        int64_t unit0, const uint32_t* mask_bits, int heads, cudaStream_t st) {
  const UnitLayout lay = heads > 0 ? unit_layout(BH / heads, heads, S, kHD, true) : unit_layout(BH, 1, S, kHD, false);
  if (rate > 0.f && mask_bits)
    return launch_fwd64<2>(out, lse, q, k, v, BH, S, lay, scale, rate, 0, 0, 0, mask_bits, st);
  if (rate > 0.f)
    return launch_fwd64<1>(out, lse, q, k, v, BH, S, lay, scale, rate, seed, offset, unit0, nullptr, st);
  return launch_fwd64<0>(out, lse, q, k, v, BH, S, lay, scale, 0.f, 0, 0, 0, nullptr, st);
}

}  // namespace dadattn
