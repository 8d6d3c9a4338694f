// bf16 fused causal attention backward for sm_100a, head size 64: dQ, dK and dV in ONE pass.
//
// The reference computes the probabilities twice, once in its dK/dV kernel and once in its dQ
// kernel (cuda/attention.cu:88-205): 7 GEMM-sized products for 5 gradients' worth. Here a CTA
// owns 128 keys of one (batch, head), streams the 128-query tiles that can see them, and per
// tile forms S = Q K^T and dP = dO V^T once, then
//     dV += P^T dO        dK += dS^T Q        dQ_tile = dS K
// with p = exp2(S scale log2e - lse log2e), ds = p (dP - delta) scale as in the reference.
// dK/dV accumulate in tensor memory over the whole loop; each tile's dQ contribution is added
// into an fp32 workspace with a TMA reduce-add (several CTAs, one per key tile, contribute to
// the same queries), and a last pass rounds the workspace to bf16. The sums into the workspace
// happen in whatever order the CTAs reach them, so dQ may differ in its last bits from run to
// run; dadattn_set_bwd_deterministic(1) selects the two-kernel path of
// flash_bwd_bf16_sm100.cu, which has no such sums.
//
// Rows of the score tile are keys (one TMEM lane each): S^T = K Q^T and dP^T = V dO^T, so that P^T and
// dS^T, packed to bf16, are the A operands of dV and dK from tensor memory. dS^T is also written to shared
// memory, [key][query] in the 128-byte swizzled layout, as the MN-major A operand of dQ. That leaves room
// for a third Q / dO stage and takes 64 KB a tile off shared memory, whose 128 bytes a clock the products,
// the stores and the TMA share (272 KB a tile). What the time was before, 4140 clocks a tile against 1660
// of the products: with two stages a tile's loads (2000 clocks beside the reduce-adds) started when dV / dK
// of the tile two back were through and held up the products of the tile between; dQ had one staging
// buffer, 3600 clocks from one use to the next. Now 2700-2800 (192 x 1024: 117 -> 84 us), set by the
// issuing thread (2500 clocks for 32 products, their waits and commits) and the arithmetic (2200) alike.
// Measured and not kept: two issuing warps, each with its own accumulators (backward 113 -> 126 us), the whole
// warp issuing (the same), the next group's tiles prefetched into L2 (117 -> 120).
//   warps 0-15   compute: four warps per TMEM lane quadrant, 32 of the 128 query columns each
//   warp 16      TMA producer           warp 17      MMA issuer + TMEM owner
//   warp 18      reducer: issues the TMA reduce-adds of dQ and the dK / dV stores
//   warp 19      row scalars: -lse log2e and -delta scale of each tile's queries
//   warps 20-23  accumulator drain: one thread per TMEM lane takes each tile's dQ, and each
//                item's dK / dV, out of tensor memory into the shared-memory staging panels,
//                while the compute warps are already on the next tile's arithmetic
// The roles are whole warpgroups so that registers can move between them (setmaxnreg): the
// compute warps hold a tile's 32 probabilities and gradients a thread and get 96 registers, the others 48.
#include <cuda_bf16.h>

#include <cfloat>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

using namespace ptx;

constexpr int kFT = 128;                  // tile edge: queries per step, keys per CTA
constexpr int kFD = 64;                   // head size
constexpr int kFPanel = 128 * 128;        // [128 rows][64 bf16] swizzled panel
constexpr int kFThreads = 24 * 32;
constexpr int kFCompute = 16 * 32;
constexpr int kFDrain = 4 * 32;           // one thread per TMEM lane
constexpr int kWarpProducer = 16, kWarpIssuer = 17, kWarpReducer = 18, kWarpDrain0 = 20;   // (19: row scalars)
// Registers per thread after the warpgroups have rebalanced. The pool is what the CTA was launched
// with (kRegsLaunch per thread, the most that 768 threads can have): an increase beyond it would
// wait for ever.
constexpr int kRegsLaunch = 80, kRegsCompute = 96, kRegsHelper = 48, kRegsDrain = 48;
static_assert(kFCompute * kRegsCompute + 128 * kRegsHelper + kFDrain * kRegsDrain <= kFThreads * kRegsLaunch,
              "the warpgroups ask for more registers than the CTA owns");
static_assert(kFThreads * kRegsLaunch <= 65536 && (kRegsLaunch + 8) * kFThreads > 65536,
              "kRegsLaunch is not what the compiler gives a CTA of this size");
constexpr int kFStages = 3;
constexpr int kFRing = 4;                 // entries of the work-item ring (a power of two)
// Rows of all units up to which they are one group. Backward alone, us, one group / groups of up to 65536
// rows: 48 x 2048 90.9 / 95.9, 24 x 4096 152 / 159; above, as groups of 98304 rows / of 65536: 192 x 1024
// 114.5 / 113.0, 144 x 700 67 / 62. Groups as even as they come: 72 x 777 as 64 + 8 units 47.5, as one 42.
constexpr int kFAllInL2 = 98304;
constexpr float kFLog2e = 1.4426950408889634f;

struct FusedSmem {
  static constexpr int kK = 0;                          // two buffers: items alternate
  static constexpr int kV = kK + 2 * kFPanel;
  static constexpr int kQ = kV + 2 * kFPanel;
  static constexpr int kDO = kQ + kFStages * kFPanel;
  static constexpr int kDS = kDO + kFStages * kFPanel;  // dS^T [128 keys][128 q] bf16, two panels
  static constexpr int kDQ = kDS + 2 * kFPanel;         // [128 q][64] fp32, two 128-byte panels
  static constexpr int kVec = kDQ + 2 * kFPanel;        // two buffers of [2][128] row scalars
  static constexpr int kBars = kVec + 2 * 2 * kFT * 4;
  static constexpr int kBarsBytes = 512;
  static constexpr int kBytes = kBars + kBarsBytes;
  static_assert(kBytes <= 232448, "shared memory budget of one CTA exceeded");
};

struct FusedBars {
  uint64_t kv_full[2], kv_empty[2], qdo_full[kFStages], qdo_empty[kFStages];
  uint64_t item_ready[kFRing], item_free[kFRing];
  uint64_t s_full[2], p_full, dp_full, w_full, acc_done, dq_drained, dkv_drained, staged[2], sent[2], settled;
  int2 ring[kFRing];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FusedBars) <= FusedSmem::kBarsBytes, "barriers overflow their shared-memory slot");

// TMA reduce-add of one [128 rows][32 fp32] panel from shared memory into the dQ workspace.
// `policy`: an L2 eviction policy (l2_policy_evict_last): the workspace is summed into up to
// T / 128 times and read once more by the rounding pass, so its lines should outlive the streamed
// Q / dO / K / V tiles in L2.
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* smem_src, int x,
                                                  int y, int z, uint64_t policy) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group.L2::cache_hint "
      "[%0, {%2, %3, %4}], [%1], %5;"
      ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// prmt with the sign-replicating selectors (8 + byte number): each selected byte of the result is 0xff or 0.
template <uint32_t SEL>
__device__ __forceinline__ uint32_t byte_signs(uint32_t w) {
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(w), "n"(SEL));
  return d;
}

// One item of work = (key tile kt, batch x head bh): the CTA that takes it streams the n_it query
// tiles that can see those keys. Items are numbered so that batch x head units come in groups of
// `group_bh` (their Q, dO and dQ rows stay in L2 while the group is worked on) and, inside a
// group, key tile by key tile: the key tiles with the most queries first.
struct Item {
  int kt, bh, n_it;
};
__device__ __forceinline__ Item decode_item(int item, int BH, int n_tiles, int group_bh) {
  const int per_group = group_bh * n_tiles;
  const int grp = item / per_group;
  const int r = item - grp * per_group;
  const int bh0 = grp * group_bh;
  const int gb = min(group_bh, BH - bh0);
  Item t;
  t.kt = r / gb;
  t.bh = bh0 + r - t.kt * gb;
  t.n_it = n_tiles - t.kt;
  return t;
}

// Items are handed out by a global counter; the producer thread takes them and publishes each, decoded
// (the divisions would sit in every role's chain), through a four-entry ring in shared memory, which the
// other roles read in the same order. An entry beyond the last item has n_it = 0.
struct ItemFeed {
  FusedBars* bars;
  volatile int* abort_flag;
  int n_tiles, n_read;
  // the next item of this CTA; n_it = 0 when there is none (or the kernel is aborting)
  __device__ __forceinline__ Item fetch() {
    const int slot = n_read & (kFRing - 1);
    if (!mbar_wait(&bars->item_ready[slot], (n_read / kFRing) & 1, abort_flag)) return Item{n_tiles, 0, 0};
    const volatile int2& e = bars->ring[slot];
    const int kt = e.x, bh = e.y;
    mbar_arrive(&bars->item_free[slot]);
    ++n_read;
    return Item{kt, bh, n_tiles - kt};
  }
};

// DROP: 0 = no dropout, 1 = Philox drawn in the kernel, 2 = keep bits read from `mask_bits`
// (dadattn_dropout_mask_bits; layout in common.cuh). F32: dK and dV leave as fp32, through maps like
// map_dqw, whose tensor is then the caller's own zero-filled fp32 dQ (nothing rounds it afterwards).
template <int DROP, bool F32>
__global__ void __launch_bounds__(kFThreads, 1)
flash_bwd_fused_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                       const __grid_constant__ CUtensorMap map_dqw, const __grid_constant__ CUtensorMap map_dk,
                       const __grid_constant__ CUtensorMap map_dv, const float* __restrict__ lse,
                       const float* __restrict__ delta, int* __restrict__ item_counter, int BH, int S,
                       int heads, int group_bh, float scale, float rate, PhiloxKey rng, int64_t unit0,
                       const uint32_t* __restrict__ mask_bits, int* __restrict__ status) {
  using L = FusedSmem;
  constexpr int D = kFD;
  constexpr uint32_t kTmemCols = 512;
  // S^T and dP^T (fp32, 128 queries each), dV, dK, dQ (64 each), P^T as packed bf16. dS^T goes back over
  // dP^T: each thread packs its 32 queries into the first 16 of the 32 columns it has read.
  constexpr uint32_t kColS = 0, kColDP = 128, kColDV = 256, kColDK = 320, kColDQ = 384, kColP = 448;

  extern __shared__ __align__(1024) uint8_t smem[];
  FusedBars* bars = reinterpret_cast<FusedBars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_tiles = (S + kFT - 1) / kFT;
  const int n_items = n_tiles * BH;

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicExch(status, DADATTN_E_CUDA);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->kv_full[s], 1);
      mbar_init(&bars->kv_empty[s], 1);
      mbar_init(&bars->s_full[s], 2);       // the product and the tile's row scalars
      mbar_init(&bars->staged[s], kFDrain);
      mbar_init(&bars->sent[s], 1);
    }
    for (int s = 0; s < kFStages; ++s) {
      mbar_init(&bars->qdo_full[s], 1);
      mbar_init(&bars->qdo_empty[s], 1);
    }
    for (int s = 0; s < kFRing; ++s) {
      mbar_init(&bars->item_ready[s], 1);
      mbar_init(&bars->item_free[s], kFCompute + kFDrain + 32 + 2);   // compute, drain, row scalars, MMA issuer, reducer
    }
    mbar_init(&bars->p_full, kFCompute);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->w_full, kFCompute);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->dq_drained, kFDrain);
    mbar_init(&bars->dkv_drained, kFDrain);
    mbar_init(&bars->settled, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == kWarpIssuer) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  pdl_wait();
  pdl_launch_dependents();

  // Registers move from the helper warpgroups to the compute warpgroups; each branch below sets
  // its own budget first.
  if (warp >= kWarpProducer && warp < kWarpDrain0) {
  setmaxnreg_dec<kRegsHelper>();
  if (warp == kWarpProducer) {
    // ------------------------------ scheduler + TMA producer ------------------------------
    if (elect_one()) {
      prefetch_tensormap(&map_q);
      prefetch_tensormap(&map_k);
      prefetch_tensormap(&map_v);
      prefetch_tensormap(&map_do);
      int n_pub = 0;
      auto publish = [&](const Item& t) -> bool {
        const int slot = n_pub & (kFRing - 1);
        if (n_pub >= kFRing &&
            !mbar_wait(&bars->item_free[slot], (n_pub / kFRing - 1) & 1, abort_flag))
          return false;
        volatile int2& e = bars->ring[slot];
        e.x = t.kt;
        e.y = t.bh;
        mbar_arrive(&bars->item_ready[slot]);
        ++n_pub;
        return true;
      };
      // the first item is the CTA's own index; the counter hands out the rest
      auto decode = [&](int item) -> Item {
        return item < n_items ? decode_item(item, BH, n_tiles, group_bh) : Item{n_tiles, 0, 0};
      };
      Item t = decode(static_cast<int>(blockIdx.x));
      bool ok = publish(t);
      int g = 0, j = 0;
      for (; ok && t.n_it > 0; ++j) {
        // K / V go to the buffer of the item before last, once its products are through
        const int kb = j & 1;
        if (ok && j >= 2) ok = mbar_wait(&bars->kv_empty[kb], ((j >> 1) - 1) & 1, abort_flag);
        if (!ok) break;
        const int ub = t.bh / heads, uh = t.bh - ub * heads;   // (batch, head) of the unit
        mbar_arrive_expect_tx(&bars->kv_full[kb], 2 * kFPanel);
        tma_load_4d(smem + L::kK + kb * kFPanel, &map_k, &bars->kv_full[kb], 0, t.kt * kFT, uh, ub);
        tma_load_4d(smem + L::kV + kb * kFPanel, &map_v, &bars->kv_full[kb], 0, t.kt * kFT, uh, ub);
        // The following item (or the end mark) is claimed only now, and published at once: the
        // other roles look one item ahead. Every item a CTA holds in advance is work that no idle
        // CTA can take near the end of the kernel, so it holds as few as it can.
        const Item nxt = decode(static_cast<int>(gridDim.x) + atomicAdd(item_counter, 1));
        ok = publish(nxt);
        for (int i = 0; ok && i < t.n_it; ++i, ++g) {
          const int s = g % kFStages, use = g / kFStages;
          if (use > 0 && !(ok = mbar_wait(&bars->qdo_empty[s], (use - 1) & 1, abort_flag))) break;
          const int q0 = (t.kt + i) * kFT;
          mbar_arrive_expect_tx(&bars->qdo_full[s], 2 * kFPanel);
          tma_load_4d(smem + L::kQ + s * kFPanel, &map_q, &bars->qdo_full[s], 0, q0, uh, ub);
          tma_load_4d(smem + L::kDO + s * kFPanel, &map_do, &bars->qdo_full[s], 0, q0, uh, ub);
        }
        t = nxt;
      }
      settle_ring(bars->kv_full, 2, j);
      settle_ring(bars->qdo_full, kFStages, g);
    }
  } else if (warp == kWarpIssuer) {
    // ------------------------------ MMA issuer ------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_x = make_idesc_bf16(128, 128, 0, 0);   // S^T, dP^T: both K-major
      constexpr uint32_t idesc_t = make_idesc_bf16(128, 64, 0, 1);    // dV, dK: A in tensor memory, B MN-major
      constexpr uint32_t idesc_q = make_idesc_bf16(128, 64, 1, 1);    // dQ: A and B MN-major
      const SmemDescBase k0_desc = make_desc_base_sw128(smem_u32(smem + L::kK), 0);
      const SmemDescBase v0_desc = make_desc_base_sw128(smem_u32(smem + L::kV), 0);
      const SmemDescBase q0_desc = make_desc_base_sw128(smem_u32(smem + L::kQ), 0);
      const SmemDescBase do0_desc = make_desc_base_sw128(smem_u32(smem + L::kDO), 0);
      // dS^T read as MN-major A (M = queries): the two 64-query panels are kFPanel apart
      const SmemDescBase ds_t = make_desc_base_sw128(smem_u32(smem + L::kDS), kFPanel);

      // S^T = K Q^T of the tile in stage s (the g-th of this CTA), K / V buffer kb
      auto issue_s = [&](int g, int s, int kb) {
        const SmemDescBase qd{q0_desc.lo + s * (kFPanel >> 4), q0_desc.hi};
        const SmemDescBase kd{k0_desc.lo + kb * (kFPanel >> 4), k0_desc.hi};
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss(tmem + kColS, desc_at(kd, kk * 32), desc_at(qd, kk * 32), idesc_x, kk > 0 ? 1u : 0u);
        mma_commit(&bars->s_full[g & 1]);
      };
      // dP^T = V dO^T
      auto issue_dp = [&](int s, int kb) {
        const SmemDescBase dd{do0_desc.lo + s * (kFPanel >> 4), do0_desc.hi};
        const SmemDescBase vd{v0_desc.lo + kb * (kFPanel >> 4), v0_desc.hi};
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss(tmem + kColDP, desc_at(vd, kk * 32), desc_at(dd, kk * 32), idesc_x, kk > 0 ? 1u : 0u);
        mma_commit(&bars->dp_full);
      };

      ItemFeed feed{bars, abort_flag, n_tiles, 0};
      int n_it = feed.fetch().n_it, n_nxt = 0;
      bool ok = n_it > 0 && mbar_wait(&bars->kv_full[0], 0, abort_flag) && mbar_wait(&bars->qdo_full[0], 0, abort_flag);
      if (ok) {
        tc_fence_after_sync();
        issue_s(0, 0, 0);
        issue_dp(0, 0);
      }
      int g = 0, s = 0;          // tile and its stage
      uint32_t par = 0;          // parity of that stage's full barrier
      for (int j = 0; ok && n_it > 0; ++j) {
        const int kb = j & 1;
        for (int i = 0; ok && i < n_it; ++i, ++g) {
          const bool last = i + 1 == n_it;
          if (last) n_nxt = feed.fetch().n_it;   // (published when the producer came to this item)
          const int sn = s + 1 == kFStages ? 0 : s + 1;
          const uint32_t parn = sn == 0 ? par ^ 1u : par;
          const bool more = !last || n_nxt > 0;
          const int kbn = last ? kb ^ 1 : kb;
          const SmemDescBase qd{q0_desc.lo + s * (kFPanel >> 4), q0_desc.hi};
          const SmemDescBase dd{do0_desc.lo + s * (kFPanel >> 4), do0_desc.hi};
          const SmemDescBase kd{k0_desc.lo + kb * (kFPanel >> 4), k0_desc.hi};
          // P^T of this tile is there, and its scores have been read: dV += P^T dO, 16 queries per MMA, and
          // the next tile's scores (across an item boundary from the other K / V buffer), while dS is being
          // formed. A new item's first products overwrite dV / dK: the drain warps must have taken the
          // previous item's out of tensor memory.
          if (!(ok = mbar_wait(&bars->p_full, g & 1, abort_flag))) break;
          if (more && !(ok = (!last || mbar_wait(&bars->kv_full[kbn], ((j + 1) >> 1) & 1, abort_flag)) &&
                             mbar_wait(&bars->qdo_full[sn], parn, abort_flag)))
            break;
          tc_fence_after_sync();
          if (more) issue_s(g + 1, sn, kbn);
          if (i == 0 && j > 0) {
            if (!(ok = mbar_wait(&bars->dkv_drained, (j - 1) & 1, abort_flag))) break;
            tc_fence_after_sync();
          }
#pragma unroll
          for (int kk = 0; kk < kFT / 16; ++kk)
            mma_ts(tmem + kColDV, tmem + kColP + kk * 8, desc_at(dd, kk * 2048), idesc_t, (i > 0 || kk > 0) ? 1u : 0u);
          // dK += dS^T Q
          if (!(ok = mbar_wait(&bars->w_full, g & 1, abort_flag))) break;
          tc_fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < kFT / 16; ++kk)
            mma_ts(tmem + kColDK, tmem + kColDP + (kk / 2) * 32 + (kk % 2) * 8, desc_at(qd, kk * 2048), idesc_t,
                   (i > 0 || kk > 0) ? 1u : 0u);
          // dS^T has been read out of its columns once dK is through: the next tile's dP^T may follow
          if (more) issue_dp(sn, kbn);
          // Q and dO of this stage are last read by the products above
          mma_commit(&bars->qdo_empty[s]);
          // dQ = dS K, 16 keys per MMA. The previous tile's dQ must have left tensor memory before.
          if (g > 0 && !(ok = mbar_wait(&bars->dq_drained, (g - 1) & 1, abort_flag))) break;
          tc_fence_after_sync();
#pragma unroll
          for (int kk = 0; kk < kFT / 16; ++kk)
            mma_ss(tmem + kColDQ, desc_at(ds_t, kk * 2048), desc_at(kd, kk * 2048), idesc_q, kk > 0 ? 1u : 0u);
          mma_commit(&bars->acc_done);
          if (last) mma_commit(&bars->kv_empty[kb]);
          s = sn;
          par = parn;
        }
        n_it = n_nxt;
      }
      settle_products(&bars->settled);
    }
  } else if (warp == kWarpReducer) {
    // ------------------------------ dQ reducer / dK, dV writer ------------------------------
    if (elect_one()) {
      prefetch_tensormap(&map_dqw);
      const uint64_t keep = l2_policy_evict_last();
      prefetch_tensormap(&map_dk);
      prefetch_tensormap(&map_dv);
      ItemFeed feed{bars, abort_flag, n_tiles, 0};
      uint32_t turn = 0;   // parity of the staging panels' use
      auto hand_back = [&]() {
        bulk_wait_read<1>();
        mbar_arrive(&bars->sent[0]);
        bulk_wait_read<0>();
        mbar_arrive(&bars->sent[1]);
        turn ^= 1u;
      };
      bool ok = true;
      for (Item t = feed.fetch(); ok && t.n_it > 0; t = feed.fetch()) {
        for (int i = 0; ok && i < t.n_it; ++i) {
          const int q0 = (t.kt + i) * kFT, k0 = t.kt * kFT;
          if (i + 1 == t.n_it) {
            // The item is complete: dV and dK take a turn of the panels ahead of the last tile's dQ (one
            // each if the panels are fp32)
            const int ub = t.bh / heads, uh = t.bh - ub * heads;
            for (int a = 0; ok && a < (F32 ? 2 : 1); ++a) {
              for (int p = 0; ok && p < 2; ++p) {
                if (!(ok = mbar_wait(&bars->staged[p], turn, abort_flag))) break;
                if (F32) tma_store_3d(a ? &map_dk : &map_dv, smem + L::kDQ + p * kFPanel, p * 32, k0, t.bh);
                else tma_store_4d(p ? &map_dk : &map_dv, smem + L::kDQ + p * kFPanel, 0, k0, uh, ub);
                bulk_commit();
              }
              if (ok) hand_back();
            }
          }
          for (int p = 0; ok && p < 2; ++p) {
            if (!(ok = mbar_wait(&bars->staged[p], turn, abort_flag))) break;
            tma_reduce_add_3d(&map_dqw, smem + L::kDQ + p * kFPanel, p * 32, q0, t.bh, keep);
            bulk_commit();
          }
          if (ok) hand_back();
        }
      }
      bulk_wait0();   // every sum and store has landed before the CTA retires
    }
  } else {
    // ------------------------------ row scalars ------------------------------
    // -lse log2e and -delta scale of each tile's 128 queries, from memory through registers (a tile
    // ahead: the SM's path to L2 is busy with the reduce-adds) into one of two buffers. Queries beyond S
    // contribute nothing: p = exp2(-inf). Buffer g % 2 is free once the products of tile g - 2, which
    // follow the arithmetic that read it, have given their stage back; that barrier's next phase needs
    // this warp's scalars of tile g + 1.
    float* vec = reinterpret_cast<float*>(smem + L::kVec);
    ItemFeed feed{bars, abort_flag, n_tiles, 0};
    Item t = feed.fetch();
    Item nxt = t.n_it > 0 ? feed.fetch() : t;
    float rl[4], rd[4];
    auto request = [&](int q_tile, int bh) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int q = q_tile * kFT + c * 32 + lane;
        const int64_t at = static_cast<int64_t>(bh) * S + q;
        rl[c] = q < S ? lse[at] : INFINITY;
        rd[c] = q < S ? delta[at] : 0.f;
      }
    };
    if (t.n_it > 0) request(t.kt, t.bh);
    bool ok = true;
    int g = 0, s2 = kFStages - 2;   // the tile; stage of tile g - 2
    uint32_t par2 = 1;              // and the parity of that use
    while (ok && t.n_it > 0) {
      for (int i = 0; i < t.n_it; ++i, ++g) {
        if (g >= 2 && !(ok = mbar_wait(&bars->qdo_empty[s2], par2, abort_flag))) break;
        if (++s2 == kFStages) s2 = 0, par2 ^= 1u;
        float* dst = vec + (g & 1) * (2 * kFT) + lane;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          dst[c * 32] = -rl[c] * kFLog2e;
          dst[kFT + c * 32] = -rd[c] * scale;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->s_full[g & 1]);
        if (i + 1 < t.n_it) {
          request(t.kt + i + 1, t.bh);
        } else if (nxt.n_it > 0) {
          request(nxt.kt, nxt.bh);
        }
      }
      t = nxt;
      if (ok && t.n_it > 0) nxt = feed.fetch();
    }
  }
  } else if (warp >= kWarpDrain0) {
    // ------------------------------ accumulator drain warps ------------------------------
    setmaxnreg_dec<kRegsDrain>();
    const int quad = warp % 4;
    const int row = quad * 32 + lane;     // TMEM lane = query row (dQ) or key row (dK / dV)
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    ItemFeed feed{bars, abort_flag, n_tiles, 0};
    bool ok = true;
    int g = 0;
    uint32_t back = 1;   // parity of the staging panels' return from their last use (none yet: passes)
    // 32 fp32 accumulator columns -> a swizzled panel [128 rows][32 fp32]
    auto stage_f32 = [&](const uint32_t (&o)[32], int p) {
      uint8_t* dst = smem + L::kDQ + p * kFPanel + row * 128;
#pragma unroll
      for (int c4 = 0; c4 < 8; ++c4)
        *reinterpret_cast<uint4*>(dst + ((c4 ^ (row & 7)) << 4)) =
            make_uint4(o[4 * c4], o[4 * c4 + 1], o[4 * c4 + 2], o[4 * c4 + 3]);
      fence_proxy_async_smem();
      mbar_arrive(&bars->staged[p]);
    };
    // 64 accumulator columns through both panels as fp32; `drained` gets an arrival once they are read
    auto turn_f32 = [&](uint32_t col, uint64_t* drained) -> bool {
#pragma unroll 1
      for (int p = 0; p < 2; ++p) {
        uint32_t o[32];
        tmem_ld32(tlane + col + p * 32, o);
        tmem_wait_ld();
        if (p == 1 && drained) {
          tc_fence_before_sync();
          mbar_arrive(drained);
        }
        if (!mbar_wait(&bars->sent[p], back, abort_flag)) return false;
        stage_f32(o, p);
      }
      back ^= 1u;
      return true;
    };
    for (Item t = feed.fetch(); ok && t.n_it > 0; t = feed.fetch()) {
      for (int i = 0; i < t.n_it; ++i, ++g) {
        if (!(ok = mbar_wait(&bars->acc_done, g & 1, abort_flag))) break;
        tc_fence_after_sync();
        if (i + 1 == t.n_it) {
          // The item is complete: dV and dK leave through the dQ staging panels, ahead of this tile's dQ.
          // (Staged in the item's own K / V buffers, they held up the K / V loads of the item after next:
          // short items waited 5000 clocks for theirs.) dkv_drained: the next item's products may overwrite.
          if (F32) {
            if (!(ok = turn_f32(kColDV, nullptr) && turn_f32(kColDK, &bars->dkv_drained))) break;
          } else {
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {   // 32 columns at a time; dV is columns [0, 64), dK [64, 128)
              uint32_t o[32];
              tmem_ld32(tlane + kColDV + c * 32, o);   // kColDK = kColDV + 64
              tmem_wait_ld();
              if (c == 3) {
                tc_fence_before_sync();
                mbar_arrive(&bars->dkv_drained);
              }
              const int p = c / 2;
              if ((c & 1) == 0 && !(ok = mbar_wait(&bars->sent[p], back, abort_flag))) break;
              uint8_t* dst = smem + L::kDQ + p * kFPanel + row * 128;
#pragma unroll
              for (int h = 0; h < 4; ++h)
                *reinterpret_cast<uint4*>(dst + ((((c & 1) * 4 + h) ^ (row & 7)) << 4)) = make_uint4(
                    pack_bf16(__uint_as_float(o[8 * h + 0]), __uint_as_float(o[8 * h + 1])),
                    pack_bf16(__uint_as_float(o[8 * h + 2]), __uint_as_float(o[8 * h + 3])),
                    pack_bf16(__uint_as_float(o[8 * h + 4]), __uint_as_float(o[8 * h + 5])),
                    pack_bf16(__uint_as_float(o[8 * h + 6]), __uint_as_float(o[8 * h + 7])));
              if (c & 1) {
                fence_proxy_async_smem();
                mbar_arrive(&bars->staged[p]);
              }
            }
            if (!ok) break;
            back ^= 1u;
          }
        }
        // dQ of the tile: tensor memory -> swizzled fp32 staging, a panel of 32 columns at a time, which
        // the reducer warp sends on: one panel is staged while the other is being read. dq_drained: the
        // next tile's dQ may overwrite this one.
        if (!(ok = turn_f32(kColDQ, &bars->dq_drained))) break;
      }
    }
  } else {
    // ------------------------------ compute warps ------------------------------
    setmaxnreg_inc<kRegsCompute>();
    const int quad = warp % 4;            // TMEM lane quadrant of this warp
    const int cg = warp / 4;              // which 32 query columns of the 128
    const int row = quad * 32 + lane;     // key row within the tile = TMEM lane
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const float scale_log2 = scale * kFLog2e;
    const float keep_scale = DROP ? 1.0f / (1.0f - rate) : 1.0f, grad_scale = scale * keep_scale;
    uint8_t* ds_row = smem + L::kDS + (cg / 2) * kFPanel + row * 128;
    const float* vec = reinterpret_cast<const float*>(smem + L::kVec) + cg * 32;
    bool ok = true;

    // Keep bits: bit 8 b + 7 - k of a lane's word is for query 4 k + b of its 32, so that k shifts to the
    // left bring those of queries 4 k .. 4 k + 3 to the four bytes' signs, from where one prmt makes a mask.
    // From a drawn mask (DROP 2) this lane fetches the word of one query for the warp's 32 keys; a 32 x 32
    // bit transposition across the warp turns it round.
    auto transpose_bits = [&](uint32_t w) -> uint32_t {
      uint32_t m = 0x0000ffffu;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1, m ^= m << d) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, w, d);
        w = (lane & d) ? ((w & ~m) | ((o >> d) & m)) : ((w & m) | ((o & m) << d));
      }
      return w;
    };

    ItemFeed feed{bars, abort_flag, n_tiles, 0};
    int g = 0;

    for (Item t = feed.fetch(); ok && t.n_it > 0; t = feed.fetch()) {
      for (int i = 0; i < t.n_it; ++i, ++g) {
        const bool diagonal = (i == 0);
        uint32_t keep_word = 0u;
        if (DROP == 2)   // (there by the time the exponentials are done)
          keep_word = __ldg(mask_bits + mask_bits_record(t.bh, t.kt + i, t.kt, cg * 32 + 4 * (7 - (lane & 7)) + (lane >> 3), n_tiles) * 4 + quad);
        // the scores and the tile's row scalars
        if (!(ok = mbar_wait(&bars->s_full[g & 1], (g >> 1) & 1, abort_flag))) break;
        tc_fence_after_sync();
        const float* v_lse = vec + (g & 1) * (2 * kFT);
        const float* v_delta = v_lse + kFT;
        uint32_t x[32];   // S^T, then p
        tmem_ld32(tlane + kColS + cg * 32, x);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          const float4 l = *reinterpret_cast<const float4*>(v_lse + c);   // (all lanes want the same four)
          const float2 e0 = ffma2(make_float2(__uint_as_float(x[c]), __uint_as_float(x[c + 1])),
                                  make_float2(scale_log2, scale_log2), make_float2(l.x, l.y));
          const float2 e1 = ffma2(make_float2(__uint_as_float(x[c + 2]), __uint_as_float(x[c + 3])),
                                  make_float2(scale_log2, scale_log2), make_float2(l.z, l.w));
          x[c] = __float_as_uint(ex2(e0.x));
          x[c + 1] = __float_as_uint(ex2(e0.y));
          x[c + 2] = __float_as_uint(ex2(e1.x));
          x[c + 3] = __float_as_uint(ex2(e1.y));
        }
        // The causal compare only exists on an item's first tile. (Behind the exponentials: a score of -inf would
        // be p = NaN where the query's lse is, and with it dV of keys that the query does not see.)
        if (diagonal) {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (row > cg * 32 + c) x[c] = 0u;
        }

        if (DROP == 1 && (!diagonal || quad <= cg)) {   // (beyond the diagonal there is nothing to drop)
          const uint64_t q = static_cast<uint64_t>(t.kt + i) * kFT + cg * 32;
          const uint64_t idx = (static_cast<uint64_t>(unit0 + t.bh) * S + q) * S + t.kt * kFT + row;
#pragma unroll 4
          for (int c = 0; c < 32; ++c)
            keep_word |= (philox_keep(rng, idx + static_cast<uint64_t>(c) * S, rate) ? 1u : 0u) << (8 * (c & 3) + 7 - (c >> 2));
        }
        if (DROP == 2) keep_word = transpose_bits(keep_word);
        // dP^T of this tile follows dV of the tile before, whose P^T has then been read
        if (!(ok = mbar_wait(&bars->dp_full, g & 1, abort_flag))) break;
        tc_fence_after_sync();
        uint32_t w[16];   // 32 queries = 16 packed columns = two K steps of the dV / dK products
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
          float2 p0 = make_float2(__uint_as_float(x[c]), __uint_as_float(x[c + 1]));
          float2 p1 = make_float2(__uint_as_float(x[c + 2]), __uint_as_float(x[c + 3]));
          if (DROP) {
            p0 = fmul2(p0, make_float2(keep_scale, keep_scale));
            p1 = fmul2(p1, make_float2(keep_scale, keep_scale));
          }
          w[c / 2] = pack_bf16(p0.x, p0.y);
          w[c / 2 + 1] = pack_bf16(p1.x, p1.y);
          if (DROP) {
            w[c / 2] &= byte_signs<0x9988>(keep_word << (c / 4));
            w[c / 2 + 1] &= byte_signs<0xbbaa>(keep_word << (c / 4));
          }
        }
        tmem_st16(tlane + kColP + cg * 16, w);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(&bars->p_full);   // (the scores are in registers, too: the next tile's may overwrite them)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t x2[16];
          tmem_ld16(tlane + kColDP + cg * 32 + h * 16, x2);
          tmem_wait_ld();
          // ds = p (dP - delta) scale as p * fma(dP, scale, -delta scale)
#pragma unroll
          for (int c = 0; c < 16; c += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(v_delta + h * 16 + c);
            uint32_t* gr = x2 + c;
            if (DROP) {
              const uint32_t k4 = keep_word << (h * 4 + c / 4);
              gr[0] &= byte_signs<0x8888>(k4);
              gr[1] &= byte_signs<0x9999>(k4);
              gr[2] &= byte_signs<0xaaaa>(k4);
              gr[3] &= byte_signs<0xbbbb>(k4);
            }
            const int at = h * 16 + c;
            const float2 ds0 = fmul2(make_float2(__uint_as_float(x[at]), __uint_as_float(x[at + 1])),
                                     ffma2(make_float2(__uint_as_float(gr[0]), __uint_as_float(gr[1])),
                                           make_float2(grad_scale, grad_scale), make_float2(d4.x, d4.y)));
            const float2 ds1 = fmul2(make_float2(__uint_as_float(x[at + 2]), __uint_as_float(x[at + 3])),
                                     ffma2(make_float2(__uint_as_float(gr[2]), __uint_as_float(gr[3])),
                                           make_float2(grad_scale, grad_scale), make_float2(d4.z, d4.w)));
            w[at / 2] = pack_bf16(ds0.x, ds0.y);
            w[at / 2 + 1] = pack_bf16(ds1.x, ds1.y);
          }
        }
        // dS^T of tile g-1 consumed
        if (g > 0) {
          if (!(ok = mbar_wait(&bars->acc_done, (g - 1) & 1, abort_flag))) break;
          tc_fence_after_sync();
        }
        tmem_st16(tlane + kColDP + cg * 32, w);
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          const int chunk = (cg & 1) * 4 + v4;  // 16-byte chunk within the 128-byte row of the panel
          *reinterpret_cast<uint4*>(ds_row + ((chunk ^ (row & 7)) << 4)) =
              make_uint4(w[4 * v4], w[4 * v4 + 1], w[4 * v4 + 2], w[4 * v4 + 3]);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        fence_proxy_async_smem();
        mbar_arrive(&bars->w_full);
      }
      if (!ok) break;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kWarpIssuer) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (threadIdx.x == 0 && bars->abort_flag) report_timeout(status, bars->abort_flag);
}

// delta[r] = sum_d dO[r,d] O[r,d] (reference flash_delta_kernel, cuda/attention.cu:76-85) and the
// zero fill of the fp32 dQ workspace, in one pass over the rows. The fill waits for the kernel ahead
// like every other access: the workspace may lie where that kernel still reads or writes (an arena
// hands its bytes on from call to call), and kernels release their dependents before they are done.
// Blocks take the rows from the end, here and in the pass that rounds: the gradient kernel starts with the first units,
// whose lines are then the last to have come into L2, and leaves those of the last ones there (192 x 1024 step 168.9
// -> 167.7 us, behind fp32 tensors 74.1 -> 73.7).
template <bool INTERLEAVED>
__global__ void fused_prepare_kernel(float* __restrict__ delta, float* __restrict__ dq_ws,
                                     int* __restrict__ item_counter,
                                     const __nv_bfloat16* __restrict__ dout,
                                     const __nv_bfloat16* __restrict__ out, int64_t rows, int S,
                                     UnitLayout lay) {
  constexpr int D = kFD, Lr = D / 8;  // 8 lanes per row
  const int64_t t = static_cast<int64_t>(gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t r = t / Lr;   // row of the [BH, S] index space: delta and the workspace are heads-split
  const int c = static_cast<int>(t % Lr) * 8;
  pdl_wait();
  pdl_launch_dependents();
  if (t == 0) *item_counter = 0;
  float sum = 0.f;
  if (r < rows) {
    zero_32_bytes(dq_ws + r * D + c);   // (whole sectors)
    // where row r = (unit, s) lies in dO and O: heads-split rows are simply consecutive
    int64_t at = r * D + c;
    if (INTERLEAVED) {
      // (32-bit: 2^31 rows would be 274 GB of bf16, and 64-bit divisions took a fifth of this pass's time)
      const int unit = static_cast<uint32_t>(r) / static_cast<uint32_t>(S), srow = static_cast<int>(r) - unit * S;
      const int ub = unit / lay.heads, uh = unit - ub * lay.heads;
      at = ub * lay.batch + uh * lay.head + srow * lay.row + c;
    }
    const uint4 a = *reinterpret_cast<const uint4*>(dout + at);
    const uint4 b = *reinterpret_cast<const uint4*>(out + at);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sum = fmaf(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), sum);
      sum = fmaf(__uint_as_float(aw[i] & 0xffff0000u), __uint_as_float(bw[i] & 0xffff0000u), sum);
    }
  }
#pragma unroll
  for (int o = Lr / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (r < rows && c == 0) delta[r] = sum;
}

// dQ workspace (fp32) -> dq (bf16). The sums are read for the last time: their lines, which would go out to memory
// in the middle of later kernels (50 MB at 192 x 1024, of the step's 490 MB of memory traffic), are dropped. Step at
// 192 x 1024 154.5 -> 152.1 us, 24 x 512 29.9 -> 28.9.
template <bool INTERLEAVED>
__global__ void fused_convert_kernel(__nv_bfloat16* __restrict__ dq, float* __restrict__ dq_ws,
                                     int64_t n8, int S, UnitLayout lay) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = static_cast<int64_t>(gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n8) return;
  float4 a, b;
  load_32_bytes(dq_ws + t * 8, a, b);
  // workspace row r = (unit, s), 8 elements at column c; heads-split dq has the same order
  int64_t at = t * 8;
  if (INTERLEAVED) {
    const int64_t r = t / (kFD / 8);
    const int c = static_cast<int>(t - r * (kFD / 8)) * 8;
    const int unit = static_cast<uint32_t>(r) / static_cast<uint32_t>(S), srow = static_cast<int>(r) - unit * S;
    const int ub = unit / lay.heads, uh = unit - ub * lay.heads;
    at = ub * lay.batch + uh * lay.head + srow * lay.row + c;
  }
  *reinterpret_cast<uint4*>(dq + at) =
      make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
  __syncwarp();   // (the line's four readers have their values; they are there together, a row being eight lanes)
  if (t % 4 == 0) discard_line(dq_ws + t * 8);
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 3-D map over the fp32 workspace [BH, S, 64] with a 32 x 128 x 1 box and 128-byte swizzle
int make_dq_workspace_map(CUtensorMap* map, float* ws, int BH, int S) {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  if (!fn) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[3] = {kFD, static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(BH)};
  const cuuint64_t strides[2] = {kFD * 4, static_cast<cuuint64_t>(S) * kFD * 4};
  const cuuint32_t box[3] = {32, kFT, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, ws, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return DADATTN_OK;
}

}  // namespace
}  // namespace dadattn
namespace dadattn {

// Workspace: delta [BH,S] fp32, then the dQ accumulator [BH,S,64] fp32 (256-byte aligned), then
// 256 bytes that hold the work-item counter.
size_t fused_bwd_workspace_bytes(int BH, int S) {
  const size_t delta_bytes = (static_cast<size_t>(BH) * S * sizeof(float) + 255) / 256 * 256;
  const size_t dq_bytes = (static_cast<size_t>(BH) * S * kFD * sizeof(float) + 255) / 256 * 256;
  return delta_bytes + dq_bytes + 256;
}

// The gradient kernel on bf16 tensors, with delta and the item counter (and a zero-filled dq_ws) ready.
// f32_dk / f32_dv: fp32 results [BH,S,64] instead of bf16 dk / dv.
static int launch_fused_kernel(float* dq_ws, uint16_t* dk, uint16_t* dv, float* f32_dk, float* f32_dv, const float* delta,
                               int* item_counter, const uint16_t* dout, const float* lse, const uint16_t* q,
                               const uint16_t* k, const uint16_t* v, int BH, int S, const UnitLayout& lay, float scale,
                               float rate, const PhiloxKey& rng, int64_t unit0, const uint32_t* mask_bits,
                               cudaStream_t st) {
  CUtensorMap mq, mk, mv, mdo, mws, mdk, mdv;
  if (int rc = make_tensor_map_bf16_units(&mq, q, BH, S, kFD, kFT, lay)) return rc;
  if (int rc = make_tensor_map_bf16_units(&mk, k, BH, S, kFD, kFT, lay)) return rc;
  if (int rc = make_tensor_map_bf16_units(&mv, v, BH, S, kFD, kFT, lay)) return rc;
  if (int rc = make_tensor_map_bf16_units(&mdo, dout, BH, S, kFD, kFT, lay)) return rc;
  if (f32_dk) {
    if (int rc = make_dq_workspace_map(&mdk, f32_dk, BH, S)) return rc;
    if (int rc = make_dq_workspace_map(&mdv, f32_dv, BH, S)) return rc;
  } else {
    if (int rc = make_tensor_map_bf16_units(&mdk, dk, BH, S, kFD, kFT, lay)) return rc;
    if (int rc = make_tensor_map_bf16_units(&mdv, dv, BH, S, kFD, kFT, lay)) return rc;
  }
  if (int rc = make_dq_workspace_map(&mws, dq_ws, BH, S)) return rc;
  if (static_cast<int64_t>(BH) * S > INT32_MAX - 1024)
    return fail(DADATTN_E_UNSUPPORTED, "BH * S = %lld rows exceed what the fused backward addresses",
                static_cast<long long>(BH) * S);
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  // One persistent CTA per SM; the CTAs draw (key tile, batch x head) items from a counter.
  // Batch x head units are worked on in even groups whose Q, dO and dQ rows (1 KiB per query) stay
  // well inside L2; in one where all of them fit, since every group but the last ends on its short items.
  const int64_t n_items = static_cast<int64_t>((S + kFT - 1) / kFT) * BH;
  if (n_items > INT32_MAX / 2) return fail(DADATTN_E_UNSUPPORTED, "too many (key tile, batch x head) items");
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  dim3 grid(static_cast<unsigned>(n_items < sms ? n_items : sms));
  const int group_bh = static_cast<int64_t>(BH) * S <= kFAllInL2 ? BH : leveled_grid(65536, S, BH).group;
  const int variant = f32_dk ? 3 : rate > 0.f ? (mask_bits ? 2 : 1) : 0;
  auto kern = variant == 3 ? flash_bwd_fused_kernel<0, true> : variant == 2 ? flash_bwd_fused_kernel<2, false>
              : variant == 1 ? flash_bwd_fused_kernel<1, false> : flash_bwd_fused_kernel<0, false>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FusedSmem::kBytes));
  static std::atomic<int> regs_seen[4];
  if (int rc = check_launch_registers(reinterpret_cast<const void*>(kern), kRegsLaunch, regs_seen[variant])) return rc;
  DAD_CUDA(launch_pdl(kern, grid, dim3(kFThreads), FusedSmem::kBytes, st, mq, mk, mv, mdo, mws, mdk, mdv,
                      lse, delta, item_counter, BH, S, lay.heads, group_bh, scale, rate,
                      rng, unit0, mask_bits, status));
  return DADATTN_OK;
}

// fp32 results on bf16 operands: dq32 (zero-filled by the caller of this function) collects dQ, delta
// and the zeroed item counter are ready in the caller's workspace.
int launch_bwd_fused_d64_f32(float* dq32, float* dk32, float* dv32, const float* delta, int* item_counter,
                             const uint16_t* dout, const float* lse, const uint16_t* q, const uint16_t* k,
                             const uint16_t* v, int BH, int S, float scale, cudaStream_t st) {
  return launch_fused_kernel(dq32, nullptr, nullptr, dk32, dv32, delta, item_counter, dout, lse, q, k, v, BH, S,
                             unit_layout(BH, 1, S, kFD, false), scale, 0.f, PhiloxKey{}, 0, nullptr, st);
}

int launch_bwd_fused_d64(uint16_t* dq, uint16_t* dk, uint16_t* dv, void* workspace, const uint16_t* dout,
                         const uint16_t* out, const float* lse, const uint16_t* q, const uint16_t* k,
                         const uint16_t* v, int BH, int S, float scale, float rate, uint64_t seed,
                         uint64_t offset, int64_t unit0, const uint32_t* mask_bits, int heads,
                         cudaStream_t st) {
  using BF = __nv_bfloat16;
  // heads > 0: every bf16 tensor is the interleaved [B*S, heads*64] activation (BH = B * heads)
  const UnitLayout lay = heads > 0 ? unit_layout(BH / heads, heads, S, kFD, true) : unit_layout(BH, 1, S, kFD, false);
  const size_t delta_bytes = (static_cast<size_t>(BH) * S * sizeof(float) + 255) / 256 * 256;
  const size_t dq_bytes = (static_cast<size_t>(BH) * S * kFD * sizeof(float) + 255) / 256 * 256;
  float* delta = static_cast<float*>(workspace);
  float* dq_ws = reinterpret_cast<float*>(static_cast<char*>(workspace) + delta_bytes);
  int* item_counter = reinterpret_cast<int*>(static_cast<char*>(workspace) + delta_bytes + dq_bytes);
  const int64_t rows = static_cast<int64_t>(BH) * S;
  const int64_t prep_threads = rows * (kFD / 8);
  stage_event(0, st);
  DAD_CUDA(launch_pdl(heads > 0 ? fused_prepare_kernel<true> : fused_prepare_kernel<false>,
                      dim3(static_cast<unsigned>((prep_threads + 255) / 256)),
                      dim3(256), 0, st, delta, dq_ws, item_counter, reinterpret_cast<const BF*>(dout),
                      reinterpret_cast<const BF*>(out), rows, S, lay));
  stage_event(1, st);
  if (int rc = launch_fused_kernel(dq_ws, dk, dv, nullptr, nullptr, delta, item_counter, dout, lse, q, k, v, BH, S, lay,
                                   scale, rate, make_philox(seed, offset), unit0, mask_bits, st))
    return rc;
  stage_event(2, st);
  const int64_t n8 = rows * kFD / 8;
  DAD_CUDA(launch_pdl(heads > 0 ? fused_convert_kernel<true> : fused_convert_kernel<false>,
                      dim3(static_cast<unsigned>((n8 + 255) / 256)), dim3(256), 0,
                      st, reinterpret_cast<BF*>(dq), dq_ws, n8, S, lay));
  stage_event(3, st);
  return DADATTN_OK;
}

}  // namespace dadattn
