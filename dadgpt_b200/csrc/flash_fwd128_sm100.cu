// bf16 fused causal attention forward for sm_100a, head size 128, launches that fill the GPU: persistent CTAs that work
// on TWO 128-row query tiles at a time, each with one thread per row.
//
// The arithmetic is that of the reference's flash_fwd_kernel (cuda/attention.cu:17-73: online softmax over key
// tiles, lse = max + ln(sum) of the scaled scores) with bf16 operands and fp32 accumulation. A 128x128 score tile
// costs 1024 clocks of tensor pipe and 1024 of the exp2 unit. What the one-tile kernel of flash_bf16_sm100.cu needs
// on top is latency: its softmax warps are all in the same phase, so that the exp2 unit is idle while they look for
// the maximum, and a CTA's start and end, some 6000 clocks, are nobody else's work. So:
//   * a work item is a PAIR of adjacent query tiles (A = tile 2p, B = tile 2p + 1) of one (batch, head). Both use
//     the same K / V tiles from one ring (shared memory: 1024 clocks a tile instead of 1280), and each has its own
//     softmax warpgroup, scores and accumulator in tensor memory and issuing thread: while A's threads compute
//     exponentials the tensor pipe runs B's products and vice versa. Sequences of one tile: that tile of two units;
//   * one thread per row: no statistics to exchange, one accumulator per tile (a second one for each half of a
//     row would not fit beside two tiles' scores). Its 128 scores are read once and stay in registers. Launches
//     that do not fill the GPU take the one-tile kernel of flash_bf16_sm100.cu, in a form that gives the same bits. (Two threads
//     per row, sixteen softmax warps, with the maximum agreed by a barrier of two warps: 192 x 1024 72.4 us instead
//     of 70, 192 x 128 10.2 instead of 9.0);
//   * the probabilities go back over the scores as packed bf16, and the P V product of the first 64 keys is issued
//     while the second 64 are being computed;
//   * CTAs are persistent and take items from the grid's own queue (clusterlaunchcontrol): the launch has one block
//     per item, heaviest first inside a group of units whose K and V fit L2 (LeveledGrid), and a CTA that is about
//     through with an item takes over the next block that has not started. K / V of the next item are on their
//     way while the current one finishes; a group's Q is loaded as soon as its results have left, which go through
//     the Q tile's shared memory and TMA.
// A pair of tiles takes about 3600 clocks (traced): both groups' exponentials end up at the same time, 2100 clocks of
// the exp2 unit for the two, and so do their products. What it measured against the one-tile kernel stands at the
// rule (fwd128_pairs_pay).
//   warp 0       scheduler + K / V producer        warp 1     issuer of group A, tensor memory
//   warp 2       issuer of group B                 warp 3     Q producer
//   warps 4-7    softmax group A                   warps 8-11 softmax group B
//
// Every mbarrier wait is bounded (sm100_ptx.cuh); on expiry the CTA raises its abort flag, all roles fall through
// to the common exit, tensor memory is freed and DADATTN_E_TIMEOUT is left in the device status word.
#include <cuda_bf16.h>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

using namespace ptx;

constexpr int kT = 128;                 // tile edge: query rows per group, keys per K/V tile
constexpr int kHD = 128;                // head size
constexpr int kPanel = 128 * 128;       // [128 rows][64 bf16]: 16 KB, 128-byte rows, swizzled
constexpr int kTileBytes = 2 * kPanel;
constexpr int kSlots = 5;               // ring of K and V tiles, K0 V0 K1 V1 ...
constexpr int kRing = 4;                // items a CTA knows of (a power of two)
constexpr int kThreads = 12 * 32;
constexpr int kGroup = 128;             // threads of a softmax group
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleAt = 8.0f;      // log2 units: O is rescaled only when the max grew by 2^8
// Registers per thread once the warpgroups have rebalanced (a softmax thread holds 128 scores).
constexpr int kRegsLaunch = 168, kRegsSoftmax = 208, kRegsHelper = 88;
static_assert(2 * kGroup * kRegsSoftmax + 128 * kRegsHelper <= kThreads * kRegsLaunch,
              "the warpgroups ask for more registers than the CTA owns");
static_assert(kThreads * kRegsLaunch <= 65536 && (kRegsLaunch + 8) * kThreads > 65536,
              "kRegsLaunch is not what the compiler gives a CTA of this size");

struct F128Smem {
  static constexpr int kQ = 0;                              // [A, B]
  static constexpr int kKV = kQ + 2 * kTileBytes;
  static constexpr int kBars = kKV + kSlots * kTileBytes;
  static constexpr int kBytes = kBars + 512;
  static_assert(kBytes <= 232448, "shared memory budget of one CTA exceeded");
};

struct F128Bars {
  __align__(16) uint4 stolen;             // answer to a request for another block
  uint64_t stolen_full;
  uint64_t item_ready[kRing], item_free[kRing];
  uint64_t q_full[2], q_empty[2], slot_full[kSlots], slot_empty[kSlots];
  uint64_t s_full[2], p_full[2][2], o_done[2], settled[2];   // [group]; p_full: [group][half of the keys]
  int2 ring[kRing];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(F128Bars) <= 512, "barrier block");

// ---- the grid's queue -------------------------------------------------------------------------------
// Asks for a block of this grid that has not started yet, in its place; the answer (16 bytes) completes on `bar`.
// Not asked again once the answer was that there is none.
__device__ __forceinline__ void request_block(uint4* answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool read_answer(const uint4* answer, dim3& block) {
  uint32_t ok, x = 0, y = 0, z = 0;
  asm volatile(
      "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 h, [%4];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, h;\n\t}"
      : "=&r"(ok), "=&r"(x), "=&r"(y), "=&r"(z)
      : "r"(smem_u32(answer))
      : "memory");
  block = dim3(x, y, z);
  return ok != 0;
}

// Level `level` of unit (or, ONE, pair of units) `u`: query tiles qa and qa + 1, the heaviest pair first, as group x
// sees it. Every role reads the CTA's items, in order, from the ring that the scheduler fills; n_kv = 0 marks the end.
struct F128Item {
  int unit, q0, n;   // n: key tiles (0: nothing to do for this group)
  int first;         // ring tile of the group's first key tile
  int n_kv;          // K / V tiles that go through the ring
};
template <bool ONE>
__device__ __forceinline__ F128Item f128_item(int u, int level, int x, int BH, int n_tiles) {
  if (level < 0) return F128Item{0, 0, 0, 0, 0};
  if (ONE) {
    const int both = 2 * u + 1 < BH;
    return F128Item{2 * u + x, 0, x ? both : 1, x ? both : 0, 1 + both};
  }
  const int qa = 2 * ((n_tiles + 1) / 2 - 1 - level), both = qa + 1 < n_tiles;
  return F128Item{u, (qa + x) * kT, x ? (both ? qa + 2 : 0) : qa + 1, 0, qa + 1 + both};
}

template <bool ONE>
struct F128Feed {
  F128Bars* bars;
  volatile int* abort_flag;
  int BH, n_tiles, n_read;
  __device__ __forceinline__ int2 next() {   // (unit, level)
    const int slot = n_read & (kRing - 1);
    if (!mbar_wait(&bars->item_ready[slot], (n_read / kRing) & 1, abort_flag)) return make_int2(0, -1);
    const volatile int2& e = bars->ring[slot];
    const int2 item = make_int2(e.x, e.y);
    mbar_arrive(&bars->item_free[slot]);
    ++n_read;
    return item;
  }
  __device__ __forceinline__ F128Item fetch(int x) {
    const int2 item = next();
    return f128_item<ONE>(item.x, item.y, x, BH, n_tiles);
  }
};

// Which slot of the ring a tile is in, and the parity of that use.
struct RingAt {
  int slot;
  uint32_t parity;
  __device__ __forceinline__ void next() {
    if (++slot == kSlots) slot = 0, parity ^= 1u;
  }
};

// ONE: sequences of one tile, a unit for each group.
template <bool ONE>
__global__ void __launch_bounds__(kThreads, 1)
flash_fwd128_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                    float* __restrict__ lse, int BH, int S, float scale, LeveledGrid order, int* __restrict__ status) {
  using L = F128Smem;
  // Tensor memory: the scores of group X at 128 X (its probabilities in the first 64 columns of them), O at 256 + 128 X.
  constexpr uint32_t kTmemCols = 512, kColS = 0, kColO = 256;

  extern __shared__ __align__(1024) uint8_t smem[];
  F128Bars* bars = reinterpret_cast<F128Bars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_tiles = (S + kT - 1) / kT;

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicExch(status, DADATTN_E_CUDA);
    return;
  }
  if (threadIdx.x == 0) {
    mbar_init(&bars->stolen_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&bars->item_ready[i], 1);
      mbar_init(&bars->item_free[i], 2 * kGroup + 3);   // softmax, issuers, Q producer
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&bars->slot_full[i], 1);
      mbar_init(&bars->slot_empty[i], 2);               // one arrival per issuer
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(&bars->q_full[x], 1);
      mbar_init(&bars->q_empty[x], 4);                  // one arrival per warp
      mbar_init(&bars->s_full[x], 1);
      mbar_init(&bars->p_full[x][0], kGroup);
      mbar_init(&bars->p_full[x][1], kGroup);
      mbar_init(&bars->o_done[x], 1);
      mbar_init(&bars->settled[x], 1);
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
  pdl_wait();
  pdl_launch_dependents();

  F128Feed<ONE> feed{bars, abort_flag, BH, n_tiles, 0};
  if (warp < 4) {
    setmaxnreg_dec<kRegsHelper>();
    if (warp == 0) {
      // ------------------------------ scheduler + K / V producer ------------------------------
      if (elect_one()) {
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        int n_pub = 0, n_asked = 0, n_loaded = 0;
        bool ok = true;
        auto publish = [&](int u, int level) -> bool {
          const int slot = n_pub & (kRing - 1);
          if (n_pub >= kRing && !mbar_wait(&bars->item_free[slot], (n_pub / kRing - 1) & 1, abort_flag)) return false;
          volatile int2& e = bars->ring[slot];
          e.x = u;
          e.y = level;
          mbar_arrive(&bars->item_ready[slot]);
          ++n_pub;
          return true;
        };
        auto ask = [&]() {
          fence_proxy_async_smem();   // (the last answer has been read)
          mbar_arrive_expect_tx(&bars->stolen_full, 16);
          request_block(&bars->stolen, &bars->stolen_full);
          ++n_asked;
        };
        // the answer; level = -1: nothing left (or given up)
        auto answer = [&](int& u, int& level) -> bool {
          level = -1;
          if (!mbar_wait(&bars->stolen_full, (n_asked - 1) & 1, abort_flag)) return false;
          dim3 b;
          if (!read_answer(&bars->stolen, b)) return true;
          if (!leveled_item(order, b, level, u)) level = -2;   // a block that pads the last group
          return true;
        };
        int u, level;
        bool mine = leveled_item(order, blockIdx, level, u);
        while (ok && !mine) {
          ask();
          ok = answer(u, level);
          mine = level != -2;
        }
        RingAt at{0, 0};
        ok = ok && publish(u, level);
        while (ok && level >= 0) {
          const int n_kv = f128_item<ONE>(u, level, 0, BH, n_tiles).n_kv;
          for (int j = 0; ok && j < n_kv; ++j) {
            const int unit = ONE ? 2 * u + j : u, row = ONE ? 0 : j * kT;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (n_loaded >= kSlots && !(ok = mbar_wait(&bars->slot_empty[at.slot], at.parity ^ 1u, abort_flag))) break;
              mbar_arrive_expect_tx(&bars->slot_full[at.slot], kTileBytes);
              for (int p = 0; p < 2; ++p)
                tma_load_3d(smem + L::kKV + at.slot * kTileBytes + p * kPanel, m ? &map_v : &map_k,
                            &bars->slot_full[at.slot], p * 64, row, unit);
              ++n_loaded;
              at.next();
            }
          }
          if (!ok) break;
          // The next block is asked for only now, with the last tiles on their way: what a CTA holds in advance no
          // idle CTA can take.
          do {
            ask();
            ok = answer(u, level);
          } while (ok && level == -2);
          ok = ok && publish(u, level);
        }
        if (n_asked > 0) settle(&bars->stolen_full, (n_asked - 1) & 1);
        settle_ring(bars->slot_full, kSlots, n_loaded);
      }
    } else if (warp == 3) {
      // ------------------------------ Q producer ------------------------------
      if (elect_one()) {
        prefetch_tensormap(&map_q);
        int n[2] = {0, 0};
        bool ok = true;
        for (int2 i = feed.next(); ok && i.y >= 0; i = feed.next()) {
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const F128Item it = f128_item<ONE>(i.x, i.y, x, BH, n_tiles);
            if (it.n == 0) continue;
            if (n[x] > 0 && !(ok = mbar_wait(&bars->q_empty[x], (n[x] - 1) & 1, abort_flag))) break;
            mbar_arrive_expect_tx(&bars->q_full[x], kTileBytes);
            for (int p = 0; p < 2; ++p)
              tma_load_3d(smem + L::kQ + x * kTileBytes + p * kPanel, &map_q, &bars->q_full[x], p * 64, it.q0, it.unit);
            ++n[x];
          }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
          if (n[x] > 0) settle(&bars->q_full[x], (n[x] - 1) & 1);
      }
    } else {
      // ------------------------------ MMA issuers ------------------------------
      const int x = warp - 1;
      if (elect_one()) {
        constexpr uint32_t idesc_s = make_idesc_bf16(kT, kT, 0, 0);    // Q, K: K-major
        constexpr uint32_t idesc_o = make_idesc_bf16(kT, kHD, 0, 1);   // P K-major, V MN-major
        const SmemDescBase q_desc = make_desc_base_sw128(smem_u32(smem + L::kQ) + x * kTileBytes, 0);
        // (read MN-major, a V tile's two 64-column panels are kPanel apart; K-major operands ignore that offset)
        const SmemDescBase kv_desc0 = make_desc_base_sw128(smem_u32(smem + L::kKV), kPanel);
        const uint32_t tS = tmem + kColS + x * 128, tO = tmem + kColO + x * 128;
        RingAt at{0, 0};
        uint32_t g = 0, u = 0;   // key tiles and items of this group so far
        bool ok = true;
        auto wait_slot = [&]() -> bool { return mbar_wait(&bars->slot_full[at.slot], at.parity, abort_flag); };
        // tiles that this group has nothing to do with: given back once they are there, as the others are
        auto skip = [&](int tiles) -> bool {
          for (int i = 0; i < 2 * tiles; ++i, at.next()) {
            if (!wait_slot()) return false;
            mbar_arrive(&bars->slot_empty[at.slot]);
          }
          return true;
        };
        auto issue_s = [&]() -> bool {
          if (!wait_slot()) return false;
          tc_fence_after_sync();
          const SmemDescBase k_desc{kv_desc0.lo + at.slot * (kTileBytes >> 4), kv_desc0.hi};
#pragma unroll
          for (int kk = 0; kk < kHD / 16; ++kk) {
            const uint32_t off = (kk / 4) * kPanel + (kk % 4) * 32;
            mma_ss(tS, desc_at(q_desc, off), desc_at(k_desc, off), idesc_s, kk > 0 ? 1u : 0u);
          }
          mma_commit(&bars->slot_empty[at.slot]);
          mma_commit(&bars->s_full[x]);
          at.next();
          return true;
        };
        for (F128Item it = feed.fetch(x); ok && it.n_kv > 0; it = feed.fetch(x)) {
          const int n = it.n;
          if (!(ok = skip(n ? it.first : it.n_kv)) || n == 0) continue;
          if (!(ok = mbar_wait(&bars->q_full[x], u & 1, abort_flag) && issue_s())) break;
          for (int j = 0; j < n; ++j, ++g) {
            if (!(ok = wait_slot())) break;
            // (a new item's first P V may overwrite O: its probabilities come after the last results have been read)
            const SmemDescBase v_desc{kv_desc0.lo + at.slot * (kTileBytes >> 4), kv_desc0.hi};
#pragma unroll
            for (int h = 0; h < 2; ++h) {   // O (+)= P[:, 64 h .. 64 h + 63] V[64 h .. 64 h + 63, :]
              if (!(ok = mbar_wait(&bars->p_full[x][h], g & 1, abort_flag))) break;
              tc_fence_after_sync();
#pragma unroll
              for (int kk = 4 * h; kk < 4 * h + 4; ++kk)
                mma_ts(tO, tS + kk * 8, desc_at(v_desc, kk * 2048), idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
            }
            if (!ok) break;
            mma_commit(&bars->slot_empty[at.slot]);
            at.next();
            if (j + 1 < n) {
              if (!(ok = issue_s())) break;   // over the probabilities, whose product is ahead in the pipe
            } else {
              mma_commit(&bars->o_done[x]);
            }
          }
          if (!ok) break;
          ++u;
          ok = skip(it.n_kv - it.first - n);
        }
        settle_products(&bars->settled[x]);
      }
    }
  } else {
    // ------------------------------ softmax ------------------------------
    setmaxnreg_inc<kRegsSoftmax>();
    const int x = warp / 4 - 1;
    const int quad = warp % 4;            // TMEM lane quadrant of this warp
    const int row = quad * 32 + lane;     // row within the tile = TMEM lane
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t tS = tlane + kColS + x * 128, tO = tlane + kColO + x * 128;
    const float scale_log2 = scale * kLog2e;
    uint8_t* stage = smem + L::kQ + x * kTileBytes + quad * 32 * 128;   // this warp's rows of the group's Q tile
    uint32_t g = 0, u = 0;                // key tiles and items of this group so far
    bool ok = true;

    for (F128Item it = feed.fetch(x); ok && it.n_kv > 0; it = feed.fetch(x)) {
      const int n = it.n, bh = it.unit, q0 = it.q0, r = q0 + row;
      if (n == 0) continue;
      float m = -INFINITY, l[2] = {0.f, 0.f};   // running max (log2 units, scaled) of the row, and its sum by halves of the tiles
      for (int j = 0; j < n; ++j, ++g) {
        const bool diagonal = j == n - 1;
        if (!(ok = mbar_wait(&bars->s_full[x], g & 1, abort_flag))) break;
        tc_fence_after_sync();
        uint32_t s[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, s[c]);
        tmem_wait_ld();
        if (diagonal) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > row) s[c][i] = 0xff800000u;  // -inf
        }
        // max of the raw scores (scale > 0 commutes with max)
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; c += 2)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            mx4[i & 3] = fmax3(mx4[i & 3], __uint_as_float(s[c][i]), __uint_as_float(s[c + 1][i]));
        const float mx = __fmul_rn(fmaxf(fmax3(mx4[0], mx4[1], mx4[2]), mx4[3]), scale_log2);
        if (j == 0) {
          m = mx;  // O is first written by a product that does not accumulate: nothing to rescale
        } else if (__any_sync(0xffffffffu, mx > m + kRescaleAt)) {
          // (P V of the tile before is through: these scores were issued behind it)
          const float m_new = fmaxf(m, mx);
          // m = -inf: nothing but zeros has been accumulated so far
          const float corr = (m == -INFINITY) ? 0.f : ex2(m - m_new);
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld32(tO + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
            tmem_st32(tO + c * 32, o);
          }
          tmem_wait_st();
          l[0] = __fmul_rn(l[0], corr);
          l[1] = __fmul_rn(l[1], corr);
          m = m_new;
        }
        // p = exp2(s scale log2e - m). A row whose scores are all -inf so far must give p = 0, not exp2(NaN).
        float2 sum2[2];
        const float2 sl = make_float2(scale_log2, scale_log2);
        const float neg_m = (m == -INFINITY) ? 0.f : -m;
        const float2 nm = make_float2(neg_m, neg_m);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];   // bf16 pairs (k, k + 1) per column
          // The keys' halves have sums of their own, as the one-tile kernel's two threads per row do. The second's begin
          // with a zero made of the first's: where they are independent the compiler interleaves the halves, and the
          // first probabilities are late (48 x 1024 24.5 -> 26.5 us, 96 x 512 17.7 -> 18.2).
          if (c == 0) sum2[0] = sum2[1] = make_float2(0.f, 0.f);
          if (c == 2) sum2[0] = fmul2(sum2[0], make_float2(0.f, 0.f)), sum2[1] = fmul2(sum2[1], make_float2(0.f, 0.f));
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 e = ffma2(make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), sl, nm);
            const float2 p = make_float2(ex2(e.x), ex2(e.y));
            sum2[(i >> 1) & 1] = fadd2(sum2[(i >> 1) & 1], p);
            pk[i / 2] = pack_bf16(p.x, p.y);
          }
          tmem_st16(tS + c * 16, pk);
          if (c & 1) {
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(&bars->p_full[x][c / 2]);
            l[c / 2] += (sum2[0].x + sum2[1].x) + (sum2[0].y + sum2[1].y);
          }
        }
      }
      if (!ok) break;

      // Results: out = O / l, lse in natural-log units of the scaled scores. They leave through the group's Q tile,
      // which nobody reads any more: every Q K^T has completed before the last s_full was observed.
      if (!(ok = mbar_wait(&bars->o_done[x], u & 1, abort_flag))) break;
      tc_fence_after_sync();
      const float l_tot = (l[0] + l[1]) * ex2(m - m);   // (NaN where the max is not finite)
      const float f = 1.0f / l_tot;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld32(tO + c * 32, o);
        tmem_wait_ld();
        uint8_t* dst = stage + (c / 2) * kPanel + lane * 128;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = __uint_as_float(o[8 * i + e]) * f;
          *reinterpret_cast<uint4*>(dst + ((((c & 1) * 4 + i) ^ (lane & 7)) << 4)) =
              make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
        }
      }
      if (r < S) lse[static_cast<size_t>(bh) * S + r] = (m + log2f(l_tot)) * kLn2;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (q0 + quad * 32 < S)
          for (int p = 0; p < 2; ++p) tma_store_3d(&map_out, stage + p * kPanel, p * 64, q0 + quad * 32, bh);
        bulk_commit();
        bulk_wait_read<0>();
        mbar_arrive(&bars->q_empty[x]);
      }
      __syncwarp();
      ++u;
    }
    if (lane == 0) bulk_wait0();
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

template <bool ONE>
int launch(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v, int BH, int S, float scale,
           cudaStream_t st) {
  CUtensorMap mq, mk, mv, mo;
  if (int rc = make_tensor_map_bf16(&mq, q, BH, S, kHD, kT)) return rc;
  if (int rc = make_tensor_map_bf16(&mk, k, BH, S, kHD, kT)) return rc;
  if (int rc = make_tensor_map_bf16(&mv, v, BH, S, kHD, kT)) return rc;
  if (int rc = make_tensor_map_bf16(&mo, out, BH, S, kHD, 32)) return rc;
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  auto kern = flash_fwd128_kernel<ONE>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F128Smem::kBytes));
  static std::atomic<int> regs_seen;
  if (int rc = check_launch_registers(reinterpret_cast<const void*>(kern), kRegsLaunch, regs_seen)) return rc;
  const int n_tiles = (S + kT - 1) / kT;
  // K and V of a group are 50 MB. (Groups of 32768 / 65536 / 98304 rows: 48 x 2048 70.3 / 60.0 / 59.9 us, 192 x 1024
  // 72.0 / 70.3 / 70.7, 128 x 777 45.2 / 45.3 / 44.4.)
  const LeveledGrid order = ONE ? LeveledGrid{(BH + 1) / 2, (BH + 1) / 2} : leveled_grid(98304, S, BH);
  DAD_CUDA(launch_pdl(kern, leveled_blocks(order, (n_tiles + 1) / 2), dim3(kThreads), F128Smem::kBytes, st, mq, mk, mv, mo,
                      lse, BH, S, scale, order, status));
  return DADATTN_OK;
}

}  // namespace

// Whether items of two query tiles are the better ones, for up to kFwd128OneSumRows rows. A short launch is over sooner
// with a tile per CTA: half the work in its longest item. So: sequences of up to three tiles, once the tiles do not fit
// the GPU at once; others, where the CTAs' mean number of K / V steps is 0.8 of the longest item's. us, one tile / two,
// by that quotient:
//     24 x 128   5.6 / 6.9 (24 tiles)   80 x 256   11.7 / 10.5 (160)  60 x 384  12.5 / 11.3 (180)  192 x 128  12.1 / 9.6 (192)
//     32 x 777  15.6 / 18.9  0.6        40 x 777   17.6 / 19.1  0.7   48 x 1024 27.5 / 24.5  0.8   48 x 777   23.2 / 21.8 0.9
//     24 x 2048 36.6 / 40.1  0.7        48 x 2048  67.3 / 59.4  1.5   96 x 512  21.9 / 17.6  1.9   192 x 1024 92.4 / 68.7 3.2
// Longer sequences keep a maximum, a sum and an accumulator for each half of a row, whatever their number: the line is in
// rows because a unit's result may not go by the units beside it. Two tiles are slower there where they leave CTAs idle
// or the launch runs at the power cap (16 x 3000 53 / 64, 24 x 8192 380 / 418, 192 x 8192 forward and backward in a loop
// 12650 / 13080) and faster between (48 x 4096 213 / 198, 192 x 4096 826-905 / 812-840).
bool fwd128_pairs_pay(int BH, int S) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  const long long n = (static_cast<long long>(S) + kT - 1) / kT, pairs = n / 2;
  if (n <= 3) return n * BH > sms;
  return 10 * (pairs * (pairs + 1) + (n % 2 ? n : 0)) * BH >= 8 * n * sms;   // (steps of a unit's items)
}

int launch_fwd_bf16_d128_pairs(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v, int BH,
                               int S, float scale, cudaStream_t st) {
  return (S <= kT ? launch<true> : launch<false>)(out, lse, q, k, v, BH, S, scale, st);
}

}  // namespace dadattn
