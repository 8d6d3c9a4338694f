// bf16 fused causal attention backward for sm_100a, head size 128: dQ, dK and dV in ONE pass.
//
// The two-kernel backward of flash_bwd_bf16_sm100.cu follows the reference (cuda/attention.cu:
// 88-205) in computing the probabilities twice: 7 GEMM-sized products for 5 gradients' worth.
// Here a CTA owns 128 keys of one (batch, head) and streams the 64-query sub-tiles that can see
// them. Rows of the score tile are keys (one TMEM lane each):
//     S^T = K Q^T,  dP^T = V dO^T                       128 keys x 64 queries, fp32 in TMEM
//     p = exp2(S^T scale log2e - lse[q] log2e),  ds = p (dP^T - delta[q]) scale
//     dV += P^T-tile dO      dK += dS^T-tile Q          accumulate in TMEM over the whole loop
//     dQ^T-tile = K^T dS^T                              128 head dims x 64 queries, per step
// P^T and dS^T go back into tensor memory as packed bf16 and are the A operands of dV / dK from
// there (tcgen05.mma with A in TMEM): an MMA with both operands in shared memory reads them at
// 128 B/clk, and with the TMA loads, the stores and the dQ staging the shared-memory traffic of
// a step (336 KB when P^T / dS^T lived there, now 224) weighs as much as the products. dS^T is
// also written, bf16, [key][query] in the 128-byte swizzled layout, as the MN-major B operand
// of dQ^T, whose A operand is the resident K tile read MN-major. Computing dQ transposed keeps
// all 128 TMEM lanes busy (M = 128 head dims) although a step has only 64 queries.
// Each step's dQ^T tile (32 KB fp32) goes from tensor memory through registers of four drain warps into an
// fp32 workspace by red.global.add.v4, laid out so that a warp's lanes, one head dim each, add 512
// consecutive bytes ([BH][64-query block][16 groups of 4 queries][128 dims][4 queries]): 1290 clocks a tile
// and SM, as fast as bulk reduce-adds from shared memory (1390; rows of 256 bytes apart, a lane on each,
// take 2400), without the 64 KB a step that staging costs where shared memory sets the pace. A last pass
// rounds the workspace to bf16. The sums happen in whatever order the CTAs reach them, so dQ may differ in
// its last bits from run to run; dadattn_set_bwd_deterministic(1) selects the two-kernel path.
//   warps 0-15   compute: four warps per TMEM lane quadrant, each taking 16 of the 64 query columns
//   warp 16      TMA producer          warp 17      MMA issuer + TMEM owner
//   warp 18      row scalars: -lse log2e and -delta scale of each step's queries      (warp 19 idle)
//   warps 20-23  drain: dQ^T out of tensor memory, one thread per lane, while the compute warps are
//                already on the next step's arithmetic
#include <cuda_bf16.h>

#include <cfloat>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace {

using namespace ptx;

// Two plain polls ahead of the suspending wait: 192 x 8192 10.30 ms, none 10.39, 8 10.39, 24 10.37 (each before
// the products were issued by a whole warp).
#define polled_wait(bar, parity, abort_flag) mbar_wait_at<2>(bar, parity, abort_flag, __LINE__)
#define polled_warp_wait(bar, parity, abort_flag) __all_sync(0xffffffffu, polled_wait(bar, parity, abort_flag))

constexpr int kGD = 128;                   // head size
constexpr int kGKeys = 128;                // keys owned by a CTA
constexpr int kGSub = 64;                  // queries per step
constexpr int kGPanel = 128 * 128;         // [128 rows][64 bf16] swizzled panel
constexpr int kGSubPanel = 64 * 128;       // [64 rows][64 bf16] swizzled panel
constexpr int kGStages = 4;                // streamed-tile ring depth
constexpr int kGThreads = 24 * 32;
constexpr int kGCompute = 16 * 32;
constexpr int kGDrain = 4 * 32;
constexpr int kGWarpProducer = 16, kGWarpIssuer = 17, kGWarpScalars = 18, kGWarpDrain0 = 20;
// Registers per thread once the warpgroups have rebalanced; the pool is what the CTA starts with. (The
// drain threads hold a row of 64 sums.)
constexpr int kGRegsLaunch = 80, kGRegsCompute = 88, kGRegsHelper = 48, kGRegsDrain = 80;
static_assert(kGCompute * kGRegsCompute + 128 * kGRegsHelper + kGDrain * kGRegsDrain <= kGThreads * kGRegsLaunch,
              "the warpgroups ask for more registers than the CTA owns");
static_assert(kGThreads * kGRegsLaunch <= 65536 && (kGRegsLaunch + 8) * kGThreads > 65536,
              "kGRegsLaunch is not what the compiler gives a CTA of this size");
constexpr int kPrepareThreads = 256;         // of the delta kernel, whose blocks zero a part of one tile
constexpr int kGDqTileBytes = kGD * kGSub * 4;   // one dQ^T tile, fp32
constexpr float kGLog2e = 1.4426950408889634f;

struct G128Smem {
  static constexpr int kTile = 2 * kGPanel;        // resident [128, 128] tile
  static constexpr int kSubTile = 2 * kGSubPanel;  // streamed [64, 128] tile
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTile;
  static constexpr int kQ = kV + kTile;
  static constexpr int kDO = kQ + kGStages * kSubTile;
  static constexpr int kDS = kDO + kGStages * kSubTile;  // [128 keys][64 q] bf16, one panel
  static constexpr int kVec = kDS + kGPanel;             // two buffers of [2][64] row scalars
  static constexpr int kBars = kVec + 2 * 2 * 64 * 4;
  static constexpr int kBytes = kBars + 256;
  static_assert(kBytes <= 232448, "shared memory budget of one CTA exceeded");
};

struct G128Bars {
  uint64_t kv_full, qdo_full[kGStages], qdo_empty[kGStages];
  uint64_t x_full[2], x_free, w_full, acc_done, dq_drained, settled;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void red_add4(float* to, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to), "f"(__uint_as_float(a)),
               "f"(__uint_as_float(b)), "f"(__uint_as_float(c)), "f"(__uint_as_float(d))
               : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(taddr)
               : "memory");
}

template <bool DROP>
__global__ void __launch_bounds__(kGThreads, 1)
flash_bwd_fused128_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                          const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                          const __grid_constant__ CUtensorMap map_dk, const __grid_constant__ CUtensorMap map_dv,
                          float* __restrict__ dq_ws, const float* __restrict__ lse,
                          const float* __restrict__ delta, int S, float scale, float rate,
                          const __grid_constant__ PhiloxRounds rng, int64_t unit0, LeveledGrid order,
                          int* __restrict__ status) {
  using L = G128Smem;
  constexpr int D = kGD;
  constexpr uint32_t kTmemCols = 512;
  // S^T, dP^T (fp32, 64 columns each), dV, dK (128 each), dQ^T (64), then P^T and dS^T as packed
  // bf16 (two queries per column: 32 columns each)
  constexpr uint32_t kColS = 0, kColDP = 64, kColDV = 128, kColDK = 256, kColDQ = 384;
  constexpr uint32_t kColP = 448, kColDSt = 480;

  extern __shared__ __align__(1024) uint8_t smem[];
  G128Bars* bars = reinterpret_cast<G128Bars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int n_sub = (S + kGSub - 1) / kGSub;
  // key tile `own` streams the query sub-tiles 2*own .. n_sub-1 (low `own` = most work = first)
  int own, bh;
  if (!leveled_block(order, own, bh)) return;
  const int first = 2 * own;
  const int n_it = n_sub - first;
  const int k0 = own * kGKeys;

  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicExch(status, DADATTN_E_CUDA);
    return;
  }
  auto load_step = [&](int s, int i) {   // Q and dO of a step, into stage s, by the producing thread
    const int q0 = (first + i) * kGSub;
    mbar_arrive_expect_tx(&bars->qdo_full[s], 2 * L::kSubTile);
    for (int p = 0; p < 2; ++p) {
      tma_load_3d(smem + L::kQ + s * L::kSubTile + p * kGSubPanel, &map_q, &bars->qdo_full[s], p * 64, q0, bh);
      tma_load_3d(smem + L::kDO + s * L::kSubTile + p * kGSubPanel, &map_do, &bars->qdo_full[s], p * 64, q0, bh);
    }
  };
  if (threadIdx.x == kGWarpProducer * 32) {
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_do);
    prefetch_tensormap(&map_dk);
    prefetch_tensormap(&map_dv);
    mbar_init(&bars->kv_full, 1);
    for (int s = 0; s < kGStages; ++s) {
      mbar_init(&bars->qdo_full[s], 1);
      mbar_init(&bars->qdo_empty[s], 1);
    }
    mbar_init(&bars->x_full[0], 2);      // the products and the step's row scalars
    mbar_init(&bars->x_full[1], 2);
    mbar_init(&bars->x_free, kGCompute);
    mbar_init(&bars->w_full, kGCompute);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->dq_drained, kGDrain);
    mbar_init(&bars->settled, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
    // The first tiles are requested here: they need this thread's barriers, and nothing of what the others set up (backward,
    // us: 72 x 777 72.4 -> 69.7, 24 x 2048 95.5 -> 91.7, 192 x 128 26.6 -> 25.2)
    pdl_wait();
    mbar_arrive_expect_tx(&bars->kv_full, 2 * L::kTile);
    for (int p = 0; p < 2; ++p) {
      tma_load_3d(smem + L::kK + p * kGPanel, &map_k, &bars->kv_full, p * 64, k0, bh);
      tma_load_3d(smem + L::kV + p * kGPanel, &map_v, &bars->kv_full, p * 64, k0, bh);
    }
    load_step(0, 0);
  }
  __syncwarp();
  if (warp == kGWarpIssuer) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  pdl_wait();
  pdl_launch_dependents();

  if (warp >= kGWarpProducer && warp < kGWarpDrain0) {
  setmaxnreg_dec<kGRegsHelper>();
  if (warp == kGWarpProducer) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int i = 1;
      for (; i < n_it; ++i) {
        const int s = i % kGStages, use = i / kGStages;
        if (use > 0 && !polled_wait(&bars->qdo_empty[s], (use - 1) & 1, abort_flag)) break;
        load_step(s, i);
      }
      settle(&bars->kv_full, 0);
      settle_ring(bars->qdo_full, kGStages, i);
    }
  } else if (warp == kGWarpIssuer) {
    // ------------------------------ MMA issuer ------------------------------
    {   // (the whole warp: mma_ss_warp)
      const uint32_t lead = elect_one(), tm = __reduce_max_sync(0xffffffffu, tmem);   // (known to be uniform, so)
      constexpr uint32_t idesc_x = make_idesc_bf16(128, 64, 0, 0);    // S^T, dP^T: both K-major
      constexpr uint32_t idesc_a = make_idesc_bf16(128, D, 0, 1);     // dV, dK: B MN-major
      constexpr uint32_t idesc_q = make_idesc_bf16(128, 64, 1, 1);    // dQ^T: A and B MN-major
      const SmemDescBase k_kmaj = make_desc_base_sw128(smem_u32(smem + L::kK), 0);
      const SmemDescBase v_kmaj = make_desc_base_sw128(smem_u32(smem + L::kV), 0);
      // K read as MN-major A (M = head dims): the two 64-dim panels are kGPanel apart
      const SmemDescBase k_mn = make_desc_base_sw128(smem_u32(smem + L::kK), kGPanel);
      const SmemDescBase ds_desc = make_desc_base_sw128(smem_u32(smem + L::kDS), 0);
      // streamed tiles: K-major B of the score GEMMs, MN-major B (panels kGSubPanel apart) of dV / dK
      const SmemDescBase q_desc0 = make_desc_base_sw128(smem_u32(smem + L::kQ), kGSubPanel);
      const SmemDescBase do_desc0 = make_desc_base_sw128(smem_u32(smem + L::kDO), kGSubPanel);
      bool ok = polled_warp_wait(&bars->kv_full, 0, abort_flag);

      auto issue_x = [&](int i) -> bool {
        const int s = i % kGStages;
        const uint32_t par = (i / kGStages) & 1;
        const SmemDescBase qd{q_desc0.lo + s * (L::kSubTile >> 4), q_desc0.hi};
        const SmemDescBase dd{do_desc0.lo + s * (L::kSubTile >> 4), do_desc0.hi};
        if (!polled_warp_wait(&bars->qdo_full[s], par, abort_flag)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss_warp(tm + kColS, desc_at(k_kmaj, (kk / 4) * kGPanel + (kk % 4) * 32),
                 desc_at(qd, (kk / 4) * kGSubPanel + (kk % 4) * 32), idesc_x, kk > 0 ? 1u : 0u, lead);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          mma_ss_warp(tm + kColDP, desc_at(v_kmaj, (kk / 4) * kGPanel + (kk % 4) * 32),
                 desc_at(dd, (kk / 4) * kGSubPanel + (kk % 4) * 32), idesc_x, kk > 0 ? 1u : 0u, lead);
        mma_commit_warp(&bars->x_full[i & 1], lead);
        return true;
      };
      auto issue_acc = [&](int i) -> bool {
        const int s = i % kGStages;
        const SmemDescBase qd{q_desc0.lo + s * (L::kSubTile >> 4), q_desc0.hi};
        const SmemDescBase dd{do_desc0.lo + s * (L::kSubTile >> 4), do_desc0.hi};
        if (!polled_warp_wait(&bars->w_full, i & 1, abort_flag)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < kGSub / 16; ++kk) {   // K dimension = 64 queries, 16 per MMA
          const uint32_t acc = (i > 0 || kk > 0) ? 1u : 0u;
          mma_ts_warp(tm + kColDV, tm + kColP + kk * 8, desc_at(dd, kk * 2048), idesc_a, acc, lead);
          mma_ts_warp(tm + kColDK, tm + kColDSt + kk * 8, desc_at(qd, kk * 2048), idesc_a, acc, lead);
        }
        mma_commit_warp(&bars->qdo_empty[s], lead);   // Q and dO of this stage are last read by the products above
        // the previous step's dQ^T must have left tensor memory before this one overwrites it
        if (i > 0 && !polled_warp_wait(&bars->dq_drained, (i - 1) & 1, abort_flag)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < kGKeys / 16; ++kk)    // K dimension = 128 keys
          mma_ss_warp(tm + kColDQ, desc_at(k_mn, kk * 2048), desc_at(ds_desc, kk * 2048), idesc_q,
                 kk > 0 ? 1u : 0u, lead);
        mma_commit_warp(&bars->acc_done, lead);
        return true;
      };

      ok = ok && issue_x(0);
      for (int i = 0; ok && i < n_it; ++i) {
        // the next step's score GEMMs go first: the arithmetic on them overlaps this step's
        // accumulating GEMMs
        if (i + 1 < n_it) ok = polled_warp_wait(&bars->x_free, i & 1, abort_flag) && issue_x(i + 1);
        ok = ok && issue_acc(i);
      }
      settle_products_warp(&bars->settled, lead);
    }
  } else if (warp == kGWarpScalars) {
    // ------------------------------ row scalars ------------------------------
    // -lse log2e and -delta scale of each step's 64 queries, requested a step ahead, into one of two buffers.
    // Queries beyond S contribute nothing: p = exp2(-inf). Buffer i % 2 is free once the products of step
    // i - 2, which follow the arithmetic that read it, have given their stage back; that barrier's next phase
    // is a later step's, which needs these scalars first.
    const size_t vec_base = static_cast<size_t>(bh) * S;
    float rl[2], rd[2];
    auto request = [&](int i) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int q = (first + i) * kGSub + c * 32 + lane;
        rl[c] = q < S ? lse[vec_base + q] : INFINITY;
        rd[c] = q < S ? delta[vec_base + q] : 0.f;
      }
    };
    request(0);
    for (int i = 0; i < n_it; ++i) {
      if (i >= 2 && !polled_wait(&bars->qdo_empty[(i - 2) % kGStages], ((i - 2) / kGStages) & 1, abort_flag)) break;
      float* dst = reinterpret_cast<float*>(smem + L::kVec) + (i & 1) * 128 + lane;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        dst[c * 32] = -rl[c] * kGLog2e;
        dst[64 + c * 32] = -rd[c] * scale;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->x_full[i & 1]);
      if (i + 1 < n_it) request(i + 1);
    }
  }
  } else if (warp >= kGWarpDrain0) {
    // ------------------------------ dQ drain ------------------------------
    setmaxnreg_dec<kGRegsDrain>();
    const int quad = warp % 4;
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    float* dst = dq_ws + (static_cast<size_t>(bh) * n_sub + first) * (kGD * kGSub) + (quad * 32 + lane) * 4;
    for (int i = 0; i < n_it; ++i, dst += kGD * kGSub) {
      if (!polled_wait(&bars->acc_done, i & 1, abort_flag)) break;
      tc_fence_after_sync();
      uint32_t o0[32], o1[32];
      tmem_ld32(tlane + kColDQ, o0);
      tmem_ld32(tlane + kColDQ + 32, o1);
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(&bars->dq_drained);
#pragma unroll
      for (int c = 0; c < 8; ++c) red_add4(dst + c * (kGD * 4), o0[4 * c], o0[4 * c + 1], o0[4 * c + 2], o0[4 * c + 3]);
#pragma unroll
      for (int c = 0; c < 8; ++c) red_add4(dst + (8 + c) * (kGD * 4), o1[4 * c], o1[4 * c + 1], o1[4 * c + 2], o1[4 * c + 3]);
    }
  } else {
    // ------------------------------ compute warps ------------------------------
    setmaxnreg_inc<kGRegsCompute>();
    const int quad = warp % 4;            // TMEM lane quadrant of this warp
    const int cg = warp / 4;              // which 16 query columns of the 64
    const int row = quad * 32 + lane;     // key within the tile = TMEM lane
    const int key = k0 + row;
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const float scale_log2 = scale * kGLog2e;
    const float keep_scale = DROP ? 1.0f / (1.0f - rate) : 1.0f;
    const float* vec = reinterpret_cast<const float*>(smem + L::kVec) + cg * 16;
    uint8_t* ds_row = smem + L::kDS + row * 128;
    bool ok = true;

    for (int i = 0; i < n_it; ++i) {
      const int q0 = (first + i) * kGSub + cg * 16;   // this thread's first query
      const float* v_lse = vec + (i & 1) * 128;
      const float* v_delta = v_lse + 64;
      if (!(ok = polled_wait(&bars->x_full[i & 1], (i >> 1) & 1, abort_flag))) break;
      tc_fence_after_sync();
      uint32_t x1[16], x2[16];
      tmem_ld16(tlane + kColS + cg * 16, x1);
      tmem_ld16(tlane + kColDP + cg * 16, x2);
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(&bars->x_free);  // scores are in registers: the next step's products may overwrite them

#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        // 128-bit broadcast reads, here and below: all lanes of a warp want the same four columns
        const float4 l4 = *reinterpret_cast<const float4*>(v_lse + c);
        const float2 e0 = ffma2(make_float2(__uint_as_float(x1[c]), __uint_as_float(x1[c + 1])),
                                make_float2(scale_log2, scale_log2), make_float2(l4.x, l4.y));
        const float2 e1 = ffma2(make_float2(__uint_as_float(x1[c + 2]), __uint_as_float(x1[c + 3])),
                                make_float2(scale_log2, scale_log2), make_float2(l4.z, l4.w));
        x1[c] = __float_as_uint(ex2(e0.x));
        x1[c + 1] = __float_as_uint(ex2(e0.y));
        x1[c + 2] = __float_as_uint(ex2(e1.x));
        x1[c + 3] = __float_as_uint(ex2(e1.y));
      }
      // Sub-tiles that straddle the diagonal. (Behind the exponentials: a score of -inf would be p = NaN where the
      // query's lse is, and with it dV of keys that the query does not see.)
      if (i < 2) {
#pragma unroll
        for (int c = 0; c < 16; ++c)
          if (key > q0 + c) x1[c] = 0u;
      }
      uint32_t keep = 0xffffu;
      if (DROP) {
        // where the warp's 32 x 16 block has visible pairs (the same number of draws in every lane: a warp's loop
        // runs as long as its longest lane's)
        if (q0 + 15 >= k0 + quad * 32)
          keep = philox_keep_bits<2>(rng, (static_cast<uint64_t>(unit0 + bh) * S + q0) * S + key, static_cast<uint32_t>(S), 16);
        __syncwarp();
      }
      uint32_t pw[8], dw[8];
#pragma unroll
      for (int c = 0; c < 16; c += 4) {
        const float4 b = *reinterpret_cast<const float4*>(v_delta + c);
        const float2 dl[2] = {make_float2(b.x, b.y), make_float2(b.z, b.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = c + 2 * h;
          const float2 p = make_float2(__uint_as_float(x1[e]), __uint_as_float(x1[e + 1]));
          float2 pd = p, g = make_float2(__uint_as_float(x2[e]), __uint_as_float(x2[e + 1]));
          if (DROP) {
            const float2 mk = make_float2((keep >> e) & 1u ? keep_scale : 0.f, (keep >> (e + 1)) & 1u ? keep_scale : 0.f);
            pd = fmul2(p, mk);
            g = fmul2(g, mk);
          }
          // ds = p (dP - delta) scale as p * fma(dP, scale, -delta scale)
          const float2 ds = fmul2(p, ffma2(g, make_float2(scale, scale), dl[h]));
          pw[e / 2] = pack_bf16(pd.x, pd.y);
          dw[e / 2] = pack_bf16(ds.x, ds.y);
        }
      }
      // P^T / dS^T of step i-1 consumed
      if (i > 0) {
        if (!(ok = polled_wait(&bars->acc_done, (i - 1) & 1, abort_flag))) break;
        tc_fence_after_sync();
      }
      // sixteen queries = eight packed columns = one K step of the dV / dK MMAs
      tmem_st8(tlane + kColP + cg * 8, pw);
      tmem_st8(tlane + kColDSt + cg * 8, dw);
#pragma unroll
      for (int v4 = 0; v4 < 2; ++v4) {
        const int chunk = cg * 2 + v4;    // 16-byte chunk within the 128-byte row
        const int off = (chunk ^ (row & 7)) << 4;
        *reinterpret_cast<uint4*>(ds_row + off) =
            make_uint4(dw[4 * v4], dw[4 * v4 + 1], dw[4 * v4 + 2], dw[4 * v4 + 3]);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      fence_proxy_async_smem();
      mbar_arrive(&bars->w_full);
    }

    // dV (column groups 0, 1) and dK (2, 3), 64 head dims each, through shared memory and TMA: a warp's 32 keys x 64 dims
    // are 4 KB of the Q ring, whose tiles the last products have read. As 16-byte stores of one row per lane, 32 rows
    // an instruction, they took 6800 clocks a CTA (backward, us: 192 x 1024 267 -> 247, 72 x 777 80 -> 73, 192 x 128 30.5 ->
    // 26.8, 24 x 2048 103 -> 95.6, 192 x 8192 9590 -> 9390).
    if (ok && polled_wait(&bars->acc_done, (n_it - 1) & 1, abort_flag)) {
      tc_fence_after_sync();
      uint8_t* stage = smem + L::kQ + cg * kGPanel + quad * 32 * 128;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
        tmem_ld32(tlane + (cg < 2 ? kColDV : kColDK) + (cg & 1) * 64 + c * 32, o);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + i) ^ (lane & 7)) << 4)) = make_uint4(
              pack_bf16(__uint_as_float(o[8 * i + 0]), __uint_as_float(o[8 * i + 1])),
              pack_bf16(__uint_as_float(o[8 * i + 2]), __uint_as_float(o[8 * i + 3])),
              pack_bf16(__uint_as_float(o[8 * i + 4]), __uint_as_float(o[8 * i + 5])),
              pack_bf16(__uint_as_float(o[8 * i + 6]), __uint_as_float(o[8 * i + 7])));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && k0 + quad * 32 < S) {   // (rows beyond S are not written)
        tma_store_3d(cg < 2 ? &map_dv : &map_dk, stage, (cg & 1) * 64, k0 + quad * 32, bh);
        bulk_commit();
        bulk_wait_read<0>();
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kGWarpIssuer) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (threadIdx.x == 0 && bars->abort_flag) report_timeout(status, bars->abort_flag);
}

// delta[r] = sum_d dO[r,d] O[r,d] (reference flash_delta_kernel, cuda/attention.cu:76-85): 16
// lanes per row of 128. Also zeros into the workspace, 32 bytes per thread (a memset of its own between two
// kernels costs short calls about 3 us). From the last row on, as the pass that rounds: the gradient kernel starts with
// the first, whose lines L2 then still holds (64 x 2048 backward 269-274 -> 261-268 us, 192 x 1024 260-264 -> 258-259).
__global__ void fused128_prepare_kernel(float* __restrict__ delta, float* __restrict__ dq_ws,
                                        const __nv_bfloat16* __restrict__ dout,
                                        const __nv_bfloat16* __restrict__ out, int64_t rows) {
  constexpr int D = kGD, Lr = D / 8;
  pdl_wait();
  pdl_launch_dependents();
  const int64_t block = gridDim.x - 1 - blockIdx.x, t = block * blockDim.x + threadIdx.x;
  const int64_t r = t / Lr;
  const int c = static_cast<int>(t % Lr) * 8;
  float4* zero = reinterpret_cast<float4*>(dq_ws) + block * (2 * kPrepareThreads);
  zero[threadIdx.x] = zero[threadIdx.x + kPrepareThreads] = make_float4(0.f, 0.f, 0.f, 0.f);
  float sum = 0.f;
  if (r < rows) {
    const uint4 a = *reinterpret_cast<const uint4*>(dout + r * D + c);
    const uint4 b = *reinterpret_cast<const uint4*>(out + r * D + c);
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

// Workspace tile [16 groups of 4 queries][128 dims][4 queries] fp32 -> dq[q][128] bf16. One CTA of 256 threads
// per tile: thread t takes head dims 2 (t % 64) and the next, so that a warp reads 1 KB and writes 128 bytes of
// a row in one piece. The sums are read for the last time: their lines need not go out to memory.
__global__ void __launch_bounds__(256)
fused128_convert_kernel(__nv_bfloat16* __restrict__ dq, float* __restrict__ dq_ws, int S, int n_sub) {
  pdl_wait();
  const int bh = gridDim.y - 1 - blockIdx.y, blk = blockIdx.x;
  float* sums = dq_ws + (static_cast<size_t>(bh) * n_sub + blk) * (kGD * kGSub);
  const float4* tile = reinterpret_cast<const float4*>(sums);
  const int d = (threadIdx.x % 64) * 2, g0 = threadIdx.x / 64;
  float4 a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = tile[(g0 + 4 * j) * kGD + d];
    b[j] = tile[(g0 + 4 * j) * kGD + d + 1];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int q = blk * kGSub + (g0 + 4 * j) * 4;
    uint32_t* dst = reinterpret_cast<uint32_t*>(dq + (static_cast<size_t>(bh) * S + q) * kGD + d);
    const uint32_t w[4] = {pack_bf16(a[j].x, b[j].x), pack_bf16(a[j].y, b[j].y), pack_bf16(a[j].z, b[j].z),
                           pack_bf16(a[j].w, b[j].w)};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (q + e < S) dst[e * (kGD / 2)] = w[e];
  }
  __syncthreads();
  static_assert(kGDqTileBytes == 256 * 128, "a line of the tile per thread");
  discard_line(sums + threadIdx.x * 32);
  pdl_launch_dependents();
}

}  // namespace

// Workspace: delta [BH,S] fp32 (padded to 256 bytes), then the dQ^T accumulator
// [BH][ceil(S/64)][16][128][4] fp32.
size_t fused128_bwd_workspace_bytes(int BH, int S) {
  const size_t delta_bytes = (static_cast<size_t>(BH) * S * sizeof(float) + 255) / 256 * 256;
  const size_t n_sub = (static_cast<size_t>(S) + kGSub - 1) / kGSub;
  return delta_bytes + static_cast<size_t>(BH) * n_sub * kGDqTileBytes;
}

int launch_bwd_fused_d128(uint16_t* dq, uint16_t* dk, uint16_t* dv, void* workspace, const uint16_t* dout,
                          const uint16_t* out, const float* lse, const uint16_t* q, const uint16_t* k,
                          const uint16_t* v, int BH, int S, float scale, float rate, uint64_t seed,
                          uint64_t offset, int64_t unit0, cudaStream_t st) {
  using BF = __nv_bfloat16;
  const size_t delta_bytes = (static_cast<size_t>(BH) * S * sizeof(float) + 255) / 256 * 256;
  const int n_sub = (S + kGSub - 1) / kGSub;
  float* delta = static_cast<float*>(workspace);
  float* dq_ws = reinterpret_cast<float*>(static_cast<char*>(workspace) + delta_bytes);
  CUtensorMap mk, mv, mq, mdo, mdk, mdv;
  if (int rc = make_tensor_map_bf16(&mk, k, BH, S, kGD, kGKeys)) return rc;
  if (int rc = make_tensor_map_bf16(&mv, v, BH, S, kGD, kGKeys)) return rc;
  if (int rc = make_tensor_map_bf16(&mq, q, BH, S, kGD, kGSub)) return rc;
  if (int rc = make_tensor_map_bf16(&mdo, dout, BH, S, kGD, kGSub)) return rc;
  if (int rc = make_tensor_map_bf16(&mdk, dk, BH, S, kGD, 32)) return rc;
  if (int rc = make_tensor_map_bf16(&mdv, dv, BH, S, kGD, 32)) return rc;
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;

  stage_event(0, st);
  const int64_t rows = static_cast<int64_t>(BH) * S;
  const int64_t blocks = static_cast<int64_t>(BH) * n_sub * (kGDqTileBytes / (32 * kPrepareThreads));
  DAD_CUDA(launch_pdl(fused128_prepare_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kPrepareThreads), 0, st, delta,
                      dq_ws, reinterpret_cast<const BF*>(dout), reinterpret_cast<const BF*>(out), rows));
  stage_event(1, st);
  const PhiloxRounds rng = make_philox_rounds(seed, offset, rate, static_cast<uint32_t>(S));
  // Key tiles level by level over groups of units, whatever the number of CTAs. Backward alone, us (medians), level
  // by level / unit by unit with a memset ahead:
  //     192 CTAs  24 x 1024     42 / 59      1800  600 x 300   190 / 199       3072  96 x 4096   1311-1329 / 1379-1389
  //     384       24 x 2048    105 / 127     2048  64 x 4096   885 / 920       3072  48 x 8192   2338-2357 / 2382-2415
  //     768       48 x 2048    205 / 220     3000  3000 x 128  320 / 328       3840  30 x 16384  5466-5522 / 5536-5553
  //    1536      192 x 1024    278 / 290     3072  192 x 2048  808 / 827      12288  192 x 8192  9441-9477 / 9500-9624
  // (6 x 65536, units one by one: 16.7-17.0 ms / 16.7.) Before the products were issued by a whole warp and dQ
  // left its staging buffer, unit by unit had been the better one beyond 2048 CTAs.
  const LeveledGrid order = leveled_grid(32768, S, BH);
  const bool drop = rate > 0.f;
  auto kern = drop ? flash_bwd_fused128_kernel<true> : flash_bwd_fused128_kernel<false>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G128Smem::kBytes));
  static std::atomic<int> regs_seen[2];
  if (int rc = check_launch_registers(reinterpret_cast<const void*>(kern), kGRegsLaunch, regs_seen[drop])) return rc;
  DAD_CUDA(launch_pdl(kern, leveled_blocks(order, (S + kGKeys - 1) / kGKeys), dim3(kGThreads),
                      G128Smem::kBytes, st, mk, mv, mq, mdo, mdk, mdv, dq_ws, lse, static_cast<const float*>(delta), S, scale, rate, rng, unit0, order, status));
  stage_event(2, st);
  DAD_CUDA(launch_pdl(fused128_convert_kernel, dim3(n_sub, BH), dim3(256), 0, st,
                      reinterpret_cast<BF*>(dq), dq_ws, S, n_sub));
  stage_event(3, st);
  return DADATTN_OK;
}

}  // namespace dadattn
