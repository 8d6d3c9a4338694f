// fp32 backward on the tensor cores (head sizes 16, 32, 64): dQ, dK and dV in one launch, exact fp32
// operands as three bf16 planes (f32_split.cuh), no atomics, bit-reproducible.
//
// As in the reference (cuda/attention.cu:88-205) the probabilities are formed twice, once where
// keys are resident and queries stream past (dK, dV) and once the other way round (dQ). Both are
// the same machine, so both kinds of work item share one grid:
//     kind    resident A1, A2   streamed B1, B2   X1 = A1 B1^T   X2 = A2 B2^T   sums
//     dK/dV   K, V              Q, dO             S^T            dP^T           dV += P^T B2, dK += dS^T B1
//     dQ      Q, dO             K, V              S              dP             dQ += dS B1
// A CTA owns 128 resident rows (one per TMEM lane) and takes the other side 64 rows at a time:
//   warps 0-15  four threads per row, 16 columns each: p = exp(s scale - lse), ds = p (dP - delta)
//               scale, both split into planes and written back to tensor memory, from where the
//               sums take them as A operands; the sums of each step are added to fp32 registers
//   warps 16-26 fetch the next step's fp32 rows, split them in registers, and put them into the
//               shared-memory stage the moment it is released; delta = rowsum(dO o O) on the way
//   warp 27     issues the products. Order on the tensor pipe: sums of step i, X2 then X1 of step
//               i + 2 (B2's stage is released before B1's, so its refill hides behind the sums'
//               last products), sums of step i + 1, ...
// A step costs 2304 (X) + 2304 (dK/dV) or 1152 (dQ) clocks of tensor pipe at head size 64 (48 for a
// 128 x 64 x 16 product; the pipe's counter takes 32) and, the mean of both kinds, about 2700 issue slots
// per scheduler, and takes about 4600 clocks (48 x 1024; 4900 before the whole warp issued the products).
// CTAs are persistent where there are more items than SMs: the streamed rings run on across items, and
// the next item's resident tiles are fetched and split, and its first products formed, while this one's
// last sums complete, so an item adds little to its steps (one CTA per item: about 5 us each; 48 x 1024 x
// 64: 154 -> 142 us, 148 x 512: 158 -> 134, 32 x 301 x 32: 20.0 -> 17.4).
// Tensor memory: X1 / X2 double buffered (buffer b at 128 b), 64 columns at 256 for the planes that
// do not fit over the scores they came from, sums at 320 and 384.
#include "f32_split.cuh"

namespace dadattn {
namespace {

using namespace f32tc;

struct BwdSmem {
  static constexpr int kA1 = 0, kA2 = 3 * kPlaneA;
  // Three stages for B2: X2 of step i + 2 is the first product after the sums of step i and must not
  // have to wait for a stage that those sums have just released (two stages: 560 clocks a step idle).
  static constexpr int kB1 = 6 * kPlaneA;                      // [2 stages][3 planes]
  static constexpr int kB2 = kB1 + 2 * 3 * kPlaneB;            // [3 stages][3 planes]
  static constexpr int kVec = kB2 + 3 * 3 * kPlaneB;           // [3 stages][lse, delta][64]; dK/dV items
  static constexpr int kOwn = kVec + 3 * 512;                  // delta of a dQ item's rows, [2 items][128]
  static constexpr int kBars = kOwn + 2 * 512;
  static constexpr int kBytes = kBars + 256;
  static_assert(kBytes <= 232448, "shared memory of a CTA exceeded");
};
struct BwdBars {
  uint64_t a_full, p_full, acc_done, settled;
  uint64_t b1_full[2], b1_empty[2], b2_full[3], b2_empty[3], x_full[2];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(BwdBars) <= 256, "barrier block");

struct BwdArgs {
  float *dq, *dk, *dv;
  const float *dout, *out, *lse, *q, *k, *v;
  float* delta;   // scratch, used only where delta_given
  int BH, S;
  float scale, rate;
  PhiloxRounds rng;
  int64_t unit0;
  bool vec_ok;
  int* status;
};

// Items in order of their number of steps, the longest first: level i holds the key tiles i and the
// query tiles n - 1 - i of every (batch, head). CTA c of G takes the items k G + (k even ? c : G-1-c).
struct BwdItem {
  bool valid, is_q;
  int bh, row0, first, n_it;   // first resident row, first streamed row, steps
};
// (A table dealt out by the host and a work queue both balance 48 x 1050 better, but what they keep in
// registers slows every step by more.)
template <bool MANY>
__device__ __forceinline__ BwdItem bwd_item(int k, int BH, int S) {
  if (!MANY && k > 0) return BwdItem{};
  const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  const int n_tiles = (S + kRows - 1) / kRows;
  const int e = k * G + ((k & 1) ? G - 1 - c : c);
  const int level = e / (2 * BH), in_level = e - level * 2 * BH;
  BwdItem it;
  it.valid = level < n_tiles;
  // (a last tile of at most one step: the level's key tiles have a step less than its query tiles)
  const bool q_first = (S - 1) % kRows < kStep;
  it.is_q = (in_level >= BH) != q_first;
  it.bh = in_level >= BH ? in_level - BH : in_level;
  it.row0 = (it.is_q ? n_tiles - 1 - level : level) * kRows;
  it.first = it.is_q ? 0 : it.row0;
  const int last = it.is_q ? min(it.row0 + kRows, S) : S;
  it.n_it = (last - it.first + kStep - 1) / kStep;
  return it;
}

// Whether delta = rowsum(dO o O) comes from a kernel ahead instead of the rows of O that this one loads
// beside those of dO. Forming it saves a launch and pays while the loaders have time for the rows: at
// head sizes below 64, whose rows are short, and while no CTA has a second item. Backward alone, us, formed here /
// given (D = 16 and 32 before whole warps issued the products):
//   D = 16   32 x 301 15.6 / 17.4   48 x 1024 95.7 / 96.6     8 x 2048 62.4 / 64.4
//   D = 32   32 x 301 17.0 / 18.7   48 x 1024 107.1 / 106.6   8 x 2048 71.6 / 71.4
//   D = 64   16 x 200 16.4 / 17.3   8 x 1024 45.5 / 45.7      (64 and 128 items)
//            32 x 301 21.1 / 21.3   8 x 2048 83-93 / 87-94    (192 and 256 items)
//            96 x 200 36.6 / 35.2   200 x 256 75.0 / 72.2     48 x 1024 143.0 / 137.2
constexpr bool delta_given(int D, bool many) { return D == 64 && many; }

template <int D, bool DROP, bool MANY>   // MANY: more items than CTAs
__global__ void __launch_bounds__(kThreads, 1) flash_bwd_f32_tc_kernel(const __grid_constant__ BwdArgs args) {
  using L = BwdSmem;
  constexpr bool kDeltaGiven = delta_given(D, MANY);
  constexpr uint32_t kExtra = 256, kSum1 = 320, kSum2 = 384;   // kSum1: dV; kSum2: dK or dQ
  constexpr int V4 = D / 4;                                    // float4 pieces of a row
  constexpr int NC = D / 4;                                    // columns of a sum per thread

  extern __shared__ __align__(1024) uint8_t smem[];
  BwdBars* bars = reinterpret_cast<BwdBars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
  const int lane = threadIdx.x % 32;
  const int S = args.S;

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicExch(args.status, DADATTN_E_CUDA);
    return;
  }
  const BwdItem item0 = bwd_item<MANY>(0, args.BH, S);   // used when there is one: formed ahead of the dependency wait
  if (threadIdx.x == 0) {
    mbar_init(&bars->a_full, kComputeThreads);
    mbar_init(&bars->p_full, kComputeThreads);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->settled, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->b1_full[s], kLoaderThreads);
      mbar_init(&bars->b1_empty[s], 1);
      mbar_init(&bars->x_full[s], 1);
    }
    for (int s = 0; s < 3; ++s) {
      mbar_init(&bars->b2_full[s], kLoaderThreads);
      mbar_init(&bars->b2_empty[s], 1);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == kWarpIssuer) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  pdl_wait();
  pdl_launch_dependents();

  if (warp >= kWarpLoader0) {
    setmaxnreg_dec<kRegsHelper>();
    if (warp < kWarpIssuer) {
      // ------------------------------ loaders ------------------------------
      // Thread t takes the same four columns of every kRowStep-th row of a streamed tile.
      const int t = threadIdx.x - kWarpLoader0 * 32;
      constexpr int kRowStep = kLoaderThreads / V4;
      constexpr int kMine = (kStep + kRowStep - 1) / kRowStep;
      const int rt = t / V4, c4 = t % V4;
      float* vec = reinterpret_cast<float*>(smem + L::kVec);
      bool ok = true;
      float4 x[kMine];
      float row_lse = 0.f, row_delta = 0.f;
      auto fetch = [&](float4 (&to)[kMine], const float* m, const BwdItem& it, int i) {
        const int r = it.first + i * kStep + rt;
        m += (static_cast<size_t>(it.bh) * S + r) * D + c4 * 4;
#pragma unroll
        for (int j = 0; j < kMine; ++j)
          to[j] = load4(m + j * kRowStep * D, rt + j * kRowStep < kStep && r + j * kRowStep < S, args.vec_ok);
      };
      BwdItem it = MANY ? bwd_item<MANY>(0, args.BH, S) : item0;
      fetch(x, it.is_q ? args.v : args.dout, it, 0);
      int s2 = 0, lap2 = 0, g = 0;   // g: steps so far, over all items
#pragma unroll(MANY ? 1 : 2)
      for (int n = 0; ok && it.valid && (MANY || n < 1); ++n) {
        const BwdItem nxt = bwd_item<MANY>(n + 1, args.BH, S);
        const bool is_q = it.is_q;
        const size_t unit = static_cast<size_t>(it.bh) * S;
        for (int i = 0; i < it.n_it; ++i, ++g) {
          const int s = g & 1;
          auto put = [&](uint8_t* to, const Split4 (&v)[kMine]) {
#pragma unroll
            for (int j = 0; j < kMine; ++j)
              if (rt + j * kRowStep < kStep) store_split<kStreamRow<D>>(to, kPlaneB, rt + j * kRowStep, c4, v[j]);
          };
          float delta[kMine];
          Split4 sp[kMine];
          if (!is_q) {
            const int rv = it.first + i * kStep + t;
            row_lse = t < kStep && rv < S ? __ldg(args.lse + unit + rv) : 0.f;
            if (kDeltaGiven) row_delta = t < kStep && rv < S ? args.delta[unit + rv] : 0.f;
          }
          if (!is_q && !kDeltaGiven) {
            float4 xo[kMine];
            fetch(xo, args.out, it, i);
#pragma unroll
            for (int j = 0; j < kMine; ++j) {
              delta[j] = dot4(x[j], xo[j]);
#pragma unroll
              for (int o = V4 / 2; o > 0; o >>= 1) delta[j] += __shfl_xor_sync(0xffffffffu, delta[j], o);
            }
          }
#pragma unroll
          for (int j = 0; j < kMine; ++j) sp[j] = split4(x[j]);
          fetch(x, is_q ? args.k : args.q, it, i);   // on its way while B2 goes to shared memory
          if (lap2 > 0 && !(ok = mbar_wait(&bars->b2_empty[s2], (lap2 - 1) & 1, abort_flag))) break;
          put(smem + L::kB2 + s2 * 3 * kPlaneB, sp);
          if (!is_q) {
            if (t < kStep) vec[s2 * 128 + t] = row_lse;
            if (kDeltaGiven && t < kStep) vec[s2 * 128 + 64 + t] = row_delta;
#pragma unroll
            for (int j = 0; j < kMine; ++j)
              if (!kDeltaGiven && c4 == 0 && rt + j * kRowStep < kStep) vec[s2 * 128 + 64 + rt + j * kRowStep] = delta[j];
          }
          fence_proxy_async_smem();
          mbar_arrive(&bars->b2_full[s2]);
          if (++s2 == 3) s2 = 0, ++lap2;
#pragma unroll
          for (int j = 0; j < kMine; ++j) sp[j] = split4(x[j]);
          const bool more = i + 1 < it.n_it;
          if (more || nxt.valid)
            fetch(x, (more ? is_q : nxt.is_q) ? args.v : args.dout, more ? it : nxt, more ? i + 1 : 0);
          if (g >= 2 && !(ok = mbar_wait(&bars->b1_empty[s], ((g >> 1) - 1) & 1, abort_flag))) break;
          put(smem + L::kB1 + s * 3 * kPlaneB, sp);
          fence_proxy_async_smem();
          mbar_arrive(&bars->b1_full[s]);
        }
        it = nxt;
      }
    } else {
      const uint32_t lead = elect_one(), tm = __reduce_max_sync(0xffffffffu, tmem);   // (known to be uniform, so)
      // ------------------------------ MMA issuer ------------------------------
      constexpr uint32_t idesc_x = make_idesc_bf16(kRows, kStep, 0, 0);   // A, B K-major
      constexpr uint32_t idesc_s = make_idesc_bf16(kRows, D, 0, 1);       // A from tensor memory, B MN-major
      const SmemDescBase a1 = make_desc_base_sw128(smem_u32(smem + L::kA1), 0);
      const SmemDescBase a2 = make_desc_base_sw128(smem_u32(smem + L::kA2), 0);
      const SmemDescBase b1_0 = make_desc_base_rows<kStreamRow<D>>(smem_u32(smem + L::kB1));
      const SmemDescBase b2_0 = make_desc_base_rows<kStreamRow<D>>(smem_u32(smem + L::kB2));
      auto issue_x = [&](int i) -> bool {
        const int s = i & 1;
        const uint32_t par = (i >> 1) & 1, tx = tm + s * 128;
        const int s2 = i % 3;
        const SmemDescBase b1{b1_0.lo + s * (3 * kPlaneB >> 4), b1_0.hi};
        const SmemDescBase b2{b2_0.lo + s2 * (3 * kPlaneB >> 4), b2_0.hi};
        auto product = [&](uint32_t td, const SmemDescBase& a, const SmemDescBase& b) {
#pragma unroll
          for (int m = 0; m < 6; ++m)
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              mma_ss_warp(td, desc_at(a, product_a(m) * kPlaneA + kk * 32), desc_at(b, product_b(m) * kPlaneB + kk * 32),
                     idesc_x, (m > 0 || kk > 0) ? 1u : 0u, lead);
        };
        if (!warp_wait(&bars->b2_full[s2], (i / 3) & 1, abort_flag)) return false;
        tc_fence_after_sync();
        product(tx + 64, a2, b2);
        if (!warp_wait(&bars->b1_full[s], par, abort_flag)) return false;
        tc_fence_after_sync();
        product(tx, a1, b1);
        mma_commit_warp(&bars->x_full[s], lead);
        return true;
      };
      auto issue_sums = [&](int i, bool is_q) -> bool {
        const int s = i & 1;
        const uint32_t tx = tm + s * 128;
        const int s2 = i % 3;
        const SmemDescBase b1{b1_0.lo + s * (3 * kPlaneB >> 4), b1_0.hi};
        const SmemDescBase b2{b2_0.lo + s2 * (3 * kPlaneB >> 4), b2_0.hi};
        if (!warp_wait(&bars->p_full, i & 1, abort_flag)) return false;
        tc_fence_after_sync();
        // the planes of 16 streamed rows kk lie over the 16 columns their scores came from
        if (!is_q) {
#pragma unroll
          for (int m = 0; m < 6; ++m)
#pragma unroll
            for (int kk = 0; kk < kStep / 16; ++kk) {
              const uint32_t at = (product_a(m) == 0 ? 0u : product_a(m) == 1 ? 8u : 64u) + kk * 16;
              mma_ts_warp(tm + kSum1, tx + at, desc_at(b2, product_b(m) * kPlaneB + kk * 16 * kStreamRow<D>), idesc_s,
                     (m > 0 || kk > 0) ? 1u : 0u, lead);
            }
        }
        mma_commit_warp(&bars->b2_empty[s2], lead);
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int kk = 0; kk < kStep / 16; ++kk) {
            const uint32_t at = product_a(m) == 0 ? tx + 64 + 8 + kk * 16 : tm + kExtra + (product_a(m) - 1) * 8 + kk * 16;
            mma_ts_warp(tm + kSum2, at, desc_at(b1, product_b(m) * kPlaneB + kk * 16 * kStreamRow<D>), idesc_s,
                   (m > 0 || kk > 0) ? 1u : 0u, lead);
          }
        mma_commit_warp(&bars->b1_empty[s], lead);
        mma_commit_warp(&bars->acc_done, lead);
        return true;
      };
      bool ok = true;
      int g = 0;   // steps so far, over all items
#pragma unroll(MANY ? 1 : 2)
      for (int n = 0; ok && (MANY || n < 1); ++n) {
        const BwdItem it = MANY ? bwd_item<MANY>(n, args.BH, S) : item0;
        if (!it.valid) break;
        ok = warp_wait(&bars->a_full, n & 1, abort_flag) && issue_x(g) && (it.n_it < 2 || issue_x(g + 1));
        for (int i = 0; ok && i < it.n_it; ++i) ok = issue_sums(g + i, it.is_q) && (i + 2 >= it.n_it || issue_x(g + i + 2));
        g += it.n_it;
      }
      settle_products_warp(&bars->settled, lead);
    }
  } else {
    setmaxnreg_inc<kRegsCompute>();
    // ------------------------------ compute ------------------------------
    const int cg = warp / 4, quad = warp % 4;   // which 16 columns of a step; TMEM lane quadrant
    const int row = quad * 32 + lane;           // resident row = TMEM lane
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    float* vec = reinterpret_cast<float*>(smem + L::kVec);
    const float scale = args.scale;
    const float keep_scale = DROP ? 1.0f / (1.0f - args.rate) : 1.0f;
    bool ok = true;
    // The resident tiles of item n, split into planes. For every item but the first this happens while
    // the sums of the item before it are still being formed (its last scores have been seen, so
    // nothing reads the tiles any more), and the rows come from L2.
    auto load_resident = [&](const BwdItem& it, int n) {
      constexpr int kRowStep = kComputeThreads / V4;
      const int rt = threadIdx.x / V4, c4 = threadIdx.x % V4;
      const size_t at = (static_cast<size_t>(it.bh) * S + it.row0 + rt) * D + c4 * 4;
      const float *a1 = (it.is_q ? args.q : args.k) + at, *a2 = (it.is_q ? args.dout : args.v) + at, *oo = args.out + at;
      float* own = reinterpret_cast<float*>(smem + L::kOwn) + (n & 1) * kRows;
      constexpr int kMine = kRows / kRowStep;
      float4 x1[kMine], x2[kMine];   // all in flight at once
#pragma unroll
      for (int j = 0; j < kMine; ++j) {
        const bool in = it.row0 + rt + j * kRowStep < S;
        x1[j] = load4(a1 + j * kRowStep * D, in, args.vec_ok);
        x2[j] = load4(a2 + j * kRowStep * D, in, args.vec_ok);
      }
      const bool form_delta = !kDeltaGiven && it.is_q;
      float4 xo[kMine];
      auto load_out = [&]() {
#pragma unroll
        for (int j = 0; j < kMine; ++j) xo[j] = load4(oo + j * kRowStep * D, it.row0 + rt + j * kRowStep < S, args.vec_ok);
      };
      if (form_delta && D < 64) load_out();
#pragma unroll
      for (int j = 0; j < kMine; ++j) store_split(smem + L::kA1, kPlaneA, rt + j * kRowStep, c4, split4(x1[j]));
      if (form_delta && D == 64) load_out();   // (into x1's registers)
#pragma unroll
      for (int j = 0; j < kMine; ++j) store_split(smem + L::kA2, kPlaneA, rt + j * kRowStep, c4, split4(x2[j]));
      if (form_delta) {
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
          float delta = dot4(x2[j], xo[j]);
#pragma unroll
          for (int o = V4 / 2; o > 0; o >>= 1) delta += __shfl_xor_sync(0xffffffffu, delta, o);
          if (c4 == 0) own[rt + j * kRowStep] = delta;
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(&bars->a_full);
    };
    // Rows of 128 bytes of the item's tiles into L2, a step or more ahead of load_resident.
    auto prefetch_resident = [&](const BwdItem& it) {
      const float* a = (threadIdx.x < kComputeThreads / 2 ? (it.is_q ? args.q : args.k) : (it.is_q ? args.dout : args.v)) +
                       (static_cast<size_t>(it.bh) * S + it.row0) * D;
      const int at = (threadIdx.x % (kComputeThreads / 2)) * 32;   // 256 lines of 32 floats at head size 64
      if (at < min(kRows, S - it.row0) * D) asm volatile("prefetch.global.L2 [%0];" ::"l"(a + at));
    };

    float sum1[NC], sum2[NC];
    auto take_sums = [&](int i, bool is_q) -> bool {
      if (!mbar_wait(&bars->acc_done, i & 1, abort_flag)) return false;
      tc_fence_after_sync();
      if (!is_q) tmem_add<NC>(tlane + kSum1 + cg * NC, sum1);
      tmem_add<NC>(tlane + kSum2 + cg * NC, sum2);
      return true;
    };
    BwdItem it{}, nxt = MANY ? bwd_item<MANY>(0, args.BH, S) : item0;
    int step = 0;   // over all items
    int left = 0;   // where a wait runs out: the first item whose barrier has not been joined
#pragma unroll(MANY ? 1 : 2)
    for (int n = 0; MANY || n < 2; ++n) {
      if (nxt.valid) load_resident(nxt, n);
      if (n > 0) {   // the results of the item before
        if (!(ok = take_sums(step - 1, it.is_q))) {
          left = n;
          break;
        }
        const int rows = min(kRows, S - it.row0);
        const size_t at = (static_cast<size_t>(it.bh) * S + it.row0) * D;
        if constexpr (MANY) {
          write_sums<D, NC>((it.is_q ? args.dq : args.dk) + at, row, cg * NC, sum2, rows, args.vec_ok);
          if (!it.is_q) write_sums<D, NC>(args.dv + at, row, cg * NC, sum1, rows, args.vec_ok);
        } else {   // (every product has completed: the stages are free)
          float* stage = reinterpret_cast<float*>(smem + L::kB1);
          stage_rows<D, NC>(stage, row, cg * NC, sum2);
          if (!it.is_q) stage_rows<D, NC>(stage + kRows * (D + 4), row, cg * NC, sum1);
          compute_sync();
          write_rows<D>((it.is_q ? args.dq : args.dk) + at, stage, rows, args.vec_ok);
          if (!it.is_q) write_rows<D>(args.dv + at, stage + kRows * (D + 4), rows, args.vec_ok);
        }
      }
      it = nxt;
      if (!it.valid) break;
      nxt = bwd_item<MANY>(n + 1, args.BH, S);
      const bool is_q = it.is_q;
      const int row0 = it.row0, first = it.first, n_it = it.n_it, bh = it.bh;
      if (nxt.valid) prefetch_resident(nxt);
      if (!kDeltaGiven && is_q) compute_sync();   // delta of all rows
      const int r_own = row0 + row;
      const size_t at_own = static_cast<size_t>(bh) * S + r_own;
      const float own_lse = is_q && r_own < S ? __ldg(args.lse + at_own) : 0.f;
      const float own_delta = !is_q ? 0.f
                              : !kDeltaGiven ? reinterpret_cast<const float*>(smem + L::kOwn)[(n & 1) * kRows + row]
                              : r_own < S ? args.delta[at_own] : 0.f;
      const uint64_t unit = static_cast<uint64_t>(args.unit0 + bh) * S;

#pragma unroll
      for (int c = 0; c < NC; ++c) sum1[c] = sum2[c] = 0.f;

      for (int i = 0; i < n_it; ++i, ++step) {
        const int s = step & 1;
        const int col0 = first + i * kStep + cg * 16;        // streamed row of this thread's first column
        if (!(ok = mbar_wait(&bars->x_full[s], (step >> 1) & 1, abort_flag))) break;
        // (the row scalars came with B2)
        if (!is_q && !(ok = mbar_wait(&bars->b2_full[step % 3], (step / 3) & 1, abort_flag))) break;
        tc_fence_after_sync();
        const uint32_t tx = tlane + s * 128 + cg * 16;
        float2 p[8], g[8];
        {
          uint32_t x1[16], x2[16];
          tmem_ld<16>(tx, x1);
          tmem_ld<16>(tx + 64, x2);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            p[c] = make_float2(__uint_as_float(x1[2 * c]), __uint_as_float(x1[2 * c + 1]));
            g[c] = make_float2(__uint_as_float(x2[2 * c]), __uint_as_float(x2[2 * c + 1]));
          }
        }
        const float2* lse_s = reinterpret_cast<const float2*>(vec + (step % 3) * 128 + cg * 16);
        const float2* delta_s = lse_s + 32;
        // p = exp(s scale - lse)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float2 l = is_q ? make_float2(own_lse, own_lse) : lse_s[c];
          p[c] = exp2_of(ffma2(p[c], make_float2(scale, scale), make_float2(-l.x, -l.y)));
        }
        // every pair of the step visible (key <= query < S)?
        const bool whole = is_q ? first + i * kStep + kStep - 1 <= row0
                                : first + i * kStep >= row0 + kRows - 1 && first + i * kStep + kStep <= S;
        if (!whole) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int rq = is_q ? r_own : col0 + c, ck = is_q ? col0 + c : r_own;
            float& x = (c & 1) ? p[c / 2].y : p[c / 2].x;
            if (ck > rq || rq >= S) x = 0.f;
          }
        }
        // ds = p (dP - delta) scale, with dropout on P and dP alike
        uint32_t keep = 0xffffu;
        if (DROP) {
          // where the warp's 32 x 16 block has visible pairs. The same number of draws in every lane: a warp's
          // loop runs as long as its longest lane's, and a constant count needs no bounds (32 x 301 x 32 with
          // dropout: 53.7 -> 52.8 us a step).
          if (is_q ? col0 <= row0 + quad * 32 + 31 : col0 + 15 >= row0 + quad * 32)
            keep = is_q ? philox_keep_bits<2>(args.rng, (unit + r_own) * S + col0, 1u, 16)
                        : philox_keep_bits<2>(args.rng, (unit + col0) * S + r_own, static_cast<uint32_t>(S), 16);
          __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float2 dl = is_q ? make_float2(own_delta, own_delta) : delta_s[c];
          const float2 pr = p[c];
          if (DROP) {
            const float2 mk = make_float2((keep >> (2 * c)) & 1u ? keep_scale : 0.f, (keep >> (2 * c + 1)) & 1u ? keep_scale : 0.f);
            p[c] = fmul2(p[c], mk);
            g[c] = fmul2(g[c], mk);
          }
          g[c] = fmul2(fmul2(pr, fadd2(g[c], make_float2(-dl.x, -dl.y))), make_float2(scale, scale));
        }
        if (i > 0 && !(ok = take_sums(step - 1, is_q))) break;   // and with it the planes of step i - 1 are free
        if (!is_q) tmem_store_split(p, tx, tx + 8, tx + 64);
        tmem_store_split(g, tx + 64 + 8, tlane + kExtra + cg * 16, tlane + kExtra + cg * 16 + 8);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(&bars->p_full);
      }
      if (!ok) {
        left = n + 1;
        break;
      }
    }
    // A warp that has given up joins the named barriers that are left: nothing bounds the wait of the others there.
    if (!ok) {
      if constexpr (!MANY) {
        compute_sync();   // (ahead of the results; that of a dQ item's delta comes before its first wait)
      } else if constexpr (!kDeltaGiven) {
        for (;; ++left) {
          const BwdItem e = bwd_item<MANY>(left, args.BH, S);
          if (!e.valid) break;
          if (e.is_q) compute_sync();
        }
      }
    }
    tc_fence_before_sync();
  }

  __syncthreads();
  if (warp == kWarpIssuer) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && bars->abort_flag) report_timeout(args.status, bars->abort_flag);
}

template <int D, bool DROP, bool MANY>
int launch(const BwdArgs& a, unsigned grid, cudaStream_t st) {
  auto kern = flash_bwd_f32_tc_kernel<D, DROP, MANY>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdSmem::kBytes));
  static std::atomic<int> regs{0};
  if (int rc = check_launch_registers(reinterpret_cast<const void*>(kern), kRegsLaunch, regs)) return rc;
  if (delta_given(D, MANY))
    if (int rc = launch_delta_f32_d64(a.delta, a.dout, a.out, static_cast<int64_t>(a.BH) * a.S, a.vec_ok, st)) return rc;
  DAD_CUDA(launch_pdl(kern, dim3(grid), dim3(kThreads), BwdSmem::kBytes, st, a));
  return DADATTN_OK;
}
template <int D, bool DROP>
int launch(const BwdArgs& a, cudaStream_t st) {
  const long long items = 2LL * a.BH * ((a.S + kRows - 1) / kRows);
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (items > INT32_MAX / 2) return fail(DADATTN_E_UNSUPPORTED, "too many (tile, batch x head) items");
  // (an item loop that runs once costs the smallest calls 1.3 us of 7)
  return items <= sms ? launch<D, DROP, false>(a, static_cast<unsigned>(items), st)
                      : launch<D, DROP, true>(a, static_cast<unsigned>(sms), st);
}

}  // namespace

int launch_bwd_f32_tc(float* dq, float* dk, float* dv, float* delta, const float* dout, const float* out, const float* lse,
                      const float* q, const float* k, const float* v, int BH, int S, int D, float scale, float rate,
                      uint64_t seed, uint64_t offset, int64_t unit0, bool vec_ok, cudaStream_t st) {
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  const BwdArgs a = {dq, dk, dv, dout, out, lse, q, k, v, delta, BH, S, scale, rate, make_philox_rounds(seed, offset, rate, static_cast<uint32_t>(S)),
                     unit0, vec_ok, status};
  const bool drop = rate > 0.f;
  if (D == 64) return drop ? launch<64, true>(a, st) : launch<64, false>(a, st);
  if (D == 32) return drop ? launch<32, true>(a, st) : launch<32, false>(a, st);
  return drop ? launch<16, true>(a, st) : launch<16, false>(a, st);
}

}  // namespace dadattn
