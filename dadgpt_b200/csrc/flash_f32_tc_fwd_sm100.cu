// fp32 forward on the tensor cores (head sizes 16, 32, 64): exact fp32 operands as three bf16 planes
// (f32_split.cuh), online softmax and output sums in fp32 registers.
//
// The arithmetic is that of the reference's flash_fwd_kernel (cuda/attention.cu:17-73). A CTA owns
// 128 query rows and takes the keys 64 at a time:
//   warps 0-15  four threads per row, 16 key columns each: row max (exchanged between them through
//               shared memory), exponentials, p split into planes and written back to tensor memory
//               over the scores, from where the P V product takes them as its A operand; each step's
//               P V is added to an fp32 register sum, so the output is never rescaled in tensor memory
//   warps 16-26 fetch fp32 K / V rows, split them in registers, fill the shared-memory rings
//   warp 27     issues the products: P V of step i, scores of step i + 2, P V of step i + 1, ...
// A step costs 2304 clocks of tensor pipe at head size 64 (24 + 24 products of 48; the pipe's counter
// takes 32) and about 2100 issue slots per scheduler, and takes about 3550 clocks (48 x 1024): the planes
// of a step are stored only after the last step's sums have been taken.
// CTAs are persistent where there are more items than SMs, as in the backward: the rings run on across
// items and the next Q is fetched and split while the last sums complete (48 x 1024 x 64: 58 -> 55.6 us,
// 148 x 512: 57.0 -> 46.6, 72 x 777: 69.9 -> 62.0).
// Tensor memory: score buffer b at 64 b, the third planes at 128, P V at 192.
#include <cfloat>

#include "f32_split.cuh"

namespace dadattn {
namespace {

using namespace f32tc;

constexpr int kStages = 3;
struct FwdSmem {
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + 3 * kPlaneA;                  // [stage][3 planes]
  static constexpr int kV = kK + kStages * 3 * kPlaneB;
  static constexpr int kMax = kV + kStages * 3 * kPlaneB;      // [2 steps][4 column groups][128]
  static constexpr int kBars = kMax + 4096;
  static constexpr int kBytes = kBars + 256;
  static_assert(kBytes <= 232448, "shared memory of a CTA exceeded");
};
struct FwdBars {
  uint64_t q_full, p_full, acc_done, x_full[2], settled;
  uint64_t k_full[kStages], v_full[kStages], k_empty[kStages], v_empty[kStages];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FwdBars) <= 256, "barrier block");

struct FwdArgs {
  float *out, *lse;
  const float *q, *k, *v;
  int BH, S;
  float scale, rate;
  PhiloxRounds rng;
  int64_t unit0;
  bool vec_ok;
  int* status;
};

// Query tiles with the most keys first; CTA c of G takes the items k G + (k even ? c : G-1-c).
struct FwdItem {
  bool valid;
  int bh, row0, n_it;   // first query row, steps
};
template <bool MANY>
__device__ __forceinline__ FwdItem fwd_item(int k, int BH, int S) {
  if (!MANY && k > 0) return FwdItem{};
  const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  const int n_tiles = (S + kRows - 1) / kRows;
  const int e = k * G + ((k & 1) ? G - 1 - c : c);
  const int level = e / BH;
  FwdItem it;
  it.valid = level < n_tiles;
  it.bh = e - level * BH;
  it.row0 = (n_tiles - 1 - level) * kRows;
  it.n_it = (min(it.row0 + kRows, S) + kStep - 1) / kStep;
  return it;
}

template <int D, bool DROP, bool MANY>   // MANY: more items than CTAs
__global__ void __launch_bounds__(kThreads, 1) flash_fwd_f32_tc_kernel(const __grid_constant__ FwdArgs args) {
  using L = FwdSmem;
  constexpr uint32_t kExtra = 128, kSum = 192;
  constexpr int V4 = D / 4;     // float4 pieces of a row
  constexpr int NC = D / 4;     // output columns per thread

  extern __shared__ __align__(1024) uint8_t smem[];
  FwdBars* bars = reinterpret_cast<FwdBars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0);
  const int lane = threadIdx.x % 32;
  const int S = args.S;

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicExch(args.status, DADATTN_E_CUDA);
    return;
  }
  const FwdItem item0 = fwd_item<MANY>(0, args.BH, S);   // used when there is one: formed ahead of the dependency wait

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, kComputeThreads);
    mbar_init(&bars->p_full, kComputeThreads);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->settled, 1);
    for (int s = 0; s < 2; ++s) mbar_init(&bars->x_full[s], 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->k_full[s], kLoaderThreads);
      mbar_init(&bars->v_full[s], kLoaderThreads);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_empty[s], 1);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == kWarpIssuer) {
    tmem_alloc(&bars->tmem_base, 256);
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
      // Thread t takes the same four columns of every kRowStep-th row of a tile.
      const int t = threadIdx.x - kWarpLoader0 * 32;
      constexpr int kRowStep = kLoaderThreads / V4;
      constexpr int kMine = (kStep + kRowStep - 1) / kRowStep;
      const int rt = t / V4, c4 = t % V4;
      bool ok = true;
      int s = 0, lap = 0;
      for (int n = 0; ok && (MANY || n < 1); ++n) {
        const FwdItem it = MANY ? fwd_item<MANY>(n, args.BH, S) : item0;
        if (!it.valid) break;
        const size_t base = static_cast<size_t>(it.bh) * S * D + c4 * 4;
        const float *kk = args.k + base, *vv = args.v + base;
        for (int i = 0; ok && i < it.n_it; ++i) {
          const int r = i * kStep + rt;
          auto fetch = [&](float4 (&x)[kMine], const float* m) {
            m += static_cast<size_t>(r) * D;
#pragma unroll
            for (int j = 0; j < kMine; ++j)
              x[j] = load4(m + j * kRowStep * D, rt + j * kRowStep < kStep && r + j * kRowStep < S, args.vec_ok);
          };
          float4 x[kMine];
          Split4 sp[kMine];
          auto put = [&](uint8_t* tile, uint64_t* empty, uint64_t* full) -> bool {
            if (lap > 0 && !mbar_wait(empty, (lap - 1) & 1, abort_flag)) return false;
#pragma unroll
            for (int j = 0; j < kMine; ++j)
              if (rt + j * kRowStep < kStep) store_split<kStreamRow<D>>(tile, kPlaneB, rt + j * kRowStep, c4, sp[j]);
            fence_proxy_async_smem();
            mbar_arrive(full);
            return true;
          };
          fetch(x, kk);
#pragma unroll
          for (int j = 0; j < kMine; ++j) sp[j] = split4(x[j]);
          fetch(x, vv);   // on its way while K goes to shared memory
          if (!(ok = put(smem + L::kK + s * 3 * kPlaneB, &bars->k_empty[s], &bars->k_full[s]))) break;
#pragma unroll
          for (int j = 0; j < kMine; ++j) sp[j] = split4(x[j]);
          ok = put(smem + L::kV + s * 3 * kPlaneB, &bars->v_empty[s], &bars->v_full[s]);
          if (++s == kStages) s = 0, ++lap;
        }
      }
    } else {
      const uint32_t lead = elect_one(), tm = __reduce_max_sync(0xffffffffu, tmem);   // (known to be uniform, so)
      // ------------------------------ MMA issuer ------------------------------
      constexpr uint32_t idesc_x = make_idesc_bf16(kRows, kStep, 0, 0);   // Q, K: K-major
      constexpr uint32_t idesc_s = make_idesc_bf16(kRows, D, 0, 1);       // P from tensor memory, V MN-major
      const SmemDescBase qd = make_desc_base_sw128(smem_u32(smem + L::kQ), 0);
      const SmemDescBase k0 = make_desc_base_rows<kStreamRow<D>>(smem_u32(smem + L::kK));
      const SmemDescBase v0 = make_desc_base_rows<kStreamRow<D>>(smem_u32(smem + L::kV));
      auto issue_x = [&](int i) -> bool {
        const int s = i % kStages;
        const uint32_t tx = tm + (i & 1) * 64;
        const SmemDescBase kd{k0.lo + s * (3 * kPlaneB >> 4), k0.hi};
        if (!warp_wait(&bars->k_full[s], (i / kStages) & 1, abort_flag)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            mma_ss_warp(tx, desc_at(qd, product_a(m) * kPlaneA + kk * 32), desc_at(kd, product_b(m) * kPlaneB + kk * 32),
                   idesc_x, (m > 0 || kk > 0) ? 1u : 0u, lead);
        mma_commit_warp(&bars->x_full[i & 1], lead);
        mma_commit_warp(&bars->k_empty[s], lead);
        return true;
      };
      auto issue_pv = [&](int i) -> bool {
        const int s = i % kStages;
        const uint32_t tx = tm + (i & 1) * 64;
        const SmemDescBase vd{v0.lo + s * (3 * kPlaneB >> 4), v0.hi};
        if (!warp_wait(&bars->v_full[s], (i / kStages) & 1, abort_flag)) return false;
        if (!warp_wait(&bars->p_full, i & 1, abort_flag)) return false;
        tc_fence_after_sync();
        // the planes of 16 keys kk lie over the 16 columns their scores came from
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int kk = 0; kk < kStep / 16; ++kk) {
            const uint32_t at = product_a(m) == 2 ? tm + kExtra + kk * 8 : tx + kk * 16 + product_a(m) * 8;
            mma_ts_warp(tm + kSum, at, desc_at(vd, product_b(m) * kPlaneB + kk * 16 * kStreamRow<D>), idesc_s,
                   (m > 0 || kk > 0) ? 1u : 0u, lead);
          }
        mma_commit_warp(&bars->v_empty[s], lead);
        mma_commit_warp(&bars->acc_done, lead);
        return true;
      };
      bool ok = true;
      int g = 0;   // steps so far, over all items
      for (int n = 0; ok && (MANY || n < 1); ++n) {
        const FwdItem it = MANY ? fwd_item<MANY>(n, args.BH, S) : item0;
        if (!it.valid) break;
        ok = warp_wait(&bars->q_full, n & 1, abort_flag) && issue_x(g) && (it.n_it < 2 || issue_x(g + 1));
        for (int i = 0; ok && i < it.n_it; ++i) ok = issue_pv(g + i) && (i + 2 >= it.n_it || issue_x(g + i + 2));
        g += it.n_it;
      }
      settle_products_warp(&bars->settled, lead);
    }
  } else {
    setmaxnreg_inc<kRegsCompute>();
    // ------------------------------ softmax ------------------------------
    const int cg = warp / 4, quad = warp % 4;   // which 16 keys of a step; TMEM lane quadrant
    const int row = quad * 32 + lane;           // query row of the tile = TMEM lane
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    float* part = reinterpret_cast<float*>(smem + L::kMax);
    // the four warps that share these 32 rows
    auto rows_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory"); };
    bool ok = true;
    // Q of an item, split into planes: for every item but the first while the last sums of the item
    // before it are still being formed (its last scores have been seen, so nothing reads Q any more).
    auto load_resident = [&](const FwdItem& it) {
      constexpr int kRowStep = kComputeThreads / V4;
      const int rt = threadIdx.x / V4, c4 = threadIdx.x % V4;
      const float* qq = args.q + (static_cast<size_t>(it.bh) * S + it.row0 + rt) * D + c4 * 4;
      constexpr int kMine = kRows / kRowStep;
      float4 x[kMine];   // all in flight at once
#pragma unroll
      for (int j = 0; j < kMine; ++j) x[j] = load4(qq + j * kRowStep * D, it.row0 + rt + j * kRowStep < S, args.vec_ok);
#pragma unroll
      for (int j = 0; j < kMine; ++j) store_split(smem + L::kQ, kPlaneA, rt + j * kRowStep, c4, split4(x[j]));
      fence_proxy_async_smem();
      mbar_arrive(&bars->q_full);
    };
    // Q of an item into L2, a step or more ahead of load_resident
    auto prefetch_resident = [&](const FwdItem& it) {
      const int at = threadIdx.x * 32;   // 128 bytes per thread
      if (at < min(kRows, S - it.row0) * D)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(args.q + (static_cast<size_t>(it.bh) * S + it.row0) * D + at));
    };
    const float scale = args.scale;
    const float keep_scale = DROP ? 1.0f / (1.0f - args.rate) : 1.0f;
    float m = -FLT_MAX, l = 0.f, o[NC];
    auto take_sums = [&](int i) -> bool {
      if (!mbar_wait(&bars->acc_done, i & 1, abort_flag)) return false;
      tc_fence_after_sync();
      tmem_add<NC>(tlane + kSum + cg * NC, o);
      return true;
    };
    FwdItem it{}, nxt = MANY ? fwd_item<MANY>(0, args.BH, S) : item0;
    int step = 0;   // over all items
    int synced = 0; // where a wait runs out: the barriers of the row's warps joined until then
#pragma unroll(MANY ? 1 : 2)
    for (int n = 0; MANY || n < 2; ++n) {
      if (nxt.valid) load_resident(nxt);
      if (n > 0) {   // the results of the item before
        if (!(ok = take_sums(step - 1))) {
          synced = step + n - 1;
          break;
        }
        float* own = part + ((step + n - 1) & 1) * 512;   // (the buffers of `part` alternate over steps and results)
        own[cg * 128 + row] = l;
        rows_sync();
        const float l_all = (own[row] + own[128 + row]) + (own[256 + row] + own[384 + row]);
        const float inv = 1.0f / l_all;
#pragma unroll
        for (int c = 0; c < NC; ++c) o[c] *= inv;
        const size_t at = static_cast<size_t>(it.bh) * S + it.row0;
        const int rows = min(kRows, S - it.row0);
        if (cg == 0 && row < rows) args.lse[at + row] = m + logf(l_all);
        if constexpr (MANY) {
          write_sums<D, NC>(args.out + at * D, row, cg * NC, o, rows, args.vec_ok);
        } else {   // (every product has completed: the rings are free)
          float* stage = reinterpret_cast<float*>(smem + L::kK);
          stage_rows<D, NC>(stage, row, cg * NC, o);
          compute_sync();
          write_rows<D>(args.out + at * D, stage, rows, args.vec_ok);
        }
      }
      it = nxt;
      if (!it.valid) break;
      nxt = fwd_item<MANY>(n + 1, args.BH, S);
      if (nxt.valid) prefetch_resident(nxt);
      const int row0 = it.row0, n_it = it.n_it, bh = it.bh, r = row0 + row;
      m = -FLT_MAX, l = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) o[c] = 0.f;

      for (int i = 0; i < n_it; ++i, ++step) {
        if (!(ok = mbar_wait(&bars->x_full[step & 1], (step >> 1) & 1, abort_flag))) {
          synced = step + n;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tx = tlane + (step & 1) * 64 + cg * 16;
        const int c0 = i * kStep + cg * 16;
        float2 p[8];
        {
          uint32_t x[16];
          tmem_ld<16>(tx, x);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            p[c] = fmul2(make_float2(__uint_as_float(x[2 * c]), __uint_as_float(x[2 * c + 1])), make_float2(scale, scale));
        }
        if (i * kStep + kStep - 1 > row0) {   // keys beyond a row's own
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float& x = (c & 1) ? p[c / 2].y : p[c / 2].x;
            if (c0 + c > r) x = -FLT_MAX;
          }
        }
        float mx0 = fmaxf(p[0].x, p[0].y), mx1 = fmaxf(p[1].x, p[1].y);
#pragma unroll
        for (int c = 2; c < 8; c += 2) {
          mx0 = fmax3(mx0, p[c].x, p[c].y);
          mx1 = fmax3(mx1, p[c + 1].x, p[c + 1].y);
        }
        float* own = part + ((step + n) & 1) * 512;
        own[cg * 128 + row] = fmaxf(mx0, mx1);
        rows_sync();
        // every row sees key 0 in step 0: the max over all columns is finite from there on
        const float m_new = fmax3(fmaxf(m, own[row]), fmaxf(own[128 + row], own[256 + row]), own[384 + row]);
        const float corr = exp2_of(make_float2(m - m_new, 0.f)).x;
        m = m_new;
        float2 sum = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          p[c] = exp2_of(fadd2(p[c], make_float2(-m_new, -m_new)));
          sum = fadd2(sum, p[c]);
        }
        if (DROP) {
          const uint64_t at = (static_cast<uint64_t>(args.unit0 + bh) * S + r) * S + c0;
          // (where the warp's block has visible pairs; the same number of draws in every lane)
          const uint32_t keep = c0 <= row0 + quad * 32 + 31 ? philox_keep_bits<4>(args.rng, at, 1u, 16) : 0u;
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 8; ++c)
            p[c] = fmul2(p[c], make_float2((keep >> (2 * c)) & 1u ? keep_scale : 0.f, (keep >> (2 * c + 1)) & 1u ? keep_scale : 0.f));
        }
        l = fmaf(l, corr, sum.x + sum.y);
        if (i > 0) {   // and with it the planes of step i - 1 are free
          if (!(ok = take_sums(step - 1))) {
            synced = step + n + 1;
            break;
          }
#pragma unroll
          for (int c = 0; c < NC; ++c) o[c] *= corr;
        }
        tmem_store_split(p, tx, tx + 8, tlane + kExtra + cg * 8);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(&bars->p_full);
      }
      if (!ok) break;
    }
    // A warp that has given up joins the named barriers that are left: nothing bounds the wait of the others there.
    if (!ok) {
      for (int n = 0; MANY || n < 1; ++n) {
        const FwdItem e = MANY ? fwd_item<MANY>(n, args.BH, S) : item0;
        if (!e.valid) break;
        for (int i = 0; i <= e.n_it; ++i)
          if (--synced < 0) rows_sync();
      }
      if (!MANY) compute_sync();
    }
    tc_fence_before_sync();
  }

  __syncthreads();
  if (warp == kWarpIssuer) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, 256);
  }
  if (threadIdx.x == 0 && bars->abort_flag) report_timeout(args.status, bars->abort_flag);
}

template <int D, bool DROP, bool MANY>
int launch(const FwdArgs& a, unsigned grid, cudaStream_t st) {
  auto kern = flash_fwd_f32_tc_kernel<D, DROP, MANY>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdSmem::kBytes));
  static std::atomic<int> regs{0};
  if (int rc = check_launch_registers(reinterpret_cast<const void*>(kern), kRegsLaunch, regs)) return rc;
  DAD_CUDA(launch_pdl(kern, dim3(grid), dim3(kThreads), FwdSmem::kBytes, st, a));
  return DADATTN_OK;
}
template <int D, bool DROP>
int launch(const FwdArgs& a, cudaStream_t st) {
  const long long items = static_cast<long long>(a.BH) * ((a.S + kRows - 1) / kRows);
  int dev = 0, sms = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  DAD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (items > INT32_MAX / 2) return fail(DADATTN_E_UNSUPPORTED, "too many (query tile, batch x head) items");
  return items <= sms ? launch<D, DROP, false>(a, static_cast<unsigned>(items), st)
                      : launch<D, DROP, true>(a, static_cast<unsigned>(sms), st);
}

}  // namespace

int launch_fwd_f32_tc(float* out, float* lse, const float* q, const float* k, const float* v, int BH, int S, int D,
                      float scale, float rate, uint64_t seed, uint64_t offset, int64_t unit0, bool vec_ok,
                      cudaStream_t st) {
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  const FwdArgs a = {out, lse, q, k, v, BH, S, scale, rate, make_philox_rounds(seed, offset, rate), unit0, vec_ok, status};
  const bool drop = rate > 0.f;
  if (D == 64) return drop ? launch<64, true>(a, st) : launch<64, false>(a, st);
  if (D == 32) return drop ? launch<32, true>(a, st) : launch<32, false>(a, st);
  return drop ? launch<16, true>(a, st) : launch<16, false>(a, st);
}

}  // namespace dadattn
