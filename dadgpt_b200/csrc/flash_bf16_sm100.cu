// bf16 fused causal attention for sm_100a: TMA-staged tiles, tcgen05 MMAs accumulating in tensor
// memory, a warp-specialised online-softmax pipeline. The arithmetic is that of the reference's
// fused kernels (cuda/attention.cu) with bf16 operands and fp32 accumulation; the interface is
// its gpu_flash_attention_forward / _backward with bf16 pointers (include/dadattn.h).
//
// Forward, one CTA per 128 query rows of one (batch, head):
//   warp 0      TMA producer: Q once, then K/V tiles of 128 keys through a 2-stage ring
//   warp 1      MMA issuer (one elected lane) and owner of the TMEM allocation:
//               S = Q K^T (128x128, fp32 in TMEM), O_h += P_h V_h per 64-key half h
//   warps 2-9   softmax, two threads per query row: warps 2-5 own key columns 0-63 of every
//               tile, warps 6-9 columns 64-127 (a warp may only touch the TMEM lane quadrant
//               warp_id % 4). Each half keeps its OWN running max / sum and its OWN output
//               accumulator in TMEM, so the two threads of a row never synchronise inside the
//               loop; the halves are merged once, in the epilogue (split-K inside the CTA). Up to
//               2048 rows of bf16 tensors without dropout they agree on one of each (ONE_SUM).
//               Eight softmax warps give every scheduler two warps to hide the FFMA -> MUFU ->
//               FADD latencies behind each other.
//               A thread reads its 64 scores with tcgen05.ld, writes P as packed bf16 over them,
//               and rescales its O half in TMEM only when its max grew by more than 2^8 (lazy
//               rescale; exact result).
// S_{j+1} is issued before P_j V_j, so the tensor core works on the next tile while the
// exponentials of the current one are computed; the scores are double-buffered in TMEM.
//
// Head size 128, launches that do not fill the GPU and dropout; the others have the persistent two-tile kernel of
// flash_fwd128_sm100.cu, head size 64 that of flash_fwd64_sm100.cu. The entry points of all are here.
//
// Every mbarrier wait is bounded (sm100_ptx.cuh). If one runs out, the CTA raises its abort
// flag, everybody falls through to the common exit, TMEM is freed, and DADATTN_E_TIMEOUT is
// left in the device status word.
#include <cuda_bf16.h>

#include <cfloat>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {

// ---------------------------------------------------------------------------------------------
// Tensor maps (host)
// ---------------------------------------------------------------------------------------------
namespace {
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) !=
            cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
}  // namespace

int make_tensor_map_bf16(CUtensorMap* map, const void* base, int BH, int S, int D, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S),
                              static_cast<cuuint64_t>(BH)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(D) * 2,
                                 static_cast<cuuint64_t>(S) * D * 2};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return DADATTN_OK;
}

static int encode_units(CUtensorMap* map, const void* base, bool f32, int units, int S, int D, int box_columns, int box_rows,
                        CUtensorMapSwizzle swizzle, const UnitLayout& lay) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const int heads = lay.heads, batch = units / lay.heads;
  const cuuint64_t size = f32 ? 4 : 2;
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S),
                              static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(batch)};
  // a dimension of extent 1 still needs a legal stride (a multiple of 16 bytes)
  const cuuint64_t head_stride = static_cast<cuuint64_t>(heads > 1 ? lay.head : D) * size;
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(lay.row) * size, head_stride,
                                 static_cast<cuuint64_t>(lay.batch) * size};
  const cuuint32_t box[4] = {static_cast<cuuint32_t>(box_columns), static_cast<cuuint32_t>(box_rows), 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DADATTN_E_CUDA, "cuTensorMapEncodeTiled (4-D) failed (%d)", (int)r);
  return DADATTN_OK;
}
int make_tensor_map_bf16_units(CUtensorMap* map, const void* base, int units, int S, int D, int box_rows,
                               const UnitLayout& lay) {
  return encode_units(map, base, false, units, S, D, 64, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, lay);
}
int make_tensor_map_rows64(CUtensorMap* map, const void* base, bool f32, int units, int S, int D, int box_rows,
                           const UnitLayout& lay) {
  return encode_units(map, base, f32, units, S, D, f32 ? 16 : 32, box_rows, CU_TENSOR_MAP_SWIZZLE_64B, lay);
}

namespace {

using namespace ptx;

#define hot_wait(bar, parity, abort_flag) mbar_wait_at<24>(bar, parity, abort_flag, __LINE__)

constexpr int kBM = 128;          // query rows per CTA
constexpr int kBN = 128;          // keys per tile
constexpr int kStages = 2;        // K/V ring depth
constexpr int kPanelBytes = 128 * 128;  // [128 rows][64 bf16], 128-byte rows, swizzled
constexpr int kFwdThreads = 320;         // producer warp, MMA warp, 8 softmax warps
constexpr int kSoftmaxThreads = 256;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.0f;  // log2 units: P stays below 2^8

constexpr int kD = 128;           // head size
constexpr int kPanels = kD / 64;  // 128-byte wide panels of a row

// The probabilities P live in tensor memory between the softmax warps and the P V MMA, written over
// the scores they were computed from and read by the MMA as its A operand: an MMA with both operands
// in shared memory reads 8 KB per 64 clocks, all of an SM's shared-memory bandwidth, so every byte of
// P kept out of shared memory counts.
template <bool ONE_SUM>
struct FwdSmem {
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + kPanels * kPanelBytes;
  static constexpr int kV = kK + kStages * kPanels * kPanelBytes;
  static constexpr int kBars = kV + kStages * kPanels * kPanelBytes;
  static constexpr int kMaxFull = kBars + 256;           // ONE_SUM: barriers [2][half][quadrant] of
  static constexpr int kMax = kMaxFull + 128;            // a tile's maxima [2][half][row]
  // An SM that is set up for 164 KB has room beside this for blocks of the next kernel (1 KB each); with the maxima's 2 KB
  // it has none: 128 x 33 behind fp32 tensors 10.8 -> 12.9 us.
  static constexpr int kBytes = ONE_SUM ? kMax + 2 * 2 * kBM * 4 : kBars + 256;
};

struct FwdBars {
  uint64_t q_full, k_full[kStages], v_full[kStages], k_empty[kStages], v_empty[kStages];
  // p_full: one per score buffer. S_{j+1} is formed before P_j is complete, so that a warp can store P_{j+1}
  // while another still works on tile j: with one barrier for both its second arrival stood in for the other's
  // first, and P_j V_j read scores for probabilities (rows of infinities in one call of five at 8 x 3080 with
  // dropout, whose draws set the warps apart). P_{j+2} needs S_{j+2}, which is issued after p_full of tile j.
  uint64_t s_full[2], p_full[2], o_done[2], stat_full, settled;  // P_j V_j commits to o_done[j & 1]
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FwdBars) <= 256, "barrier block");

// ONE_SUM: a row's two halves agree on its maximum, tile by tile, and add into one accumulator, as the rows of
// flash_fwd128_sm100.cu do, in the same order: launches of up to kFwd128OneSumRows rows take that kernel or this one by
// the number of their units, and a unit's result is the same bit for bit. (The maxima go through shared memory and are
// looked at behind half of the exponentials: 24 x 2048 36.0 -> 36.6 us, 4 x 2048 17.8 -> 18.1; looked at ahead of them, by
// a barrier of the two warps, 37.7 and 19.7. Against float64 at 192 x 1024: out 2.04e-3 of its norm either way of dealing,
// lse 2.9e-7 rms; with two sums 2.02e-3, because the largest probability of each half is then an exact 1, and 2.9e-7.)
// Else each half has a maximum, a sum and an accumulator of its own, merged
// at the end.
template <bool DROP, bool ONE_SUM>
__global__ void __launch_bounds__(kFwdThreads, 1)
flash_fwd_bf16_kernel(const __grid_constant__ CUtensorMap map_q,
                      const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                      float* __restrict__ lse, int S, float scale, float rate, const __grid_constant__ PhiloxRounds rng,
                      int64_t unit0, LeveledGrid order, int* __restrict__ status) {
  using L = FwdSmem<ONE_SUM>;
  // TMEM columns: two S buffers [0,256) so that Q K^T of the next tile runs while this tile's softmax
  // still reads its scores, O_0 [256,384), O_1 [384,512).
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColS = 0, kColO = 256;

  extern __shared__ __align__(1024) uint8_t smem[];
  FwdBars* bars = reinterpret_cast<FwdBars*>(smem + L::kBars);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  int level, bh;
  if (!leveled_block(order, level, bh)) return;
  const int qt = (S + kBM - 1) / kBM - 1 - level;   // heaviest tiles first
  const int q0 = qt * kBM;
  const int n_kv = qt + 1;  // causal: key tiles 0..qt

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicExch(status, DADATTN_E_CUDA);
    return;
  }

  // The tiles of the ring's stage s, by the producing thread
  auto load_k = [&](int s, int j) {
    mbar_arrive_expect_tx(&bars->k_full[s], kPanels * kPanelBytes);
    for (int p = 0; p < kPanels; ++p)
      tma_load_3d(smem + L::kK + (s * kPanels + p) * kPanelBytes, &map_k, &bars->k_full[s], p * 64, j * kBN, bh);
  };
  auto load_v = [&](int s, int j) {
    mbar_arrive_expect_tx(&bars->v_full[s], kPanels * kPanelBytes);
    for (int p = 0; p < kPanels; ++p)
      tma_load_3d(smem + L::kV + (s * kPanels + p) * kPanelBytes, &map_v, &bars->v_full[s], p * 64, j * kBN, bh);
  };
  auto load_first = [&]() {
    pdl_wait();
    mbar_arrive_expect_tx(&bars->q_full, kPanels * kPanelBytes);
    for (int p = 0; p < kPanels; ++p)
      tma_load_3d(smem + L::kQ + p * kPanelBytes, &map_q, &bars->q_full, p * 64, q0, bh);
    load_k(0, 0);
    load_v(0, 0);
  };
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    prefetch_tensormap(&map_out);
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) mbar_init(&bars->s_full[b], 1);
    mbar_init(&bars->p_full[0], kSoftmaxThreads);
    mbar_init(&bars->p_full[1], kSoftmaxThreads);
    mbar_init(&bars->o_done[0], 1);
    mbar_init(&bars->o_done[1], 1);
    mbar_init(&bars->stat_full, kSoftmaxThreads);
    mbar_init(&bars->settled, 1);
    if (ONE_SUM)
      for (int i = 0; i < 16; ++i) mbar_init(reinterpret_cast<uint64_t*>(smem + L::kMaxFull) + i, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
    // The first tiles are requested here: they need this thread's barriers, and nothing of what the others set up (192 x
    // 1024 93.4 -> 91.9 us, 192 x 128 11.8 -> 11.3). With dropout the others have draws to make meanwhile, and do not wait
    // for it (48 x 57 9.79 -> 9.60 us, 72 x 777 103.4 -> 103.1).
    if (!DROP) load_first();
  }
  __syncwarp();
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  // Set-up is done; from here on global memory is read, which the previous grid in the stream
  // may have produced. Once every CTA of this grid is here the next grid may start its set-up.
  pdl_wait();
  pdl_launch_dependents();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      if (DROP) load_first();
      int n_k = 1, n_v = 1;   // tiles loaded
      for (int j = 1; j < n_kv; ++j) {
        const int s = j % kStages, use = j / kStages;
        // K's slot frees when Q K^T of its previous tenant is done, V's when P V is done
        if (use > 0 && !hot_wait(&bars->k_empty[s], (use - 1) & 1, abort_flag)) break;
        load_k(s, j);
        ++n_k;
        if (use > 0 && !hot_wait(&bars->v_empty[s], (use - 1) & 1, abort_flag)) break;
        load_v(s, j);
        ++n_v;
      }
      settle(&bars->q_full, 0);
      settle_ring(bars->k_full, kStages, n_k);
      settle_ring(bars->v_full, kStages, n_v);
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(kBM, kBN, 0, 0);  // Q, K: K-major
      constexpr uint32_t idesc_o = make_idesc_bf16(kBM, kD, 0, 1);   // P K-major, V MN-major
      const SmemDescBase q_desc = make_desc_base_sw128(smem_u32(smem + L::kQ), 0);
      const SmemDescBase k_desc0 = make_desc_base_sw128(smem_u32(smem + L::kK), 0);
      const SmemDescBase v_desc0 = make_desc_base_sw128(smem_u32(smem + L::kV), kPanelBytes);
      constexpr uint32_t kStageBytes = kPanels * kPanelBytes;
      bool ok = hot_wait(&bars->q_full, 0, abort_flag);

      // O_h[:, 64 pn .. 64 pn + 63] (+)= P_i[:, 64 h .. 64 h + 63] V_i[64 h .. 64 h + 63, :]; ONE_SUM: one O for both
      auto issue_pv = [&](int i) -> bool {
        const int s = i % kStages;
        if (!hot_wait(&bars->v_full[s], (i / kStages) & 1, abort_flag)) return false;
        if (!hot_wait(&bars->p_full[i & 1], (i >> 1) & 1, abort_flag)) return false;
        tc_fence_after_sync();
        const SmemDescBase v_desc{v_desc0.lo + s * (kStageBytes >> 4), v_desc0.hi};
        // One MMA per 16 keys covers all 128 output columns: the V tile is MN-major, its 64-column
        // panels are kPanelBytes apart, which is what the descriptor's leading byte offset says.
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)   // P_i sits in the first 32 columns of each half of score buffer i % 2
            mma_ts(tmem + kColO + (ONE_SUM ? 0 : h * kD), tmem + kColS + (i % 2) * 128 + h * 64 + kk * 8,
                   desc_at(v_desc, (h * 4 + kk) * 2048), idesc_o, (i > 0 || kk > 0 || (ONE_SUM && h > 0)) ? 1u : 0u);
        }
        mma_commit(&bars->v_empty[s]);
        mma_commit(&bars->o_done[i & 1]);
        return true;
      };

      for (int j = 0; ok && j < n_kv; ++j) {
        const int s = j % kStages;
        // Score buffer sb is overwritten by S_j only after P_{j-2} V_{j-2}, which was issued earlier
        // by this same thread: the tensor pipe keeps them in order.
        const int sb = j % 2;
        if (!(ok = hot_wait(&bars->k_full[s], (j / kStages) & 1, abort_flag))) break;
        tc_fence_after_sync();
        const SmemDescBase k_desc{k_desc0.lo + s * (kStageBytes >> 4), k_desc0.hi};
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk) {
          const uint32_t off = (kk / 4) * kPanelBytes + (kk % 4) * 32;
          mma_ss(tmem + kColS + sb * 128, desc_at(q_desc, off), desc_at(k_desc, off), idesc_s,
                 kk > 0 ? 1u : 0u);
        }
        mma_commit(&bars->k_empty[s]);
        mma_commit(&bars->s_full[sb]);
        if (j > 0) ok = issue_pv(j - 1);
      }
      if (ok) issue_pv(n_kv - 1);
      settle_products(&bars->settled);
    }
  } else {
    // ------------------------------ softmax ------------------------------
    const int quad = warp % 4;            // TMEM lane quadrant this warp may touch
    const int half = (warp - 2) / 4;      // which 64 key columns of every tile
    const int row = quad * 32 + lane;     // row within the tile = TMEM lane
    const int r = q0 + row;               // query index
    const uint32_t tlane = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    // what this thread rescales: its half's accumulator, or half the columns of the only one
    const uint32_t tO = tlane + kColO + half * (ONE_SUM ? kD / 2 : kD);
    float* maxima = reinterpret_cast<float*>(smem + L::kMax) + row;
    uint64_t* max_full = reinterpret_cast<uint64_t*>(smem + L::kMaxFull) + quad;   // a warp's 32 maxima are there
    const float scale_log2 = scale * kLog2e;
    const float keep_scale = DROP ? 1.0f / (1.0f - rate) : 1.0f;
    // waits for P_i V_i (tile i) to have completed
    auto wait_pv = [&](int i) { return hot_wait(&bars->o_done[i & 1], (i >> 1) & 1, abort_flag); };
    float m = -INFINITY, l = 0.f;  // running max (log2 units, scaled) and sum of this half-row
    bool ok = true;

    for (int j = 0; j < n_kv; ++j) {
      const int sb = j % 2;
      const uint32_t tS = tlane + kColS + sb * 128 + half * 64;
      uint32_t keep[2] = {0u, 0u};
      if (DROP) {
        // The words of the warp's 32 x 32 blocks that have visible pairs, while the scores are on their way, by
        // the shared form of the draws: 24 x 1000 with dropout 104 -> 56 us. (The same number in every lane: a
        // warp's loop runs as long as its longest lane's.)
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          const int col = j * kBN + half * 64 + ch * 32;
          if (col <= q0 + quad * 32 + 31)
            keep[ch] = philox_keep_bits<8>(rng, (static_cast<uint64_t>(unit0 + bh) * S + r) * S + col, 1u, 32);
        }
        __syncwarp();
      }
      if (!(ok = hot_wait(&bars->s_full[sb], (j / 2) & 1, abort_flag))) break;
      tc_fence_after_sync();
      const int c0 = j * kBN + half * 64;  // first key of this thread's 64 columns
      // Only the diagonal tile needs the causal mask: columns beyond `limit` are dropped.
      const bool diagonal = (j == n_kv - 1);
      const int limit = r - c0;

      // The thread's 64 scores, both 32-column loads in flight together; they stay in registers for the
      // max and for the exponentials.
      uint32_t xa[32], xb[32];
      tmem_ld32(tS, xa);
      tmem_ld32(tS + 32, xb);
      tmem_wait_ld();
      if (diagonal) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i > limit) xa[i] = 0xff800000u;  // -inf
          if (32 + i > limit) xb[i] = 0xff800000u;
        }
      }
      // max of the raw scores (scale > 0 commutes with max)
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i)
        mx4[i & 3] = fmax3(mx4[i & 3], __uint_as_float(xa[i]), __uint_as_float(xb[i]));
      float mx = __fmul_rn(fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])), scale_log2);

      // ONE_SUM: the other half's maximum of the row. (A buffer is written again two tiles on, behind the wait for the
      // other half's next maxima, which come after it has read these.)
      auto agree = [&]() -> bool {
        if (!hot_wait(&max_full[(sb * 2 + 1 - half) * 4], (j >> 1) & 1, abort_flag)) return false;
        mx = fmaxf(mx, maxima[(sb * 2 + 1 - half) * kBM]);
        return true;
      };
      // the accumulators and the sum get the scale of the larger maximum
      auto rescale = [&]() -> bool {
        if (!wait_pv(j - 1)) return false;
        tc_fence_after_sync();
        const float m_new = fmaxf(m, mx);
        // m = -inf: nothing but zeros has been accumulated so far (every earlier column masked)
        const float corr = (m == -INFINITY) ? 0.f : ex2(m - m_new);
#pragma unroll 1
        for (int c = 0; c < (ONE_SUM ? kD / 2 : kD) / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
          tmem_st32(tO + c * 32, o);
        }
        tmem_wait_st();
        l = __fmul_rn(l, corr);
        m = m_new;
        return true;
      };
      if (ONE_SUM) {
        maxima[(sb * 2 + half) * kBM] = mx;
        __syncwarp();
        if (lane == 0) mbar_arrive(&max_full[(sb * 2 + half) * 4]);
        if (j == 0 && !(ok = agree())) break;
      }
      if (j == 0)
        m = mx;  // O is first written by an MMA with accumulate = 0: nothing to rescale
      else if (!ONE_SUM && __any_sync(0xffffffffu, mx > m + kRescaleThreshold) && !(ok = rescale()))
        break;

      // ---- p = exp2(s * scale * log2e - m), packed two-float FMAs and sums (192 x 8192: 3.41 -> 3.32 ms,
      // 24 x 8192 419 -> 405 us, 24 x 2048 37.1 -> 36.8; a share of the exponentials on the FMA pipe was no faster). A half-row with no visible key yet has
      // m = -inf: its scores are all -inf and must give p = 0, not exp2(nan). ----
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const float2 sl = make_float2(scale_log2, scale_log2);
      uint32_t pk[32];  // packed P of this thread
      auto process = [&](uint32_t (&x)[32], int ch) {
        float pv[32];
        const float neg_m = (m == -INFINITY) ? 0.f : -m;
        const float2 nm = make_float2(neg_m, neg_m);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 e = ffma2(make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), sl, nm);
          const float2 p = make_float2(ex2(e.x), ex2(e.y));
          pv[i] = p.x, pv[i + 1] = p.y;
          sum2[(i >> 1) & 1] = fadd2(sum2[(i >> 1) & 1], p);
        }
        if (DROP) {
#pragma unroll
          for (int i = 0; i < 32; ++i) pv[i] = (keep[ch] >> i) & 1u ? pv[i] * keep_scale : 0.f;
        }
        // bf16 pairs (k, k+1) per 32-bit TMEM column: 16 columns for these 32 probabilities
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[ch * 16 + i] = pack_bf16(pv[2 * i], pv[2 * i + 1]);
      };
      process(xa, 0);
      if (ONE_SUM && j > 0) {
        // The other half's maximum is looked at only now. The exponentials above were computed with the one before, which
        // stands for nearly every tile; where it does not they are computed again.
        if (!(ok = agree())) break;
        if (__any_sync(0xffffffffu, mx > m + kRescaleThreshold)) {
          if (!(ok = rescale())) break;
          sum2[0] = sum2[1] = make_float2(0.f, 0.f);
          process(xa, 0);
        }
      }
      process(xb, 1);
      l += (sum2[0].x + sum2[1].x) + (sum2[0].y + sum2[1].y);
      tmem_st32(tS, pk);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&bars->p_full[sb]);
    }

    // Epilogue: merge the two halves of each row. out = (O_0 w_0 + O_1 w_1) / (l_0 w_0 + l_1 w_1)
    // with w_h = exp2(m_h - max(m_0, m_1)); lse in natural-log units of the scaled scores.
    // Each thread of the pair writes half of the row's 128 outputs.
    // The (max, sum) pairs are exchanged through the Q tile's shared memory, which nobody reads
    // any more: every Q K^T has completed before the last s_full was observed.
    float2* stat = reinterpret_cast<float2*>(smem + L::kQ);  // [2][128]
    if (ok) {
      stat[half * 128 + row] = make_float2(m, l);
      mbar_arrive(&bars->stat_full);
      ok = hot_wait(&bars->stat_full, 0, abort_flag) &&
           wait_pv(n_kv - 1);
    }
    if (ok) {
      tc_fence_after_sync();
      const float2 s0 = stat[row], s1 = stat[128 + row];
      const float m_tot = fmaxf(s0.x, s1.x);  // half 0 always sees key 0: finite
      const float w0 = ex2(s0.x - m_tot);
      const float w1 = (s1.x == -INFINITY) ? 0.f : ex2(s1.x - m_tot);
      const float l_tot = s0.y * w0 + s1.y * w1;
      const float f0 = w0 / l_tot, f1 = w1 / l_tot;
      constexpr int kCols = kD / 2;  // output columns per thread
      // Through shared memory and TMA: a warp's 32 rows x 64 columns are 4 KB of the K ring, whose tiles the last
      // products have read. As 16-byte stores of one row per lane they took 2300 clocks a CTA (192 x 1024
      // 95.4 -> 93.4 us).
      uint8_t* stage = smem + L::kK + half * kPanelBytes + quad * 32 * 128;
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) {
        uint32_t oa[32], ob[32];
        tmem_ld32(tlane + kColO + half * kCols + c * 32, oa);
        if (!ONE_SUM) tmem_ld32(tlane + kColO + kD + half * kCols + c * 32, ob);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            y[e] = ONE_SUM ? __uint_as_float(oa[8 * i + e]) * f0
                           : __uint_as_float(oa[8 * i + e]) * f0 + __uint_as_float(ob[8 * i + e]) * f1;
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + i) ^ (lane & 7)) << 4)) =
              make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]),
                         pack_bf16(y[6], y[7]));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && q0 + quad * 32 < S) {   // (rows beyond S are not written)
        tma_store_3d(&map_out, stage, half * kCols, q0 + quad * 32, bh);
        bulk_commit();
      }
      if (half == 0 && r < S) lse[static_cast<size_t>(bh) * S + r] = (m_tot + log2f(l_tot)) * kLn2;
      if (lane == 0) bulk_wait_read<0>();   // (behind lse: 24 x 33 4.61 -> 4.52 us, 8 x 700 9.04 -> 8.96)
    }
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

template <bool DROP, bool ONE_SUM>
int launch_fwd_bf16(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k,
                    const uint16_t* v, int BH, int S, float scale, float rate, uint64_t seed,
                    uint64_t offset, int64_t unit0, cudaStream_t st) {
  CUtensorMap mq, mk, mv, mo;
  if (int rc = make_tensor_map_bf16(&mq, q, BH, S, kD, kBM)) return rc;
  if (int rc = make_tensor_map_bf16(&mk, k, BH, S, kD, kBN)) return rc;
  if (int rc = make_tensor_map_bf16(&mv, v, BH, S, kD, kBN)) return rc;
  if (int rc = make_tensor_map_bf16(&mo, out, BH, S, kD, 32)) return rc;
  int* status = device_status_word();
  if (!status) return DADATTN_E_CUDA;
  auto kern = flash_fwd_bf16_kernel<DROP, ONE_SUM>;
  DAD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                FwdSmem<ONE_SUM>::kBytes));
  const LeveledGrid order = leveled_grid(32768, S, BH);   // (16384 and 65536: 0-4 % slower or the same)
  DAD_CUDA(launch_pdl(kern, leveled_blocks(order, (S + kBM - 1) / kBM), dim3(kFwdThreads), FwdSmem<ONE_SUM>::kBytes, st,
                      mq, mk, mv, mo, lse, S, scale, rate,
                      make_philox_rounds(seed, offset, rate), unit0, order, status));
  return DADATTN_OK;
}

}  // namespace

int launch_fwd_bf16_d128_two_sums(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v,
                                  int BH, int S, float scale, cudaStream_t st) {
  return launch_fwd_bf16<false, false>(out, lse, q, k, v, BH, S, scale, 0.f, 0, 0, 0, st);
}

}  // namespace dadattn

using namespace dadattn;

extern "C" int dadattn_flash_bf16_supported(int d_head) { return d_head == 64 || d_head == 128; }

extern "C" int dadattn_flash_fwd_bf16(uint16_t* out, float* lse, const uint16_t* q,
                                      const uint16_t* k, const uint16_t* v, int BH, int S, int D,
                                      float scale, float rate, uint64_t seed, uint64_t offset,
                                      int64_t unit0, dadattn_stream_t stream) {
  if (!out || !lse || !q || !k || !v) return fail(DADATTN_E_ARG, "null tensor pointer");
  if (BH <= 0 || S <= 0) return fail(DADATTN_E_ARG, "BH=%d and S=%d must be positive", BH, S);
  if (BH > 65535) return fail(DADATTN_E_UNSUPPORTED, "BH=%d exceeds 65535 per call", BH);
  if (!dadattn_flash_bf16_supported(D))
    return fail(DADATTN_E_UNSUPPORTED, "flash attention bf16: unsupported d_head %d", D);
  if (!(rate >= 0.0f && rate < 1.0f))
    return fail(DADATTN_E_ARG, "dropout rate %f outside [0,1)", static_cast<double>(rate));
  if (!(scale > 0.0f)) return fail(DADATTN_E_ARG, "bf16 forward needs scale > 0");
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) ||
      !aligned(lse, 4))
    return fail(DADATTN_E_ARG, "bf16 tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool drop = rate > 0.f;
  if (D == 64)   // head size 64 has a kernel of its own (flash_fwd64_sm100.cu)
    return launch_fwd_bf16_d64(out, lse, q, k, v, BH, S, scale, rate, seed, offset, unit0, nullptr, 0, st);
  // (a draw costs more than the rest of the arithmetic: with dropout the larger number of smaller items is the better
  // one, 192 x 512 119 us against 142)
  if (drop) return launch_fwd_bf16<true, false>(out, lse, q, k, v, BH, S, scale, rate, seed, offset, unit0, st);
  // The arithmetic goes by S alone, so that a unit's result does not depend on the units it is computed with.
  if (S > kFwd128OneSumRows) return launch_fwd_bf16_d128_two_sums(out, lse, q, k, v, BH, S, scale, st);
  if (fwd128_pairs_pay(BH, S)) return launch_fwd_bf16_d128_pairs(out, lse, q, k, v, BH, S, scale, st);
  return launch_fwd_bf16<false, true>(out, lse, q, k, v, BH, S, scale, 0.f, 0, 0, 0, st);
}

extern "C" int dadattn_flash_fwd_bf16_masked(uint16_t* out, float* lse, const uint16_t* q,
                                             const uint16_t* k, const uint16_t* v, int BH, int S, int D,
                                             float scale, float rate, const uint32_t* mask_bits,
                                             dadattn_stream_t stream) {
  if (!out || !lse || !q || !k || !v) return fail(DADATTN_E_ARG, "null tensor pointer");
  if (!mask_bits || !aligned(mask_bits, 16))
    return fail(DADATTN_E_ARG, "mask_bits must be a 16-byte aligned device pointer");
  if (BH <= 0 || S <= 0) return fail(DADATTN_E_ARG, "BH=%d and S=%d must be positive", BH, S);
  if (BH > 65535) return fail(DADATTN_E_UNSUPPORTED, "BH=%d exceeds 65535 per call", BH);
  if (D != 64)
    return fail(DADATTN_E_UNSUPPORTED, "a bit-packed dropout mask is taken at head size 64 only (got %d)", D);
  if (!(rate > 0.0f && rate < 1.0f))
    return fail(DADATTN_E_ARG, "the masked forward needs the rate the mask was drawn with, in (0,1)");
  if (!(scale > 0.0f)) return fail(DADATTN_E_ARG, "bf16 forward needs scale > 0");
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) || !aligned(lse, 4))
    return fail(DADATTN_E_ARG, "bf16 tensors must be 16-byte aligned");
  return launch_fwd_bf16_d64(out, lse, q, k, v, BH, S, scale, rate, 0, 0, 0, mask_bits, 0,
                             static_cast<cudaStream_t>(stream));
}

extern "C" int dadattn_flash_fwd_bf16_strided(uint16_t* out, float* lse, const uint16_t* q,
                                              const uint16_t* k, const uint16_t* v, int B, int H, int S,
                                              int D, float scale, float rate, uint64_t seed,
                                              uint64_t offset, int64_t unit0, dadattn_stream_t stream) {
  if (!out || !lse || !q || !k || !v) return fail(DADATTN_E_ARG, "null tensor pointer");
  if (B <= 0 || H <= 0 || S <= 0) return fail(DADATTN_E_ARG, "B=%d, H=%d and S=%d must be positive", B, H, S);
  if (static_cast<long long>(B) * H > 65535)
    return fail(DADATTN_E_UNSUPPORTED, "B*H=%lld exceeds 65535 per call", static_cast<long long>(B) * H);
  if (D != 64)
    return fail(DADATTN_E_UNSUPPORTED, "interleaved [B*S, H*D] activations are taken at head size 64 only (got %d)", D);
  if (!(rate >= 0.0f && rate < 1.0f))
    return fail(DADATTN_E_ARG, "dropout rate %f outside [0,1)", static_cast<double>(rate));
  if (!(scale > 0.0f)) return fail(DADATTN_E_ARG, "bf16 forward needs scale > 0");
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) || !aligned(lse, 4))
    return fail(DADATTN_E_ARG, "bf16 tensors must be 16-byte aligned");
  return launch_fwd_bf16_d64(out, lse, q, k, v, B * H, S, scale, rate, seed, offset, unit0, nullptr, H,
                             static_cast<cudaStream_t>(stream));
}
