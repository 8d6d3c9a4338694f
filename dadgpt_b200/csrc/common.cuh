// Shared host/device helpers for the dadattn kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "dadattn.h"

namespace dadattn {

// Thread-local error text behind dadattn_last_error().
char* error_buffer();
int fail(int code, const char* fmt, ...);

#define DAD_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return ::dadattn::fail(DADATTN_E_CUDA, "%s failed: %s (%s:%d)", #call,            \
                             cudaGetErrorString(e_), __FILE__, __LINE__);               \
  } while (0)

#define DAD_LAUNCH_CHECK(name)                                                          \
  do {                                                                                  \
    cudaError_t e_ = cudaGetLastError();                                                \
    if (e_ != cudaSuccess)                                                              \
      return ::dadattn::fail(DADATTN_E_CUDA, "launch of %s failed: %s", name,           \
                             cudaGetErrorString(e_));                                   \
  } while (0)

// Device-side sticky status word (one per device that loads the library). Kernels record a
// DADATTN_E_* code here instead of trapping; dadattn_device_status() reads and clears it.
int* device_status_word();  // device pointer for the current device, nullptr on failure

// Kernels whose warpgroups move registers between them (setmaxnreg) budget with the count the CTA is
// launched with; were the compiler to give the kernel fewer, an increase would wait for registers
// that nobody can give back. Refuses such a launch. `seen` belongs to the kernel.
int check_launch_registers(const void* kernel, int expected, std::atomic<int>& seen);

// ---- Philox4x32-10 with cuRAND's curand_init(seed, subsequence, offset) counter set-up -------
// The reference draws one uniform per attention probability with subsequence = flat element
// index (cuda/gpu_ops.cu:712-727). key = seed; counter = {offset/4 (64 bit), subsequence}.
struct PhiloxKey {
  uint32_t k0, k1;       // seed
  uint32_t c0, c1;       // offset / 4
  uint32_t word;         // offset % 4
};

__host__ __device__ inline PhiloxKey make_philox(uint64_t seed, uint64_t offset) {
  PhiloxKey p;
  p.k0 = static_cast<uint32_t>(seed);
  p.k1 = static_cast<uint32_t>(seed >> 32);
  p.c0 = static_cast<uint32_t>(offset >> 2);
  p.c1 = static_cast<uint32_t>(offset >> 34);
  p.word = static_cast<uint32_t>(offset & 3);
  return p;
}

__device__ __forceinline__ uint32_t philox_draw(const PhiloxKey& p, uint64_t subsequence) {
  uint32_t c0 = p.c0, c1 = p.c1, c2 = static_cast<uint32_t>(subsequence),
           c3 = static_cast<uint32_t>(subsequence >> 32);
  uint32_t k0 = p.k0, k1 = p.k1;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return p.word == 0 ? c0 : p.word == 1 ? c1 : p.word == 2 ? c2 : c3;
}

// The same draw when the wanted word is the first of the block (offset a multiple of 4, as in
// every call the reference makes): both halves of each 32 x 32 product come from one widening
// multiply, the round keys are compile-time offsets of the seed, and the last round computes
// only the word that is used.
__device__ __forceinline__ uint32_t philox_draw_word0(const PhiloxKey& p, uint64_t subsequence) {
  uint32_t c0 = p.c0, c1 = p.c1, c2 = static_cast<uint32_t>(subsequence),
           c3 = static_cast<uint32_t>(subsequence >> 32);
#pragma unroll
  for (int r = 0; r < 9; ++r) {
    const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0;
    const uint64_t p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2;
    const uint32_t k0 = p.k0 + static_cast<uint32_t>(r) * 0x9E3779B9u;
    const uint32_t k1 = p.k1 + static_cast<uint32_t>(r) * 0xBB67AE85u;
    const uint32_t n0 = static_cast<uint32_t>(p1 >> 32) ^ c1 ^ k0;
    const uint32_t n2 = static_cast<uint32_t>(p0 >> 32) ^ c3 ^ k1;
    c1 = static_cast<uint32_t>(p1);
    c3 = static_cast<uint32_t>(p0);
    c0 = n0;
    c2 = n2;
  }
  return __umulhi(0xCD9E8D57u, c2) ^ c1 ^ (p.k0 + 9u * 0x9E3779B9u);
}

// true = keep. Same float arithmetic as curand_uniform followed by the reference's `r < rate`.
__device__ __forceinline__ bool philox_keep(const PhiloxKey& p, uint64_t subsequence,
                                            float rate) {
  float u = fmaf(static_cast<float>(philox_draw(p, subsequence)), 2.3283064e-10f,
                 2.3283064e-10f / 2.0f);
  return !(u < rate);
}

// The keep bits of several draws at once, for kernels whose time is the drawing: the mask, stripped to
// what it needs.
//  * The round keys come precomputed from the host (kernel parameters: constant-bank operands), both
//    halves of each 32 x 32 product from one widening multiply, the last rounds compute only what the
//    first output word depends on, and "uniform < rate" is decided on the integer draw: the uniform
//    is a non-decreasing function of it (cvt.rn, one fma), so the dropped draws are those below a
//    threshold that the host finds with the same float arithmetic.
//  * Of the counter only the low subsequence word changes from draw to draw. The first round's
//    product with the offset word is one number for the call, the second round's product with what
//    comes of it one for the thread, and neither reaches the other lane before the third round: 13
//    widening products, three high and one low are left of 20. The pipe that multiplies integers sets the
//    pace: at 192 x 1024 the mask kernel takes 250 us (265 with 19 widening products) and keeps it busy
//    84 % of the time, at 54 % of the issue slots.
struct PhiloxRounds {
  uint32_t k0[10], k1[9];   // key words of rounds 0..9 (the last round needs only k0)
  uint32_t c0, c1;          // low counter words: offset / 4
  uint32_t m_lo, m_hi;      // round 0: 0xD2511F53 * c0
  uint32_t word;            // offset % 4: which word of the block is the draw; 4 more where strides do not fit
  uint32_t drop_below;      // draws below this are dropped (uniform < rate)
};
// Whether 31 strides stay within 32 bits, as the shared form of philox_keep_bits takes for granted.
constexpr bool philox_strides_fit(uint32_t stride) { return 31ull * stride <= 0xffffffffu; }
static_assert(philox_strides_fit(1) && philox_strides_fit(138547332) && !philox_strides_fit(138547333) &&
              !philox_strides_fit(0x7fffffff), "the line lies at 2^32 / 31");
PhiloxRounds make_philox_rounds(uint64_t seed, uint64_t offset, float rate, uint32_t stride = 1);

// Bit i (i < n <= 32): whether the probability of flat index at + i * stride is kept. `stride` is at most the one
// that `p` was made for.
template <int UNROLL>
__device__ __forceinline__ uint32_t philox_keep_bits(const PhiloxRounds& p, uint64_t at, uint32_t stride, int n) {
  const uint32_t lo = static_cast<uint32_t>(at), hi = static_cast<uint32_t>(at >> 32);
  uint32_t bits = 0;
  if (p.word == 0 && lo <= 0xffffffffu - 31ull * stride) {   // (the high word stays put)
    const uint64_t t = static_cast<uint64_t>(0xCD9E8D57u) * (p.m_hi ^ hi ^ p.k1[0]);
    const uint32_t x0 = static_cast<uint32_t>(t >> 32) ^ p.k0[1], x1 = static_cast<uint32_t>(t), x2 = p.m_lo ^ p.k1[1];
#pragma unroll UNROLL
    for (int i = 0; i < n; ++i) {
      const uint64_t a = static_cast<uint64_t>(0xCD9E8D57u) * (lo + static_cast<uint32_t>(i) * stride);
      const uint64_t b = static_cast<uint64_t>(0xD2511F53u) * (static_cast<uint32_t>(a >> 32) ^ p.c1 ^ p.k0[0]);
      uint32_t c0 = x0 ^ static_cast<uint32_t>(a), c1 = x1;
      uint32_t c2 = static_cast<uint32_t>(b >> 32) ^ x2, c3 = static_cast<uint32_t>(b);
#pragma unroll
      for (int r = 2; r < 8; ++r) {
        const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0, p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2;
        c0 = static_cast<uint32_t>(p1 >> 32) ^ c1 ^ p.k0[r];
        c2 = static_cast<uint32_t>(p0 >> 32) ^ c3 ^ p.k1[r];
        c1 = static_cast<uint32_t>(p1);
        c3 = static_cast<uint32_t>(p0);
      }
      const uint32_t n2 = __umulhi(0xD2511F53u, c0) ^ c3 ^ p.k1[8];
      const uint32_t draw = __umulhi(0xCD9E8D57u, n2) ^ (0xCD9E8D57u * c2) ^ p.k0[9];
      bits |= (draw >= p.drop_below ? 1u : 0u) << i;
    }
    return bits;
  }
  const PhiloxKey key = {p.k0[0], p.k1[0], p.c0, p.c1, p.word & 3u};
#pragma unroll 1
  for (int i = 0; i < n; ++i)
    bits |= (philox_draw(key, at + static_cast<uint64_t>(i) * stride) >= p.drop_below ? 1u : 0u) << i;
  return bits;
}

// ---- bit-packed dropout mask (dadattn_dropout_mask_bits) ----------------------------------------
// One 16-byte record per (batch x head, 128-query tile qt, 128-key tile kt <= qt, query row of
// the tile): bit i of 32-bit word w says whether the probability of key 32 w + i of the key tile
// is kept (1) or dropped (0). Records of a tile are contiguous (2 KB), tiles of a (batch, head)
// are numbered qt (qt + 1) / 2 + kt: only the causal lower triangle exists.
constexpr int kMaskTile = 128;
__host__ __device__ inline size_t mask_bits_record(int bh, int qt, int kt, int row, int n_tiles) {
  const size_t n_tri = static_cast<size_t>(n_tiles) * (n_tiles + 1) / 2;
  return (static_cast<size_t>(bh) * n_tri + static_cast<size_t>(qt) * (qt + 1) / 2 + kt) * kMaskTile + row;
}
inline size_t dropout_mask_bits_bytes(int BH, int S) {
  const size_t n_tiles = (static_cast<size_t>(S) + kMaskTile - 1) / kMaskTile;
  return static_cast<size_t>(BH) * (n_tiles * (n_tiles + 1) / 2) * kMaskTile * 16;
}

// Forward at head size 128 without dropout. Up to kFwd128OneSumRows rows: one maximum, sum and accumulator per row, two query
// tiles per CTA (flash_fwd128_sm100.cu) where that is the better, else one (flash_bf16_sm100.cu), with the same results.
// Beyond: flash_bf16_sm100.cu with those of each half of a row, which launch_fwd_bf16_d128_two_sums takes at every S.
constexpr int kFwd128OneSumRows = 2048;
bool fwd128_pairs_pay(int BH, int S);
int launch_fwd_bf16_d128_pairs(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v, int BH,
                               int S, float scale, cudaStream_t st);
int launch_fwd_bf16_d128_two_sums(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v,
                                  int BH, int S, float scale, cudaStream_t st);
// Forward at head size 64 (flash_fwd64_sm100.cu). mask_bits != nullptr with rate > 0: keep bits
// from dadattn_dropout_mask_bits; mask_bits == nullptr with rate > 0: the Philox mask is drawn
// inside the kernel. heads > 0: tensors are the interleaved [B*S, heads*64] activations.
int launch_fwd_bf16_d64(uint16_t* out, float* lse, const uint16_t* q, const uint16_t* k,
                        const uint16_t* v, int BH, int S, float scale, float rate, uint64_t seed,
                        uint64_t offset, int64_t unit0, const uint32_t* mask_bits, int heads,
                        cudaStream_t st);

// Whether the calling thread's backward is the single-pass one (dadattn_set_bwd_deterministic).
bool bwd_single_pass();

// bf16 operands, fp32 results (flash_f32_via_bf16.cu), head size 64.
int launch_fwd_bf16_d64_f32(float* out, float* lse, const uint16_t* q, const uint16_t* k, const uint16_t* v, int BH,
                            int S, float scale, cudaStream_t st);
int launch_bwd_fused_d64_f32(float* dq32, float* dk32, float* dv32, const float* delta, int* item_counter,
                             const uint16_t* dout, const float* lse, const uint16_t* q, const uint16_t* k,
                             const uint16_t* v, int BH, int S, float scale, cudaStream_t st);

// fp32 tensors on the tensor cores, exact operands (flash_f32_tc_*.cu): head sizes 16, 32, 64.
int launch_fwd_f32_tc(float* out, float* lse, const float* q, const float* k, const float* v, int BH, int S, int D,
                      float scale, float rate, uint64_t seed, uint64_t offset, int64_t unit0, bool vec_ok,
                      cudaStream_t st);
// delta: scratch of BH * S floats for rowsum(dO o O), which launch_delta_f32_d64 (flash_f32.cu) forms at
// head size 64.
int launch_bwd_f32_tc(float* dq, float* dk, float* dv, float* delta, const float* dout, const float* out, const float* lse,
                      const float* q, const float* k, const float* v, int BH, int S, int D, float scale, float rate,
                      uint64_t seed, uint64_t offset, int64_t unit0, bool vec_ok, cudaStream_t st);
int launch_delta_f32_d64(float* delta, const float* dout, const float* out, int64_t rows, bool vec_ok, cudaStream_t st);

// Launch with programmatic stream serialization: the grid may become resident while its
// predecessor in the stream drains, runs its set-up (barriers, TMEM, descriptor prefetch), and
// parks in pdl_wait() until the predecessor has completed and flushed its memory. Kernels
// launched this way call pdl_wait() before their first access to global memory.
template <typename Kernel, typename... Args>
cudaError_t launch_pdl(Kernel kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
// Grids of (tile level, batch x head) blocks, level 0 = the tiles with the most work: units in groups
// (whose tensors then stay in L2 while they are worked on), inside a group level by level. Blocks are
// handed out in index order, so the long ones start first and the short ones fill the gaps at the end.
// With one unit after the other, a launch of a few waves ended on whatever tile came last: the forward
// at 24 x 2048 x 128 took 44.1 us, level by level 37.1, 96 x 512 23.6 and 22.6, 24 x 8192 433 and 417,
// 192 x 8192 3427 and 3405. Grid dimensions rather than a division of one block index: those stay in
// uniform registers (2 % of the forward's time).
struct LeveledGrid {
  int group, units;
};
// Groups of about `rows` rows, as even as they come.
inline LeveledGrid leveled_grid(int rows, int S, int BH) {
  const int most = rows / S < 1 ? 1 : rows / S, groups = (BH + most - 1) / most;
  return LeveledGrid{(BH + groups - 1) / groups, BH};
}
#ifdef __CUDACC__
// (x is the only grid dimension that holds more than 65535 levels: longer sequences are in groups of 1)
inline dim3 leveled_blocks(const LeveledGrid& g, int n_levels) {
  const int groups = (g.units + g.group - 1) / g.group;
  return g.group == 1 ? dim3(n_levels, 1, groups) : dim3(g.group, n_levels, groups);
}
// False for the blocks that pad the last group.
template <typename Index>
__device__ __forceinline__ bool leveled_item(const LeveledGrid& g, const Index& block, int& level, int& bh) {
  level = g.group == 1 ? block.x : block.y;
  bh = block.z * g.group + (g.group == 1 ? 0 : block.x);
  return bh < g.units;
}
__device__ __forceinline__ bool leveled_block(const LeveledGrid& g, int& level, int& bh) {
  return leveled_item(g, blockIdx, level, bh);
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// Optional timing hooks of the bf16 backward (dadattn_set_stage_events): event i is recorded on
// the call's stream before its i-th kernel, and one more after the last kernel.
extern thread_local cudaEvent_t* g_stage_events;
extern thread_local int g_stage_event_count;
inline void stage_event(int i, cudaStream_t st) {
  if (g_stage_events && i < g_stage_event_count) cudaEventRecord(g_stage_events[i], st);
}

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

}  // namespace dadattn
