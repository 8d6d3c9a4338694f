// Exact fp32 operands on the bf16 tensor cores, shared by the forward and backward of
// flash_f32_tc_*.cu.
//
// An fp32 number is the sum of three bf16 numbers, x = x0 + x1 + x2 with x0 = bf16(x), x1 =
// bf16(x - x0), x2 = x - x0 - x1: each takes 8 of the 24 significand bits, both subtractions are
// exact and so is the last conversion. A product of two fp32 matrices is then the sum of the nine
// products of their planes. The three smallest (x1 y2, x2 y1, x2 y2) are at most 2^-26 of |x||y|,
// a quarter of what one rounding of an fp32 multiply-add may lose, and are left out; the other six
// are accumulated in fp32, smallest first, at most 64 products deep, and the accumulator is then
// added to a register sum in fp32 with round-to-nearest. Nothing is rounded to bf16: the result is
// that of an fp32 dot product with another order of summation (measured against float64: no larger
// error than the FFMA kernels of flash_f32.cu).
//
// Range. Every finite x: the first plane saturates at bf16's largest number, 3.3895e38, what a larger x
// has beyond it goes to the second. Below 2^-110 the last bits of the third plane fall under bf16's
// smallest number, an absolute error of at most 2^-134. An infinite or NaN element (its planes hold a
// NaN) makes NaN of every result that its tile's products add it to: the rows and columns that see it,
// and for V, K in the dQ product, dO and Q in the dK / dV products also rows or keys of the same tile
// for which its weight is a masked 0 (0 x NaN).
#pragma once

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace dadattn {
namespace f32tc {

using namespace ptx;

constexpr int kRows = 128;          // rows of the resident tile: one per TMEM lane
constexpr int kStep = 64;           // rows of the streamed tile per step
constexpr int kPlaneA = kRows * 128;   // one bf16 plane, 128-byte rows (64 elements), swizzled
constexpr int kPlaneB = kStep * 128;
constexpr int kComputeThreads = 512;   // four per row, 16 of a step's 64 columns each
constexpr int kLoaderThreads = 11 * 32;
constexpr int kThreads = 896;          // 16 compute warps, 11 loader warps, 1 issuer warp
constexpr int kWarpLoader0 = 16, kWarpIssuer = 27;
// Registers per thread once the warpgroups have rebalanced; the pool is what the CTA starts with.
constexpr int kRegsLaunch = 72, kRegsCompute = 88, kRegsHelper = 48;
static_assert(kComputeThreads * kRegsCompute + (kThreads - kComputeThreads) * kRegsHelper <= kThreads * kRegsLaunch, "register pool exceeded");

// Plane pairs of the six products, smallest first.
__device__ __forceinline__ constexpr int product_a(int i) { return i == 0 ? 2 : i == 1 ? 0 : i == 2 ? 1 : i == 3 ? 1 : 0; }
__device__ __forceinline__ constexpr int product_b(int i) { return i == 0 ? 0 : i == 1 ? 2 : i == 2 ? 1 : i == 3 ? 0 : i == 4 ? 1 : 0; }

// (lo, hi) -> packed bf16 as plane i of a split
template <int I>
__device__ __forceinline__ uint32_t pack_plane(float lo, float hi) {
  if (I > 0) return pack_bf16(lo, hi);   // (not saturating: an infinity may not end as a finite sum)
  uint32_t r;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// Four fp32 values -> three planes of four packed bf16.
struct Split4 {
  uint2 p[3];
};
__device__ __forceinline__ Split4 split4(float4 x) {
  Split4 s;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    s.p[i] = i == 0 ? make_uint2(pack_plane<0>(x.x, x.y), pack_plane<0>(x.z, x.w))
                    : make_uint2(pack_plane<1>(x.x, x.y), pack_plane<1>(x.z, x.w));
    const float2 minus = make_float2(-1.f, -1.f);
    const float2 a = ffma2(make_float2(__uint_as_float(s.p[i].x << 16), __uint_as_float(s.p[i].x & 0xffff0000u)), minus,
                           make_float2(x.x, x.y));   // exact
    const float2 b = ffma2(make_float2(__uint_as_float(s.p[i].y << 16), __uint_as_float(s.p[i].y & 0xffff0000u)), minus,
                           make_float2(x.z, x.w));
    x = make_float4(a.x, a.y, b.x, b.y);
  }
  return s;
}
// Rows of a streamed tile are as wide as the head, so that the sums' products, which read them MN-major, are too: at
// 64 columns for every head size those of 32 and 16 took 33 clocks a product instead of 17 and 10 (backward, us:
// 48 x 1024 x 16 87 -> 73, x 32 99 -> 94; forward and backward 64 x 300 x 16 39.4 -> 33, 32 x 301 x 32 24.5 -> 23.2, 16 x
// 64 x 16 9.9 -> 9.3).
template <int D>
constexpr int kStreamRow = 2 * D;
// Columns 4 c4 .. 4 c4 + 3 of a row into the three planes of a tile with rows of ROW_BYTES and the swizzle of that width.
template <int ROW_BYTES = 128>
__device__ __forceinline__ void store_split(uint8_t* tile, int plane_bytes, int row, int c4, const Split4& s) {
  const int swizzle = ROW_BYTES == 128 ? row & 7 : ROW_BYTES == 64 ? (row >> 1) & 3 : (row >> 2) & 1;
  uint8_t* at = tile + row * ROW_BYTES + ((((c4 >> 1) ^ swizzle) << 4) | ((c4 & 1) << 3));
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * plane_bytes) = s.p[i];
}

// Four consecutive fp32 values at any 4-byte alignment; zeros when !in.
__device__ __forceinline__ float4 load4(const float* __restrict__ p, bool in, bool vec_ok) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in) {
    if (vec_ok)
      x = __ldg(reinterpret_cast<const float4*>(p));
    else
      x = make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
  }
  return x;
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
}

// N consecutive columns of the thread's TMEM lane (N = 16, 8 or 4)
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 16)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
  else if constexpr (N == 8)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr)
        : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
      : "memory");
}
// 16 values of a row -> three planes of packed pairs in tensor memory, 8 columns each.
__device__ __forceinline__ void tmem_store_split(float2 (&x)[8], uint32_t t0, uint32_t t1, uint32_t t2) {
  const uint32_t t[3] = {t0, t1, t2};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint32_t pk[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      pk[j] = i == 0 ? pack_plane<0>(x[j].x, x[j].y) : pack_plane<1>(x[j].x, x[j].y);
      if (i < 2)
        x[j] = ffma2(make_float2(__uint_as_float(pk[j] << 16), __uint_as_float(pk[j] & 0xffff0000u)),
                     make_float2(-1.f, -1.f), x[j]);   // exact
    }
    tmem_st8(t[i], pk);
  }
}
// sum[c] += the accumulator's columns taddr + c
template <int N>
__device__ __forceinline__ void tmem_add(uint32_t taddr, float (&sum)[N]) {
  uint32_t a[N];
  tmem_ld<N>(taddr, a);
  tmem_wait_ld();
#pragma unroll
  for (int c = 0; c < N; ++c) sum[c] += __uint_as_float(a[c]);
}
// e^x for x <= 0 (or a masked score's -FLT_MAX, which gives 0)
__device__ __forceinline__ float2 exp2_of(float2 x) {
  const float2 t = fmul2(x, make_float2(1.4426950408889634f, 1.4426950408889634f));
  return make_float2(ex2(t.x), ex2(t.y));
}
// The 128 x D results of a CTA, N columns of a row per compute thread, through shared memory (free by
// then) to global memory: written straight from the registers, every lane on a row of its own, a
// warp's store touches 32 lines and the stores of a tile take as long as two of its steps.
template <int D, int N>
__device__ __forceinline__ void stage_rows(float* stage, int row, int col, const float (&x)[N]) {
#pragma unroll
  for (int c = 0; c < N; c += 4)
    *reinterpret_cast<float4*>(stage + row * (D + 4) + col + c) = make_float4(x[c], x[c + 1], x[c + 2], x[c + 3]);
}
template <int D>
__device__ __forceinline__ void write_rows(float* __restrict__ dst, const float* stage, int rows, bool vec_ok) {
  constexpr int V4 = D / 4;
#pragma unroll
  for (int j = 0; j < kRows * V4 / kComputeThreads; ++j) {
    const int e = threadIdx.x + j * kComputeThreads, r = e / V4, c = (e % V4) * 4;
    if (r >= rows) continue;
    const float4 x = *reinterpret_cast<const float4*>(stage + r * (D + 4) + c);
    float* p = dst + static_cast<size_t>(r) * D + c;
    if (vec_ok)
      *reinterpret_cast<float4*>(p) = x;
    else
      p[0] = x.x, p[1] = x.y, p[2] = x.z, p[3] = x.w;
  }
}
// N consecutive results per thread (lane = row of the tile) to global memory. Groups of N/4 lanes first
// exchange their 16-byte pieces, so that a group's lanes write N consecutive floats of one row: written
// as they are, every lane on a row of its own, a store touches 32 lines and a tile's stores take as
// long as two of its steps.
template <int D, int N>
__device__ __forceinline__ void write_sums(float* __restrict__ dst, int row, int col, float (&x)[N], int rows, bool vec_ok) {
  constexpr int kPieces = N / 4;
  const int a = row & (kPieces - 1);
#pragma unroll
  for (int b = 1; b < kPieces; b <<= 1)
#pragma unroll
    for (int i = 0; i < kPieces; ++i)
      if (!(i & b))
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float &lo = x[i * 4 + e], &hi = x[(i | b) * 4 + e];
          const float got = __shfl_xor_sync(0xffffffffu, (a & b) ? lo : hi, b);
          if (a & b) lo = got; else hi = got;
        }
#pragma unroll
  for (int j = 0; j < kPieces; ++j) {   // piece `a` of row j of the group
    const int r = row - a + j;
    if (r >= rows) continue;
    float* p = dst + static_cast<size_t>(r) * D + col + a * 4;
    if (vec_ok)
      *reinterpret_cast<float4*>(p) = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
    else
      p[0] = x[4 * j], p[1] = x[4 * j + 1], p[2] = x[4 * j + 2], p[3] = x[4 * j + 3];
  }
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 9, %0;" ::"n"(kComputeThreads) : "memory"); }

}  // namespace f32tc
}  // namespace dadattn
