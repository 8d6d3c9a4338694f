// fp32 tensors in, fp32 tensors out, tensor-core arithmetic in between.
//
// DadGPT keeps every activation in fp32 and selects reduced precision per operation: its
// gpu_set_matmul_precision(BF16) (reference cuda/gpu_ops.cuh:43-44, the training default in
// src/train.hpp:29) makes cuBLAS round the GEMM operands to bf16 and accumulate in fp32. The
// entry points here give the fused attention the same contract: q, k, v (and dO, O) are rounded
// to bf16 on the fly into a workspace and the tcgen05 kernels of flash_*_sm100.cu run on them with
// fp32 softmax and accumulation. At head size 64 those kernels write the caller's fp32 tensors
// themselves (dQ is summed straight into the caller's tensor), and one pass over the fp32 inputs
// rounds them, forms delta and clears dQ: at 48 x 1024 the conversions before and after the kernels
// took as long as the kernels (136 us a step). At head size 128 the bf16 results are widened by a
// pass of their own. lse is written in fp32 directly. The drop-in shim
// (gpu_ops_attention.cpp) routes the reference's fp32 signatures here when the precision mode
// says so; the exact-fp32 kernels of flash_f32.cu remain the default.
#include <cuda_bf16.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "common.cuh"

namespace dadattn {
namespace {

constexpr int kMaxCast = 5;
struct CastList {
  const void* src[kMaxCast];
  void* dst[kMaxCast];
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// blockIdx.y selects the tensor; eight elements per thread
__global__ void cast_f32_to_bf16_kernel(CastList list, int64_t n8) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n8) return;
  const float4* s = reinterpret_cast<const float4*>(list.src[blockIdx.y]) + 2 * t;
  const float4 a = s[0], b = s[1];
  reinterpret_cast<uint4*>(list.dst[blockIdx.y])[t] =
      make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
}

__global__ void cast_bf16_to_f32_kernel(CastList list, int64_t n8) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n8) return;
  const uint4 w = reinterpret_cast<const uint4*>(list.src[blockIdx.y])[t];
  float4* d = reinterpret_cast<float4*>(list.dst[blockIdx.y]) + 2 * t;
  d[0] = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u),
                     __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
  d[1] = make_float4(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u),
                     __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
}

__device__ __forceinline__ uint4 round8(const float4& a, const float4& b) {
  return make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
}

// q, k, v -> bf16: eight elements of each per thread, six 16-byte loads in flight. HBM bound.
__global__ void __launch_bounds__(256) via_forward_inputs_kernel(CastList list, int64_t n8) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n8) return;
  float4 x[3][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float4* s = static_cast<const float4*>(list.src[i]) + 2 * t;
    x[i][0] = __ldg(s);
    x[i][1] = __ldg(s + 1);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) static_cast<uint4*>(list.dst[i])[t] = round8(x[i][0], x[i][1]);
}

// Everything the gradient kernel needs, in one pass over the rows (head size 64, eight lanes per row):
// q, k, v, dout -> bf16, delta = rowsum(bf16(dout) o out) in fp32, zeros into dq and the item counter.
// From the last row on: the gradient kernel starts with the first, whose lines L2 then still holds.
__global__ void __launch_bounds__(256)
via_backward_inputs_kernel(CastList list, const float* __restrict__ out, float* __restrict__ dq,
                           float* __restrict__ delta, int* __restrict__ item_counter, int64_t n8) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t t = static_cast<int64_t>(gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x;
  if (t == 0) *item_counter = 0;
  const bool in = t < n8;
  float4 x[4][2], o[2];
  float sum = 0.f;
  if (in) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4* s = static_cast<const float4*>(list.src[i]) + 2 * t;
      x[i][0] = __ldg(s);
      x[i][1] = __ldg(s + 1);
    }
    o[0] = __ldg(reinterpret_cast<const float4*>(out) + 2 * t);
    o[1] = __ldg(reinterpret_cast<const float4*>(out) + 2 * t + 1);
    float4* z = reinterpret_cast<float4*>(dq) + 2 * t;
    z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    uint4 w;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w = round8(x[i][0], x[i][1]);
      static_cast<uint4*>(list.dst[i])[t] = w;
    }
    // with dout as rounded: what the kernel's dP is made of, so that dP - delta cancels where it should
    const uint32_t d[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 2; ++i)
      sum += __uint_as_float(d[2 * i] << 16) * o[i].x + __uint_as_float(d[2 * i] & 0xffff0000u) * o[i].y +
             __uint_as_float(d[2 * i + 1] << 16) * o[i].z + __uint_as_float(d[2 * i + 1] & 0xffff0000u) * o[i].w;
  }
#pragma unroll
  for (int d = 4; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  if (in && t % 8 == 0) delta[t / 8] = sum;
}

int launch_cast(bool to_bf16, const CastList& list, int count, int64_t elems, cudaStream_t st) {
  const int64_t n8 = elems / 8;
  dim3 grid(static_cast<unsigned>((n8 + 255) / 256), count);
  if (to_bf16)
    DAD_CUDA(launch_pdl(cast_f32_to_bf16_kernel, grid, dim3(256), 0, st, list, n8));
  else
    DAD_CUDA(launch_pdl(cast_bf16_to_f32_kernel, grid, dim3(256), 0, st, list, n8));
  return DADATTN_OK;
}

size_t tensor_bytes(int BH, int S, int D) {
  return (static_cast<size_t>(BH) * S * D * sizeof(uint16_t) + 255) / 256 * 256;
}

int check_common(int BH, int S, int D, float scale, const void* workspace, size_t given) {
  if (BH <= 0 || S <= 0) return fail(DADATTN_E_ARG, "via bf16: bad sizes BH=%d S=%d", BH, S);
  if (BH > 65535) return fail(DADATTN_E_UNSUPPORTED, "BH=%d exceeds 65535 per call", BH);
  if (D != 64 && D != 128) return fail(DADATTN_E_UNSUPPORTED, "via bf16: unsupported d_head %d", D);
  if (!(scale > 0.f)) return fail(DADATTN_E_ARG, "via bf16: scale must be positive");
  if (!workspace || !aligned(workspace, 256))
    return fail(DADATTN_E_ARG, "via bf16: workspace must be a 256-byte aligned device pointer");
  const size_t need = dadattn_flash_f32_via_bf16_workspace_bytes(BH, S, D);
  if (given < need) return fail(DADATTN_E_WORKSPACE, "via bf16: workspace %zu < %zu bytes", given, need);
  return DADATTN_OK;
}

std::atomic<int> g_precision{-1};  // -1: not decided yet (environment consulted on first read)

constexpr int kMaxDevices = 64;
void* g_scratch[kMaxDevices] = {};
size_t g_scratch_bytes[kMaxDevices] = {};
std::mutex g_scratch_mutex;

}  // namespace
}  // namespace dadattn

using namespace dadattn;

extern "C" size_t dadattn_flash_f32_via_bf16_workspace_bytes(int BH, int S, int D) {
  if (BH <= 0 || S <= 0 || D <= 0) return 0;
  // bf16 copies of q, k, v, out, dout and dq, dk, dv, then the bf16 backward's own workspace
  const size_t bwd = (dadattn_flash_bwd_bf16_workspace_bytes(BH, S, D) + 255) / 256 * 256;
  return 8 * tensor_bytes(BH, S, D) + bwd;
}

extern "C" int dadattn_flash_fwd_f32_via_bf16(float* out, float* lse, const float* q, const float* k,
                                              const float* v, int BH, int S, int D, float scale,
                                              void* workspace, size_t workspace_bytes,
                                              dadattn_stream_t stream) {
  if (!out || !lse || !q || !k || !v) return fail(DADATTN_E_ARG, "via bf16: null pointer");
  if (int rc = check_common(BH, S, D, scale, workspace, workspace_bytes)) return rc;
  if (!aligned(out, 16) || !aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16))
    return fail(DADATTN_E_ARG, "via bf16: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t tb = tensor_bytes(BH, S, D);
  char* w = static_cast<char*>(workspace);
  uint16_t *bq = reinterpret_cast<uint16_t*>(w), *bk = reinterpret_cast<uint16_t*>(w + tb),
           *bv = reinterpret_cast<uint16_t*>(w + 2 * tb), *bo = reinterpret_cast<uint16_t*>(w + 3 * tb);
  const int64_t elems = static_cast<int64_t>(BH) * S * D;
  CastList in = {{q, k, v}, {bq, bk, bv}};
  if (D == 64) {
    const int64_t n8 = elems / 8;
    DAD_CUDA(launch_pdl(via_forward_inputs_kernel, dim3(static_cast<unsigned>((n8 + 255) / 256)), dim3(256), 0, st, in,
                        n8));
    return launch_fwd_bf16_d64_f32(out, lse, bq, bk, bv, BH, S, scale, st);
  }
  if (int rc = launch_cast(true, in, 3, elems, st)) return rc;
  if (!aligned(lse, 4)) return fail(DADATTN_E_ARG, "via bf16: lse must be 4-byte aligned");
  // Sums by halves of a row at every S: the results are fp32 tensors, which callers compare as such, and their bits are
  // those that this entry point has always given.
  if (int rc = launch_fwd_bf16_d128_two_sums(bo, lse, bq, bk, bv, BH, S, scale, st)) return rc;
  CastList back = {{bo}, {out}};
  return launch_cast(false, back, 1, elems, st);
}

extern "C" int dadattn_flash_bwd_f32_via_bf16(float* dq, float* dk, float* dv, const float* dout,
                                              const float* out, const float* lse, const float* q,
                                              const float* k, const float* v, int BH, int S, int D,
                                              float scale, void* workspace, size_t workspace_bytes,
                                              dadattn_stream_t stream) {
  if (!dq || !dk || !dv || !dout || !out || !lse || !q || !k || !v)
    return fail(DADATTN_E_ARG, "via bf16: null pointer");
  if (int rc = check_common(BH, S, D, scale, workspace, workspace_bytes)) return rc;
  if (!aligned(dq, 16) || !aligned(dk, 16) || !aligned(dv, 16) || !aligned(dout, 16) ||
      !aligned(out, 16) || !aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16))
    return fail(DADATTN_E_ARG, "via bf16: tensors must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t tb = tensor_bytes(BH, S, D);
  char* w = static_cast<char*>(workspace);
  uint16_t* b[8];
  for (int i = 0; i < 8; ++i) b[i] = reinterpret_cast<uint16_t*>(w + i * tb);
  void* bwd_ws = w + 8 * tb;
  const size_t bwd_bytes = dadattn_flash_bwd_bf16_workspace_bytes(BH, S, D);
  const int64_t elems = static_cast<int64_t>(BH) * S * D;
  if (D == 64 && bwd_single_pass()) {
    // delta and the item counter take the place of the bf16 copy of `out`, which this path has no use for
    CastList in = {{q, k, v, dout}, {b[0], b[1], b[2], b[4]}};
    float* delta = reinterpret_cast<float*>(b[3]);
    int* item_counter = reinterpret_cast<int*>(b[5]);
    const int64_t n8 = elems / 8;
    DAD_CUDA(launch_pdl(via_backward_inputs_kernel, dim3(static_cast<unsigned>((n8 + 255) / 256)), dim3(256), 0, st, in,
                        out, dq, delta, item_counter, n8));
    return launch_bwd_fused_d64_f32(dq, dk, dv, delta, item_counter, b[4], lse, b[0], b[1], b[2], BH, S, scale, st);
  }
  CastList in = {{q, k, v, out, dout}, {b[0], b[1], b[2], b[3], b[4]}};
  if (int rc = launch_cast(true, in, 5, elems, st)) return rc;
  if (int rc = dadattn_flash_bwd_bf16(b[5], b[6], b[7], bwd_ws, bwd_bytes, b[4], b[3], lse, b[0], b[1],
                                      b[2], BH, S, D, scale, 0.f, 0, 0, 0, stream))
    return rc;
  CastList back = {{b[5], b[6], b[7]}, {dq, dk, dv}};
  return launch_cast(false, back, 3, elems, st);
}

extern "C" int dadattn_set_f32_precision(int mode) {
  if (mode != 0 && mode != 1) return fail(DADATTN_E_ARG, "precision mode %d (0 = fp32, 1 = bf16)", mode);
  g_precision.store(mode);
  return DADATTN_OK;
}

extern "C" int dadattn_get_f32_precision(void) {
  int mode = g_precision.load();
  if (mode < 0) {
    const char* env = std::getenv("DADATTN_PRECISION");
    mode = (env && (!std::strcmp(env, "bf16") || !std::strcmp(env, "BF16"))) ? 1 : 0;
    g_precision.store(mode);
  }
  return mode;
}

extern "C" int dadattn_library_scratch(size_t bytes, void** ptr) {
  if (!ptr) return fail(DADATTN_E_ARG, "scratch: null pointer");
  int dev = 0;
  DAD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(DADATTN_E_UNSUPPORTED, "device ordinal %d not supported", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_bytes[dev] < bytes) {
    // Work already enqueued on the old buffer must finish before it is released.
    if (g_scratch[dev]) {
      DAD_CUDA(cudaDeviceSynchronize());
      DAD_CUDA(cudaFree(g_scratch[dev]));
      g_scratch[dev] = nullptr;
      g_scratch_bytes[dev] = 0;
    }
    void* p = nullptr;
    DAD_CUDA(cudaMalloc(&p, bytes));
    g_scratch[dev] = p;
    g_scratch_bytes[dev] = bytes;
  }
  *ptr = g_scratch[dev];
  return DADATTN_OK;
}
