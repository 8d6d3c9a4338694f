// Library-wide pieces of the C ABI: error text, version, the device-side status word.
#include <cstring>

#include "common.cuh"

namespace dadattn {

namespace {
thread_local char g_error[512] = "";
constexpr int kMaxDevices = 64;
// Status, and a detail for it: the source line of a wait that ran out. Part of the library image on
// every device, zero when it is loaded.
__device__ int g_status_words[2];
std::atomic<int*> g_status[kMaxDevices] = {};
}  // namespace

char* error_buffer() { return g_error; }

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof g_error, fmt, ap);
  va_end(ap);
  return code;
}

// In host code the name g_status_words is only a handle; the address a kernel can use is looked up per
// device, with that device current. No allocation, so a first call may come while a stream is being
// captured, its own or another.
int* device_status_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    fail(DADATTN_E_CUDA, "no current CUDA device");
    return nullptr;
  }
  int* word = g_status[dev].load(std::memory_order_relaxed);
  if (!word) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_status_words) != cudaSuccess) {
      fail(DADATTN_E_CUDA, "cannot find the device status word: %s", cudaGetErrorString(cudaGetLastError()));
      return nullptr;
    }
    word = static_cast<int*>(p);
    g_status[dev].store(word, std::memory_order_relaxed);   // (the same address whoever looks it up)
  }
  return word;
}

int check_launch_registers(const void* kernel, int expected, std::atomic<int>& seen) {
  int regs = seen.load(std::memory_order_relaxed);
  if (regs == 0) {
    cudaFuncAttributes attr;
    DAD_CUDA(cudaFuncGetAttributes(&attr, kernel));
    regs = attr.numRegs;   // the same value for every device
    seen.store(regs, std::memory_order_relaxed);
  }
  if (regs != expected)
    return fail(DADATTN_E_UNSUPPORTED, "a kernel was compiled with %d registers per thread, its register budgets "
                "assume %d", regs, expected);
  return DADATTN_OK;
}

}  // namespace dadattn

using namespace dadattn;

extern "C" const char* dadattn_last_error(void) { return error_buffer(); }

extern "C" const char* dadattn_version(void) { return "dadattn 0.1 sm_100a"; }

extern "C" int dadattn_device_status(dadattn_stream_t stream) {
  int* word = device_status_word();
  if (!word) return DADATTN_E_CUDA;
  int host[2] = {0, 0};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  DAD_CUDA(cudaMemcpyAsync(host, word, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  DAD_CUDA(cudaMemsetAsync(word, 0, 2 * sizeof(int), st));
  DAD_CUDA(cudaStreamSynchronize(st));
  if (host[0] == DADATTN_E_TIMEOUT)
    fail(host[0], "a bounded device-side wait ran out (wait at source line %d of its kernel)", host[1]);
  else if (host[0] == DADATTN_E_ARG)
    fail(host[0], "a kernel skipped work: sequence length outside [0, max_len)");
  else if (host[0] != 0)
    fail(host[0], "device status %d", host[0]);
  return host[0];
}
