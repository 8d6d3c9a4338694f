"""A kernel to put ahead of the library's in a stream: it releases its dependents at once
(griddepcontrol.launch_dependents), so that a kernel launched with programmatic stream serialization may
start beside it, and only some time later touches memory. What the library's kernels do before they have
waited for it then shows in the results."""
import functools

import torch
from cuda.bindings import driver, nvrtc

SOURCE = rb"""
extern "C" __global__ void ahead(int* dst, const int* src, long long n, int value, int pause) {
  asm volatile("griddepcontrol.launch_dependents;");
  for (int i = 0; i < pause; ++i) __nanosleep(1000);
  for (long long i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src ? src[i] : value;
}
"""


def _ok(result):
    assert int(result[0]) == 0, result[0]
    return result[1] if len(result) > 1 else None


@functools.cache
def _kernel():
    torch.cuda.current_stream().synchronize()   # makes the context current
    program = _ok(nvrtc.nvrtcCreateProgram(SOURCE, b"ahead.cu", 0, [], []))
    _ok(nvrtc.nvrtcCompileProgram(program, 1, [b"--gpu-architecture=sm_100a"]))
    image = b" " * _ok(nvrtc.nvrtcGetCUBINSize(program))
    _ok(nvrtc.nvrtcGetCUBIN(program, image))
    module = _ok(driver.cuModuleLoadData(image))
    return _ok(driver.cuModuleGetFunction(module, b"ahead"))


def launch(dst, src=None, value=0, pause=400):
    """After about `pause` microseconds: dst[i] = src[i], or `value` without src (4-byte words). One block
    of 256 threads on the current stream."""
    import ctypes
    n = dst.numel() * dst.element_size() // 4
    assert dst.is_contiguous() and (src is None or src.numel() * src.element_size() // 4 >= n)
    args = ((dst.data_ptr(), src.data_ptr() if src is not None else 0, n, value, pause),
            (ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_int))
    _ok(driver.cuLaunchKernel(_kernel(), 1, 1, 1, 256, 1, 1, 0, torch.cuda.current_stream().cuda_stream, args, 0))
