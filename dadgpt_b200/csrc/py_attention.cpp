// CPython module behind dadgpt_b200/attention.py: argument checks, the current stream and the C
// call of include/dadattn.h, for torch tensors.
//
// Why native: the smallest calls (a tiny fp32 step, a short prompt, one decoded token) are bound by
// the host. Checked in Python and called through ctypes, a call cost 10-13 us of host time, of
// which the launches themselves are 2-3 us each; here the checks and argument conversion are
// about 0.3 us. Tensors are unpacked with torch's own C++ accessor, never through attribute
// look-ups; the GIL is released around the C call (a launch can block on a full queue).
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <functional>
#include <initializer_list>
#include <string>
#include <utility>

#include "dadattn.h"

namespace {

PyObject* g_error_class = nullptr;   // DadAttnError(code, message), set by set_error_class

const char* type_name(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return "torch.float32";
    case at::kBFloat16: return "torch.bfloat16";
    case at::kByte: return "torch.uint8";
    case at::kInt: return "torch.int32";
    default: return c10::toString(t);
  }
}

struct Bad {};   // a Python exception is set

// Positional arguments of a METH_FASTCALL function, converted in order.
class Args {
 public:
  Args(PyObject* const* a, Py_ssize_t n, Py_ssize_t want, const char* fn) : a_(a) {
    if (n != want) {
      PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", fn, want, n);
      throw Bad{};
    }
  }
  const at::Tensor& tensor(const char* name) {
    PyObject* o = a_[i_++];
    if (!THPVariable_Check(o)) {
      PyErr_Format(PyExc_ValueError, "%s must be a torch tensor, got %s", name, Py_TYPE(o)->tp_name);
      throw Bad{};
    }
    return THPVariable_Unpack(o);
  }
  // a contiguous CUDA tensor of the given type
  const at::Tensor& need(const char* name, at::ScalarType type) {
    const at::Tensor& t = tensor(name);
    if (!t.is_cuda()) {
      PyErr_Format(PyExc_ValueError, "%s must be a CUDA tensor (there is no CPU path)", name);
      throw Bad{};
    }
    if (t.scalar_type() != type || !t.is_contiguous()) {
      PyErr_Format(PyExc_ValueError, "%s must be contiguous %s, got %s contiguous=%s", name, type_name(type),
                   type_name(t.scalar_type()), t.is_contiguous() ? "True" : "False");
      throw Bad{};
    }
    return t;
  }
  bool none() {
    if (a_[i_] != Py_None) return false;
    ++i_;
    return true;
  }
  int integer() {   // a size: larger ones than an int fit no tensor
    const int64_t v = integer64();
    if (v != static_cast<int>(v)) {
      PyErr_Format(PyExc_ValueError, "size %lld out of range", static_cast<long long>(v));
      throw Bad{};
    }
    return static_cast<int>(v);
  }
  int64_t integer64() {
    const long long v = PyLong_AsLongLong(a_[i_++]);
    if (v == -1 && PyErr_Occurred()) throw Bad{};
    return v;
  }
  uint64_t bits64() {
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(a_[i_++]);
    if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) throw Bad{};
    return v;
  }
  float real() {
    const double v = PyFloat_AsDouble(a_[i_++]);
    if (v == -1.0 && PyErr_Occurred()) throw Bad{};
    return static_cast<float>(v);
  }

 private:
  PyObject* const* a_;
  Py_ssize_t i_ = 0;
};

void need_shape(const char* name, const at::Tensor& t, std::initializer_list<int64_t> shape) {
  if (t.sizes() == at::IntArrayRef(shape.begin(), shape.size())) return;
  auto text = [](at::IntArrayRef s) {
    std::string r = "(";
    for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
    return r + (s.size() == 1 ? ",)" : ")");
  };
  PyErr_Format(PyExc_ValueError, "%s has shape %s, expected %s", name, text(t.sizes()).c_str(),
               text(at::IntArrayRef(shape.begin(), shape.size())).c_str());
  throw Bad{};
}

void need_shapes(std::initializer_list<std::pair<const char*, std::reference_wrapper<const at::Tensor>>> tensors,
                 std::initializer_list<int64_t> shape) {
  for (const auto& [name, t] : tensors) need_shape(name, t.get(), shape);
}

void* ptr(const at::Tensor& t) { return t.data_ptr(); }
float* f32(const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); }
uint16_t* b16(const at::Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()); }
dadattn_stream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

PyObject* done(int rc) {
  if (rc == 0) Py_RETURN_NONE;
  PyObject* e = PyObject_CallFunction(g_error_class ? g_error_class : PyExc_RuntimeError, "is", rc,
                                      dadattn_last_error());
  if (e) {
    PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(e)), e);
    Py_DECREF(e);
  }
  return nullptr;
}

template <typename F>
int without_gil(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}

// Runs a body that may throw Bad (exception already set) or a c10 error.
template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const Bad&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

constexpr at::ScalarType kF = at::kFloat, kB = at::kBFloat16;

// out, lse, q, k, v, BH, S, D, scale, rate, seed, offset, unit0
PyObject* fwd_f32(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 13, "fwd_f32");
    const at::Tensor &out = p.need("out", kF), &lse = p.need("lse", kF), &q = p.need("q", kF), &k = p.need("k", kF),
                     &v = p.need("v", kF);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"out", out}, {"q", q}, {"k", k}, {"v", v}}, {BH, S, D});
    need_shape("lse", lse, {BH, S});
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_fwd_f32_dropout(f32(out), f32(lse), f32(q), f32(k), f32(v), BH, S, D, scale, rate, seed,
                                           offset, unit0, st);
    }));
  });
}

// dq, dk, dv, delta, dout, out, lse, q, k, v, BH, S, D, scale, rate, seed, offset, unit0
PyObject* bwd_f32(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 18, "bwd_f32");
    const at::Tensor &dq = p.need("dq", kF), &dk = p.need("dk", kF), &dv = p.need("dv", kF),
                     &delta = p.need("delta", kF), &dout = p.need("dout", kF), &out = p.need("out", kF),
                     &lse = p.need("lse", kF), &q = p.need("q", kF), &k = p.need("k", kF), &v = p.need("v", kF);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"dq", dq}, {"dk", dk}, {"dv", dv}, {"dout", dout}, {"out", out}, {"q", q}, {"k", k}, {"v", v}},
                {BH, S, D});
    need_shape("lse", lse, {BH, S});
    if (delta.numel() < static_cast<int64_t>(BH) * S) {
      PyErr_SetString(PyExc_ValueError, "delta scratch smaller than BH*S");
      return nullptr;
    }
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_bwd_f32_dropout(f32(dq), f32(dk), f32(dv), f32(delta), f32(dout), f32(out), f32(lse),
                                           f32(q), f32(k), f32(v), BH, S, D, scale, rate, seed, offset, unit0, st);
    }));
  });
}

// out, lse, q, k, v, BH, S, D, scale, rate, seed, offset, unit0, mask_bits or None
PyObject* fwd_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 14, "fwd_bf16");
    const at::Tensor &out = p.need("out", kB), &lse = p.need("lse", kF), &q = p.need("q", kB), &k = p.need("k", kB),
                     &v = p.need("v", kB);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"out", out}, {"q", q}, {"k", k}, {"v", v}}, {BH, S, D});
    need_shape("lse", lse, {BH, S});
    const bool masked = !p.none();   // (an empty tensor's pointer is null: the library refuses it)
    const uint32_t* bits = masked ? static_cast<const uint32_t*>(ptr(p.tensor("mask_bits"))) : nullptr;
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return masked ? dadattn_flash_fwd_bf16_masked(b16(out), f32(lse), b16(q), b16(k), b16(v), BH, S, D, scale, rate,
                                                    bits, st)
                    : dadattn_flash_fwd_bf16(b16(out), f32(lse), b16(q), b16(k), b16(v), BH, S, D, scale, rate, seed,
                                             offset, unit0, st);
    }));
  });
}

// dq, dk, dv, workspace, dout, out, lse, q, k, v, BH, S, D, scale, rate, seed, offset, unit0, mask_bits or None
PyObject* bwd_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 19, "bwd_bf16");
    const at::Tensor &dq = p.need("dq", kB), &dk = p.need("dk", kB), &dv = p.need("dv", kB),
                     &ws = p.tensor("workspace"), &dout = p.need("dout", kB), &out = p.need("out", kB),
                     &lse = p.need("lse", kF), &q = p.need("q", kB), &k = p.need("k", kB), &v = p.need("v", kB);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"dq", dq}, {"dk", dk}, {"dv", dv}, {"dout", dout}, {"out", out}, {"q", q}, {"k", k}, {"v", v}},
                {BH, S, D});
    need_shape("lse", lse, {BH, S});
    const bool masked = !p.none();   // (an empty tensor's pointer is null: the library refuses it)
    const uint32_t* bits = masked ? static_cast<const uint32_t*>(ptr(p.tensor("mask_bits"))) : nullptr;
    void* const w = ptr(ws);
    const size_t bytes = ws.nbytes();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return masked ? dadattn_flash_bwd_bf16_masked(b16(dq), b16(dk), b16(dv), w, bytes, b16(dout), b16(out), f32(lse),
                                                    b16(q), b16(k), b16(v), BH, S, D, scale, rate, bits, st)
                    : dadattn_flash_bwd_bf16(b16(dq), b16(dk), b16(dv), w, bytes, b16(dout), b16(out), f32(lse),
                                             b16(q), b16(k), b16(v), BH, S, D, scale, rate, seed, offset, unit0, st);
    }));
  });
}

// out, lse, q, k, v, B, H, S, D, scale, rate, seed, offset, unit0
PyObject* fwd_bf16_strided(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 14, "fwd_bf16_strided");
    const at::Tensor &out = p.need("out", kB), &lse = p.need("lse", kF), &q = p.need("q", kB), &k = p.need("k", kB),
                     &v = p.need("v", kB);
    const int B = p.integer(), H = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"out", out}, {"q", q}, {"k", k}, {"v", v}}, {int64_t(B) * S, int64_t(H) * D});
    need_shape("lse", lse, {int64_t(B) * H, S});
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_fwd_bf16_strided(b16(out), f32(lse), b16(q), b16(k), b16(v), B, H, S, D, scale, rate, seed,
                                            offset, unit0, st);
    }));
  });
}

// dq, dk, dv, workspace, dout, out, lse, q, k, v, B, H, S, D, scale, rate, seed, offset, unit0
PyObject* bwd_bf16_strided(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 19, "bwd_bf16_strided");
    const at::Tensor &dq = p.need("dq", kB), &dk = p.need("dk", kB), &dv = p.need("dv", kB),
                     &ws = p.tensor("workspace"), &dout = p.need("dout", kB), &out = p.need("out", kB),
                     &lse = p.need("lse", kF), &q = p.need("q", kB), &k = p.need("k", kB), &v = p.need("v", kB);
    const int B = p.integer(), H = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real(), rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    need_shapes({{"dq", dq}, {"dk", dk}, {"dv", dv}, {"dout", dout}, {"out", out}, {"q", q}, {"k", k}, {"v", v}},
                {int64_t(B) * S, int64_t(H) * D});
    need_shape("lse", lse, {int64_t(B) * H, S});
    void* const w = ptr(ws);
    const size_t bytes = ws.nbytes();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_bwd_bf16_strided(b16(dq), b16(dk), b16(dv), w, bytes, b16(dout), b16(out), f32(lse),
                                            b16(q), b16(k), b16(v), B, H, S, D, scale, rate, seed, offset, unit0, st);
    }));
  });
}

// out, lse, q, k, v, BH, S, D, scale, workspace
PyObject* fwd_via_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 10, "fwd_via_bf16");
    const at::Tensor &out = p.need("out", kF), &lse = p.need("lse", kF), &q = p.need("q", kF), &k = p.need("k", kF),
                     &v = p.need("v", kF);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real();
    const at::Tensor& ws = p.tensor("workspace");
    need_shapes({{"out", out}, {"q", q}, {"k", k}, {"v", v}}, {BH, S, D});
    need_shape("lse", lse, {BH, S});
    void* const w = ptr(ws);
    const size_t bytes = ws.nbytes();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_fwd_f32_via_bf16(f32(out), f32(lse), f32(q), f32(k), f32(v), BH, S, D, scale, w, bytes, st);
    }));
  });
}

// dq, dk, dv, dout, out, lse, q, k, v, BH, S, D, scale, workspace
PyObject* bwd_via_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 14, "bwd_via_bf16");
    const at::Tensor &dq = p.need("dq", kF), &dk = p.need("dk", kF), &dv = p.need("dv", kF),
                     &dout = p.need("dout", kF), &out = p.need("out", kF), &lse = p.need("lse", kF),
                     &q = p.need("q", kF), &k = p.need("k", kF), &v = p.need("v", kF);
    const int BH = p.integer(), S = p.integer(), D = p.integer();
    const float scale = p.real();
    const at::Tensor& ws = p.tensor("workspace");
    need_shapes({{"dq", dq}, {"dk", dk}, {"dv", dv}, {"dout", dout}, {"out", out}, {"q", q}, {"k", k}, {"v", v}},
                {BH, S, D});
    need_shape("lse", lse, {BH, S});
    void* const w = ptr(ws);
    const size_t bytes = ws.nbytes();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_flash_bwd_f32_via_bf16(f32(dq), f32(dk), f32(dv), f32(dout), f32(out), f32(lse), f32(q), f32(k),
                                            f32(v), BH, S, D, scale, w, bytes, st);
    }));
  });
}

// bits, BH, S, rate, seed, offset, unit0
PyObject* mask_bits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 7, "mask_bits");
    const at::Tensor& bits = p.need("mask bits", at::kInt);
    const int BH = p.integer(), S = p.integer();
    const float rate = p.real();
    const uint64_t seed = p.bits64(), offset = p.bits64();
    const int64_t unit0 = p.integer64();
    uint32_t* const dst = static_cast<uint32_t*>(ptr(bits));
    const size_t bytes = bits.nbytes();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] { return dadattn_dropout_mask_bits(dst, bytes, BH, S, rate, seed, offset, unit0, st); }));
  });
}

// out, q, k_new, v_new, k_cache, v_cache, pos, scale
PyObject* decode_f32(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 8, "decode_f32");
    const at::Tensor &out = p.need("out", kF), &q = p.need("q", kF), &kn = p.need("k_new", kF),
                     &vn = p.need("v_new", kF), &k = p.need("k_cache", kF), &v = p.need("v_cache", kF);
    const int64_t pos = p.integer64();
    const float scale = p.real();
    if (k.dim() != 3) {
      PyErr_SetString(PyExc_ValueError, "k_cache must be [H, max_len, D]");
      return nullptr;
    }
    const int H = static_cast<int>(k.size(0)), max_len = static_cast<int>(k.size(1)), D = static_cast<int>(k.size(2));
    if (pos < 0 || pos >= max_len) {
      PyErr_Format(PyExc_IndexError, "model_forward_cached: pos %lld outside context length %d",
                   static_cast<long long>(pos), max_len);
      return nullptr;
    }
    need_shape("v_cache", v, {H, max_len, D});
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_decode_f32(f32(out), f32(q), f32(kn), f32(vn), f32(k), f32(v), H, max_len, D,
                                static_cast<int>(pos), scale, st);
    }));
  });
}

// out, q, k_new, v_new, k_cache, v_cache, lengths, B, H, D, max_len, scale, workspace
PyObject* decode_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args p(a, n, 13, "decode_bf16");
    const at::Tensor &out = p.need("out", kB), &q = p.need("q", kB), &kn = p.need("k_new", kB),
                     &vn = p.need("v_new", kB), &k = p.tensor("k_cache"), &v = p.tensor("v_cache"),
                     &len = p.tensor("lengths");
    const int B = p.integer(), H = p.integer(), D = p.integer(), max_len = p.integer();
    const float scale = p.real();
    const at::Tensor& ws = p.tensor("workspace");
    need_shapes({{"out", out}, {"q", q}, {"k_new", kn}, {"v_new", vn}}, {B, H, D});
    int32_t* const lengths = static_cast<int32_t*>(ptr(len));
    void* const w = ptr(ws);
    const size_t bytes = ws.numel();
    const dadattn_stream_t st = stream();
    return done(without_gil([&] {
      return dadattn_decode_bf16(b16(out), b16(q), b16(kn), b16(vn), b16(k), b16(v), lengths, B, H, D, max_len, scale,
                                 w, bytes, st);
    }));
  });
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_XINCREF(cls);
  Py_XDECREF(g_error_class);
  g_error_class = cls;
  Py_RETURN_NONE;
}

#define FAST(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(fwd_f32), FAST(bwd_f32), FAST(fwd_bf16), FAST(bwd_bf16), FAST(fwd_bf16_strided),
                           FAST(bwd_bf16_strided), FAST(fwd_via_bf16), FAST(bwd_via_bf16), FAST(mask_bits),
                           FAST(decode_f32), FAST(decode_bf16),
                           {"set_error_class", set_error_class, METH_O, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&g_module); }
