// Shared by the host extension's translation units: argument checks, the launch stopwatch, device status words and
// the (B, H, T, D) view of a torch tensor that the C ABI takes.
#pragma once
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <atomic>
#include <string>

#include "../../include/fox_b200.h"

namespace foxh {

using at::Tensor;

constexpr int64_t kSms = 148;

// Python exceptions from code that may run without the interpreter lock (the autograd engine's threads among it).
[[noreturn]] void raise_assert(const std::string& msg);   // AssertionError, as the Python mirror's asserts
[[noreturn]] void raise_fox(const std::string& msg);      // forgetting_transformer_b200.FoxError

inline void check_that(bool ok, const char* msg = "") {
  if (!ok) raise_assert(msg);
}

// fox_* return codes
void check_rc(int rc, const char* what);

// One stopwatch interval around a launch while a KernelTimer is active (in any thread: an interval belongs to the launch that
// opened it, and one whose launch fails is dropped).
struct Interval {
  const char* name = nullptr;
  cudaEvent_t a = nullptr, b = nullptr;
};
extern std::atomic<bool> g_timing;
Interval timer_begin(const char* name, cudaStream_t st);
void timer_end(const Interval& iv, cudaStream_t st);
void timer_drop(const Interval& iv);

template <typename F>
inline void launch(const char* name, cudaStream_t st, F&& f) {
  if (!g_timing.load(std::memory_order_relaxed)) {
    check_rc(f(), name);
    return;
  }
  const Interval iv = timer_begin(name, st);
  const int rc = f();
  if (rc == FOX_OK) timer_end(iv, st);
  else timer_drop(iv);
  check_rc(rc, name);
}

// int32[4] in pinned host memory that a kernel writes when a bounded wait runs out (never otherwise), so that looking
// at it costs the host a load instead of a queued copy and an event per step.  Every call looks: the kernels that write may
// still run at the first call after them.
int32_t* status_words(int device);
void status_poll(int device);      // raises FoxError when there is a record, unless a graph is being captured
void status_check(int device);     // synchronising look

inline int dtype_code(at::ScalarType t) {
  if (t == at::kBFloat16) return FOX_DTYPE_BF16;
  if (t == at::kHalf) return FOX_DTYPE_FP16;
  if (t == at::kFloat) return FOX_DTYPE_FP32;
  raise_fox(std::string("unsupported dtype ") + c10::toString(t));
}

// Addressable by TMA as it is: unit inner stride, 16-byte aligned base and byte strides.
inline bool tma_ready(const Tensor& x) {
  const auto st = x.strides();
  const auto sz = x.sizes();
  if (st.back() != 1 || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16) return false;
  const int64_t es = x.element_size();
  for (size_t i = 0; i + 1 < st.size(); ++i)
    if (sz[i] != 1 && ((st[i] * es) % 16 || st[i] <= 0)) return false;
  return true;
}
inline Tensor tma_view(const Tensor& x) { return tma_ready(x) ? x : x.contiguous(); }
inline Tensor empty_like_tma(const Tensor& x) {
  Tensor o = at::empty_like(x);
  return tma_ready(o) ? o : at::empty(x.sizes(), x.options());
}

// head_first: (B,H,T,D), else (B,T,H,D)
inline fox_tensor4 t4(const Tensor& x, bool head_first) {
  const int ih = head_first ? 1 : 2, it = head_first ? 2 : 1;
  const int64_t d = x.size(3);
  // (an axis of extent 1 may carry any stride; give it one the kernels accept)
  auto stride = [&](int i) { return x.size(i) == 1 ? d : x.stride(i); };
  return fox_tensor4{x.data_ptr(), stride(0), stride(ih), stride(it)};
}

// A tangent of forward-mode differentiation.  The native nodes have none to give: their callers leave such calls to the
// Python autograd functions, which refuse them.
inline bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

// Under torch.jit.trace a native result would be recorded as the at::empty that made it: uninitialised memory in the
// traced graph.  The autograd functions are recorded as Python operators.
inline bool tracing() { return torch::jit::tracer::isTracing(); }

// A Tensor or Parameter itself.  A subclass (a quantised weight, a distributed or a not yet waited-for tensor) may have
// other semantics and no storage: its data pointer is null.
inline bool plain_tensor(PyObject* o) { return THPVariable_CheckExact(o); }

inline const Tensor& unpack(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) raise_assert(std::string(what) + " must be a tensor");
  return THPVariable_Unpack(o);
}
inline Tensor unpack_opt(PyObject* o, const char* what) { return o == Py_None ? Tensor() : unpack(o, what); }

}  // namespace foxh

// Entry points by translation unit (METH_FASTCALL)
#define FOX_PY(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t nargs)
FOX_PY(py_attention);
FOX_PY(py_attention_forward);
FOX_PY(py_attention_backward);
FOX_PY(py_set_block_classes);
FOX_PY(py_block);
FOX_PY(py_block_step);
