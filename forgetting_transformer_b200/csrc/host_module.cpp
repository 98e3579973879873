// Python module _fox_host: the host side of the operators in native code.  A training step of the short shapes spent
// 0.4 to 3 ms in Python (argument handling, ctypes calls, one autograd node and a dozen small torch calls per
// operator) against some 50 us of kernels; here the same work is direct C++ calls.
#include "host_common.h"

#include <c10/cuda/CUDAGraphsC10Utils.h>

#include <mutex>
#include <vector>

namespace foxh {

static PyObject* g_fox_error = nullptr;

[[noreturn]] static void raise(PyObject* type, const std::string& msg) {
  PyGILState_STATE g = PyGILState_Ensure();
  PyErr_SetString(type ? type : PyExc_RuntimeError, msg.c_str());
  python_error e;
  e.persist();
  PyGILState_Release(g);
  throw e;
}
void raise_assert(const std::string& msg) { raise(PyExc_AssertionError, msg); }
void raise_fox(const std::string& msg) { raise(g_fox_error, msg); }

void check_rc(int rc, const char* what) {
  if (rc == FOX_OK) return;
  static const char* names[] = {"", "FOX_ERR_BAD_ARG", "FOX_ERR_HEAD_DIM", "FOX_ERR_ALIGNMENT", "FOX_ERR_DRIVER",
                                "FOX_ERR_TENSORMAP", "FOX_ERR_LAUNCH", "FOX_ERR_DEVICE", "FOX_ERR_TOO_LARGE",
                                "FOX_ERR_THRESHOLD", "FOX_ERR_NO_MEMORY"};
  raise_fox(std::string(what) + " failed: " + (rc < 0 && rc >= -10 ? std::string(names[-rc]) : std::to_string(rc)));
}

// ---------------------------------------------------------------- stopwatch
std::atomic<bool> g_timing{false};
namespace {
std::mutex g_timer_mu;
std::vector<Interval> g_intervals;
}  // namespace

Interval timer_begin(const char* name, cudaStream_t st) {
  Interval iv{name, nullptr, nullptr};
  C10_CUDA_CHECK(cudaEventCreate(&iv.a));
  C10_CUDA_CHECK(cudaEventCreate(&iv.b));
  C10_CUDA_CHECK(cudaEventRecord(iv.a, st));
  return iv;
}
void timer_end(const Interval& iv, cudaStream_t st) {
  C10_CUDA_CHECK(cudaEventRecord(iv.b, st));
  std::lock_guard<std::mutex> g(g_timer_mu);
  g_intervals.push_back(iv);
}
void timer_drop(const Interval& iv) {
  cudaEventDestroy(iv.a);
  cudaEventDestroy(iv.b);
}

// ---------------------------------------------------------------- status words
namespace {
constexpr int kMaxDevices = 64;
struct Status {
  Tensor words;
  std::atomic<int32_t*> ptr{nullptr};   // of `words`, once they are there
};
Status g_status[kMaxDevices];
std::mutex g_status_mu;
Status& status_of(int device) {
  if (device < 0 || device >= kMaxDevices) raise_fox("device ordinal out of range");
  return g_status[device];
}
}  // namespace

static const Tensor& status_tensor(int device) {
  Status& s = status_of(device);
  std::lock_guard<std::mutex> g(g_status_mu);
  if (!s.words.defined()) {
    s.words = at::zeros({4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    s.ptr = static_cast<int32_t*>(s.words.data_ptr());
  }
  return s.words;
}
int32_t* status_words(int device) {
  int32_t* p = status_of(device).ptr;
  return p ? p : static_cast<int32_t*>(status_tensor(device).data_ptr());
}

static void report(int device, const char* when) {
  // (a record's first word is claimed before the others are written: let the kernel end)
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  (void)cudaDeviceSynchronize();
  volatile int32_t* w = status_words(device);
  const int32_t v[4] = {w[0], w[1], w[2], w[3]};
  for (int i = 0; i < 4; ++i) w[i] = 0;
  raise_fox(std::string("kernel wait timed out") + when + ": site=" + std::to_string(v[0]) + " cta=" + std::to_string(v[1]) +
            " thread=" + std::to_string(v[2]) + " detail=" + std::to_string(v[3]));
}
void status_poll(int device) {
  volatile int32_t* w = status_of(device).ptr;
  // (a report synchronises, which a capture does not allow: the record stays for the next call)
  if (!w || w[0] == 0 || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return;
  report(device, " in an earlier step");
}
void status_check(int device) {
  volatile int32_t* w = status_of(device).ptr;
  if (!w) return;
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  C10_CUDA_CHECK(cudaDeviceSynchronize());
  if (w[0] != 0) report(device, "");
}

// ---------------------------------------------------------------- module
static FOX_PY(py_set_error) {
  HANDLE_TH_ERRORS
  Py_XINCREF(args[0]);
  g_fox_error = args[0];
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
static FOX_PY(py_status_words) {
  HANDLE_TH_ERRORS
  return THPVariable_Wrap(status_tensor(static_cast<int>(PyLong_AsLong(args[0]))));
  END_HANDLE_TH_ERRORS
}
static FOX_PY(py_status_poll) {
  HANDLE_TH_ERRORS
  status_poll(static_cast<int>(PyLong_AsLong(args[0])));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
// check_status(device or -1 for every device that has status words)
static FOX_PY(py_status_check) {
  HANDLE_TH_ERRORS
  const int only = static_cast<int>(PyLong_AsLong(args[0]));
  for (int d = 0; d < kMaxDevices; ++d)
    if (only < 0 || only == d) status_check(d);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
static FOX_PY(py_timer) {   // timer(True): start recording; timer(False): stop
  HANDLE_TH_ERRORS
  g_timing = PyObject_IsTrue(args[0]) == 1;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
static FOX_PY(py_timer_take) {   // [(kernel, milliseconds), ...] of everything recorded, which is then forgotten
  HANDLE_TH_ERRORS
  std::vector<Interval> got;
  {
    std::lock_guard<std::mutex> g(g_timer_mu);
    got.swap(g_intervals);
  }
  PyObject* out = PyList_New(0);
  for (auto& iv : got) {
    float ms = 0.f;
    C10_CUDA_CHECK(cudaEventSynchronize(iv.b));
    C10_CUDA_CHECK(cudaEventElapsedTime(&ms, iv.a, iv.b));
    timer_drop(iv);
    PyObject* t = Py_BuildValue("(sd)", iv.name, static_cast<double>(ms));
    PyList_Append(out, t);
    Py_DECREF(t);
  }
  return out;
  END_HANDLE_TH_ERRORS
}

#define FOX_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
static PyMethodDef g_methods[] = {
    FOX_METHOD("set_error", py_set_error),
    FOX_METHOD("status_words", py_status_words),
    FOX_METHOD("status_poll", py_status_poll),
    FOX_METHOD("status_check", py_status_check),
    FOX_METHOD("timer", py_timer),
    FOX_METHOD("timer_take", py_timer_take),
    FOX_METHOD("attention", py_attention),
    FOX_METHOD("attention_forward", py_attention_forward),
    FOX_METHOD("attention_backward", py_attention_backward),
    FOX_METHOD("set_block_classes", py_set_block_classes),
    FOX_METHOD("block", py_block),
    FOX_METHOD("block_step", py_block_step),
    {nullptr, nullptr, 0, nullptr}};
static PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fox_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace foxh

PyMODINIT_FUNC PyInit__fox_host(void) { return PyModule_Create(&foxh::g_module); }
