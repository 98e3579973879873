// FoxProBlock on the host: one forward and one backward for the whole block (attn_norm -> attention layer -> residual ->
// mlp_norm -> SwiGLU MLP -> residual; upstream's modeling_forgetting_transformer.py:98-430, 467-516, 552-622).
//
// The modules' own forward calls some twenty operators through Python, each with an autograd node, and its backward adds
// seven gradients of the normalised input with a kernel each: 2.6 ms per step of host work for B4 T512, 0.5 ms of
// kernels.  Here the seven projections are one product with the stacked weights (fox_pack, one pass over them) and their
// gradients one product each way, taken apart by fox_unpack.  Forward: 8 kernels (9 pruned) and 4 products; backward: 10 (11
// at head dim 128) and 8.
#include "host_block.h"
#include "host_gemm.h"

#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/graph_task.h>

#include <cmath>

namespace foxh {

// ---------------------------------------------------------------- the module tree
namespace {
enum Class { kLayerCls, kMlpCls, kRmsCls, kGroupCls, kGatedCls, kShiftCls, kLinearCls, kCacheCls, kStoreCls, kClasses };
constexpr int kModuleClasses = kCacheCls;   // those before it are modules
PyObject* g_classes[kClasses] = {};
PyObject* g_forwards[kModuleClasses] = {};   // their forward functions
PyObject* g_module_call[2] = {};             // torch.nn.Module and its __call__
PyObject* g_global_hooks[4] = {};   // torch.nn's global forward / pre / backward / backward pre hooks

// interned attribute names
#define FOX_NAMES(X)                                                                                                        \
  X(_modules) X(_parameters) X(_forward_hooks) X(_forward_pre_hooks) X(_backward_hooks) X(_backward_pre_hooks) X(forward)     \
  X(weight) X(bias) X(attn_norm) X(attn) X(mlp_norm) X(mlp) X(q_proj) X(k_proj) X(v_proj) X(o_proj) X(fgate_proj)             \
  X(ogate_proj) X(output_norm) X(q_norm) X(k_norm) X(linear) X(shift_proj) X(gate_proj) X(down_proj) X(eps) X(num_heads)      \
  X(log_pruning_tolerance) X(qk_norm) X(use_k_shift) X(use_v_shift) X(activation) X(is_rms_norm) X(num_groups)     \
  X(_layers) X(key_shift_cache) X(value_shift_cache) X(_seen_tokens) X(k) X(v) X(g) X(length) X(__call__)
#define FOX_DECL(n) PyObject* s_##n;
FOX_NAMES(FOX_DECL)
#undef FOX_DECL

// A module's attribute dictionaries (borrowed while the module lives; read under the interpreter lock)
struct Mod {
  PyObject* dict = nullptr;
  PyObject* get(PyObject* name) const { return PyDict_GetItem(dict, name); }
  bool flag(PyObject* name) const { PyObject* v = get(name); return v && PyObject_IsTrue(v) == 1; }
  double number(PyObject* name) const {   // -1 for anything but a number, which is left to the modules
    PyObject* v = get(name);
    return v && (PyFloat_Check(v) || PyLong_Check(v)) ? PyFloat_AsDouble(v) : -1.;
  }
  bool none(PyObject* name) const { PyObject* v = get(name); return v == Py_None; }
  PyObject* child(PyObject* name) const {
    PyObject* m = get(s__modules);
    return m ? PyDict_GetItem(m, name) : nullptr;
  }
  PyObject* param(PyObject* name) const {
    PyObject* m = get(s__parameters);
    return m ? PyDict_GetItem(m, name) : nullptr;
  }
};

bool open(PyObject* obj, Mod& m) {
  PyObject* d = PyObject_GenericGetDict(obj, nullptr);
  if (!d) {
    PyErr_Clear();
    return false;
  }
  m.dict = d;
  Py_DECREF(d);   // (the module keeps it)
  return true;
}
bool empty_dict(PyObject* d) { return !d || d == Py_None || (PyDict_Check(d) && PyDict_GET_SIZE(d) == 0); }

// Is a class's attribute still the function it was when the package was loaded?  (Another one may have been put there.)
bool unpatched(PyObject* cls, PyObject* name, PyObject* function) {
  return PyDict_GetItem(reinterpret_cast<PyTypeObject*>(cls)->tp_dict, name) == function;
}

bool open_plain(const Mod& parent, PyObject* name, Class cls, Mod& m) {
  PyObject* obj = parent.child(name);
  if (!obj || reinterpret_cast<PyObject*>(Py_TYPE(obj)) != g_classes[cls] || !unpatched(g_classes[cls], s_forward, g_forwards[cls]) ||
      !open(obj, m))
    return false;
  return empty_dict(m.get(s__forward_hooks)) && empty_dict(m.get(s__forward_pre_hooks)) && empty_dict(m.get(s__backward_hooks)) &&
         empty_dict(m.get(s__backward_pre_hooks)) && !m.get(s_forward);
}

bool tensor(PyObject* o, Tensor& t) {
  if (!o || !plain_tensor(o)) return false;
  t = THPVariable_Unpack(o);
  return true;
}
bool matrix(const Mod& m, const Tensor& x, int64_t rows, int64_t cols, Tensor& t) {
  return tensor(m.param(s_weight), t) && t.dim() == 2 && t.size(0) == rows && t.size(1) == cols && t.is_contiguous() &&
         t.scalar_type() == x.scalar_type() && t.device() == x.device() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}
bool vector(PyObject* o, const Tensor& x, int64_t n, Tensor& t) {
  if (!tensor(o, t) || t.dim() != 1 || t.size(0) != n || !t.is_contiguous() || t.device() != x.device()) return false;
  const auto d = t.scalar_type();
  return d == at::kFloat || d == at::kHalf || d == at::kBFloat16;
}
bool no_bias(const Mod& m) { PyObject* b = m.param(s_bias); return !b || b == Py_None; }
bool linear(const Mod& parent, PyObject* name, const Tensor& x, int64_t rows, int64_t cols, Tensor& t) {
  Mod m;
  return open_plain(parent, name, kLinearCls, m) && no_bias(m) && matrix(m, x, rows, cols, t);
}
bool norm(const Mod& parent, PyObject* name, Class cls, const Tensor& x, int64_t n, int64_t groups, Tensor& t, float& eps) {
  Mod m;
  if (!open_plain(parent, name, cls, m) || !no_bias(m) || !vector(m.param(s_weight), x, n, t)) return false;
  eps = static_cast<float>(m.number(s_eps));
  if (cls == kRmsCls) return eps >= 0.f;
  if (!m.flag(s_is_rms_norm) || m.number(s_num_groups) != static_cast<double>(groups)) return false;
  if (cls == kGatedCls) {
    PyObject* a = m.get(s_activation);
    if (!a || !PyUnicode_Check(a) || PyUnicode_CompareWithASCIIString(a, "sigmoid") != 0) return false;
  }
  return eps >= 0.f;
}
bool shift_linear(const Mod& parent, PyObject* name, const Tensor& x, int64_t C, int64_t H, Tensor& w, Tensor& mix) {
  Mod m;
  return open_plain(parent, name, kShiftCls, m) && m.number(s_num_heads) == static_cast<double>(H) &&
         linear(m, s_linear, x, C, C, w) && linear(m, s_shift_proj, x, H, C, mix);
}
bool row_norm_size(int64_t C) {   // what fox_rmsnorm is built for
  const int64_t v = C / 256;
  return C % 256 == 0 && v >= 1 && v <= 8 && v != 7;
}
}  // namespace

bool read_block(PyObject* self, const Tensor& x, Block& b) {
  using B = Block;
  if (!g_classes[0] || tracing() || !x.is_cuda() || x.dim() != 3) return false;
  const auto dt = x.scalar_type();
  if ((dt != at::kHalf && dt != at::kBFloat16) || at::autocast::is_autocast_enabled(at::kCUDA)) return false;
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;   // (they are there to see the products)
  for (PyObject* h : g_global_hooks)
    if (!empty_dict(h)) return false;
  if (!unpatched(g_module_call[0], s___call__, g_module_call[1])) return false;
  Mod blk, attn, mlp, m;
  if (!open(self, blk) || !open_plain(blk, s_attn, kLayerCls, attn) || !open_plain(blk, s_mlp, kMlpCls, mlp)) return false;
  const int64_t C = b.C = x.size(2), H = b.H = static_cast<int64_t>(attn.number(s_num_heads));
  if (!row_norm_size(C) || H <= 0 || C % H) return false;
  const int64_t D = b.D = C / H;
  if (D != 16 && D != 32 && D != 64 && D != 128) return false;
  if (!attn.flag(s_qk_norm) || !attn.flag(s_use_k_shift) || !attn.flag(s_use_v_shift)) return false;
  b.pruned = !attn.none(s_log_pruning_tolerance);
  float k_eps = 0.f;
  if (!norm(blk, s_attn_norm, kRmsCls, x, C, 1, b.p[B::kAttnNorm], b.attn_eps) ||
      !norm(blk, s_mlp_norm, kRmsCls, x, C, 1, b.p[B::kMlpNorm], b.mlp_eps) || !linear(attn, s_q_proj, x, C, C, b.p[B::kQ]) ||
      !shift_linear(attn, s_k_proj, x, C, H, b.p[B::kK], b.p[B::kKMix]) ||
      !shift_linear(attn, s_v_proj, x, C, H, b.p[B::kV], b.p[B::kVMix]) ||
      !linear(attn, s_ogate_proj, x, C, C, b.p[B::kOGate]) || !linear(attn, s_o_proj, x, C, C, b.p[B::kO]) ||
      !norm(attn, s_q_norm, kGroupCls, x, C, H, b.p[B::kQNorm], b.qk_eps) ||
      !norm(attn, s_k_norm, kGroupCls, x, C, H, b.p[B::kKNorm], k_eps) || k_eps != b.qk_eps ||
      !norm(attn, s_output_norm, kGatedCls, x, C, H, b.p[B::kONorm], b.o_eps))
    return false;
  if (!open_plain(attn, s_fgate_proj, kLinearCls, m) || !matrix(m, x, H, C, b.p[B::kFGate])) return false;
  PyObject* fb = m.param(s_bias);
  if (fb && fb != Py_None && (!vector(fb, x, H, b.p[B::kFBias]) || b.p[B::kFBias].scalar_type() != dt)) return false;
  if (!open_plain(mlp, s_gate_proj, kLinearCls, m) || !no_bias(m) || !tensor(m.param(s_weight), b.p[B::kGate])) return false;
  const Tensor& g = b.p[B::kGate];
  if (g.dim() != 2 || g.size(0) % 16 || !matrix(m, x, g.size(0), C, b.p[B::kGate])) return false;
  b.inter = g.size(0) / 2;
  if (!linear(mlp, s_down_proj, x, C, b.inter, b.p[B::kDown]) || has_tangent(x)) return false;
  for (const Tensor& t : b.p)
    if (has_tangent(t)) return false;
  return true;
}

// ---------------------------------------------------------------- working memory
namespace {
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Shape {
  int64_t B = 0, T = 0, C = 0, H = 0, D = 0, inter = 0, tokens = 0, ld = 0;   // ld: columns of the stacked projection
  bool bias = false, pruned = false, mask = false;
};
Shape shape_of(const Block& b, const Tensor& x, bool mask) {
  Shape s;
  s.B = x.size(0); s.T = x.size(1); s.C = b.C; s.H = b.H; s.D = b.D; s.inter = b.inter;
  s.tokens = s.B * s.T;
  s.ld = (4 * b.C + 3 * b.H + 7) / 8 * 8;
  s.bias = b.p[Block::kFBias].defined();
  s.pruned = b.pruned;
  s.mask = mask;
  return s;
}
AttnShape attn_shape(const Shape& s) { return AttnShape{s.B, s.H, s.T, s.T, s.D}; }

// Arrays laid out one after another in one allocation, each on a 256-byte boundary: a tensor per array costs the host
// an allocation, a saved variable and a release.
struct Arena {
  char* base = nullptr;   // null: only the size is wanted
  size_t used = 0;
  template <typename T>
  T* take(int64_t n) {
    T* p = reinterpret_cast<T*>(base + used);
    used += (static_cast<size_t>(n) * sizeof(T) + 255) / 256 * 256;
    return base ? p : nullptr;
  }
};

// what the forward makes, and leaves for the backward where there is one
struct Acts {
  uint16_t *stack, *hn, *y, *qn, *kn, *vs, *o, *gated, *z, *m, *packed;
  uint16_t *proj, *act;                               // o_proj's result and the MLP's product: not kept
  float *w_attn, *w_q, *w_k, *w_o, *w_mlp;            // norm weights as fp32, one after another
  uint16_t* bias;                                     // of the stacked product (ld), or null
  float *r_attn, *r_mlp, *r_q, *r_k, *r_o;            // reciprocal norms
  float *lam, *L, *norms;
  int64_t *start, *end, *seq;
};
void lay_out_small(const Shape& s, Arena& m, Acts& a, bool keep) {
  const int64_t n = s.tokens, BH = s.B * s.H;
  a.stack = m.take<uint16_t>(s.ld * s.C);
  a.w_attn = m.take<float>(5 * s.C);
  a.w_q = a.w_attn + s.C;
  a.w_k = a.w_q + s.C;
  a.w_o = a.w_k + s.C;
  a.w_mlp = a.w_o + s.C;
  a.bias = s.bias ? m.take<uint16_t>(s.ld) : nullptr;
  a.r_attn = m.take<float>(n);
  a.r_mlp = m.take<float>(n);
  a.r_q = keep ? m.take<float>(n * s.H) : nullptr;
  a.r_k = keep ? m.take<float>(n * s.H) : nullptr;
  a.r_o = m.take<float>(n * s.H);
  a.lam = m.take<float>(BH * s.T);
  a.L = m.take<float>(BH * s.T);
  a.norms = m.take<float>(attn_norms(attn_shape(s), false).floats(BH));
  a.seq = s.mask ? m.take<int64_t>(s.B) : nullptr;
  a.start = s.pruned ? m.take<int64_t>(BH * attn_blocks(s.T)) : nullptr;
  a.end = s.pruned && keep ? m.take<int64_t>(BH * attn_blocks(s.T)) : nullptr;
}
// For a backward everything lies beside everything, what the MLP's part of it reads apart: that is released first.
size_t lay_out_mlp(const Shape& s, char* base, Acts& a) {
  Arena m{base};
  const int64_t n = s.tokens;
  a.z = m.take<uint16_t>(n * s.C);
  a.m = m.take<uint16_t>(n * s.C);
  a.packed = m.take<uint16_t>(n * 2 * s.inter);
  return m.used;
}
size_t lay_out_attn(const Shape& s, char* base, Acts& a) {
  Arena m{base};
  const int64_t n = s.tokens;
  lay_out_small(s, m, a, true);
  a.hn = m.take<uint16_t>(n * s.C);
  a.y = m.take<uint16_t>(n * s.ld);
  a.qn = m.take<uint16_t>(n * s.C);
  a.kn = m.take<uint16_t>(n * s.C);
  a.vs = m.take<uint16_t>(n * s.C);
  a.o = m.take<uint16_t>(n * s.C);
  a.gated = m.take<uint16_t>(n * s.C);
  return m.used;
}
// Without one: what is done with makes room.  The attention layer's arrays and the MLP's take turns in the same memory, o
// lies over the normalised input, the gated output over q, o_proj's result over k.
size_t lay_out_transient(const Shape& s, char* base, Acts& a) {
  Arena m{base};
  const int64_t n = s.tokens;
  lay_out_small(s, m, a, false);
  const size_t shared = m.used;
  a.proj = a.kn = m.take<uint16_t>(n * s.C);   // (first: read while m and z behind it are written)
  a.y = m.take<uint16_t>(n * s.ld);
  a.o = a.hn = m.take<uint16_t>(n * s.C);
  a.gated = a.qn = m.take<uint16_t>(n * s.C);
  a.vs = m.take<uint16_t>(n * s.C);
  const size_t attn_end = m.used;
  m.used = shared;
  a.act = m.take<uint16_t>(n * std::max(s.inter, s.C));   // (over proj, which the norm in front has read by then)
  a.m = m.take<uint16_t>(n * s.C);
  a.z = m.take<uint16_t>(n * s.C);
  a.packed = m.take<uint16_t>(n * 2 * s.inter);
  return std::max(attn_end, m.used);
}

// The backward's temporaries: what both parts use, the MLP's, the attention layer's.  The last two are never there together.
struct Temps {
  void* gemm;
  float* parts;
  uint16_t* dz;
  uint16_t *dact, *dpacked, *act, *dm;                           // MLP (dm over dact)
  uint16_t *dgated, *dy, *d_o, *dq, *dk, *dv, *dhn, *dstack;     // attention layer (dq over dgated, dhn over d_o)
  float* attn_work;
};
size_t lay_out_shared(const Shape& s, char* base, int64_t part_floats, Temps& t) {
  Arena m{base};
  t.gemm = m.take<char>(static_cast<int64_t>(kGemmWorkspace));
  t.parts = m.take<float>(part_floats);
  t.dz = m.take<uint16_t>(s.tokens * s.C);
  return m.used;
}
size_t lay_out_mlp(const Shape& s, char* base, Temps& t) {
  Arena m{base};
  const int64_t n = s.tokens;
  t.dm = t.dact = m.take<uint16_t>(n * std::max(s.inter, s.C));
  t.dpacked = m.take<uint16_t>(n * 2 * s.inter);
  t.act = m.take<uint16_t>(n * s.inter);
  return m.used;
}
size_t lay_out_attn(const Shape& s, char* base, bool two_kernel, Temps& t) {
  Arena m{base};
  const int64_t n = s.tokens;
  t.dq = t.dgated = m.take<uint16_t>(n * s.C);
  t.dy = m.take<uint16_t>(n * s.ld);
  t.dhn = t.d_o = m.take<uint16_t>(n * s.C);
  t.dk = m.take<uint16_t>(n * s.C);
  t.dv = m.take<uint16_t>(n * s.C);
  t.dstack = m.take<uint16_t>(s.ld * s.C);
  t.attn_work = m.take<float>(attn_backward_floats(attn_shape(s), two_kernel));
  return m.used;
}
// memory for one of the layouts above, which lay(nullptr) sizes and lay(base) places
template <typename F>
Tensor allocate(const at::TensorOptions& bytes, F&& lay) {
  const Tensor t = at::empty({static_cast<int64_t>(lay(nullptr))}, bytes);
  lay(static_cast<char*>(t.data_ptr()));
  return t;
}

AttnCall attn_call(const Shape& s, const Acts& a, int dev, cudaStream_t st, int code) {
  AttnCall c;
  c.device = dev;
  c.st = st;
  c.code = code;
  c.s = attn_shape(s);
  auto t4 = [&](uint16_t* p) { return fox_tensor4{p, s.T * s.C, s.D, s.C}; };
  c.q = t4(a.qn);
  c.k = t4(a.kn);
  c.v = t4(a.vs);
  c.o = t4(a.o);
  c.sm_scale = static_cast<float>(1. / std::sqrt(static_cast<double>(s.D)));
  c.seq_start = a.seq;
  c.gate_kind = code;
  c.gate = a.y + 4 * s.C;
  c.gate_st[0] = s.T * s.ld;
  c.gate_st[1] = 1;
  c.gate_st[2] = s.ld;
  c.lam = a.lam;
  c.L = a.L;
  c.start = a.start;
  c.end = a.end;
  return c;
}

// ---------------------------------------------------------------- forward
void pack(int dev, cudaStream_t st, const Block& b, const Shape& s, const Acts& a) {
  using B = Block;
  const B::Param mats[] = {B::kQ, B::kK, B::kV, B::kOGate, B::kFGate, B::kKMix, B::kVMix};
  const void* mp[7];
  int64_t rows[7];
  for (int i = 0; i < 7; ++i) {
    mp[i] = b.p[mats[i]].const_data_ptr();
    rows[i] = b.p[mats[i]].size(0);
  }
  const B::Param vs[] = {B::kAttnNorm, B::kQNorm, B::kKNorm, B::kONorm, B::kMlpNorm};
  const void* vp[5];
  int64_t len[5];
  int32_t vd[5];
  for (int i = 0; i < 5; ++i) {
    vp[i] = b.p[vs[i]].const_data_ptr();
    len[i] = b.p[vs[i]].size(0);
    vd[i] = dtype_code(b.p[vs[i]].scalar_type());
  }
  launch("fox_pack", st, [&] {
    return fox_pack(dev, st, 7, mp, rows, s.ld, s.C, a.stack, 5, vp, len, vd, a.w_attn,
                    s.bias ? b.p[B::kFBias].const_data_ptr() : nullptr, s.H, 4 * s.C, a.bias);
  });
}

struct Forward {
  Tensor out, acts, mlp_acts, mask;
};

Forward forward(const Block& b, const Shape& s, const Tensor& x_in, const Tensor& mask, const Tensor& threshold, bool needs_grad) {
  const c10::cuda::CUDAGuard guard(x_in.device());
  const at::AutoDispatchBelowADInplaceOrView no_autograd;
  const int dev = x_in.device().index();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const int code = dtype_code(x_in.scalar_type());
  const auto bytes = x_in.options().dtype(at::kByte);
  status_poll(dev);
  Forward f;
  const Tensor x = x_in.contiguous();
  Acts a;
  if (needs_grad) {
    f.acts = allocate(bytes, [&](char* base) { return lay_out_attn(s, base, a); });
    f.mlp_acts = allocate(bytes, [&](char* base) { return lay_out_mlp(s, base, a); });
  } else {
    f.acts = allocate(bytes, [&](char* base) { return lay_out_transient(s, base, a); });
  }
  // [product workspace | with a backward: o_proj's result, then the MLP's product]
  const Tensor temp = at::empty({static_cast<int64_t>(kGemmWorkspace) + (needs_grad ? 2 * s.tokens * std::max(s.inter, s.C) : 0)}, bytes);
  Gemm g{dev, code, st, temp.data_ptr()};
  if (needs_grad) a.proj = a.act = reinterpret_cast<uint16_t*>(static_cast<char*>(temp.data_ptr()) + kGemmWorkspace);
  f.out = at::empty(x_in.sizes(), x_in.options());

  pack(dev, st, b, s, a);
  launch("fox_rmsnorm_fwd", st, [&] {
    return fox_rmsnorm_fwd(dev, st, code, s.tokens, s.C, x.const_data_ptr(), nullptr, a.w_attn, b.attn_eps, a.hn, nullptr, a.r_attn);
  });
  gemm(g, s.tokens, s.ld, s.C, a.hn, s.C, false, a.stack, s.C, true, nullptr, 0, a.y, s.ld, a.bias);
  const int64_t* mask_p = nullptr;
  if (mask.defined()) {
    f.mask = mask.to(at::kLong).contiguous();
    mask_p = f.mask.const_data_ptr<int64_t>();
  }
  launch("fox_mix_fwd", st, [&] {
    return fox_mix_fwd(dev, st, code, s.B, s.T, s.H, s.D, a.y, s.ld, a.w_q, a.w_k, b.qk_eps, mask_p, a.qn, a.kn, a.vs, a.r_q, a.r_k,
                       a.seq);
  });
  Tensor thr;
  if (threshold.defined()) thr = threshold.detach().to(x_in.device(), at::kFloat).expand({s.B, s.H});
  AttnCall c = attn_call(s, a, dev, st, code);
  attn_forward_launch(c, attn_norms(c.s, false), a.norms, thr.defined() ? Threshold::kTensor : Threshold::kNone, 0.,
                      thr.defined() ? static_cast<float*>(thr.data_ptr()) : nullptr, thr.defined() ? thr.stride(0) : 0,
                      thr.defined() ? thr.stride(1) : 0);
  launch("fox_normgate_fwd", st, [&] {
    return fox_normgate_fwd_ld(dev, st, code, s.tokens, s.H, s.D, a.o, a.y + 3 * s.C, s.ld, a.w_o, b.o_eps, a.gated, a.r_o);
  });
  gemm(g, s.tokens, s.C, s.C, a.gated, s.C, false, b.p[Block::kO].const_data_ptr(), s.C, true, nullptr, 0, a.proj, s.C);
  launch("fox_rmsnorm_fwd", st, [&] {
    return fox_rmsnorm_fwd(dev, st, code, s.tokens, s.C, a.proj, x.const_data_ptr(), a.w_mlp, b.mlp_eps, a.m, a.z, a.r_mlp);
  });
  gemm(g, s.tokens, 2 * s.inter, s.C, a.m, s.C, false, b.p[Block::kGate].const_data_ptr(), s.C, true, nullptr, 0, a.packed, 2 * s.inter);
  launch("fox_swiglu_fwd", st, [&] {
    return fox_swiglu_fwd(dev, st, code, s.tokens, s.inter, a.packed, 2 * s.inter, a.packed + s.inter, 2 * s.inter, a.act, s.inter);
  });
  gemm(g, s.tokens, s.C, s.inter, a.act, s.inter, false, b.p[Block::kDown].const_data_ptr(), s.inter, true, a.z, s.C,
       f.out.mutable_data_ptr(), s.C);
  return f;
}

// ---------------------------------------------------------------- backward
struct BlockBackward : public torch::autograd::Node {
  SavedVariable x, acts, mlp_acts, mask, w_o, w_gate, w_down;
  at::ScalarType dtypes[Block::kCount];
  bool released = false;
  Shape s;

  std::string name() const override { return "FoxProBlockBackward"; }
  void release_variables() override {
    for (SavedVariable* v : {&x, &acts, &mlp_acts, &mask, &w_o, &w_gate, &w_down}) v->reset_data();
    released = true;
  }

  variable_list apply(variable_list&& grads) override {
    using B = Block;
    variable_list out(1 + B::kCount);
    if (!grads[0].defined()) return out;
    if (released) throw std::runtime_error(torch::autograd::ERR_BACKWARD_TWICE);
    const Tensor xt = x.unpack().contiguous(), at_ = acts.unpack(), mt = mask.unpack();
    Tensor mlp_at = mlp_acts.unpack();
    const Tensor wo = w_o.unpack(), wg = w_gate.unpack(), wd = w_down.unpack();
    const c10::cuda::CUDAGuard guard(xt.device());
    const at::AutoDispatchBelowADInplaceOrView no_autograd;
    const int dev = xt.device().index();
    C10_CUDA_CHECK(cudaSetDevice(dev));   // (gives an engine thread the device's context before the library's first call)
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
    const int code = dtype_code(xt.scalar_type());
    const auto o16 = xt.options();
    const int64_t n = s.tokens, C = s.C, I = s.inter;
    Acts a;
    lay_out_attn(s, static_cast<char*>(at_.data_ptr()), a);
    lay_out_mlp(s, static_cast<char*>(mlp_at.data_ptr()), a);
    auto want = [&](int i) { return task_should_compute_output(1 + i); };
    const Tensor dout = grads[0].contiguous();

    // partial sums of the norm weights' gradients and of the gate bias's, joined in one launch at the end
    const int64_t rn = std::min<int64_t>((n + 7) / 8, 148 * 4), ng = std::min<int64_t>(n, 148 * 4);
    const int64_t mx = fox_mix_bwd_partials(n);
    const bool two_kernel = default_two_kernel(s.D);
    const int64_t part_floats = C * (2 * rn + ng + 2 * mx) + s.B * s.H;
    const auto bytes = o16.dtype(at::kByte);
    Temps t;
    const Tensor shared = allocate(bytes, [&](char* base) { return lay_out_shared(s, base, part_floats, t); });
    Tensor temp = allocate(bytes, [&](char* base) { return lay_out_mlp(s, base, t); });
    float* part_attn = t.parts;
    float* part_mlp = part_attn + rn * C;
    float* part_o = part_mlp + rn * C;
    float* part_q = part_o + ng * C;
    float* part_k = part_q + mx * C;
    float* part_bias = part_k + mx * C;
    Gemm g{dev, code, st, t.gemm};
    // dW (rows, cols) = dY^T X, where it is asked for
    auto weight_grad = [&](B::Param w, int64_t rows, int64_t cols, const void* dy, const void* in) {
      if (!want(w)) return;
      out[1 + w] = at::empty({rows, cols}, o16);
      gemm(g, rows, cols, n, dy, rows, true, in, cols, false, nullptr, 0, out[1 + w].mutable_data_ptr(), cols);
    };

    // ---- MLP
    const void* gout = dout.const_data_ptr();
    gemm(g, n, I, C, gout, C, false, wd.const_data_ptr(), I, false, nullptr, 0, t.dact, I);
    launch("fox_swiglu_bwd", st, [&] {
      return fox_swiglu_bwd(dev, st, code, n, I, a.packed, 2 * I, a.packed + I, 2 * I, t.dact, I, t.dpacked, 2 * I, t.dpacked + I,
                            2 * I, t.act, I);
    });
    weight_grad(B::kDown, C, I, gout, t.act);
    gemm(g, n, C, 2 * I, t.dpacked, 2 * I, false, wg.const_data_ptr(), C, false, nullptr, 0, t.dm, C);
    weight_grad(B::kGate, 2 * I, C, t.dpacked, a.m);
    launch("fox_rmsnorm_bwd", st, [&] {
      return fox_rmsnorm_bwd(dev, st, code, n, C, a.z, a.w_mlp, a.r_mlp, t.dm, gout, t.dz, part_mlp, rn);
    });
    // ---- attention layer, in the memory that the MLP's part no longer needs (this stream's, so that reuse keeps the order)
    temp.reset();
    mlp_at.reset();
    if (!torch::autograd::get_current_graph_task_keep_graph()) mlp_acts.reset_data();
    temp = allocate(bytes, [&](char* base) { return lay_out_attn(s, base, two_kernel, t); });
    gemm(g, n, C, C, t.dz, C, false, wo.const_data_ptr(), C, false, nullptr, 0, t.dgated, C);
    weight_grad(B::kO, C, C, t.dz, a.gated);
    launch("fox_normgate_bwd", st, [&] {
      return fox_normgate_bwd_ld(dev, st, code, n, s.H, s.D, a.o, a.y + 3 * C, s.ld, a.w_o, a.r_o, t.dgated, t.d_o, t.dy + 3 * C,
                                 s.ld, part_o, ng);
    });
    const AttnCall c = attn_call(s, a, dev, st, code);
    AttnGradCall gc;
    auto t4 = [&](uint16_t* p) { return fox_tensor4{p, s.T * C, s.D, C}; };
    gc.g = t4(t.d_o);
    gc.dq = t4(t.dq);
    gc.dk = t4(t.dk);
    gc.dv = t4(t.dv);
    gc.work = t.attn_work;
    gc.dgate = t.dy + 4 * C;
    for (int i = 0; i < 3; ++i) gc.dgate_st[i] = c.gate_st[i];
    gc.dbias = s.bias ? part_bias : nullptr;
    gc.two_kernel = two_kernel;
    attn_backward_launch(c, gc);
    launch("fox_mix_bwd", st, [&] {
      return fox_mix_bwd(dev, st, code, s.B, s.T, s.H, s.D, a.y, s.ld, a.w_q, a.w_k, mt.defined() ? mt.const_data_ptr<int64_t>() : nullptr,
                         a.r_q, a.r_k, t.dq, t.dk, t.dv, t.dy, part_q, part_k, mx);
    });
    static const B::Param mats[] = {B::kQ, B::kK, B::kV, B::kOGate, B::kFGate, B::kKMix, B::kVMix};
    bool any = false;
    for (B::Param m : mats) any = any || want(m);
    if (any) {   // one product, taken apart
      gemm(g, s.ld, C, n, t.dy, s.ld, true, a.hn, C, false, nullptr, 0, t.dstack, C);
      void* dst[7];
      int64_t rows[7];
      for (int i = 0; i < 7; ++i) {
        rows[i] = i < 4 ? C : s.H;
        if (want(mats[i])) out[1 + mats[i]] = at::empty({rows[i], C}, o16);
        dst[i] = want(mats[i]) ? out[1 + mats[i]].mutable_data_ptr() : nullptr;
      }
      launch("fox_unpack", st, [&] { return fox_unpack(dev, st, 7, dst, rows, C, t.dstack); });
    }
    gemm(g, n, C, s.ld, t.dy, s.ld, false, a.stack, C, false, nullptr, 0, t.dhn, C);
    const Tensor dx = at::empty(xt.sizes(), o16);
    launch("fox_rmsnorm_bwd", st, [&] {
      return fox_rmsnorm_bwd(dev, st, code, n, C, xt.const_data_ptr(), a.w_attn, a.r_attn, t.dhn, t.dz, dx.mutable_data_ptr(),
                             part_attn, rn);
    });
    if (task_should_compute_output(0)) out[0] = dx;
    // ---- norm weights and gate bias
    const float* part[6] = {part_attn, part_q, part_k, part_o, part_mlp, part_bias};
    const int64_t rows[6] = {rn, mx, mx, ng, rn, s.B}, cols[6] = {C, C, C, C, C, s.H};
    static const B::Param vec[6] = {B::kAttnNorm, B::kQNorm, B::kKNorm, B::kONorm, B::kMlpNorm, B::kFBias};
    const int nv = s.bias ? 6 : 5;
    int32_t od[6];
    void* op[6];
    Tensor sums[6];
    for (int i = 0; i < nv; ++i) {
      sums[i] = at::empty({cols[i]}, o16.dtype(dtypes[vec[i]]));
      od[i] = dtype_code(dtypes[vec[i]]);
      op[i] = sums[i].data_ptr();
      if (want(vec[i])) out[1 + vec[i]] = sums[i];
    }
    launch("fox_column_sums", st, [&] { return fox_column_sums(dev, st, nv, part, rows, cols, od, op); });
    return out;
  }
};
}  // namespace

}  // namespace foxh

// ---------------------------------------------------------------- Python entry points
using namespace foxh;

// set_block_classes(FoxProAttentionLayer, FoxMLP, RMSNorm, GroupNorm, FusedGroupNormGated, ShiftLinear, nn.Linear, FgateCache,
//                   its layer store, the four global hook dictionaries of torch.nn.modules.module, nn.Module, its __call__,
//                   the forward functions of the first seven)
FOX_PY(py_set_block_classes) {
  HANDLE_TH_ERRORS
#define FOX_INTERN(n) s_##n = PyUnicode_InternFromString(#n);
  FOX_NAMES(FOX_INTERN)
#undef FOX_INTERN
  for (int i = 0; i < kClasses; ++i) {
    Py_INCREF(args[i]);
    g_classes[i] = args[i];
  }
  for (int i = 0; i < 4; ++i) {
    Py_INCREF(args[kClasses + i]);
    g_global_hooks[i] = args[kClasses + i];
  }
  PyObject* const* rest = args + kClasses + 4;
  for (int i = 0; i < 2; ++i) {
    Py_INCREF(rest[i]);
    g_module_call[i] = rest[i];
  }
  for (int i = 0; i < kModuleClasses; ++i) {
    Py_INCREF(rest[2 + i]);
    g_forwards[i] = rest[2 + i];
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// block(self, hidden_states, attention_mask or None, threshold) -> out, or None where the modules' own forward has to run.
// threshold(hidden_states) gives the pruning threshold; it is called where there is one and the block runs here.
FOX_PY(py_block) {
  HANDLE_TH_ERRORS
  Tensor x;
  Block b;
  if (!tensor(args[1], x) || !read_block(args[0], x, b)) Py_RETURN_NONE;
  if (args[2] != Py_None && !plain_tensor(args[2])) Py_RETURN_NONE;
  const Tensor mask = unpack_opt(args[2], "attention_mask");
  if (x.size(1) < 2 || x.size(0) < 1) Py_RETURN_NONE;
  if (mask.defined()) {
    const auto d = mask.scalar_type();
    if (mask.dim() != 2 || mask.size(0) != x.size(0) || mask.size(1) != x.size(1) || mask.device() != x.device() ||
        (d != at::kLong && d != at::kBool && d != at::kInt))
      Py_RETURN_NONE;
  }
  Tensor threshold;
  if (b.pruned) {
    PyObject* t = PyObject_CallOneArg(args[3], args[1]);
    if (!t) throw python_error();
    const bool ok = tensor(t, threshold);
    Py_DECREF(t);
    if (!ok) Py_RETURN_NONE;
  }
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    bool needs = false;
    if (at::GradMode::is_enabled()) {
      needs = x.requires_grad();
      for (const Tensor& t : b.p) needs = needs || (t.defined() && t.requires_grad());
    }
    const Shape s = shape_of(b, x, mask.defined());
    Forward f = forward(b, s, x, mask, threshold, needs);
    out = f.out;
    if (needs) {
      std::shared_ptr<BlockBackward> node(new BlockBackward(), torch::autograd::deleteNode);
      torch::autograd::edge_list edges;
      auto edge = [&](const Tensor& t) {
        edges.push_back(t.defined() && t.requires_grad() ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge());
      };
      edge(x);
      for (const Tensor& t : b.p) edge(t);
      node->set_next_edges(std::move(edges));
      torch::autograd::set_history(out, node);
      node->x = SavedVariable(x, false);
      node->acts = SavedVariable(f.acts, false);
      node->mlp_acts = SavedVariable(f.mlp_acts, false);
      node->mask = SavedVariable(f.mask, false);
      node->w_o = SavedVariable(b.p[Block::kO], false);
      node->w_gate = SavedVariable(b.p[Block::kGate], false);
      node->w_down = SavedVariable(b.p[Block::kDown], false);
      for (int i = 0; i < Block::kCount; ++i) node->dtypes[i] = b.p[i].defined() ? b.p[i].scalar_type() : at::kFloat;
      node->s = s;
    }
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- one generated token
namespace {
// Layer i of an FgateCache: its buffers, length and shift states, where a token fits without growing them.
struct CacheLayer {
  Tensor k, v, g, k_state, v_state;
  int64_t length = 0;
  Mod cache, store;
};
bool list_tensor(const Mod& m, PyObject* name, int64_t i, Tensor& t) {
  PyObject* l = m.get(name);
  return l && PyList_Check(l) && i < PyList_GET_SIZE(l) && tensor(PyList_GET_ITEM(l, i), t);
}
bool open_cache(PyObject* cache, int64_t i, const Tensor& x, const Block& b, CacheLayer& c) {
  if (reinterpret_cast<PyObject*>(Py_TYPE(cache)) != g_classes[kCacheCls] || i < 0 || !open(cache, c.cache)) return false;
  PyObject* layers = c.cache.get(s__layers);
  if (!layers || !PyList_Check(layers) || i >= PyList_GET_SIZE(layers)) return false;
  PyObject* store = PyList_GET_ITEM(layers, i);
  if (reinterpret_cast<PyObject*>(Py_TYPE(store)) != g_classes[kStoreCls] || !open(store, c.store)) return false;
  PyObject* len = c.store.get(s_length);
  if (!len || !PyLong_Check(len) || !tensor(c.store.get(s_k), c.k) || !tensor(c.store.get(s_v), c.v) || !tensor(c.store.get(s_g), c.g) ||
      !list_tensor(c.cache, s_key_shift_cache, i, c.k_state) || !list_tensor(c.cache, s_value_shift_cache, i, c.v_state))
    return false;
  c.length = PyLong_AsLongLong(len);
  const int64_t B = x.size(0);
  auto plain = [&](const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt && t.is_contiguous() && t.device() == x.device(); };
  for (const Tensor* t : {&c.k, &c.v})
    if (!plain(*t, x.scalar_type()) || t->dim() != 4 || t->size(0) != B || t->size(1) != b.H || t->size(3) != b.D) return false;
  for (const Tensor* t : {&c.k_state, &c.v_state})
    if (!plain(*t, x.scalar_type()) || t->numel() != B * b.C) return false;
  const int64_t cap = c.k.size(2);
  return plain(c.g, at::kFloat) && c.g.dim() == 3 && c.g.size(0) == B && c.g.size(1) == b.H && c.g.size(2) == cap && c.v.size(2) == cap &&
         c.length + 1 <= cap;
}

Tensor step(const Block& b, const Tensor& x_in, const Tensor& mask, const CacheLayer& c) {
  using B = Block;
  const c10::cuda::CUDAGuard guard(x_in.device());
  const at::AutoDispatchBelowADInplaceOrView no_autograd;
  const int dev = x_in.device().index();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev).stream();
  const int code = dtype_code(x_in.scalar_type());
  status_poll(dev);
  const Tensor x = x_in.contiguous();
  Tensor out = at::empty(x_in.sizes(), x_in.options()), mask64;
  if (mask.defined()) mask64 = mask.to(at::kLong).contiguous();
  // written in place: what has saved one of them for a backward has to notice
  for (const Tensor* t : {&c.k, &c.v, &c.g, &c.k_state, &c.v_state}) t->unsafeGetTensorImpl()->bump_version();
  const int64_t n = x.size(0), C = b.C, H = b.H, D = b.D, N = c.length + 1, cap = c.k.size(2);
  const AttnShape as{n, H, 1, N, D};
  uintptr_t bits = 0;   // (fox_step_attn takes 16-byte pieces of states and cache; the two kernels take any state)
  for (const Tensor* t : {&c.k, &c.v, &c.k_state, &c.v_state}) bits |= reinterpret_cast<uintptr_t>(t->data_ptr());
  int64_t splits = bits % 16 ? 0 : fox_step_attn_splits(n, H, N);
  // Long ranges at head dim 128 are faster by the two kernels, except one or two CTAs to an SM (16 heads, one sequence of 6000 keys
  // 61 and 58 us a layer, two 70 and 78, three 93 and 91, eight of 2000 110 and 103, of 12000 219 and 205; one of 2000 49 and 50).
  if (D == 128 && N > splits * 512 && (n * H * splits < kSms || n * H * splits > 2 * kSms)) splits = 0;
  const int64_t ld = (4 * C + 3 * H + 3) / 4 * 4;
  Tensor memory;
  float *y, *z, *L, *work;
  uint16_t *q, *o, *act;
  int64_t* seq;
  for (char* base = nullptr;;) {   // first the size, then the pieces
    Arena m{base};
    y = m.take<float>(n * ld);
    z = m.take<float>(n * C);
    L = m.take<float>(n * H);
    work = m.take<float>(splits > 0 ? 0 : attn_decode_floats(as));
    q = m.take<uint16_t>(n * C);
    o = m.take<uint16_t>(n * C);
    act = m.take<uint16_t>(n * b.inter);
    seq = m.take<int64_t>(n);
    if (base) break;
    memory = at::empty({static_cast<int64_t>(m.used)}, x.options().dtype(at::kByte));
    base = static_cast<char*>(memory.data_ptr());
  }
  int32_t* status = status_words(dev);
  auto dt = [&](B::Param p) { return dtype_code(b.p[p].scalar_type()); };
  auto ptr = [&](B::Param p) { return b.p[p].const_data_ptr(); };

  const B::Param first[] = {B::kQ, B::kK, B::kV, B::kOGate, B::kFGate, B::kKMix, B::kVMix};
  const void* mats[7];
  int64_t rows[7];
  for (int i = 0; i < 7; ++i) {
    mats[i] = ptr(first[i]);
    rows[i] = b.p[first[i]].size(0);
  }
  launch("fox_step_product", st, [&] {
    return fox_step_product_ahead(dev, st, code, 0, 0, n, C, x.const_data_ptr(), 0, ptr(B::kAttnNorm), dt(B::kAttnNorm), b.attn_eps, 0,
                                  nullptr, 0, 7, mats, rows, nullptr, y, ld, nullptr, 0, status);
  });
  const bool bias = b.p[B::kFBias].defined();
  const int64_t* mask_p = mask64.defined() ? mask64.const_data_ptr<int64_t>() : nullptr;
  const float sm_scale = static_cast<float>(1. / std::sqrt(static_cast<double>(D)));
  if (splits > 0) {
    launch("fox_step_attn", st, [&] {
      return fox_step_attn(dev, st, code, n, H, D, y, ld, ptr(B::kQNorm), dt(B::kQNorm), ptr(B::kKNorm), dt(B::kKNorm), b.qk_eps,
                           bias ? ptr(B::kFBias) : nullptr, bias ? dt(B::kFBias) : 0, mask_p, c.k_state.data_ptr(), c.v_state.data_ptr(),
                           c.k.data_ptr(), c.v.data_ptr(), c.g.mutable_data_ptr<float>(), cap, c.length, sm_scale, o, splits);
    });
  } else {
    launch("fox_step_mix", st, [&] {
      return fox_step_mix(dev, st, code, n, H, D, y, ld, ptr(B::kQNorm), dt(B::kQNorm), ptr(B::kKNorm), dt(B::kKNorm), b.qk_eps,
                          bias ? ptr(B::kFBias) : nullptr, bias ? dt(B::kFBias) : 0,
                          mask_p, seq, c.k_state.data_ptr(), c.v_state.data_ptr(), q,
                          c.k.data_ptr(), c.v.data_ptr(), c.g.mutable_data_ptr<float>(), cap, c.length);
    });
    AttnCall a;
    a.device = dev;
    a.st = st;
    a.code = code;
    a.s = as;
    a.q = fox_tensor4{q, C, D, D};
    a.o = fox_tensor4{o, C, D, D};
    a.k = fox_tensor4{c.k.data_ptr(), H * cap * D, cap * D, D};
    a.v = fox_tensor4{c.v.data_ptr(), H * cap * D, cap * D, D};
    a.sm_scale = sm_scale;
    a.seq_start = mask64.defined() ? seq : nullptr;
    a.gate = c.g.data_ptr();
    a.gate_st[0] = H * cap;
    a.gate_st[1] = cap;
    a.gate_st[2] = 1;
    a.L = L;
    attn_decode_launch(a, false, work, true);
  }
  const void* m1[1] = {ptr(B::kO)};
  const int64_t r1[1] = {C};
  launch("fox_step_product", st, [&] {
    return fox_step_product_ahead(dev, st, code, 1, 1, n, C, o, 0, ptr(B::kONorm), dt(B::kONorm), b.o_eps, D, y + 3 * C, ld, 1, m1, r1,
                                  x.const_data_ptr(), z, C, nullptr, 0, status);
  });
  const void* m2[1] = {ptr(B::kGate)};
  const int64_t r2[1] = {2 * b.inter};
  const void* m3[1] = {ptr(B::kDown)};
  launch("fox_step_product", st, [&] {
    return fox_step_product_ahead(dev, st, code, 0, 2, n, C, z, 1, ptr(B::kMlpNorm), dt(B::kMlpNorm), b.mlp_eps, 0, nullptr, 0, 1, m2, r2,
                                  nullptr, act, b.inter, m3[0], C * b.inter * 2, status);
  });
  launch("fox_step_product", st, [&] {
    return fox_step_product_ahead(dev, st, code, 2, 3, n, b.inter, act, 0, nullptr, 0, 0.f, 0, nullptr, 0, 1, m3, r1, z,
                                  out.mutable_data_ptr(), C, nullptr, 0, status);
  });
  return out;
}
}  // namespace

// block_step(self, hidden_states (B, 1, hidden), attention_mask (B, N + 1) or None, cache, layer_idx) -> out, with the token
// appended to the cache, or None where the modules' own forward has to run
FOX_PY(py_block_step) {
  HANDLE_TH_ERRORS
  Tensor x;
  Block b;
  CacheLayer c;
  const int64_t layer = PyLong_AsLongLong(args[4]);
  if (PyErr_Occurred()) throw python_error();
  if (!tensor(args[1], x) || x.dim() != 3 || x.size(1) != 1 || x.size(0) < 1 || x.size(0) > 16 || !read_block(args[0], x, b) || b.pruned ||
      b.inter % 32 || x.size(0) * (std::max(b.C, b.inter) / 8 + 12) * 16 > 200 * 1024 || !open_cache(args[3], layer, x, b, c))
    Py_RETURN_NONE;
  // (fox_step_product reads norm weights in 16-byte pieces; views of a flat buffer need not start on one.  Seen here, before
  // the first launch writes to the cache)
  for (Block::Param w : {Block::kAttnNorm, Block::kONorm, Block::kMlpNorm})
    if (reinterpret_cast<uintptr_t>(b.p[w].const_data_ptr()) % 16) Py_RETURN_NONE;
  if (at::GradMode::is_enabled()) {
    bool needs = x.requires_grad();
    for (const Tensor& t : b.p) needs = needs || (t.defined() && t.requires_grad());
    for (const Tensor* t : {&c.k, &c.v, &c.g, &c.k_state, &c.v_state}) needs = needs || t->requires_grad();
    if (needs) Py_RETURN_NONE;
  }
  if (args[2] != Py_None && !plain_tensor(args[2])) Py_RETURN_NONE;
  const Tensor mask = unpack_opt(args[2], "attention_mask");
  if (mask.defined()) {
    const auto d = mask.scalar_type();
    if (mask.dim() != 2 || mask.size(0) != x.size(0) || mask.size(1) != c.length + 1 || mask.device() != x.device() ||
        (d != at::kLong && d != at::kBool && d != at::kInt))
      Py_RETURN_NONE;
  }
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = step(b, x, mask, c);
  }
  auto set = [](const Mod& m, PyObject* name, int64_t v) {
    PyObject* n = PyLong_FromLongLong(v);
    PyDict_SetItem(m.dict, name, n);
    Py_DECREF(n);
  };
  set(c.store, s_length, c.length + 1);
  if (layer == 0) set(c.cache, s__seen_tokens, static_cast<int64_t>(c.cache.number(s__seen_tokens)) + 1);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}
