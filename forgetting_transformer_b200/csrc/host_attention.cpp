// forgetting_attention on the host: checks, allocations, launches and the autograd node.
//
// Same contract as upstream's ForgettingAttention function and forgetting_attention wrapper
// (src/forgetting_transformer/ops/forgetting_attention.py:44-455).  A forward is one launch for the prefix sum and the
// norm maxima, one for the pruning indices when a threshold is given, one for the attention; a backward is one for
// delta (and clearing the accumulators), one or two for the attention and one for the gate gradient (and dQ's
// conversion).  Working arrays come from the caching allocator in one piece per direction.
#include "host_attention.h"

#include <ATen/ExpandUtils.h>

#include <cmath>
#include <cstdlib>
#include <sstream>

namespace foxh {

namespace {
constexpr int64_t kBlock = FOX_FWD_BLOCK_M;
static_assert(FOX_FWD_BLOCK_M == FOX_BWD_BLOCK_M && FOX_FWD_BLOCK_N == FOX_BWD_BLOCK_N, "one grid for both directions");

bool env_is(const char* name, char c) {
  const char* v = std::getenv(name);
  return v && v[0] == c && v[1] == 0;
}
bool debug_sync() {
  static const bool on = env_is("FOX_B200_DEBUG_SYNC", '1');
  return on;
}
}  // namespace

bool default_two_kernel(int64_t D) {
  static const bool one_pass = env_is("FOX_B200_ONE_PASS_BWD", '1');
  return D == 128 && !one_pass;
}

// ---------------------------------------------------------------- argument checks (upstream lines 81-91)
AttnShape check_attention(const AttnInputs& in) {
  const bool hf = in.head_first;
  check_that(in.q.dim() == 4 && in.k.dim() == 4 && in.v.dim() == 4 && in.gate.dim() == 3,
             "q, k, v must have 4 dimensions and log_fgate 3");
  const int ih = hf ? 1 : 2, it = hf ? 2 : 1;
  AttnShape s{in.q.size(0), in.q.size(ih), in.q.size(it), in.k.size(it), in.q.size(3)};
  check_that(s.D == in.k.size(3) && s.D == in.v.size(3), "feature size of q, k, v should be equal");
  check_that(s.D == 16 || s.D == 32 || s.D == 64 || s.D == 128, "We only support head dims in {16, 32, 64, 128}");
  check_that(in.gate.size(0) == s.B && in.gate.size(hf ? 1 : 2) == s.H && in.gate.size(hf ? 2 : 1) == s.N);
  const auto gt = in.gate.scalar_type();
  if (in.gate_is_logit) {
    if (gt != at::kHalf && gt != at::kBFloat16 && gt != at::kFloat)
      raise_assert("gate logits must be fp16, bf16 or fp32, but got " + std::string(c10::toString(gt)));
  } else {
    check_that(gt == at::kFloat,
               "log_fgate must be in torch.float32. It is best to do this cast before logsigmoid, e.g., "
               "torch.nn.functional.logsigmoid(fgate_logit.float()).");
  }
  check_that(in.k.size(ih) == in.v.size(ih), "num of heads in k and v should be equal");
  check_that(s.H == in.k.size(ih),
             "groupped query attention has not been tested. You can uncomment this if you know what you are doing.");
  check_that(s.M <= s.N, "The key/value tensors must be longer than the query tensor");
  check_that(in.k.size(0) == s.B && in.v.size(0) == s.B && in.v.size(it) == s.N,
             "q, k, v should have equal batch sizes and k, v equal lengths");
  if (in.seq_start.defined()) check_that(in.seq_start.dim() == 1 && in.seq_start.size(0) == s.B);
  if (!in.q.is_cuda())
    raise_fox("forgetting_attention needs CUDA tensors on an sm_100 device; there is no CPU path");
  return s;
}

Threshold parse_threshold(PyObject* o) {
  Threshold t;
  if (o == Py_None) return t;
  if (PyUnicode_Check(o)) {
    const char* c = PyUnicode_AsUTF8(o);
    if (!c || std::string(c) != "auto")
      raise_assert("adaptive_threshold must be either the string \"auto\", a float, or a Tensor, but got " +
                   std::string(c ? c : "?") + ".");
    t.kind = Threshold::kAuto;
  } else if (THPVariable_Check(o)) {
    t.kind = Threshold::kTensor;
    t.tensor = THPVariable_Unpack(o);
  } else {
    t.kind = Threshold::kValue;
    t.value = PyFloat_AsDouble(o);
    if (PyErr_Occurred()) throw python_error();
  }
  return t;
}

static void gate_strides(const Tensor& g, bool hf, int64_t* st) {
  st[0] = g.stride(0);
  st[1] = g.stride(hf ? 1 : 2);
  st[2] = g.stride(hf ? 2 : 1);
}

// ---------------------------------------------------------------- launches
int64_t attn_blocks(int64_t n) { return (n + kBlock - 1) / kBlock; }

// largest key norm per (b,h): the forward kernel's bound that lets most tiles skip the row-maximum pass
AttnNorms attn_norms(const AttnShape& s, bool is_auto) {
  AttnNorms n;
  if (is_auto) {
    n.n_k = fox_norm_parts(s.B, s.H, s.N, s.D);
    n.n_q = fox_norm_parts(s.B, s.H, s.M, s.D);
  } else if (s.N >= 8 * kBlock && s.M > 1) {
    n.n_k = fox_key_norm_parts(s.B, s.H, s.N, s.D);
  }
  return n;
}

static void prepare_launch(const AttnCall& c, const AttnNorms& n, float* norms, Threshold::Kind kind, double threshold_value,
                           float* threshold, int64_t thr_sb, int64_t thr_sh) {
  const AttnShape& s = c.s;
  float* k_parts = n.n_k ? norms : nullptr;
  float* q_parts = n.n_q ? norms + c.BH() * n.n_k : nullptr;
  launch("fox_attn_prologue", c.st, [&] {
    return fox_attn_prologue(c.device, c.st, c.code, c.gate_kind, s.B, s.H, s.M, s.N, s.D, c.gate, c.gate_st[0], c.gate_st[1],
                             c.gate_st[2], c.seq_start, c.lam, n.n_k ? &c.k : nullptr, k_parts, n.n_k,
                             n.n_q ? &c.q : nullptr, q_parts, n.n_q);
  });
  if (kind == Threshold::kNone) return;
  launch("fox_find_index", c.st, [&] {
    if (kind == Threshold::kTensor)
      return fox_find_index(c.device, c.st, s.B, s.H, s.M, s.N, kBlock, kBlock, c.lam, threshold, thr_sb, thr_sh, c.start, c.end);
    return fox_attn_index(c.device, c.st, c.code, s.B, s.H, s.M, s.N, kBlock, kBlock, c.lam, static_cast<float>(threshold_value),
                          q_parts, n.n_q, q_parts ? k_parts : nullptr, n.n_k, c.sm_scale, c.start, c.end, threshold);
  });
}

void attn_forward_launch(const AttnCall& c, const AttnNorms& n, float* norms, Threshold::Kind kind, double threshold_value,
                         float* threshold, int64_t thr_sb, int64_t thr_sh) {
  prepare_launch(c, n, norms, kind, threshold_value, threshold, thr_sb, thr_sh);
  int32_t* status = status_words(c.device);
  launch("fox_attn_fwd", c.st, [&] {
    return fox_attn_fwd_parts(c.device, c.st, c.code, c.s.B, c.s.H, c.s.M, c.s.N, c.s.D, &c.q, &c.k, &c.v, c.lam, c.seq_start,
                              c.start, c.sm_scale, &c.o, c.L, n.n_k ? norms : nullptr, n.n_k, status);
  });
  if (debug_sync()) status_check(c.device);
}

// [dq accumulator (B,H,M,max(D,64)), one-pass only | delta, dlam_row (B,H,M) each | dlam_col (B,H,N)]
static int64_t accum_floats(const AttnShape& s, bool two_kernel) {
  return two_kernel ? 0 : s.B * s.H * s.M * std::max<int64_t>(s.D, 64);
}
int64_t attn_backward_floats(const AttnShape& s, bool two_kernel) {
  return accum_floats(s, two_kernel) + s.B * s.H * (2 * s.M + s.N);
}

void attn_backward_launch(const AttnCall& c, const AttnGradCall& g) {
  const AttnShape& s = c.s;
  const int64_t B = s.B, H = s.H, M = s.M, N = s.N, D = s.D, BH = B * H;
  float* dq_accum = g.work;
  float* delta = dq_accum + accum_floats(s, g.two_kernel);
  float* dlam_row = delta + BH * M;
  float* dlam_col = dlam_row + BH * M;
  const int dev = c.device;
  const cudaStream_t st = c.st;
  int32_t* status = status_words(dev);
  if (g.two_kernel) {
    // key side (dk, dv, column sums) without a dQ product, query side as its own kernel: no fp32 dQ partials to
    // add-reduce into L2, which is what bounds the one-pass kernel at head dim 128
    launch("fox_bwd_delta", st, [&] { return fox_bwd_delta(dev, st, c.code, B, H, M, D, &c.o, &g.g, delta); });
    launch("fox_attn_bwd", st, [&] {
      return fox_attn_bwd(dev, st, c.code, B, H, M, N, D, &c.q, &c.k, &c.v, &g.g, c.lam, c.L, delta, c.seq_start, c.end, c.sm_scale,
                          nullptr, nullptr, dlam_col, &g.dk, &g.dv, status);
    });
    launch("fox_attn_bwd_dq", st, [&] {
      return fox_attn_bwd_dq(dev, st, c.code, B, H, M, N, D, &c.q, &c.k, &c.v, &g.g, c.lam, c.L, delta, c.seq_start, c.start,
                             c.sm_scale, &g.dq, dlam_row, status);
    });
  } else {
    launch("fox_bwd_delta", st,
           [&] { return fox_bwd_prepare(dev, st, c.code, B, H, M, D, &c.o, &g.g, delta, dq_accum, dlam_row); });
    launch("fox_attn_bwd", st, [&] {
      return fox_attn_bwd(dev, st, c.code, B, H, M, N, D, &c.q, &c.k, &c.v, &g.g, c.lam, c.L, delta, c.seq_start, c.end, c.sm_scale,
                          dq_accum, dlam_row, dlam_col, &g.dk, &g.dv, status);
    });
  }
  // reverse prefix sum of the two halves of dlog_lambda (upstream lines 390-392); for gate logits also the chain rule
  // through log sigmoid, in the logits' dtype and layout
  launch("fox_bwd_finish", st, [&] {
    return fox_bwd_finish(dev, st, c.code, B, H, M, N, D, dlam_col, dlam_row, c.gate_kind, c.gate, c.gate_st[0], c.gate_st[1],
                          c.gate_st[2], g.dgate, g.dgate_st[0], g.dgate_st[1], g.dgate_st[2], g.dbias,
                          g.two_kernel ? nullptr : dq_accum, c.sm_scale, g.two_kernel ? nullptr : &g.dq);
  });
  if (debug_sync()) status_check(dev);
}

int64_t attn_decode_floats(const AttnShape& s) {
  return fox_attn_decode_workspace_floats(s.B, s.H, s.D, fox_attn_decode_splits(s.B, s.H, s.N));
}
void attn_decode_launch(const AttnCall& c, bool prefix, float* work, bool programmatic) {
  const AttnShape& s = c.s;
  const int64_t splits = fox_attn_decode_splits(s.B, s.H, s.N);
  launch("fox_attn_decode", c.st, [&] {
    if (prefix)
      return fox_attn_decode(c.device, c.st, c.code, s.B, s.H, s.N, s.D, &c.q, &c.k, &c.v, c.lam, c.seq_start, c.start, c.sm_scale,
                             &c.o, c.L, work, splits);
    return fox_attn_decode_gates(c.device, c.st, c.code, s.B, s.H, s.N, s.D, &c.q, &c.k, &c.v, static_cast<const float*>(c.gate),
                                 c.gate_st[0], c.gate_st[1], c.gate_st[2], c.seq_start, c.sm_scale, &c.o, c.L, work, splits,
                                 programmatic);
  });
}

// ---------------------------------------------------------------- forward
static AttnCall call_of(const AttnSaved& r, cudaStream_t st) {
  AttnCall c;
  c.device = r.q.device().index();
  c.st = st;
  c.code = dtype_code(r.q.scalar_type());
  c.s = r.shape;
  c.q = t4(r.q, r.head_first);
  c.k = t4(r.k, r.head_first);
  c.v = t4(r.v, r.head_first);
  c.o = t4(r.o, r.head_first);
  c.sm_scale = static_cast<float>(r.sm_scale);
  if (r.seq_start.defined()) c.seq_start = r.seq_start.const_data_ptr<int64_t>();
  c.lam = const_cast<float*>(r.lam());
  c.L = const_cast<float*>(r.L());
  return c;
}

AttnSaved attention_forward(const AttnInputs& in, const AttnShape& s, bool needs_grad) {
  const c10::cuda::CUDAGuard guard(in.q.device());
  const at::AutoDispatchBelowADInplaceOrView no_autograd;
  const int dev = in.q.device().index();
  const bool hf = in.head_first;
  const int64_t B = s.B, H = s.H, M = s.M, N = s.N, D = s.D, BH = B * H;
  status_poll(dev);   // did a kernel of an earlier step give up on a wait? (no synchronisation)

  AttnSaved r;
  r.shape = s;
  r.head_first = hf;
  r.gate_is_logit = in.gate_is_logit;
  r.sm_scale = in.sm_scale;
  r.set_gate_layout(in.gate.sizes(), in.gate.is_non_overlapping_and_dense() ? in.gate.strides() : at::IntArrayRef());
  r.q = tma_view(in.q);
  r.k = tma_view(in.k);
  r.v = tma_view(in.v);
  if (in.seq_start.defined()) r.seq_start = in.seq_start.to(in.q.device(), at::kLong).contiguous();
  const bool pruned = in.threshold.kind != Threshold::kNone;
  const AttnNorms norms = attn_norms(s, in.threshold.kind == Threshold::kAuto);
  // [log_lambda (B,H,N) | L (B,H,M) | norm parts]
  r.vectors = at::empty({BH * (N + M) + norms.floats(BH)}, in.q.options().dtype(at::kFloat));
  float* norm_parts = r.vectors.mutable_data_ptr<float>() + BH * (N + M);
  r.o = empty_like_tma(r.q);

  AttnCall c = call_of(r, c10::cuda::getCurrentCUDAStream(dev).stream());
  c.gate = in.gate.data_ptr();
  gate_strides(in.gate, hf, c.gate_st);
  if (in.gate_is_logit) c.gate_kind = dtype_code(in.gate.scalar_type());
  if (pruned) {
    r.index = at::empty({BH * (attn_blocks(M) + (needs_grad ? attn_blocks(N) : 0))}, in.q.options().dtype(at::kLong));
    c.start = r.index.mutable_data_ptr<int64_t>();
    c.end = needs_grad ? c.start + BH * attn_blocks(M) : nullptr;
    if (in.threshold.kind == Threshold::kTensor) {
      r.threshold = in.threshold.tensor.to(in.q.device(), at::kFloat);
      if (!at::is_expandable_to(r.threshold.sizes(), {B, H})) {
        std::ostringstream os;
        os << r.threshold.sizes();
        throw std::runtime_error(
            "adaptive_threshold must be either the string \"auto\" or broadcastable to (batch_size, num_heads) = (" +
            std::to_string(B) + ", " + std::to_string(H) + "), but got torch.Size(" + os.str() + ").");
      }
    } else {
      r.threshold = at::empty({B, H}, in.q.options().dtype(at::kFloat));
    }
  }
  const Tensor thr_bh = pruned ? r.threshold.expand({B, H}) : Tensor();
  float* thr = pruned ? static_cast<float*>(thr_bh.data_ptr()) : nullptr;
  const int64_t thr_sb = pruned ? thr_bh.stride(0) : 0, thr_sh = pruned ? thr_bh.stride(1) : 0;
  if (M == 1 && !needs_grad) {
    // generation step: one query row against the cache, no gradients -> split-KV kernels.  Only a threshold's index scan
    // (or gate logits) needs the prefix sum; otherwise the decode kernel works from the gates.
    const bool prefix = pruned || in.gate_is_logit;
    if (prefix) prepare_launch(c, norms, norm_parts, in.threshold.kind, in.threshold.value, thr, thr_sb, thr_sh);
    const Tensor work = at::empty({attn_decode_floats(s)}, r.q.options().dtype(at::kFloat));
    attn_decode_launch(c, prefix, work.mutable_data_ptr<float>(), false);
    return r;
  }
  attn_forward_launch(c, norms, norm_parts, in.threshold.kind, in.threshold.value, thr, thr_sb, thr_sh);
  return r;
}

// ---------------------------------------------------------------- backward
AttnGrads attention_backward(const AttnSaved& r, const Tensor& d_o, bool two_kernel) {
  const c10::cuda::CUDAGuard guard(r.q.device());
  const at::AutoDispatchBelowADInplaceOrView no_autograd;
  const int dev = r.q.device().index();
  const bool hf = r.head_first;
  const Tensor grad = tma_view(d_o);
  AttnCall c = call_of(r, c10::cuda::getCurrentCUDAStream(dev).stream());
  const int64_t nmb = attn_blocks(c.s.M), nnb = attn_blocks(c.s.N);

  Tensor index = r.index;
  if (r.threshold.defined()) {
    const bool have = index.defined() && index.numel() == c.BH() * (nmb + nnb);
    if (!have) index = at::empty({c.BH() * (nmb + nnb)}, r.q.options().dtype(at::kLong));
    c.start = index.mutable_data_ptr<int64_t>();
    c.end = c.start + c.BH() * nmb;
    if (!have) {
      const Tensor thr = r.threshold.expand({c.s.B, c.s.H});
      launch("fox_find_index", c.st, [&] {
        return fox_find_index(dev, c.st, c.s.B, c.s.H, c.s.M, c.s.N, kBlock, kBlock, c.lam, thr.const_data_ptr<float>(), thr.stride(0),
                              thr.stride(1), c.start, c.end);
      });
    }
  }
  AttnGrads out;
  out.dq = empty_like_tma(r.q);
  out.dk = empty_like_tma(r.k);
  out.dv = empty_like_tma(r.v);
  AttnGradCall g;
  g.two_kernel = two_kernel && c.s.D >= 64;
  const Tensor work = at::empty({attn_backward_floats(c.s, g.two_kernel)}, r.q.options().dtype(at::kFloat));
  g.work = work.mutable_data_ptr<float>();
  g.g = t4(grad, hf);
  g.dq = t4(out.dq, hf);
  g.dk = t4(out.dk, hf);
  g.dv = t4(out.dv, hf);
  if (r.gate_is_logit) {
    c.gate_kind = dtype_code(r.gate.scalar_type());
    c.gate = r.gate.data_ptr();
    gate_strides(r.gate, hf, c.gate_st);
    out.dgate = at::empty_like(r.gate);
  } else {   // in the gates' own layout, which the gradient's accumulation would otherwise copy it into
    out.dgate = at::empty_strided(r.gate_sizes, r.gate_strides, r.q.options().dtype(at::kFloat));
  }
  g.dgate = out.dgate.data_ptr();
  gate_strides(out.dgate, hf, g.dgate_st);
  attn_backward_launch(c, g);
  return out;
}

// ---------------------------------------------------------------- autograd node
namespace {
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct AttentionBackward : public torch::autograd::Node {
  // Everything with memory goes through saved variables: they check that nothing was written to in between (a caller's
  // seq_start or threshold is used as it is where its type allows) and pass the hooks that move or drop saved tensors.
  // gate: the logits, where they are what was given.
  SavedVariable q, k, v, o, gate, seq_start, vectors, threshold, index;
  AttnSaved rest;   // (its tensors are left empty)
  bool released = false;

  std::string name() const override { return "ForgettingAttentionBackward"; }
  void release_variables() override {
    for (SavedVariable* s : {&q, &k, &v, &o, &gate, &seq_start, &vectors, &threshold, &index}) s->reset_data();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(4);
    if (!grads[0].defined()) return out;
    if (released) throw std::runtime_error(torch::autograd::ERR_BACKWARD_TWICE);
    AttnSaved r = rest;
    r.q = q.unpack();
    r.k = k.unpack();
    r.v = v.unpack();
    r.o = o.unpack(shared_from_this());
    if (r.gate_is_logit) r.gate = gate.unpack();
    r.seq_start = seq_start.unpack();
    r.vectors = vectors.unpack();
    r.threshold = threshold.unpack();
    r.index = index.unpack();
    AttnGrads g = attention_backward(r, grads[0], default_two_kernel(r.shape.D));
    if (task_should_compute_output(0)) out[0] = g.dq;
    if (task_should_compute_output(1)) out[1] = g.dk;
    if (task_should_compute_output(2)) out[2] = g.dv;
    if (task_should_compute_output(3)) out[3] = g.dgate;
    return out;
  }
};
}  // namespace

Tensor attention(const AttnInputs& in) {
  const AttnShape s = check_attention(in);
  const bool needs = at::GradMode::is_enabled() && (in.q.requires_grad() || in.k.requires_grad() || in.v.requires_grad() ||
                                                    in.gate.requires_grad());
  AttnSaved r = attention_forward(in, s, needs);
  if (!needs) return r.o;
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(in.q, in.k, in.v, in.gate));
  Tensor o = r.o;
  torch::autograd::set_history(o, node);
  node->q = SavedVariable(r.q, false);
  node->k = SavedVariable(r.k, false);
  node->v = SavedVariable(r.v, false);
  node->o = SavedVariable(o, true);
  if (in.gate_is_logit) node->gate = SavedVariable(in.gate, false);
  node->seq_start = SavedVariable(r.seq_start, false);
  node->vectors = SavedVariable(r.vectors, false);
  node->threshold = SavedVariable(r.threshold, false);
  node->index = SavedVariable(r.index, false);
  for (Tensor* t : {&r.q, &r.k, &r.v, &r.o, &r.seq_start, &r.vectors, &r.threshold, &r.index}) t->reset();
  node->rest = std::move(r);
  return o;
}

}  // namespace foxh

// ---------------------------------------------------------------- Python entry points
using namespace foxh;

static AttnInputs parse_inputs(PyObject* const* a) {   // q, k, v, gate, head_first, seq_start, sm_scale, threshold, gate_is_logit
  AttnInputs in;
  in.q = unpack(a[0], "q");
  in.k = unpack(a[1], "k");
  in.v = unpack(a[2], "v");
  in.gate = unpack(a[3], "log_fgate");
  in.head_first = PyObject_IsTrue(a[4]) == 1;
  in.seq_start = unpack_opt(a[5], "seq_start");
  in.threshold = parse_threshold(a[7]);
  in.gate_is_logit = a[8] == Py_True;
  if (a[6] == Py_None) {
    in.sm_scale = 1. / std::sqrt(static_cast<double>(in.q.size(-1)));
  } else {
    in.sm_scale = PyFloat_AsDouble(a[6]);
    if (PyErr_Occurred()) throw python_error();
  }
  return in;
}

// the nine arguments -> out, or None where the autograd function has to be called
FOX_PY(py_attention) {
  HANDLE_TH_ERRORS
  if (tracing()) Py_RETURN_NONE;
  for (int i = 0; i < 4; ++i)
    if (THPVariable_Check(args[i]) && !plain_tensor(args[i])) Py_RETURN_NONE;
  const AttnInputs in = parse_inputs(args);
  for (const Tensor* t : {&in.q, &in.k, &in.v, &in.gate, &in.seq_start, &in.threshold.tensor})
    if (has_tangent(*t)) Py_RETURN_NONE;
  Tensor out;
  {
    pybind11::gil_scoped_release no_gil;
    out = attention(in);
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

static PyObject* tensor_tuple(std::initializer_list<const Tensor*> ts) {   // (an undefined tensor becomes None)
  PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
  Py_ssize_t i = 0;
  for (const Tensor* t : ts) PyTuple_SET_ITEM(out, i++, THPVariable_Wrap(*t));
  return out;
}

// (the nine arguments of attention, needs_grad) -> (out, L, log_lambda, seq_start, threshold, start_index, end_index)
FOX_PY(py_attention_forward) {
  HANDLE_TH_ERRORS
  const AttnInputs in = parse_inputs(args);
  const bool needs = args[9] == Py_True;
  AttnSaved r;
  Tensor L, lam, start, end;
  {
    pybind11::gil_scoped_release no_gil;
    const AttnShape s = check_attention(in);
    r = attention_forward(in, s, needs);
    const int64_t BH = s.B * s.H, nmb = (s.M + kBlock - 1) / kBlock, nnb = (s.N + kBlock - 1) / kBlock;
    lam = r.vectors.narrow(0, 0, BH * s.N).view({s.B, s.H, s.N});
    L = r.vectors.narrow(0, BH * s.N, BH * s.M).view({s.B, s.H, s.M});
    if (r.index.defined()) {
      start = r.index.narrow(0, 0, BH * nmb).view({s.B, s.H, nmb});
      if (needs) end = r.index.narrow(0, BH * nmb, BH * nnb).view({s.B, s.H, nnb});
    }
  }
  return tensor_tuple({&r.o, &L, &lam, &r.seq_start, &r.threshold, &start, &end});
  END_HANDLE_TH_ERRORS
}

// head-first (q, k, v, out, L, log_lambda, seq_start, threshold, dout, gate logits or None, sm_scale, two_kernel)
// -> (dq, dk, dv, dgate)
FOX_PY(py_attention_backward) {
  HANDLE_TH_ERRORS
  AttnSaved r;
  r.q = tma_view(unpack(args[0], "q"));
  r.k = tma_view(unpack(args[1], "k"));
  r.v = tma_view(unpack(args[2], "v"));
  r.o = tma_view(unpack(args[3], "out"));
  r.head_first = true;
  r.shape = AttnShape{r.q.size(0), r.q.size(1), r.q.size(2), r.k.size(2), r.q.size(3)};
  r.set_gate_layout({r.shape.B, r.shape.H, r.shape.N}, {});
  r.separate_L = unpack(args[4], "L").contiguous();
  r.separate_lam = unpack(args[5], "log_lambda").contiguous();
  r.seq_start = unpack_opt(args[6], "seq_start");
  r.threshold = unpack_opt(args[7], "threshold");
  const Tensor d_o = unpack(args[8], "dout");
  r.gate = unpack_opt(args[9], "gate logits");
  r.gate_is_logit = r.gate.defined();
  r.sm_scale = PyFloat_AsDouble(args[10]);
  const bool two_kernel = args[11] == Py_True;
  AttnGrads g;
  {
    pybind11::gil_scoped_release no_gil;
    g = attention_backward(r, d_o, two_kernel);
  }
  return tensor_tuple({&g.dq, &g.dk, &g.dv, &g.dgate});
  END_HANDLE_TH_ERRORS
}
