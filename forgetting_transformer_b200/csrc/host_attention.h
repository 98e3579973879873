// Attention on the host: what a call gets, what its forward keeps, what its backward returns.
#pragma once
#include "host_common.h"

#include <array>

namespace foxh {

struct Threshold {
  enum Kind { kNone, kValue, kTensor, kAuto } kind = kNone;
  double value = 0.;
  Tensor tensor;
};

struct AttnInputs {
  Tensor q, k, v, gate, seq_start;
  bool head_first = true, gate_is_logit = false;
  double sm_scale = 0.;
  Threshold threshold;
};

struct AttnShape {
  int64_t B = 0, H = 0, M = 0, N = 0, D = 0;
};

struct AttnSaved {
  AttnShape shape;
  bool head_first = true, gate_is_logit = false;
  double sm_scale = 0.;
  Tensor q, k, v, o, gate, seq_start;
  Tensor vectors;                    // [log_lambda (B,H,N) | L (B,H,M) | norm parts]
  Tensor threshold;                  // fp32, expands to (B,H), with a threshold (a caller's tensor as it is where it can be)
  Tensor index;                      // [start (B,H,ceil(M/128)) | end (B,H,ceil(N/128)), with gradients], with a threshold
  Tensor separate_lam, separate_L;   // instead of `vectors`, where the caller holds the two as tensors

  std::array<int64_t, 3> gate_sizes{}, gate_strides{};   // of the gate gradient

  void set_gate_layout(at::IntArrayRef sizes, at::IntArrayRef strides) {   // no strides: contiguous
    for (int i = 0; i < 3; ++i) gate_sizes[i] = sizes[i];
    gate_strides = {gate_sizes[1] * gate_sizes[2], gate_sizes[2], 1};
    for (size_t i = 0; i < strides.size(); ++i) gate_strides[i] = strides[i];
  }
  const float* lam() const {
    return vectors.defined() ? vectors.const_data_ptr<float>() : separate_lam.const_data_ptr<float>();
  }
  const float* L() const {
    return vectors.defined() ? vectors.const_data_ptr<float>() + shape.B * shape.H * shape.N
                             : separate_L.const_data_ptr<float>();
  }
};

// One call of the kernels on raw device pointers; every array is the caller's.
struct AttnCall {
  int device = 0, code = 0;          // FOX_DTYPE_* of q, k, v
  cudaStream_t st = nullptr;
  AttnShape s;
  fox_tensor4 q, k, v, o;
  float sm_scale = 0.f;
  const int64_t* seq_start = nullptr;
  int gate_kind = FOX_GATE_LOG;      // or the dtype of gate logits
  const void* gate = nullptr;
  int64_t gate_st[3] = {0, 0, 0};    // b, h, t strides
  float *lam = nullptr, *L = nullptr;              // (B,H,N), (B,H,M)
  int64_t *start = nullptr, *end = nullptr;        // with a threshold (end: with gradients)

  int64_t BH() const { return s.B * s.H; }
};
struct AttnNorms {   // parts of the row-norm maxima a forward needs: n_k, n_q floats per (b,h)
  int64_t n_k = 0, n_q = 0;
  int64_t floats(int64_t BH) const { return BH * (n_k + n_q); }
};
AttnNorms attn_norms(const AttnShape& s, bool is_auto);
int64_t attn_blocks(int64_t n);   // tiles of the pruning grid

// norms: attn_norms().floats() floats.  threshold: where kind is not kNone; its (B,H) values for a tensor, or the place
// that receives them.
void attn_forward_launch(const AttnCall& c, const AttnNorms& n, float* norms, Threshold::Kind kind, double threshold_value,
                         float* threshold, int64_t thr_sb, int64_t thr_sh);
// one query row without gradients; prefix: c.lam (and c.start) have been formed, else the log gates c.gate are used
int64_t attn_decode_floats(const AttnShape& s);
void attn_decode_launch(const AttnCall& c, bool prefix, float* work, bool programmatic);
struct AttnGradCall {
  fox_tensor4 g, dq, dk, dv;         // dout and the gradients
  float* work = nullptr;             // attn_backward_floats()
  void* dgate = nullptr;
  int64_t dgate_st[3] = {0, 0, 0};
  float* dbias = nullptr;            // (B*H) or nullptr
  bool two_kernel = false;
};
int64_t attn_backward_floats(const AttnShape& s, bool two_kernel);
void attn_backward_launch(const AttnCall& c, const AttnGradCall& g);

struct AttnGrads {
  Tensor dq, dk, dv, dgate;
};

AttnShape check_attention(const AttnInputs& in);
Threshold parse_threshold(PyObject* o);
bool default_two_kernel(int64_t D);
AttnSaved attention_forward(const AttnInputs& in, const AttnShape& s, bool needs_grad);
AttnGrads attention_backward(const AttnSaved& r, const Tensor& d_o, bool two_kernel);
Tensor attention(const AttnInputs& in);   // with its autograd node where gradients are needed

}  // namespace foxh
