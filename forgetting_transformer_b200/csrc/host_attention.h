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
  Tensor threshold;                  // (B,H) fp32 view, with a threshold
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
