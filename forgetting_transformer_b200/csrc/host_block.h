// A FoX-Pro block as the host sees it: the parameters of the Python module tree and what may run natively.
#pragma once
#include "host_attention.h"

namespace foxh {

struct Block {
  // in the order of the autograd node's inputs (after the hidden states)
  enum Param { kAttnNorm, kQ, kK, kKMix, kV, kVMix, kOGate, kFGate, kFBias, kQNorm, kKNorm, kONorm, kO, kMlpNorm, kGate, kDown, kCount };
  Tensor p[kCount];   // kFBias may be undefined
  int64_t C = 0, H = 0, D = 0, inter = 0;
  float attn_eps = 0.f, qk_eps = 0.f, o_eps = 0.f, mlp_eps = 0.f;
  bool pruned = false;   // log_pruning_tolerance is set
};

// Reads the module tree; false where any part of it is not the plain module this code stands in for (another class, a
// hook, a patched forward of the object or its class, a tensor subclass, other dtypes or layouts, autocast, a forward-mode
// tangent) or under torch.jit.trace or a dispatch mode: the modules' own forward then runs.
bool read_block(PyObject* self, const Tensor& x, Block& b);

}  // namespace foxh
