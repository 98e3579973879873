// Fused cross-entropy loss over a (rows, classes) logit matrix, forward and backward.  HBM-bound: the forward
// reads every logit once, the backward reads it once more and writes the gradient (in place if asked to).
//
// Stands in for upstream's Triton kernels cross_entropy_fwd_kernel / cross_entropy_bwd_kernel
// (src/forgetting_transformer/model/forgetting_transformer/fused_cross_entropy.py:24-134) behind
// FusedCrossEntropyLoss, as the model's loss uses it (modeling_forgetting_transformer.py:877-884,
// inplace_backward=True, reduction='none'):
//
//   z      = logit_scale * logits[row, :]                       (fp32)
//   lse    = log sum_c exp(z_c)
//   loss   = lse - (1 - eps) z_label - eps mean_c z_c + lse_square_scale lse^2        (0 where label == ignore_index)
//   z_loss = lse_square_scale lse^2                                                    (0 where label == ignore_index)
//   dlogits_c = dloss logit_scale ( exp(z_c - lse) (1 + 2 lse_square_scale lse) - (1 - eps) [c == label] - eps / C )
//
// With the classes split over ranks (upstream lines 150-151, 196-226: every rank holds n_cols of C = world * n_cols
// classes, starting at class_start) the forward writes the rank's own lse and the part of the loss that does not
// need the global one, -(1 - eps) z_label [label on this rank] - eps sum_c z_c / C; the host joins the ranks' lse
// (log-sum-exp of an all-gather), sums the parts and adds the global lse; the backward takes the global lse.
//
// Forward: every thread runs an online (maximum, sum) pair over its 16-byte pieces of the row (and the plain sum of
// the logits when label smoothing is on); the pairs are merged through shuffles and shared memory.  Logits are fp32,
// bf16 or fp16; the row stride is in elements and the rows must be 16-byte aligned.
//
// One CTA per row.  Both kernels are bound by HBM as long as the arithmetic stays under it: a load brings 8 logits, and
// at the copy rate an SM has about 10 cycles per scheduler for each warp-wide element.  So the arithmetic is packed two
// wide, the exponential is the bare ex2 unit (results under 2^-126 are zero), the label is compared once per 16-byte
// piece, indices are 32-bit, and each thread has kCeDepth loads in flight.  Several small CTAs share an SM, so that the
// others read while one merges its sums.  The backward walks the rows from the last to the first, so that it begins with
// those the forward left in L2, and does not read a row whose gradient is zero whatever its (finite) logits are.
// 8192 x 50304 bf16, a seventh of the rows without a target: forward 220 -> 149 us (5.5 TB/s), backward 269 -> 226 us
// (6.8 TB/s).  256 threads x 4 loads at 5 CTAs per SM: 432 us for a loss step; 512 threads at 2 CTAs 472, 128 threads at 10
// 450, 2 loads at 8 CTAs 435.  Copies by cp.async into a ring that runs on across rows: 551 to 600, the ring's bookkeeping
// costs more issue slots than the loads' latency did.
#include <cooperative_groups.h>

#include <type_traits>

#include "fox_common.cuh"
#include "fox_host.h"

namespace fox {

constexpr int kCeThreads = 256;
constexpr int kCeDepth = 4;   // 16-byte loads of a thread in flight
constexpr int kCeCtas = 5;    // per SM, at least: the registers that the loads in flight need

constexpr float kCeLog2e = 1.4426950408889634f;
__device__ __forceinline__ float ce_exp(float x) { return fast_exp2(x * kCeLog2e); }
__device__ __forceinline__ float2 ce_exp(float2 x) {
  const float2 t = __fmul2_rn(x, make_float2(kCeLog2e, kCeLog2e));
  return make_float2(fast_exp2(t.x), fast_exp2(t.y));
}

template <int kDtype>   // 0 fp16, 1 bf16, 2 fp32
struct CeVec;
template <>
struct CeVec<2> {
  static constexpr int kElems = 4;
  __device__ static void unpack(uint4 v, float2* f) {
    f[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
    f[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w));
  }
  __device__ static uint4 pack(const float2* f) {
    return make_uint4(__float_as_uint(f[0].x), __float_as_uint(f[0].y), __float_as_uint(f[1].x), __float_as_uint(f[1].y));
  }
  __device__ static float load1(const void* base, int64_t i) { return reinterpret_cast<const float*>(base)[i]; }
  __device__ static void store1(void* base, int64_t i, float v) { reinterpret_cast<float*>(base)[i] = v; }
};
template <int kDtype>
struct CeVec {
  static constexpr bool kBf16 = kDtype == 1;
  static constexpr int kElems = 8;
  __device__ static void unpack(uint4 v, float2* f) {
    f[0] = unpack2<kBf16>(v.x);
    f[1] = unpack2<kBf16>(v.y);
    f[2] = unpack2<kBf16>(v.z);
    f[3] = unpack2<kBf16>(v.w);
  }
  __device__ static uint4 pack(const float2* f) {
    return make_uint4(pack2<kBf16>(f[0].x, f[0].y), pack2<kBf16>(f[1].x, f[1].y), pack2<kBf16>(f[2].x, f[2].y),
                      pack2<kBf16>(f[3].x, f[3].y));
  }
  __device__ static float load1(const void* base, int64_t i) {
    const uint32_t w = reinterpret_cast<const uint16_t*>(base)[i];
    return unpack2<kBf16>(w).x;
  }
  __device__ static void store1(void* base, int64_t i, float v) {
    reinterpret_cast<uint16_t*>(base)[i] = static_cast<uint16_t>(pack2<kBf16>(v, 0.f) & 0xffffu);
  }
};

// (m, s) <- merge of two online pairs: sum of exp(z - m)
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
  const float mn = fmaxf(m, m2);
  s = (m == -INFINITY ? 0.f : s * ce_exp(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * ce_exp(m2 - mn));
  m = mn;
}

// kTot: the plain sum of the logits is wanted (label smoothing)
template <int kDtype, bool kTot>
__global__ void __launch_bounds__(kCeThreads, kCeCtas)
fox_ce_fwd_kernel(const void* __restrict__ logits, int64_t row_stride, const int64_t* __restrict__ labels,
                  float* __restrict__ losses, float* __restrict__ z_losses, float* __restrict__ lse_out,
                  int64_t n_cols, float label_smoothing, float logit_scale, float lse_square_scale,
                  int64_t ignore_index, int64_t total_classes, int64_t class_start, int split) {
  using V = CeVec<kDtype>;
  constexpr int E = V::kElems;
  const int64_t row = blockIdx.x;
  const char* base = reinterpret_cast<const char*>(logits) + row * row_stride * (kDtype == 2 ? 4 : 2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // (read here: their latency would otherwise stand at the end of the row)
  const int64_t label = labels[row];
  const int64_t local = label - class_start;     // index among this rank's classes
  const bool mine = label != ignore_index && local >= 0 && local < n_cols;
  const float zlab = tid == 0 && mine ? V::load1(base, local) * logit_scale : 0.f;
  float m = -INFINITY, s = 0.f, tot = 0.f;
  const int n_vec = static_cast<int>(n_cols / E);
  const uint4* vec = reinterpret_cast<const uint4*>(base);
  const float2 scale2 = make_float2(logit_scale, logit_scale);
  auto pieces = [&](const uint4* raw, auto count) {   // `count` loaded pieces
    constexpr int C = decltype(count)::value;
    float2 f[C * E / 2];
    float mx = m;
#pragma unroll
    for (int d = 0; d < C; ++d) V::unpack(raw[d], f + d * (E / 2));
#pragma unroll
    for (int j = 0; j < C * E / 2; ++j) {
      f[j] = __fmul2_rn(f[j], scale2);
      mx = fmax3(mx, f[j].x, f[j].y);
      if (kTot) tot += f[j].x + f[j].y;
    }
    const float ref = mx == -INFINITY ? 0.f : mx;   // (classes masked with -inf add nothing)
    const float2 neg = make_float2(-ref, -ref);
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < C * E / 2; ++j) acc = __fadd2_rn(acc, ce_exp(__fadd2_rn(f[j], neg)));
    s = s * ce_exp(m - ref) + (acc.x + acc.y);
    m = mx;
  };
  int i = tid;
  for (; i + (kCeDepth - 1) * kCeThreads < n_vec; i += kCeDepth * kCeThreads) {
    uint4 raw[kCeDepth];
#pragma unroll
    for (int d = 0; d < kCeDepth; ++d) raw[d] = ldg_v4_here(vec + i + d * kCeThreads);
    pieces(raw, std::integral_constant<int, kCeDepth>());
  }
  for (; i < n_vec; i += kCeThreads) {
    const uint4 raw = vec[i];
    pieces(&raw, std::integral_constant<int, 1>());
  }
  for (int64_t c = static_cast<int64_t>(n_vec) * E + tid; c < n_cols; c += kCeThreads) {   // ragged end of the row
    const float z = V::load1(base, c) * logit_scale;
    if (kTot) tot += z;
    ce_merge(m, s, z, 1.f);
  }
  auto merge = [&](int width) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if (o >= width) continue;
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
      if (kTot) tot += __shfl_xor_sync(0xffffffffu, tot, o);
      ce_merge(m, s, m2, s2);
    }
  };
  merge(32);
  constexpr int kWarps = kCeThreads / 32;
  __shared__ float sm[kWarps], ss[kWarps], st[kWarps];
  if (lane == 0) { sm[warp] = m; ss[warp] = s; st[warp] = tot; }
  __syncthreads();
  if (warp == 0) {
    m = sm[lane % kWarps];
    s = ss[lane % kWarps];
    tot = st[lane % kWarps];
    merge(kWarps);
  }
  if (tid == 0) {
    const float lse = logf(s) + m;
    lse_out[row] = lse;
    const float n_all = static_cast<float>(total_classes);
    float loss = 0.f, zl = 0.f;
    if (label != ignore_index && split) {
      // the part of the loss that needs no global lse (upstream lines 84-92)
      loss = (label_smoothing > 0.f ? -label_smoothing * tot / n_all : 0.f) - (mine ? (1.f - label_smoothing) * zlab : 0.f);
    } else if (label != ignore_index) {
      if (mine) {
        loss = label_smoothing > 0.f ? lse - label_smoothing * tot / n_all - (1.f - label_smoothing) * zlab
                                     : lse - zlab;
      } else {   // a label outside the classes contributes only the smoothing term (upstream lines 74-78)
        loss = label_smoothing > 0.f ? label_smoothing * (lse - tot / n_all) : 0.f;
      }
      zl = lse_square_scale * lse * lse;
      loss += zl;
    }
    losses[row] = loss;
    if (z_losses) z_losses[row] = zl;
  }
}

template <int kDtype>
__global__ void __launch_bounds__(kCeThreads, kCeCtas)
fox_ce_bwd_kernel(const void* __restrict__ logits, int64_t row_stride, const int64_t* __restrict__ labels,
                  const float* __restrict__ lse_in, const float* __restrict__ dloss, int64_t dloss_stride,
                  void* __restrict__ dlogits, int64_t d_row_stride, int64_t n_cols, float label_smoothing,
                  float logit_scale, float lse_square_scale, int64_t ignore_index, int64_t total_classes,
                  int64_t class_start, const float* __restrict__ count) {
  using V = CeVec<kDtype>;
  constexpr int E = V::kElems;
  constexpr int kBytes = kDtype == 2 ? 4 : 2;
  const int64_t row = static_cast<int64_t>(gridDim.x) - 1 - blockIdx.x;
  const char* base = reinterpret_cast<const char*>(logits) + row * row_stride * kBytes;
  char* dbase = reinterpret_cast<char*>(dlogits) + row * d_row_stride * kBytes;
  const int tid = threadIdx.x;
  const int64_t label_all = labels[row];
  float dl_row = dloss[row * dloss_stride];   // (not behind the label's latency)
  if (count) dl_row /= *count;                // (of the mean)
  const float lse = lse_in[row];
  const int64_t label = label_all - class_start;   // index among this rank's classes (outside [0, n_cols): none)
  const float dl = (label_all != ignore_index) ? dl_row : 0.f;
  const float pscale = 1.f + 2.f * lse_square_scale * lse;
  const float g = dl * logit_scale;
  const float smooth_neg = label_smoothing / static_cast<float>(total_classes);
  const float at_label = 1.f - label_smoothing;
  const int n_vec = static_cast<int>(n_cols / E);
  uint4* dvec = reinterpret_cast<uint4*>(dbase);
  // Every element is 0 * (finite): with a finite lse no logit is NaN or +inf, and exp(z - lse) <= 1.  With any other lse
  // the products below decide (0 * NaN).
  if (g == 0.f && fabsf(lse) < INFINITY && fabsf(pscale) < INFINITY && fabsf(smooth_neg) < INFINITY) {
    for (int i = tid; i < n_vec; i += kCeThreads) dvec[i] = make_uint4(0, 0, 0, 0);
    for (int64_t c = static_cast<int64_t>(n_vec) * E + tid; c < n_cols; c += kCeThreads) V::store1(dbase, c, 0.f);
    return;
  }
  const uint4* vec = reinterpret_cast<const uint4*>(base);
  const float2 scale2 = make_float2(logit_scale, logit_scale), neg_lse = make_float2(-lse, -lse),
               pscale2 = make_float2(pscale, pscale), neg_smooth = make_float2(-smooth_neg, -smooth_neg),
               g2 = make_float2(g, g);
  const int label_vec = label >= 0 && label < n_cols ? static_cast<int>(label / E) : -1;
  const int label_elem = static_cast<int>(label % E);
  auto piece = [&](uint4 raw, int i) {
    float2 f[E / 2];
    V::unpack(raw, f);
#pragma unroll
    for (int j = 0; j < E / 2; ++j) f[j] = __fmul2_rn(ce_exp(__fadd2_rn(__fmul2_rn(f[j], scale2), neg_lse)), pscale2);
    if (i == label_vec) {
#pragma unroll
      for (int j = 0; j < E / 2; ++j) {
        if (2 * j == label_elem) f[j].x -= at_label;
        if (2 * j + 1 == label_elem) f[j].y -= at_label;
      }
    }
#pragma unroll
    for (int j = 0; j < E / 2; ++j) f[j] = __fmul2_rn(g2, __fadd2_rn(f[j], neg_smooth));
    dvec[i] = V::pack(f);
  };
  int i = tid;
  for (; i + (kCeDepth - 1) * kCeThreads < n_vec; i += kCeDepth * kCeThreads) {
    uint4 raw[kCeDepth];
    // (dlogits may be the logits' own memory: a thread reads its pieces before it writes them)
#pragma unroll
    for (int d = 0; d < kCeDepth; ++d) raw[d] = ld_v4_here(vec + i + d * kCeThreads);
#pragma unroll
    for (int d = 0; d < kCeDepth; ++d) piece(raw[d], i + d * kCeThreads);
  }
  for (; i < n_vec; i += kCeThreads) piece(ld_v4_here(vec + i), i);
  for (int64_t c = static_cast<int64_t>(n_vec) * E + tid; c < n_cols; c += kCeThreads) {
    float pr = ce_exp(V::load1(base, c) * logit_scale - lse) * pscale;
    if (c == label) pr -= at_label;
    V::store1(dbase, c, g * (pr - smooth_neg));
  }
}

// The mean of the rows' losses over the rows with a target, and their number, for the backward to divide by.  One launch in
// place of five elementwise and reduction kernels; sums in fp64, a cluster's CTAs through its shared memory.  Bound by
// latency: 1024 threads take up to 8192 rows in one trip of eight loads each, more rows are spread over a cluster of eight
// CTAs (a loss step of 8192 x 50304 bf16 413 -> 394 us; the kernels of one of 1000 x 16000 36 -> 23).
// (Begins before the losses are written: no __restrict__, which would let its loads move in front of the wait.)
constexpr int kMeanThreads = 1024, kMeanCluster = 8, kMeanRows = 8192;

__global__ void __launch_bounds__(kMeanThreads)
fox_ce_mean_kernel(const float* losses, const int64_t* labels, int64_t n_rows, int64_t ignore_index, float* mean, float* count) {
  __shared__ double s_sum[32], s_total;
  __shared__ long long s_n[32], s_rows;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double sum = 0.;
  long long n = 0;
#pragma unroll 8
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * kMeanThreads + tid; r < n_rows; r += static_cast<int64_t>(gridDim.x) * kMeanThreads) {
    sum += static_cast<double>(losses[r]);
    n += labels[r] != ignore_index;
  }
  auto reduce = [&] {
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      n += __shfl_xor_sync(0xffffffffu, n, o);
    }
  };
  reduce();
  if (lane == 0) {
    s_sum[warp] = sum;
    s_n[warp] = n;
  }
  __syncthreads();
  if (warp == 0) {
    sum = s_sum[lane];
    n = s_n[lane];
    reduce();
    if (lane == 0) {
      s_total = sum;
      s_rows = n;
    }
  }
  if (gridDim.x > 1) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    if (blockIdx.x == 0 && tid == 0) {
      for (int c = 1; c < kMeanCluster; ++c) {
        sum += *cluster.map_shared_rank(&s_total, c);
        n += *cluster.map_shared_rank(&s_rows, c);
      }
    }
    cluster.sync();   // (the others' shared memory is read until here)
  }
  if (blockIdx.x == 0 && tid == 0) {
    const float rows = static_cast<float>(n);
    *mean = static_cast<float>(sum) / rows;
    *count = rows;
  }
}

}  // namespace fox

static int ce_dtype_index(int dtype) {
  return dtype == FOX_DTYPE_FP16 ? 0 : dtype == FOX_DTYPE_BF16 ? 1 : dtype == FOX_DTYPE_FP32 ? 2 : -1;
}

static int ce_fwd_launch(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols, const void* logits,
                         int64_t row_stride, const int64_t* labels, float label_smoothing, float logit_scale,
                         float lse_square_scale, int64_t ignore_index, int64_t total_classes, int64_t class_start,
                         int split, float* losses, float* z_losses, float* lse) {
  using namespace fox;
  const int di = ce_dtype_index(dtype);
  if (!logits || !labels || !losses || (!z_losses && !split) || !lse || n_rows <= 0 || n_cols <= 0 || di < 0)
    return FOX_ERR_BAD_ARG;
  if (total_classes < n_cols || class_start < 0 || class_start + n_cols > total_classes) return FOX_ERR_BAD_ARG;
  const int bytes = di == 2 ? 4 : 2;
  if (n_rows > 2147483647LL || n_cols / (16 / bytes) > 2147483647LL / 2) return FOX_ERR_TOO_LARGE;   // (16-byte pieces are counted in 32 bits)
  if (reinterpret_cast<uintptr_t>(logits) % 16 || (row_stride * bytes) % 16 || row_stride < n_cols) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto kern = di == 0 ? (label_smoothing > 0.f ? fox_ce_fwd_kernel<0, true> : fox_ce_fwd_kernel<0, false>)
              : di == 1 ? (label_smoothing > 0.f ? fox_ce_fwd_kernel<1, true> : fox_ce_fwd_kernel<1, false>)
                        : (label_smoothing > 0.f ? fox_ce_fwd_kernel<2, true> : fox_ce_fwd_kernel<2, false>);
  kern<<<static_cast<unsigned>(n_rows), kCeThreads, 0, st>>>(logits, row_stride, labels, losses, z_losses, lse, n_cols, label_smoothing, logit_scale,
                              lse_square_scale, ignore_index, total_classes, class_start, split);
  return cudaGetLastError() == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

static int ce_bwd_launch(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols, const void* logits,
                         int64_t row_stride, const int64_t* labels, const float* lse, const float* dloss,
                         int64_t dloss_stride, float label_smoothing, float logit_scale, float lse_square_scale,
                         int64_t ignore_index, int64_t total_classes, int64_t class_start, void* dlogits,
                         int64_t dlogits_row_stride, const float* count = nullptr) {
  using namespace fox;
  const int di = ce_dtype_index(dtype);
  if (!logits || !labels || !lse || !dloss || !dlogits || n_rows <= 0 || n_cols <= 0 || di < 0) return FOX_ERR_BAD_ARG;
  if (total_classes < n_cols || class_start < 0 || class_start + n_cols > total_classes) return FOX_ERR_BAD_ARG;
  const int bytes = di == 2 ? 4 : 2;
  if (n_rows > 2147483647LL || n_cols / (16 / bytes) > 2147483647LL / 2) return FOX_ERR_TOO_LARGE;   // (16-byte pieces are counted in 32 bits)
  if (reinterpret_cast<uintptr_t>(logits) % 16 || (row_stride * bytes) % 16 || row_stride < n_cols ||
      reinterpret_cast<uintptr_t>(dlogits) % 16 || (dlogits_row_stride * bytes) % 16 || dlogits_row_stride < n_cols)
    return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto kern = di == 0 ? fox_ce_bwd_kernel<0>
              : di == 1 ? fox_ce_bwd_kernel<1>
                        : fox_ce_bwd_kernel<2>;
  kern<<<static_cast<unsigned>(n_rows), kCeThreads, 0, st>>>(logits, row_stride, labels, lse, dloss, dloss_stride, dlogits, dlogits_row_stride, n_cols,
                              label_smoothing, logit_scale, lse_square_scale, ignore_index, total_classes, class_start, count);
  return cudaGetLastError() == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

extern "C" int fox_cross_entropy_fwd(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols,
                                     const void* logits, int64_t row_stride, const int64_t* labels,
                                     float label_smoothing, float logit_scale, float lse_square_scale,
                                     int64_t ignore_index, float* losses, float* z_losses, float* lse) {
  return ce_fwd_launch(device, stream, dtype, n_rows, n_cols, logits, row_stride, labels, label_smoothing, logit_scale,
                       lse_square_scale, ignore_index, n_cols, 0, 0, losses, z_losses, lse);
}

extern "C" int fox_cross_entropy_bwd(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols,
                                     const void* logits, int64_t row_stride, const int64_t* labels, const float* lse,
                                     const float* dloss, int64_t dloss_stride, float label_smoothing,
                                     float logit_scale, float lse_square_scale, int64_t ignore_index, void* dlogits,
                                     int64_t dlogits_row_stride) {
  return ce_bwd_launch(device, stream, dtype, n_rows, n_cols, logits, row_stride, labels, lse, dloss, dloss_stride,
                       label_smoothing, logit_scale, lse_square_scale, ignore_index, n_cols, 0, dlogits,
                       dlogits_row_stride);
}

extern "C" int fox_cross_entropy_fwd_split(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols,
                                           const void* logits, int64_t row_stride, const int64_t* labels,
                                           float label_smoothing, float logit_scale, int64_t ignore_index,
                                           int64_t total_classes, int64_t class_start, float* loss_parts,
                                           float* lse_local) {
  // (the z-loss needs the global lse: the host forms it)
  return ce_fwd_launch(device, stream, dtype, n_rows, n_cols, logits, row_stride, labels, label_smoothing, logit_scale,
                       0.f, ignore_index, total_classes, class_start, 1, loss_parts, nullptr, lse_local);
}

extern "C" int fox_cross_entropy_bwd_split(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols,
                                           const void* logits, int64_t row_stride, const int64_t* labels,
                                           const float* lse_global, const float* dloss, int64_t dloss_stride,
                                           float label_smoothing, float logit_scale, float lse_square_scale,
                                           int64_t ignore_index, int64_t total_classes, int64_t class_start,
                                           void* dlogits, int64_t dlogits_row_stride) {
  return ce_bwd_launch(device, stream, dtype, n_rows, n_cols, logits, row_stride, labels, lse_global, dloss,
                       dloss_stride, label_smoothing, logit_scale, lse_square_scale, ignore_index, total_classes,
                       class_start, dlogits, dlogits_row_stride);
}

extern "C" int fox_cross_entropy_mean(int device, void* stream, int64_t n_rows, const float* losses, const int64_t* labels,
                                      int64_t ignore_index, float* mean, float* count) {
  using namespace fox;
  if (!losses || !labels || !mean || !count || n_rows <= 0) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attrs[2] = {};
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = kMeanCluster;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  const bool cluster = n_rows > kMeanRows;
  cfg.gridDim = dim3(cluster ? kMeanCluster : 1);
  cfg.blockDim = dim3(kMeanThreads);
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cfg.attrs = attrs;
  cfg.numAttrs = cluster ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, fox_ce_mean_kernel, losses, labels, n_rows, ignore_index, mean, count) == cudaSuccess
             ? FOX_OK : FOX_ERR_LAUNCH;
}

extern "C" int fox_cross_entropy_bwd_mean(int device, void* stream, int dtype, int64_t n_rows, int64_t n_cols, const void* logits,
                                          int64_t row_stride, const int64_t* labels, const float* lse, const float* dmean,
                                          const float* count, float label_smoothing, float logit_scale, float lse_square_scale,
                                          int64_t ignore_index, void* dlogits, int64_t dlogits_row_stride) {
  if (!count) return FOX_ERR_BAD_ARG;
  return ce_bwd_launch(device, stream, dtype, n_rows, n_cols, logits, row_stride, labels, lse, dmean, 0, label_smoothing,
                       logit_scale, lse_square_scale, ignore_index, n_cols, 0, dlogits, dlogits_row_stride, count);
}
