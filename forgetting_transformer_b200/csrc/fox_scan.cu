// HBM-bound helpers around the attention kernels: log-gate prefix sum with the
// seq_start masking folded in, block-pruning index scans, reverse prefix sum
// for the gate gradient, max row norms for the automatic threshold, the
// delta = rowsum(O * dO) pre-pass and the fp32 -> 16-bit dQ conversion.
//
// Upstream counterparts (src/forgetting_transformer/ops/forgetting_attention.py):
//   masked clone + torch.cumsum ............ lines 117-127
//   _find_start_index_kernel ............... lines 695-745
//   _find_end_index_kernel ................. lines 747-795
//   _bwd_preprocess ........................ lines 902-943
//   reverse cumsum of dlog_lambda .......... lines 390-392
//   vector_norm(...).max(...) .............. lines 95-96
#include <math.h>

#include <type_traits>

#include "fox_common.cuh"
#include "fox_host.h"

namespace fox {

// ------------------------------------------------------------------ block scan
constexpr int kScanThreads = 1024;
constexpr int kScanPerThread = 4;
constexpr int kScanChunk = kScanThreads * kScanPerThread;

// inclusive scan of one value per thread across the CTA; returns the inclusive
// prefix and (via total) the CTA total.  red[] holds 32 floats.
__device__ __forceinline__ float block_inclusive_scan(float v, float* red, float& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  if (lane == 31) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float w = red[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += n;
    }
    red[lane] = w;
  }
  __syncthreads();
  const float prefix = warp > 0 ? red[warp - 1] : 0.f;
  total = red[31];
  __syncthreads();
  return v + prefix;
}

// One gate value: kIn = 3 reads an fp32 log gate; kIn = 0 / 1 / 2 reads an fp16 / bf16 / fp32 gate LOGIT, of which log_gate
// returns log sigmoid(x) = min(x, 0) - log1p(exp(-|x|)) in fp32 (the F.logsigmoid(fgate_logit.float()) of
// upstream's layer, modeling_forgetting_transformer.py:343-346).
template <int kIn>
__device__ __forceinline__ float load_gate(const void* base, int64_t idx) {   // (16-bit values: their bits)
  if constexpr (kIn >= 2) return reinterpret_cast<const float*>(base)[idx];
  else return __uint_as_float(reinterpret_cast<const uint16_t*>(base)[idx]);
}
template <int kIn>
__device__ __forceinline__ float log_gate(float raw) {
  if constexpr (kIn == 3) {
    return raw;
  } else {
    float x = raw;
    if constexpr (kIn < 2) x = unpack2<kIn == 1>(__float_as_uint(raw)).x;
    return fminf(x, 0.f) - log1pf(expf(-fabsf(x)));
  }
}

// log_lambda[b,h,t] = carry_in[b,h] + sum_{u<=t, u>=seq_start[b]} log_fgate[b,h,u]
// One CTA per (b,h); chunks of 4096 elements with a carried running total.  With gate logits as input
// (kIn < 3) the log gates themselves are formed on the fly and, if lf_out is given, written out (unmasked).
// Bound by the chain of a chunk's load, scan and three barriers, 2.2 us of which the load is a third: with kAhead the next chunk's gates
// are asked for before the scan (prologue, bf16: one row of 65536 gates 35.9 -> 22.9 us, 24 rows of 11000 13.5 -> 11.3, 4 of 9000 8.7 ->
// 7.0; up to 4096, one chunk, unchanged).  From logits the chunk in hand is then formed by every thread, with gates or without; without
// kAhead a thread that has none (past the row's end, in front of seq_start) leaves the logarithms out, which is worth more up to
// eleven quarters of a chunk (24 rows of 4097 7.9 us before, 9.9 ahead, 8.2 so; 8192 10.8, 11.3, 10.3; 11000 12.8, 14.5, 13.6, with half of it
// padding 11.8, 14.7, 12.4; but 16 of 12000 17.0, 16.3, 17.0, 8 of 16384 20.0, 17.4, 18.8, one of 65536 38.1, 34.6, 37.7); from fp32 logits, whose
// loads take longer, up to seven (4 of 8192 7.6, 6.9, 8.2).  In the reverse scan, with three arrays, it takes more registers than two
// blocks of 1024 threads have, spills, and loses: 24 rows of 16384 24.0 and 24.0 us, from logits 24.5 and 28.7.
template <int kIn, bool kAhead>
__device__ __forceinline__ void cumsum_rows(const void* lf, int64_t sb, int64_t sh, int64_t sn, const int64_t* seq_start,
                                            const float* carry_in, float* out, float* total_out, float* lf_out, int H, int N, int bh, float* red) {
  const int b = bh / H, h = bh % H;
  const int64_t src0 = b * sb + h * sh;
  float* dst = out + static_cast<int64_t>(bh) * N;
  const int s0 = seq_start ? static_cast<int>(seq_start[b]) : 0;
  float carry = carry_in ? carry_in[bh] : 0.f;
  float next[kScanPerThread];
  auto load = [&](int base) {
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
      const int t = base + threadIdx.x * kScanPerThread + j;   // (may have run past 2^31)
      next[j] = 0.f;
      if (static_cast<unsigned>(t) < static_cast<unsigned>(N) && (t >= s0 || (kIn < 3 && lf_out))) next[j] = load_gate<kIn>(lf, src0 + static_cast<int64_t>(t) * sn);
    }
  };
  if (kAhead) load(0);
  for (int base = 0; base < N; base += kScanChunk) {
    const int t0 = base + threadIdx.x * kScanPerThread;
    float x[kScanPerThread];
    if (!kAhead) load(base);
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) x[j] = next[j];
    if (kAhead) load(base + kScanChunk);
    if (kIn == 3 || kAhead || (t0 < N && (t0 + kScanPerThread > s0 || lf_out))) {   // (a thread without gates has no logarithms to take)
#pragma unroll
      for (int j = 0; j < kScanPerThread; ++j) {
        const int t = t0 + j;
        const float g = log_gate<kIn>(x[j]);
        if (kIn < 3 && lf_out && t < N) lf_out[static_cast<int64_t>(bh) * N + t] = g;
        // (a log gate that was not loaded is 0 already; with the next ones in flight the choice costs nothing and without it the
        // additions wait for them: 148 rows of 16384 7.4 us, 7.9 without)
        x[j] = (kIn == 3 && !kAhead) || (t < N && t >= s0) ? g : 0.f;
      }
    }
#pragma unroll
    for (int j = 1; j < kScanPerThread; ++j) x[j] += x[j - 1];
    float total;
    const float incl = block_inclusive_scan(x[kScanPerThread - 1], red, total);
    const float excl = incl - x[kScanPerThread - 1] + carry;
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
      const int t = t0 + j;
      if (t < N) dst[t] = x[j] + excl;
    }
    carry += total;
  }
  if (total_out && threadIdx.x == 0) total_out[bh] = carry;
}

template <int kIn, bool kAhead>
__global__ void __launch_bounds__(kScanThreads, kAhead ? 0 : 2)
fox_cumsum_kernel(const void* __restrict__ lf, int64_t sb, int64_t sh, int64_t sn,
                  const int64_t* __restrict__ seq_start, const float* __restrict__ carry_in,
                  float* __restrict__ out, float* __restrict__ total_out, float* __restrict__ lf_out, int H, int N) {
  __shared__ float red[32];
  cumsum_rows<kIn, kAhead>(lf, sb, sh, sn, seq_start, carry_in, out, total_out, lf_out, H, N, blockIdx.x, red);
}

// dlog_fgate[t] = carry_in + sum_{u >= t} (dcol[u] + drow[u - P] if u >= P)
// Reverse inclusive scan, one CTA per (b,h).  kIn < 3: the chain rule through log sigmoid is applied on the way
// out, dlogit[t] = dlog_fgate[t] * sigmoid(-logit[t]), written in the logits' dtype with the logits' strides.
struct RevParams {
  const float *dcol, *drow, *carry_in;
  float *out, *total_out;
  int M, N;
  const void* logit;       // kIn < 3
  void* dlogit;
  int64_t sb, sh, sn;      // strides of logit
  int64_t osb, osh, osn;   // strides of out / dlogit
  int H;
  float* dbias;            // (B*H) or nullptr: sum of each (b,h)'s dlogit
};

template <int kIn>
__device__ __forceinline__ void revcumsum_rows(const RevParams& p, int bh, float* red) {
  const float *dcol = p.dcol, *drow = p.drow, *carry_in = p.carry_in;
  float *out = p.out, *total_out = p.total_out;
  const int M = p.M, N = p.N, H = p.H;
  const void* logit = p.logit;
  void* dlogit = p.dlogit;
  const int64_t sb = p.sb, sh = p.sh, sn = p.sn;
  const float* c = dcol + static_cast<int64_t>(bh) * N;
  const float* r = drow ? drow + static_cast<int64_t>(bh) * M : nullptr;
  const int64_t o0 = static_cast<int64_t>(bh / H) * p.osb + static_cast<int64_t>(bh % H) * p.osh;
  const int P = N - M;
  float dsum = 0.f;
  float carry = carry_in ? carry_in[bh] : 0.f;
  // walk chunks from the right; inside a chunk index i runs right-to-left
  for (int base = 0; base < N; base += kScanChunk) {
    const int i0 = base + threadIdx.x * kScanPerThread;
    float x[kScanPerThread];
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
      const int t = N - 1 - (i0 + j);
      float v = 0.f;
      if (t >= 0) {
        v = c[t];
        if (r && t >= P) v += r[t - P];
      }
      x[j] = v;
    }
#pragma unroll
    for (int j = 1; j < kScanPerThread; ++j) x[j] += x[j - 1];
    float total;
    const float incl = block_inclusive_scan(x[kScanPerThread - 1], red, total);
    const float excl = incl - x[kScanPerThread - 1] + carry;
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
      const int t = N - 1 - (i0 + j);
      if (t >= 0) {
        const float gsum = x[j] + excl;
        if constexpr (kIn == 3) {
          out[o0 + static_cast<int64_t>(t) * p.osn] = gsum;
        } else {
          const int64_t idx = static_cast<int64_t>(bh / H) * sb + static_cast<int64_t>(bh % H) * sh + static_cast<int64_t>(t) * sn;
          float xl;
          if constexpr (kIn == 2) xl = reinterpret_cast<const float*>(logit)[idx];
          else xl = unpack2<kIn == 1>(static_cast<uint32_t>(reinterpret_cast<const uint16_t*>(logit)[idx])).x;
          const float dl = gsum / (1.f + expf(xl));     // d/dx log sigmoid(x) = sigmoid(-x)
          dsum += dl;
          const int64_t odx = o0 + static_cast<int64_t>(t) * p.osn;
          if constexpr (kIn == 2) reinterpret_cast<float*>(dlogit)[odx] = dl;
          else reinterpret_cast<uint16_t*>(dlogit)[odx] = static_cast<uint16_t>(pack2<kIn == 1>(dl, 0.f) & 0xffffu);
        }
      }
    }
    carry += total;
  }
  if (total_out && threadIdx.x == 0) total_out[bh] = carry;
  if (kIn < 3 && p.dbias) {
    float total;
    (void)block_inclusive_scan(dsum, red, total);
    if (threadIdx.x == 0) p.dbias[bh] = total;
  }
}

// ------------------------------------------------------------ pruning indices
// Threshold of one (b,h): a value (kThrTensor: read from a (B,H) view), or upstream's automatic rule
// -(2 max||q|| max||k|| sm_scale + log N) - 10 evaluated step by step in the input dtype
// (src/forgetting_transformer/ops/forgetting_attention.py:91-109) from fp32 norm maxima.
enum ThresholdKind { kThrTensor = 0, kThrScalar = 1, kThrAutoFp16 = 2, kThrAutoBf16 = 3 };

template <bool kBf16>
__device__ __forceinline__ float round16(float x) {
  return unpack2<kBf16>(pack2<kBf16>(x, 0.f)).x;
}
template <bool kBf16>
__device__ __forceinline__ float auto_threshold(float qn, float kn, float sm_scale, float log_n) {
  const float bound = round16<kBf16>(round16<kBf16>(round16<kBf16>(qn) * round16<kBf16>(kn)) * sm_scale);
  const float s = round16<kBf16>(round16<kBf16>(2.f * bound) + log_n);
  return round16<kBf16>(-s - 10.f);
}

struct IndexParams {
  const float* lam;
  const float* thr;            // kThrTensor
  int64_t thr_sb, thr_sh;
  float thr_value;             // kThrScalar
  const float *q_parts, *k_parts;   // automatic: per-(b,h) partial norm maxima
  int n_q_parts, n_k_parts;
  float sm_scale, log_n;
  int kind;
  int64_t *start, *end;
  float* thr_out;              // (B,H) or nullptr: the threshold that was used
  int H, M, N, BM, BN, nmb, nnb;
};

// First index in [from, n) at which stop() holds, or n: 32 at a time by a warp, whose lanes all get it.
template <typename F>
__device__ __forceinline__ int warp_first(int from, int n, int lane, F stop) {
  for (int c0 = from; c0 < n; c0 += 32) {
    const unsigned hit = __ballot_sync(0xffffffffu, c0 + lane < n && stop(min(c0 + lane, n - 1)));
    if (hit) return c0 + __ffs(hit) - 1;
  }
  return n;
}
// Inclusive running maximum over a CTA's threads, behind `carry`; last: the maximum of all.  red: 32 ints.
__device__ __forceinline__ int block_running_max(int v, int carry, int* red, int& last) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = max(v, n);
  }
  __syncthreads();
  if (lane == 31) red[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; ++w) v = max(v, red[w]);
  v = max(v, carry);
  last = carry;
  for (int w = 0; w < warps; ++w) last = max(last, red[w]);
  return v;
}

// One CTA per (b,h).  The scans only look at log_lambda on block boundaries, so those values are staged in shared memory.
// Upstream's scans carry their position: a row's search begins where the row before it stopped, and advances while the
// condition holds.  Where the staged prefix never rises (every log gate is at most 0), neither does a row's difference to a
// later column fall, so that the condition fails from one column on and the carried scan is the running maximum of searches
// that begin at 0: a thread takes a row, by bisection.  The comparisons are the same ones on the same values, so the arrays
// are bit-identical.  A prefix that rises or is NaN somewhere, a threshold that no column of some row stops at, or few blocks go through
// the carried scan itself, 32 blocks at a time by one warp (0: start_index (B,H,ceil(M/BM)); 1: end_index (B,H,ceil(N/BN))),
// bound by its dependent steps:
// 64 (b,h) of 128 x 128 blocks take 37-40 us by the scan and 6.6 by the searches.
constexpr int kIndexThreads = 128;
constexpr int kIndexScan = 4;   // up to so many blocks the scan is shorter than the searches' barriers (2 x 2: 2.8 us against 3.7)
__global__ void __launch_bounds__(kIndexThreads)
fox_find_index_kernel(const IndexParams p) {
  extern __shared__ float sm[];
  __shared__ int red[32];
  const int nmb = p.nmb, nnb = p.nnb, M = p.M, N = p.N, BM = p.BM, BN = p.BN;
  float* row_first = sm;        // lam[P + mb*BM]            (nmb)
  float* col_last = sm + nmb;   // lam[min(N-1, nb*BN+BN-1)] (nnb)
  float* row_e = col_last + nnb;  // lam[min(mb*BM, M-1)], mb in [0, nmb]  (nmb + 1)
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* l = p.lam + static_cast<int64_t>(bh) * N;
  wait_for_kernel_in_front();
  const int P = N - M;
  for (int i = threadIdx.x; i < nmb; i += blockDim.x) row_first[i] = l[P + i * BM];
  for (int i = threadIdx.x; i < nnb; i += blockDim.x) col_last[i] = l[min(N - 1, i * BN + BN - 1)];
  for (int i = threadIdx.x; i <= nmb; i += blockDim.x) row_e[i] = l[min(min(i * BM, M), M - 1)];
  float t;
  if (p.kind == kThrTensor) {
    t = p.thr[b * p.thr_sb + h * p.thr_sh];
  } else if (p.kind == kThrScalar) {
    t = p.thr_value;
  } else {
    float qn = 0.f, kn = 0.f;
    for (int i = lane; i < p.n_q_parts; i += 32) qn = fmaxf(qn, p.q_parts[bh * p.n_q_parts + i]);
    for (int i = lane; i < p.n_k_parts; i += 32) kn = fmaxf(kn, p.k_parts[bh * p.n_k_parts + i]);
    for (int o = 16; o > 0; o >>= 1) {
      qn = fmaxf(qn, __shfl_xor_sync(0xffffffffu, qn, o));
      kn = fmaxf(kn, __shfl_xor_sync(0xffffffffu, kn, o));
    }
    t = p.kind == kThrAutoBf16 ? auto_threshold<true>(qn, kn, p.sm_scale, p.log_n)
                               : auto_threshold<false>(qn, kn, p.sm_scale, p.log_n);
  }
  if (p.thr_out && threadIdx.x == 0) p.thr_out[bh] = t;
  __syncthreads();
  int64_t* start = p.start ? p.start + static_cast<int64_t>(bh) * nmb : nullptr;
  int64_t* end = p.end ? p.end + static_cast<int64_t>(bh) * nnb : nullptr;
  bool falling = false;
  if (max(nmb, nnb) > kIndexScan) {
    falling = t == t && col_last[0] == col_last[0];
    for (int i = threadIdx.x; i + 1 < nnb; i += blockDim.x) falling = falling && col_last[i + 1] <= col_last[i];
    for (int i = threadIdx.x; i < nmb; i += blockDim.x) {
      falling = falling && row_e[i + 1] <= row_e[i] && row_first[i] == row_first[i];
      falling = falling && !(row_first[i] - col_last[nnb - 1] < t);   // (some column stops every row)
    }
    falling = __syncthreads_and(falling);
  }
  if (falling) {
    if (start) {
      int carry = 0;
      for (int m0 = 0; m0 < nmb; m0 += kIndexThreads) {
        const int mb = m0 + static_cast<int>(threadIdx.x);
        int lo = 0, hi = nnb - 1;   // the first column that stops this row
        if (mb < nmb) {
          const float x = row_first[mb];
          while (lo < hi) {
            const int c = (lo + hi) >> 1;
            if (!(x - col_last[c] < t)) hi = c;
            else lo = c + 1;
          }
        }
        const int s = block_running_max(mb < nmb ? lo : 0, carry, red, carry);
        if (mb < nmb) start[mb] = static_cast<int64_t>(s) * BN;
      }
    }
    if (end) {
      int carry = 0;
      for (int n0 = 0; n0 < nnb; n0 += kIndexThreads) {
        const int nb = n0 + static_cast<int>(threadIdx.x);
        int lo = 0, hi = nmb;       // the first row block that stops this column, or nmb
        if (nb < nnb) {
          const float x = col_last[nb];
          while (lo < hi) {
            const int c = (lo + hi) >> 1;
            if (!(row_e[c] - x >= t)) hi = c;
            else lo = c + 1;
          }
        }
        const int e = block_running_max(nb < nnb ? lo : 0, carry, red, carry);
        if (nb < nnb) end[nb] = min(e * BM, M);
      }
    }
    return;
  }
  if (warp == 0 && start) {
    int s = 0;  // in blocks of BN
    for (int mb = 0; mb < nmb; ++mb) {
      const float lo = row_first[mb];
      // upstream: while (lo - lam[min(N-1, s+BN-1)] < thr) s += BN.  Past the last block the clamped column stays
      // N-1, which is col_last[nnb-1]: a condition that still holds there holds for ever (upstream would not
      // return; here s moves on by nnb + 2 blocks past it).
      const int c = warp_first(s, nnb, lane, [&](int i) { return !(lo - col_last[i] < t); });
      if (c < nnb) s = c;
      else if (lo - col_last[nnb - 1] < t) s = s < nnb ? 2 * nnb + 1 : s + nnb + 2;
      if (lane == 0) start[mb] = static_cast<int64_t>(s) * BN;
    }
  }
  if (warp == 1 && end) {
    int eb = 0;  // row block: the row index is min(eb * BM, M)
    for (int nb = 0; nb < nnb; ++nb) {
      const float li = col_last[nb];
      if (eb < nmb) eb = warp_first(eb, nmb, lane, [&](int i) { return !(row_e[i] - li >= t); });
      if (lane == 0) end[nb] = min(eb * BM, M);
    }
  }
}

// ----------------------------------------------------------- max row L2 norm
// out[b,h] = max_t ||x[b,h,t,:]||_2 as fp32 (the caller rounds to the input dtype,
// which commutes with the max).  out must be zero-initialised; the maximum is
// taken with an integer atomicMax on the non-negative float bit pattern.
template <bool kBf16>
__global__ void __launch_bounds__(256)
fox_max_row_norm_kernel(const uint16_t* __restrict__ x, int64_t sb, int64_t sh, int64_t st, int H, int T, int D,
                        float* __restrict__ out) {
  const int lanes_per_row = D / 8;              // one 16-byte load per lane
  const int rows_per_block = 256 / lanes_per_row;
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const int sub = threadIdx.x % lanes_per_row;
  const int r_in = threadIdx.x / lanes_per_row;
  const uint16_t* base = x + b * sb + h * sh;
  float best = 0.f;
  // every lane runs the same number of iterations (the shuffles below need the full warp)
  // four rows per iteration with their loads issued first; the maximum is taken over the squared norms and the
  // square root once at the end (sqrt is monotone and correctly rounded: same result as the maximum of the roots)
  constexpr int kU = 4;
  for (int t0 = blockIdx.x * rows_per_block; t0 < T; t0 += kU * gridDim.x * rows_per_block) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * gridDim.x * rows_per_block + r_in;
      v[u] = make_uint4(0, 0, 0, 0);
      if (t < T) v[u] = *reinterpret_cast<const uint4*>(base + static_cast<int64_t>(t) * st + sub * 8);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack2<kBf16>(w[j]);
        acc = fmaf(f.x, f.x, acc);
        acc = fmaf(f.y, f.y, acc);
      }
      for (int o = lanes_per_row / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      best = fmaxf(best, acc);
    }
  }
  best = sqrtf(best);
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(out + bh), __float_as_int(best));
}

// ------------------------------------------------------ before the attention forward
// The prefix sum of the log gates and the largest key (and, for the automatic threshold, query) row norms in one
// launch: they are independent, and each alone leaves most of the chip idle (one CTA per (b,h) scans, a scan of
// 16384 gates takes 10 us).  Block 0 of a (b, h) scans; blocks 1 .. n_k (n_k+1 .. n_k+n_q) each take every n_k-th
// (n_q-th) group of rows and write ONE partial maximum, so nothing has to be zeroed first; the reader takes the
// maximum of the parts.  All blocks lie on the grid's x axis, one (b, h) behind the other: y ends at 65535, and with the
// parts on the slow axis the scans start first but the norms' reads spread over all (b, h), 1.5 % slower where they are long.
// Two blocks to an SM, at most 32 registers a thread: bf16 took 42 by itself and had one, whose loads and reductions took turns
// (keys alone, 48 (b,h) of 16384 x 64: 30.0 -> 25.0 us, 512 of 2048 x 64 43.2 -> 34.4, 32 of 2048 x 128 9.5 -> 7.2; with queries, 64 of
// 16384 x 128: 113.8 -> 101.4; 4 of 9000 x 128, whose scans are the longest, 8.4 and 8.7).
// From some 24 (b, h) on two scans then share an SM here and there, and the launch waits for them (24 of 16384 x 64 from a block's
// logits 21.3 us with one block to an SM, 29.1 with two).  With kFirst the scans are the first blocks, one to an SM: 18.5.  It is taken
// where blocks share SMs at all and each scan finds one of its own, from logits (8 (b,h) 5 % less, 12 and 16 6 %, 32 13 %; strided ones
// of 64 3 %) and from strided log gates (24 of 16384 26.8 -> 18.9, 32 8 %, 8 to 16 within 2 %); contiguous log gates lose 1 to 5 %,
// the compiler's order of their loads being a worse one there.
struct NormSource {
  const uint16_t* x;
  int64_t sb, sh, st;
  int T, n_parts;
  float* parts;   // (B*H, n_parts)
};

// max over this block's rows of the squared norm, then its root: D / 8 lanes share a row (one 16-byte load each),
// four rows per iteration with their loads issued first
template <bool kBf16>
__device__ __forceinline__ void norm_part(const NormSource& s, int D, int H, int bh, int part, float* red) {
  const int lanes_per_row = D / 8;
  const int rows_per_block = kScanThreads / lanes_per_row;
  const int sub = threadIdx.x % lanes_per_row, r_in = threadIdx.x / lanes_per_row;
  const uint16_t* base = s.x + (bh / H) * s.sb + (bh % H) * s.sh + sub * 8;
  const int stride = s.n_parts * rows_per_block;
  float best = 0.f;
  constexpr int kU = 4;
  for (int t0 = part * rows_per_block; t0 < s.T; t0 += kU * stride) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * stride + r_in;
      v[u] = make_uint4(0, 0, 0, 0);
      if (t < s.T) v[u] = *reinterpret_cast<const uint4*>(base + static_cast<int64_t>(t) * s.st);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack2<kBf16>(w[j]);
        acc = fmaf(f.x, f.x, acc);
        acc = fmaf(f.y, f.y, acc);
      }
      for (int o = lanes_per_row / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      best = fmaxf(best, acc);
    }
  }
  for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    // (sqrt is monotone and correctly rounded: same result as the maximum of the roots)
    if (threadIdx.x == 0) s.parts[static_cast<int64_t>(bh) * s.n_parts + part] = sqrtf(best);
  }
}

template <int kIn, bool kBf16, bool kAhead, bool kFirst>
__global__ void __launch_bounds__(kScanThreads, 2)
fox_prologue_kernel(const void* lf, int64_t sb, int64_t sh, int64_t sn, const int64_t* seq_start, float* lam, const NormSource k, const NormSource q, int units, int H, int N, int D) {
  __shared__ float red[32];
  if constexpr (kFirst) {
    wait_for_kernel_in_front();
    if (static_cast<int>(blockIdx.x) < units) {
      cumsum_rows<kIn, kAhead>(lf, sb, sh, sn, seq_start, nullptr, lam, nullptr, nullptr, H, N, blockIdx.x, red);
    } else {
      const int parts = k.n_parts + q.n_parts, i = blockIdx.x - units, bh = i / parts, x = i % parts;
      if (x < k.n_parts) norm_part<kBf16>(k, D, H, bh, x, red);
      else norm_part<kBf16>(q, D, H, bh, x - k.n_parts, red);
    }
  } else {
    const int parts = 1 + k.n_parts + q.n_parts, bh = blockIdx.x / parts, x = blockIdx.x % parts;
    wait_for_kernel_in_front();
    if (x == 0) cumsum_rows<kIn, kAhead>(lf, sb, sh, sn, seq_start, nullptr, lam, nullptr, nullptr, H, N, bh, red);
    else if (x <= k.n_parts) norm_part<kBf16>(k, D, H, bh, x - 1, red);
    else norm_part<kBf16>(q, D, H, bh, x - 1 - k.n_parts, red);
  }
}

// ------------------------------------------------------ delta = rowsum(O * dO)
// D / 8 lanes share a row (16 bytes each); a thread takes kDeltaRows rows a block-stride apart and issues all
// its loads before using any (two loads per thread left the kernel at a third of the copy rate).  For the one-pass
// backward the same threads clear the fp32 accumulators of their rows (acc_cols floats a row of dq_acc, dlam_row),
// which a fill kernel of its own did in front of it.
constexpr int kDeltaRows = 4;
constexpr int kAccumCols = 64;
template <bool kBf16>
__global__ void __launch_bounds__(256)
fox_delta_kernel(const uint16_t* o, int64_t o_sb, int64_t o_sh, int64_t o_st, const uint16_t* d_o, int64_t d_sb, int64_t d_sh,
                 int64_t d_st, int H, int M, int D, float* delta, float* dq_acc, int acc_cols, float* dlam_row) {
  const int lanes_per_row = D / 8;
  const int rows_per_pass = 256 / lanes_per_row;
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const int sub = threadIdx.x % lanes_per_row;
  const int row0 = blockIdx.x * rows_per_pass * kDeltaRows + threadIdx.x / lanes_per_row;
  const uint16_t* ob = o + b * o_sb + h * o_sh + sub * 8;
  const uint16_t* gb = d_o + b * d_sb + h * d_sh + sub * 8;
  uint4 a[kDeltaRows], g[kDeltaRows];
  wait_for_kernel_in_front();
#pragma unroll
  for (int i = 0; i < kDeltaRows; ++i) {
    const int row = row0 + i * rows_per_pass;
    a[i] = g[i] = make_uint4(0, 0, 0, 0);
    if (row < M) {
      a[i] = *reinterpret_cast<const uint4*>(ob + static_cast<int64_t>(row) * o_st);
      g[i] = *reinterpret_cast<const uint4*>(gb + static_cast<int64_t>(row) * d_st);
    }
  }
  if (dq_acc) {   // (under the loads) whole rows by the lanes that share one, neighbouring lanes 16 bytes apart
#pragma unroll
    for (int i = 0; i < kDeltaRows; ++i) {
      const int row = row0 + i * rows_per_pass;
      if (row < M) {
        float4* z = reinterpret_cast<float4*>(dq_acc + (static_cast<int64_t>(bh) * M + row) * acc_cols);
        for (int c = sub; c < acc_cols / 4; c += lanes_per_row) z[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (sub == 0) dlam_row[static_cast<int64_t>(bh) * M + row] = 0.f;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kDeltaRows; ++i) {
    const int row = row0 + i * rows_per_pass;
    const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 fa = unpack2<kBf16>(aw[j]), fg = unpack2<kBf16>(gw[j]);
      acc = fmaf(fa.x, fg.x, acc);
      acc = fmaf(fa.y, fg.y, acc);
    }
    for (int o2 = lanes_per_row / 2; o2 > 0; o2 >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
    if (row < M && sub == 0) delta[static_cast<int64_t>(bh) * M + row] = acc;
  }
}

// ------------------------------------------- after the attention backward
// The reverse prefix sum of the gate gradient and, for the one-pass backward, dq = (fp32 accumulator) * scale in
// 16 bits.  One launch: the first scan_blocks CTAs scan (one (b,h) each, started first because they are the long
// ones), the others convert, each thread 8 channels of kConvRows rows with its loads issued first.
struct ConvParams {
  const float* acc;       // (B,H,M,acc_cols)
  uint16_t* dq;
  int64_t sb, sh, st;
  int H, M, D, acc_cols;
  float scale;
  int blocks_per_bh, units;   // units = B * H; 0: nothing to convert
};
constexpr int kConvRows = 2;

template <bool kBf16>
__device__ __forceinline__ void convert_rows(const ConvParams& p, int block) {
  const int lanes_per_row = p.D / 8;
  const int rows_per_pass = kScanThreads / lanes_per_row;
  const int bh = block / p.blocks_per_bh, b = bh / p.H, h = bh % p.H;
  const int sub = threadIdx.x % lanes_per_row;
  const int row0 = (block % p.blocks_per_bh) * rows_per_pass * kConvRows + threadIdx.x / lanes_per_row;
  float4 a[kConvRows], c[kConvRows];
#pragma unroll
  for (int i = 0; i < kConvRows; ++i) {
    const int row = row0 + i * rows_per_pass;
    if (row < p.M) {
      const float4* src = reinterpret_cast<const float4*>(p.acc + (static_cast<int64_t>(bh) * p.M + row) * p.acc_cols + sub * 8);
      a[i] = src[0];
      c[i] = src[1];
    }
  }
#pragma unroll
  for (int i = 0; i < kConvRows; ++i) {
    const int row = row0 + i * rows_per_pass;
    if (row < p.M) {
      uint4 w;
      w.x = pack2<kBf16>(a[i].x * p.scale, a[i].y * p.scale);
      w.y = pack2<kBf16>(a[i].z * p.scale, a[i].w * p.scale);
      w.z = pack2<kBf16>(c[i].x * p.scale, c[i].y * p.scale);
      w.w = pack2<kBf16>(c[i].z * p.scale, c[i].w * p.scale);
      *reinterpret_cast<uint4*>(p.dq + b * p.sb + h * p.sh + static_cast<int64_t>(row) * p.st + sub * 8) = w;
    }
  }
}

template <int kIn, bool kBf16>
__global__ void __launch_bounds__(kScanThreads)
fox_bwd_finish_kernel(const RevParams rev, const ConvParams conv, int scan_blocks) {
  __shared__ float red[32];
  wait_for_kernel_in_front();
  if (static_cast<int>(blockIdx.x) < scan_blocks) revcumsum_rows<kIn>(rev, blockIdx.x, red);
  else convert_rows<kBf16>(conv, blockIdx.x - scan_blocks);
}

static inline bool head_dim_ok(int64_t D) { return D == 16 || D == 32 || D == 64 || D == 128; }
static inline bool aligned16(const fox_tensor4* t) {
  return t && t->ptr && reinterpret_cast<uintptr_t>(t->ptr) % 16 == 0 && (t->sb * 2) % 16 == 0 &&
         (t->sh * 2) % 16 == 0 && (t->st * 2) % 16 == 0;
}
// The prefix sums by themselves.  Loading ahead takes 38 to 41 registers, one block to an SM instead of two: log gates where the rows
// have an SM each or are so long that it pays all the same (148 rows of 4097 4.4 us without, 4.2 ahead, of 16384 9.1 and 7.4; 149 of 8192 8.1
// and 7.6, but 1024 23.6 and 26.1; 1024 of 16384 45.4 and 42.6; 512 of 100 6.0 and 8.8); logits, whose threads without gates have no
// logarithms to take without it, later and in one round of blocks only (148 of 8192 7.1 and 6.6, of 16384 12.8 and 12.1; 149 of 16384 19.9 and 21.4;
// 1024 of 4096 21.9 and 27.8).
template <int kIn>
static void launch_cumsum(cudaStream_t st, unsigned rows, const void* gates, int64_t sb, int64_t sh, int64_t sn, const int64_t* seq_start,
                          const float* carry_in, float* out, float* total_out, float* lf_out, int H, int N) {
  const bool ahead = kIn == 3 ? N > kScanChunk && (rows <= kSms || N >= 4 * kScanChunk) : rows <= kSms && N >= 3 * kScanChunk;
  (ahead ? fox_cumsum_kernel<kIn, true> : fox_cumsum_kernel<kIn, false>)<<<rows, kScanThreads, 0, st>>>(
      gates, sb, sh, sn, seq_start, carry_in, out, total_out, lf_out, H, N);
}

static inline int launch_rc() { return cudaGetLastError() == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH; }

}  // namespace fox

using namespace fox;

extern "C" const char* fox_version(void) { return "fox_b200 0.1 (sm_100a; tcgen05 + TMA)"; }

extern "C" int fox_cumsum_fwd(int device, void* stream, int64_t B, int64_t H, int64_t N, const float* log_fgate,
                              int64_t sb, int64_t sh, int64_t sn, const int64_t* seq_start,
                              const float* carry_in, float* log_lambda, float* total_out) {
  if (!log_fgate || !log_lambda || B <= 0 || H <= 0 || N <= 0) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  launch_cumsum<3>((cudaStream_t)stream, (unsigned)(B * H), log_fgate, sb, sh, sn, seq_start, carry_in, log_lambda, total_out, nullptr,
                   (int)H, (int)N);
  return launch_rc();
}

extern "C" int fox_gate_prefix_fwd(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t N,
                                   const void* fgate_logit, int64_t sb, int64_t sh, int64_t sn,
                                   const int64_t* seq_start, float* log_fgate_out, float* log_lambda) {
  if (!fgate_logit || !log_lambda || B <= 0 || H <= 0 || N <= 0) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_FP16 && dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP32) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const unsigned grid = (unsigned)(B * H);
  cudaStream_t st = (cudaStream_t)stream;
  auto launch = dtype == FOX_DTYPE_FP16 ? launch_cumsum<0> : dtype == FOX_DTYPE_BF16 ? launch_cumsum<1> : launch_cumsum<2>;
  launch(st, grid, fgate_logit, sb, sh, sn, seq_start, nullptr, log_lambda, nullptr, log_fgate_out, (int)H, (int)N);
  return launch_rc();
}

static ConvParams make_conv(int64_t B, int64_t H, int64_t M, int64_t D, const float* acc, int64_t acc_cols, float scale,
                            const fox_tensor4* dq) {
  ConvParams c{};
  c.acc = acc; c.dq = (uint16_t*)dq->ptr; c.sb = dq->sb; c.sh = dq->sh; c.st = dq->st;
  c.H = (int)H; c.M = (int)M; c.D = (int)D; c.acc_cols = (int)acc_cols; c.scale = scale;
  const int64_t rows_per_block = kConvRows * kScanThreads / (D / 8);
  c.blocks_per_bh = (int)((M + rows_per_block - 1) / rows_per_block);
  c.units = (int)(B * H);
  return c;
}

// (reverse scan and / or dQ conversion; every public entry point below ends here)
static int launch_finish(cudaStream_t st, int gate_kind, bool bf16, const RevParams& rev, int scan_blocks,
                         const ConvParams& conv) {
  const int64_t grid = scan_blocks + static_cast<int64_t>(conv.units) * conv.blocks_per_bh;
  if (grid <= 0 || grid > 2147483647LL) return FOX_ERR_TOO_LARGE;
  switch (gate_kind) {
#define FOX_FIN(K)                                                                                              \
  return launch_behind(bf16 ? fox_bwd_finish_kernel<K, true> : fox_bwd_finish_kernel<K, false>, dim3((unsigned)grid), \
                       kScanThreads, 0, st, rev, conv, scan_blocks)
    case FOX_DTYPE_FP16: FOX_FIN(0);
    case FOX_DTYPE_BF16: FOX_FIN(1);
    case FOX_DTYPE_FP32: FOX_FIN(2);
    case FOX_GATE_LOG: FOX_FIN(3);
#undef FOX_FIN
    default: return FOX_ERR_BAD_ARG;
  }
}

extern "C" int fox_revcumsum(int device, void* stream, int64_t B, int64_t H, int64_t M, int64_t N,
                             const float* dlam_col, const float* dlam_row, const float* carry_in,
                             float* dlog_fgate, float* total_out) {
  if (!dlam_col || !dlog_fgate || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const RevParams rev{dlam_col, dlam_row, carry_in, dlog_fgate, total_out, (int)M, (int)N, nullptr, nullptr, 0, 0, 0, H * N, N, 1, (int)H, nullptr};
  return launch_finish((cudaStream_t)stream, FOX_GATE_LOG, false, rev, (int)(B * H), ConvParams{});
}

extern "C" int fox_gate_prefix_bwd(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t N,
                                   const float* dlam_col, const float* dlam_row, const void* fgate_logit,
                                   int64_t sb, int64_t sh, int64_t sn, void* dfgate_logit) {
  if (!dlam_col || !fgate_logit || !dfgate_logit || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_FP16 && dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP32) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const RevParams rev{dlam_col, dlam_row, nullptr, nullptr, nullptr, (int)M, (int)N, fgate_logit, dfgate_logit, sb, sh, sn, sb, sh, sn, (int)H, nullptr};
  return launch_finish((cudaStream_t)stream, dtype, false, rev, (int)(B * H), ConvParams{});
}

extern "C" int fox_bwd_finish(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t N, int64_t D,
                              const float* dlam_col, const float* dlam_row, int gate_kind, const void* fgate_logit,
                              int64_t sb, int64_t sh, int64_t sn, void* dgate, int64_t osb, int64_t osh,
                              int64_t osn, float* dbias, const float* dq_accum, float scale, const fox_tensor4* dq) {
  if (!dlam_col || !dgate || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N) return FOX_ERR_BAD_ARG;
  if (gate_kind != FOX_GATE_LOG && !fgate_logit) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if ((dq_accum == nullptr) != (dq == nullptr)) return FOX_ERR_BAD_ARG;
  if (!head_dim_ok(D)) return FOX_ERR_HEAD_DIM;
  if (dq && (!aligned16(dq) || reinterpret_cast<uintptr_t>(dq_accum) % 16)) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const bool log_gate = gate_kind == FOX_GATE_LOG;
  const RevParams rev{dlam_col, dlam_row, nullptr, log_gate ? (float*)dgate : nullptr, nullptr, (int)M, (int)N,
                      fgate_logit, dgate, sb, sh, sn, osb, osh, osn, (int)H, dbias};
  ConvParams conv{};
  if (dq) conv = make_conv(B, H, M, D, dq_accum, D > kAccumCols ? D : kAccumCols, scale, dq);
  return launch_finish((cudaStream_t)stream, gate_kind, dtype == FOX_DTYPE_BF16, rev, (int)(B * H), conv);
}

// Parts a (b,h)'s row-norm maximum is split into: about two blocks of 1024 threads per SM over all (b,h), never more
// than the row groups there are, at most 32 (a warp of the reader takes one each).
extern "C" int64_t fox_norm_parts(int64_t B, int64_t H, int64_t T, int64_t D) {
  if (B <= 0 || H <= 0 || D < 8) return 1;   // (fox_attn_prologue refuses such a call)
  const int64_t rows_per_block = kScanThreads / (D / 8);
  int64_t n = (T + rows_per_block - 1) / rows_per_block;
  const int64_t per_unit = (kSms * 2) / (B * H) > 0 ? (kSms * 2) / (B * H) : 1;
  n = n < per_unit ? n : per_unit;
  return n < 32 ? n : 32;
}

// The same for keys alone, whose blocks share a launch with those of the prefix scans, one a (b,h).  Where fewer parts make two
// blocks per SM nearly full, that is faster than a few blocks more behind them (fp16; 24 (b,h) of 11000 x 64: 16 -> 13 us),
// unless the parts left have to be much longer: 2 -> 1 part never (148 of 4096 x 128: 42 -> 51), 3 -> 2 not with long rows in many
// (96 of 8192 x 128: 49 -> 53, of 4096 29 -> 28), and 4 -> 3 only in a fuller wave (70 of 4096 x 128, 280 blocks: 20 -> 22; 71, 284
// blocks: 22.3 -> 21.6).  Long rows of 16 or 32 channels keep theirs as well: their blocks are bound by instructions (fp16, 24 of
// 12300 x 16: 16.9 -> 23.3, 20 of 16384 x 16 a third more).
extern "C" int64_t fox_key_norm_parts(int64_t B, int64_t H, int64_t N, int64_t D) {
  if (B <= 0 || H <= 0) return 1;
  const int64_t n = fox_norm_parts(B, H, N, D), bh = B * H, places = 2 * kSms, fewer = places / bh - 1, blocks = (fewer + 1) * bh;
  if (fewer >= n) return n;
  const bool full = blocks >= places - (fewer >= 4 ? 16 : 12) && (N <= 4096 || D >= 64);
  return full && (fewer >= 3 || (fewer == 2 && (N <= 4096 || D == 64))) ? fewer : n;
}

extern "C" int fox_attn_prologue(int device, void* stream, int dtype, int gate_kind, int64_t B, int64_t H, int64_t M,
                                 int64_t N, int64_t D, const void* gates, int64_t sb, int64_t sh, int64_t sn,
                                 const int64_t* seq_start, float* log_lambda, const fox_tensor4* k, float* k_parts,
                                 int64_t n_k_parts, const fox_tensor4* q, float* q_parts, int64_t n_q_parts) {
  if (!gates || !log_lambda || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if (n_k_parts > 32767 || n_q_parts > 32767 || B * H > 2147483647LL / (1 + (k ? n_k_parts : 0) + (q ? n_q_parts : 0)))
    return FOX_ERR_TOO_LARGE;
  if (!head_dim_ok(D)) return FOX_ERR_HEAD_DIM;
  NormSource ks{}, qs{};
  if (k) {
    if (!aligned16(k)) return FOX_ERR_ALIGNMENT;
    if (!k_parts || n_k_parts <= 0) return FOX_ERR_BAD_ARG;
    ks = NormSource{(const uint16_t*)k->ptr, k->sb, k->sh, k->st, (int)N, (int)n_k_parts, k_parts};
  }
  if (q) {
    if (!aligned16(q)) return FOX_ERR_ALIGNMENT;
    if (!q_parts || n_q_parts <= 0) return FOX_ERR_BAD_ARG;
    qs = NormSource{(const uint16_t*)q->ptr, q->sb, q->sh, q->st, (int)M, (int)n_q_parts, q_parts};
  }
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const unsigned grid = (unsigned)(B * H * (1 + ks.n_parts + qs.n_parts));
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == FOX_DTYPE_BF16;
  const int64_t units = B * H, quarters = (N * 4 + kScanChunk - 1) / kScanChunk;   // (of a chunk)
  const bool first = grid > kSms && units <= kSms && (gate_kind != FOX_GATE_LOG || (sn != 1 && units > 16));
  const bool ahead = gate_kind == FOX_GATE_LOG || quarters > (gate_kind == FOX_DTYPE_FP32 ? 7 : 11);
  auto launch = [&](auto gates_in, auto ahead_c) {
    constexpr int kIn = decltype(gates_in)::value;
    constexpr bool kAhead = decltype(ahead_c)::value;
    auto kern = first ? (bf ? fox_prologue_kernel<kIn, true, kAhead, true> : fox_prologue_kernel<kIn, false, kAhead, true>)
                      : (bf ? fox_prologue_kernel<kIn, true, kAhead, false> : fox_prologue_kernel<kIn, false, kAhead, false>);
    return launch_behind(kern, dim3(grid), kScanThreads, 0, st, gates, sb, sh, sn, seq_start, log_lambda, ks, qs, (int)units, (int)H, (int)N, (int)D);
  };
  auto either = [&](auto gates_in) { return ahead ? launch(gates_in, std::true_type{}) : launch(gates_in, std::false_type{}); };
  switch (gate_kind) {
    case FOX_DTYPE_FP16: return either(std::integral_constant<int, 0>{});
    case FOX_DTYPE_BF16: return either(std::integral_constant<int, 1>{});
    case FOX_DTYPE_FP32: return either(std::integral_constant<int, 2>{});
    case FOX_GATE_LOG: return launch(std::integral_constant<int, 3>{}, std::true_type{});
    default: return FOX_ERR_BAD_ARG;
  }
}

static int launch_index(int device, cudaStream_t st, int64_t B, IndexParams p) {
  p.nmb = (p.M + p.BM - 1) / p.BM;
  p.nnb = (p.N + p.BN - 1) / p.BN;
  const size_t smem = sizeof(float) * (2 * (size_t)p.nmb + (size_t)p.nnb + 1);
  if (smem > 200 * 1024) return FOX_ERR_TOO_LARGE;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  if (smem > 48 * 1024) {
    if (cudaFuncSetAttribute(fox_find_index_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return FOX_ERR_LAUNCH;
  }
  return launch_behind(fox_find_index_kernel, dim3((unsigned)(B * p.H)), kIndexThreads, (int)smem, st, p);
}

extern "C" int fox_attn_index(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t N,
                              int64_t block_m, int64_t block_n, const float* log_lambda, float threshold,
                              const float* q_parts, int64_t n_q_parts, const float* k_parts, int64_t n_k_parts,
                              float sm_scale, int64_t* start_index, int64_t* end_index, float* threshold_out) {
  if (!log_lambda || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N || block_m <= 0 || block_n <= 0)
    return FOX_ERR_BAD_ARG;
  if ((q_parts == nullptr) != (k_parts == nullptr)) return FOX_ERR_BAD_ARG;
  if (!start_index && !end_index && !threshold_out) return FOX_OK;
  IndexParams p{};
  p.lam = log_lambda; p.start = start_index; p.end = end_index; p.thr_out = threshold_out;
  p.H = (int)H; p.M = (int)M; p.N = (int)N; p.BM = (int)block_m; p.BN = (int)block_n;
  p.kind = kThrScalar;
  p.thr_value = threshold;
  if (q_parts) {
    p.kind = dtype == FOX_DTYPE_BF16 ? kThrAutoBf16 : kThrAutoFp16;
    p.q_parts = q_parts; p.n_q_parts = (int)n_q_parts;
    p.k_parts = k_parts; p.n_k_parts = (int)n_k_parts;
    p.sm_scale = sm_scale;
    p.log_n = (float)log((double)N);
  }
  return launch_index(device, (cudaStream_t)stream, B, p);
}

extern "C" int fox_find_index(int device, void* stream, int64_t B, int64_t H, int64_t M, int64_t N,
                              int64_t block_m, int64_t block_n, const float* log_lambda, const float* threshold,
                              int64_t thr_sb, int64_t thr_sh, int64_t* start_index, int64_t* end_index) {
  if (!log_lambda || !threshold || B <= 0 || H <= 0 || N <= 0 || M <= 0 || M > N || block_m <= 0 || block_n <= 0)
    return FOX_ERR_BAD_ARG;
  if (!start_index && !end_index) return FOX_OK;
  IndexParams p{};
  p.lam = log_lambda; p.thr = threshold; p.thr_sb = thr_sb; p.thr_sh = thr_sh; p.kind = kThrTensor;
  p.start = start_index; p.end = end_index;
  p.H = (int)H; p.M = (int)M; p.N = (int)N; p.BM = (int)block_m; p.BN = (int)block_n;
  return launch_index(device, (cudaStream_t)stream, B, p);
}

extern "C" int fox_max_row_norm(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t T, int64_t D,
                                const fox_tensor4* x, float* out_zeroed) {
  if (!x || !out_zeroed || B <= 0 || H <= 0 || T <= 0) return FOX_ERR_BAD_ARG;
  if (B > 65535 || H > 65535 || B * H > 65535) return FOX_ERR_TOO_LARGE;   // (b, h) is the grid's y index
  if (!head_dim_ok(D)) return FOX_ERR_HEAD_DIM;
  if (!aligned16(x)) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const int rows_per_block = 256 / (int)(D / 8);
  // one wave of resident blocks (8 of 256 threads per SM on 148 SMs) shared among the (b, h) rows of the grid:
  // more blocks than that run as a second, partly filled wave
  int64_t gx = (T + rows_per_block - 1) / rows_per_block;
  const int64_t per_unit = (148 * 8) / (B * H) > 0 ? (148 * 8) / (B * H) : 1;
  if (gx > per_unit) gx = per_unit;
  dim3 grid((unsigned)gx, (unsigned)(B * H));
  if (dtype == FOX_DTYPE_BF16)
    fox_max_row_norm_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>((const uint16_t*)x->ptr, x->sb, x->sh, x->st, (int)H, (int)T, (int)D, out_zeroed);
  else
    fox_max_row_norm_kernel<false><<<grid, 256, 0, (cudaStream_t)stream>>>((const uint16_t*)x->ptr, x->sb, x->sh, x->st, (int)H, (int)T, (int)D, out_zeroed);
  return launch_rc();
}

static int launch_delta(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t D,
                        const fox_tensor4* o, const fox_tensor4* d_o, float* delta, float* dq_accum, float* dlam_row) {
  if (!o || !d_o || !delta || B <= 0 || H <= 0 || M <= 0) return FOX_ERR_BAD_ARG;
  if (B > 65535 || H > 65535 || B * H > 65535) return FOX_ERR_TOO_LARGE;   // (b, h) is the grid's y index
  if (!head_dim_ok(D)) return FOX_ERR_HEAD_DIM;
  if (!aligned16(o) || !aligned16(d_o) || reinterpret_cast<uintptr_t>(dq_accum) % 16) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const int rows_per_block = kDeltaRows * 256 / (int)(D / 8);
  const int acc_cols = (int)(D > kAccumCols ? D : kAccumCols);
  dim3 grid((unsigned)((M + rows_per_block - 1) / rows_per_block), (unsigned)(B * H));
  return launch_behind(dtype == FOX_DTYPE_BF16 ? fox_delta_kernel<true> : fox_delta_kernel<false>, grid, 256, 0, (cudaStream_t)stream,
                       (const uint16_t*)o->ptr, o->sb, o->sh, o->st, (const uint16_t*)d_o->ptr, d_o->sb, d_o->sh, d_o->st, (int)H,
                       (int)M, (int)D, delta, dq_accum, acc_cols, dlam_row);
}

extern "C" int fox_bwd_delta(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t D,
                             const fox_tensor4* o, const fox_tensor4* d_o, float* delta) {
  return launch_delta(device, stream, dtype, B, H, M, D, o, d_o, delta, nullptr, nullptr);
}

extern "C" int fox_bwd_prepare(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t D,
                               const fox_tensor4* o, const fox_tensor4* d_o, float* delta, float* dq_accum,
                               float* dlam_row) {
  if (!dq_accum || !dlam_row) return FOX_ERR_BAD_ARG;
  return launch_delta(device, stream, dtype, B, H, M, D, o, d_o, delta, dq_accum, dlam_row);
}

extern "C" int fox_dq_convert(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t M, int64_t D,
                              const float* dq_accum, float scale, const fox_tensor4* dq) {
  if (!dq_accum || !dq || B <= 0 || H <= 0 || M <= 0) return FOX_ERR_BAD_ARG;
  if (B > 65535 || H > 65535 || B * H > 65535) return FOX_ERR_TOO_LARGE;
  if (!head_dim_ok(D)) return FOX_ERR_HEAD_DIM;
  if (!aligned16(dq)) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  return launch_finish((cudaStream_t)stream, FOX_GATE_LOG, dtype == FOX_DTYPE_BF16, RevParams{}, 0,
                       make_conv(B, H, M, D, dq_accum, D, scale, dq));
}
