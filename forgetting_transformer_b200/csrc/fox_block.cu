// Kernels between the matrix products of a FoX-Pro block's training step, with the operators that touch the same rows
// fused: the projections q, k, v, output gate and the narrow ones (forget gate, shift mixing weights) of all heads come
// out of ONE product whose rows are [q | k | v | ogate | fgate | k mix | v mix | pad], and go back into one.
//
// Stands in for what upstream's layer does with separate operators
// (src/forgetting_transformer/model/forgetting_transformer/modeling_forgetting_transformer.py:44-95, 296-346): the
// token shift of k and v (token_shift.py:21-158), the per-head RMSNorm of q and k (layernorm.py:183-245, 328-423).
//
//   k' = a_k k[t-1] + (1 - a_k) k[t],  a_k = sigmoid(k mix);   v' likewise
//   q_n = q rstd(q) w_q;   k_n = k' rstd(k') w_k               (per head)
//
// All are bound by HBM: every row is read once and written once.  Thread = 8 channels of one head (16-byte accesses),
// a CTA walks consecutive tokens so that the previous (forward) or next (backward) token's row is the one it has just
// had in registers, and a head's reduction is a shuffle over D / 8 lanes.
#include "fox_common.cuh"
#include "fox_host.h"

namespace fox {

template <bool kBf16>
__device__ __forceinline__ void blk_unpack(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = unpack2<kBf16>(w[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
template <bool kBf16>
__device__ __forceinline__ uint4 blk_pack(const float* f) {
  return make_uint4(pack2<kBf16>(f[0], f[1]), pack2<kBf16>(f[2], f[3]), pack2<kBf16>(f[4], f[5]), pack2<kBf16>(f[6], f[7]));
}
template <bool kBf16>
__device__ __forceinline__ float blk_load1(const uint16_t* p) {
  return unpack2<kBf16>(static_cast<uint32_t>(*p)).x;
}
// The two mixing weights of a head: its even lanes hold the logit of k's, the odd ones of v's, each warp forms both with one
// sigmoid and hands them round.
__device__ __forceinline__ float2 blk_mix_weights(float logit, int lanes) {
  const float w = sigmoid_fp32(logit);
  const int lane0 = (threadIdx.x & 31) & ~(lanes - 1);
  return make_float2(__shfl_sync(0xffffffffu, w, lane0), __shfl_sync(0xffffffffu, w, lane0 + 1));
}
__device__ __forceinline__ float head_sum(float x, int lanes) {
  for (int o = lanes >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

constexpr int kMixThreads = 256;   // rows of up to 2048 channels

struct MixParams {
  const uint16_t* y;      // (tokens, ld): [q | k | v | ogate | fgate | k mix | v mix | pad]
  int64_t ld;
  const float *wq, *wk;   // (C)
  const int64_t* mask;    // (tokens) or nullptr: 0 = padding, whose k and v rows count as zero
  float *rstd_q, *rstd_k; // (tokens, H)
  uint16_t *q, *k, *v;    // (tokens, C)
  int64_t* seq_start;     // (B) or nullptr: receives T - sum of the sequence's mask (left padding)
  int mix_blocks;         // CTAs that take tokens; the ones after them count a sequence's mask each
  float eps;
  int H, D, T, rows;      // rows: tokens a CTA takes
  int64_t tokens;
};

// k, v rows of one token (zero where masked or out of range)
__device__ __forceinline__ void mix_load(const MixParams& p, int64_t t, bool on, int ch, int C, uint4& k, uint4& v) {
  k = v = make_uint4(0, 0, 0, 0);
  if (on && (!p.mask || p.mask[t] != 0)) {
    k = *reinterpret_cast<const uint4*>(p.y + t * p.ld + C + ch);
    v = *reinterpret_cast<const uint4*>(p.y + t * p.ld + 2 * C + ch);
  }
}

// One CTA of 192 threads per 3 tokens' loads in flight is too little to cover the chain load - sum over a head's lanes -
// store, so it takes one token at a time in 64 registers and has 5 CTAs per SM, where two tokens in 116 registers left 2: 16384 x 1536 bf16 96 -> 71.5 us (4.2 TB/s), 2048 x 768 7.5 ->
// 7.3 us.  (Two tokens in 80 registers: 67 and 8.1 us; one in 48 registers: 91 and 9.5 us; 4 channels a thread, which doubles
// the instructions for addresses and sums: 199 and 13 us.)
template <bool kBf16>
__global__ void __launch_bounds__(kMixThreads, 4) fox_mix_fwd_kernel(const MixParams p) {
  if (static_cast<int>(blockIdx.x) >= p.mix_blocks) {
    __shared__ unsigned long long s_sum;
    const int b = blockIdx.x - p.mix_blocks;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    long long n = 0;
    for (int t = threadIdx.x; t < p.T; t += blockDim.x) n += p.mask[static_cast<int64_t>(b) * p.T + t];
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, static_cast<unsigned long long>(n));
    __syncthreads();
    if (threadIdx.x == 0) p.seq_start[b] = p.T - static_cast<int64_t>(s_sum);
    return;
  }
  const int lanes = p.D >> 3, C = p.H * p.D;
  const int h = threadIdx.x / lanes, sub = threadIdx.x % lanes;
  const bool active = h < p.H;
  const int ch = active ? h * p.D + sub * 8 : 0;
  const float inv_d = 1.f / static_cast<float>(p.D);
  float wq[8], wk[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    wq[j] = active ? p.wq[ch + j] : 0.f;
    wk[j] = active ? p.wk[ch + j] : 0.f;
  }
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * p.rows, t1 = min(t0 + p.rows, p.tokens);
  uint4 kp, vp;
  int pos = static_cast<int>(t0 % p.T);   // of the token in its sequence
  mix_load(p, t0 - 1, active && pos != 0, ch, C, kp, vp);
  for (int64_t t = t0; t < t1; ++t) {
    uint4 qr = make_uint4(0, 0, 0, 0), kr, vr;
    float mix = 0.f;
    mix_load(p, t, active, ch, C, kr, vr);
    if (active) {
      const uint16_t* row = p.y + t * p.ld;
      qr = *reinterpret_cast<const uint4*>(row + ch);
      mix = blk_load1<kBf16>(row + 4 * C + (1 + (sub & 1)) * p.H + h);
    }
    const bool first = pos == 0;   // no token before it
    pos = pos + 1 == p.T ? 0 : pos + 1;
    float q[8], k[8], v[8], kq[8], vq[8];
    blk_unpack<kBf16>(qr, q);
    blk_unpack<kBf16>(kr, k);
    blk_unpack<kBf16>(vr, v);
    blk_unpack<kBf16>(kp, kq);
    blk_unpack<kBf16>(vp, vq);
    const float2 w = blk_mix_weights(mix, lanes);
    const float a = w.x, c = w.y;
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      k[j] = k[j] * (1.f - a) + (first ? 0.f : kq[j] * a);
      v[j] = v[j] * (1.f - c) + (first ? 0.f : vq[j] * c);
      sq = fmaf(q[j], q[j], sq);
      sk = fmaf(k[j], k[j], sk);
    }
    const float rq = rsqrtf(head_sum(sq, lanes) * inv_d + p.eps), rk = rsqrtf(head_sum(sk, lanes) * inv_d + p.eps);
    if (active) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        q[j] *= rq * wq[j];
        k[j] *= rk * wk[j];
      }
      const int64_t o = t * C + ch;
      *reinterpret_cast<uint4*>(p.q + o) = blk_pack<kBf16>(q);
      *reinterpret_cast<uint4*>(p.k + o) = blk_pack<kBf16>(k);
      *reinterpret_cast<uint4*>(p.v + o) = blk_pack<kBf16>(v);
      if (sub == 0 && p.rstd_q) {
        p.rstd_q[t * p.H + h] = rq;
        p.rstd_k[t * p.H + h] = rk;
      }
    }
    kp = kr;
    vp = vr;
  }
}

struct MixBwdParams {
  MixParams f;                       // y, ld, weights, mask, rstd, sizes
  const uint16_t *dq, *dk, *dv;      // (tokens, C)
  uint16_t* dy;                      // (tokens, ld): writes q, k, v, k mix, v mix and the pad columns
  float *dwq, *dwk;                  // (gridDim.x, C) partials
  int pad0, pad1;                    // pad columns of dy
};

struct MixRow {
  uint4 q, dq, dk, dv;   // of token t
  uint4 kp, vp;          // k, v of token t - 1
  float mix, rq, rk;
};

template <bool kBf16>
__device__ __forceinline__ void mix_bwd_load(const MixBwdParams& p, int64_t t, bool on, int ch, int C, int h, int sub, MixRow& r) {
  r.q = r.dq = r.dk = r.dv = make_uint4(0, 0, 0, 0);
  r.mix = r.rq = r.rk = 0.f;
  mix_load(p.f, t - 1, on && t > 0, ch, C, r.kp, r.vp);
  if (on) {
    const uint16_t* row = p.f.y + t * p.f.ld;
    const int64_t o = t * C + ch;
    r.q = *reinterpret_cast<const uint4*>(row + ch);
    r.dq = *reinterpret_cast<const uint4*>(p.dq + o);
    r.dk = *reinterpret_cast<const uint4*>(p.dk + o);
    r.dv = *reinterpret_cast<const uint4*>(p.dv + o);
    r.mix = blk_load1<kBf16>(row + 4 * C + (1 + (sub & 1)) * p.f.H + h);
    r.rq = p.f.rstd_q[t * p.f.H + h];
    r.rk = p.f.rstd_k[t * p.f.H + h];
  }
}

// Tokens are walked backwards: the gradient of k[t] is (1 - a[t]) dk'[t] + a[t+1] dk'[t+1], the second term carried from
// the token before in this order.  A CTA first forms the token after its range for that carry (1 / rows more reads).
// The next token's rows are fetched before the current one is worked on.
template <bool kBf16>
__global__ void __launch_bounds__(kMixThreads, 2) fox_mix_bwd_kernel(const MixBwdParams p) {
  const MixParams& f = p.f;
  const int lanes = f.D >> 3, C = f.H * f.D;
  const int h = threadIdx.x / lanes, sub = threadIdx.x % lanes;
  const bool active = h < f.H;
  const int ch = active ? h * f.D + sub * 8 : 0;
  const float inv_d = 1.f / static_cast<float>(f.D);
  float wq[8], wk[8], dwq[8], dwk[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    wq[j] = active ? f.wq[ch + j] : 0.f;
    wk[j] = active ? f.wk[ch + j] : 0.f;
    dwq[j] = dwk[j] = 0.f;
  }
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * f.rows; t0 < f.tokens; t0 += static_cast<int64_t>(gridDim.x) * f.rows) {
    const int64_t t1 = min(t0 + f.rows, f.tokens);
    const bool halo = t1 < f.tokens && t1 % f.T != 0;
    const int64_t last = halo ? t1 : t1 - 1;
    float ck[8], cv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) ck[j] = cv[j] = 0.f;
    uint4 kc, vc;   // k, v of the current token
    mix_load(f, last, active, ch, C, kc, vc);
    MixRow nx;
    mix_bwd_load<kBf16>(p, last, active, ch, C, h, sub, nx);
    for (int64_t t = last; t >= t0; --t) {
      const MixRow r = nx;
      mix_bwd_load<kBf16>(p, t - 1, active && t > t0, ch, C, h, sub, nx);
      const bool first = t % f.T == 0;
      const bool own = t < t1;
      float k[8], v[8], kq[8], vq[8], dk[8], dv[8];
      blk_unpack<kBf16>(kc, k);
      blk_unpack<kBf16>(vc, v);
      blk_unpack<kBf16>(r.kp, kq);
      blk_unpack<kBf16>(r.vp, vq);
      blk_unpack<kBf16>(r.dk, dk);
      blk_unpack<kBf16>(r.dv, dv);
      const float2 w = blk_mix_weights(r.mix, lanes);
      const float a = w.x, c = w.y;
      float ks[8], wdy[8], c1 = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (first) kq[j] = vq[j] = 0.f;   // (the row before is another sequence's)
        ks[j] = (k[j] * (1.f - a) + kq[j] * a) * r.rk;   // normalised k'
        wdy[j] = wk[j] * dk[j];
        if (own) dwk[j] = fmaf(dk[j], ks[j], dwk[j]);
        c1 = fmaf(ks[j], wdy[j], c1);
      }
      c1 = head_sum(c1, lanes) * inv_d;
      float da = 0.f, dc = 0.f;
      float ok[8], ov[8];
      const bool live = !f.mask || f.mask[t] != 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = (wdy[j] - ks[j] * c1) * r.rk;   // dk'
        da = fmaf(g, kq[j] - k[j], da);
        dc = fmaf(dv[j], vq[j] - v[j], dc);
        ok[j] = live ? fmaf(g, 1.f - a, ck[j]) : 0.f;
        ov[j] = live ? fmaf(dv[j], 1.f - c, cv[j]) : 0.f;
        ck[j] = first ? 0.f : a * g;
        cv[j] = first ? 0.f : c * dv[j];
      }
      da = head_sum(da, lanes);
      dc = head_sum(dc, lanes);
      if (own) {
        float q[8], dq[8], c2 = 0.f;
        blk_unpack<kBf16>(r.q, q);
        blk_unpack<kBf16>(r.dq, dq);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          q[j] *= r.rq;
          dwq[j] = fmaf(dq[j], q[j], dwq[j]);
          dq[j] *= wq[j];
          c2 = fmaf(q[j], dq[j], c2);
        }
        c2 = head_sum(c2, lanes) * inv_d;
        if (active) {
#pragma unroll
          for (int j = 0; j < 8; ++j) dq[j] = (dq[j] - q[j] * c2) * r.rq;
          uint16_t* row = p.dy + t * f.ld;
          *reinterpret_cast<uint4*>(row + ch) = blk_pack<kBf16>(dq);
          *reinterpret_cast<uint4*>(row + C + ch) = blk_pack<kBf16>(ok);
          *reinterpret_cast<uint4*>(row + 2 * C + ch) = blk_pack<kBf16>(ov);
          if (sub == 0) {
            row[4 * C + f.H + h] = static_cast<uint16_t>(pack2<kBf16>(da * a * (1.f - a), 0.f) & 0xffffu);
            row[4 * C + 2 * f.H + h] = static_cast<uint16_t>(pack2<kBf16>(dc * c * (1.f - c), 0.f) & 0xffffu);
          }
        }
        if (threadIdx.x < p.pad1 - p.pad0) p.dy[t * f.ld + p.pad0 + threadIdx.x] = 0;
      }
      kc = r.kp;
      vc = r.vp;
    }
  }
  if (active) {
    float* o = p.dwq + static_cast<int64_t>(blockIdx.x) * C + ch;
    *reinterpret_cast<float4*>(o) = make_float4(dwq[0], dwq[1], dwq[2], dwq[3]);
    *reinterpret_cast<float4*>(o + 4) = make_float4(dwq[4], dwq[5], dwq[6], dwq[7]);
    o = p.dwk + static_cast<int64_t>(blockIdx.x) * C + ch;
    *reinterpret_cast<float4*>(o) = make_float4(dwk[0], dwk[1], dwk[2], dwk[3]);
    *reinterpret_cast<float4*>(o + 4) = make_float4(dwk[4], dwk[5], dwk[6], dwk[7]);
  }
}

// ------------------------------------------------------------ parameters of a block, laid out for its products
// One launch instead of a concatenation and a cast per parameter: the projection weights stacked into one (rows, C)
// matrix (padding rows zero), the norm weights as fp32, the gate bias as the product's bias vector: added there in fp32 it
// is rounded once with its projection, where a bias added to a 16-bit projection keeps the projection's rounding error when
// the two nearly cancel.
constexpr int kPackMats = 8, kPackVecs = 6;
struct PackParams {
  const uint16_t* mat[kPackMats];   // (mat_rows[i], C) contiguous
  int mat_row0[kPackMats + 1];      // first row of each in the stack; [n_mats] = rows of the stack without padding
  int n_mats, rows, C;              // rows: with padding
  uint16_t* stack;
  const void* vec[kPackVecs];
  int vec_len[kPackVecs], vec_off[kPackVecs], vec_dtype[kPackVecs];
  int n_vecs, vec_blocks;
  float* vecs;
  const uint16_t* bias;     // (n_bias), into bias_out (rows) from bias_row on
  int n_bias, bias_row;
  uint16_t* bias_out;       // or nullptr
};

__global__ void __launch_bounds__(256) fox_pack_kernel(const PackParams p) {
  if (static_cast<int>(blockIdx.x) < p.vec_blocks) {
    for (int i = 0; i < p.n_vecs; ++i) {
      for (int e = blockIdx.x * 256 + threadIdx.x; e < p.vec_len[i]; e += p.vec_blocks * 256) {
        float x;
        if (p.vec_dtype[i] == FOX_DTYPE_FP32) x = static_cast<const float*>(p.vec[i])[e];
        else if (p.vec_dtype[i] == FOX_DTYPE_BF16) x = unpack2<true>(static_cast<const uint16_t*>(p.vec[i])[e]).x;
        else x = unpack2<false>(static_cast<const uint16_t*>(p.vec[i])[e]).x;
        p.vecs[p.vec_off[i] + e] = x;
      }
    }
    if (p.bias_out)
      for (int e = blockIdx.x * 256 + threadIdx.x; e < p.rows; e += p.vec_blocks * 256)
        p.bias_out[e] = e >= p.bias_row && e - p.bias_row < p.n_bias ? p.bias[e - p.bias_row] : static_cast<uint16_t>(0);
    return;
  }
  const int per_row = p.C / 8;
  const int64_t total = static_cast<int64_t>(p.rows) * per_row, step = static_cast<int64_t>(gridDim.x - p.vec_blocks) * 256;
  constexpr int kU = 4;
  for (int64_t e0 = static_cast<int64_t>(blockIdx.x - p.vec_blocks) * 256 + threadIdx.x; e0 < total; e0 += kU * step) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t e = e0 + u * step;
      v[u] = make_uint4(0, 0, 0, 0);
      if (e < total) {
        const int row = static_cast<int>(e / per_row), c = static_cast<int>(e % per_row);
        int m = 0;
        while (m < p.n_mats && row >= p.mat_row0[m + 1]) ++m;
        if (m < p.n_mats)
          v[u] = *reinterpret_cast<const uint4*>(p.mat[m] + static_cast<int64_t>(row - p.mat_row0[m]) * p.C + c * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t e = e0 + u * step;
      if (e < total) *reinterpret_cast<uint4*>(p.stack + e * 8) = v[u];
    }
  }
}

// The weight gradients come out of one product as a stack of the same layout; every parameter gets memory of its own, so that
// a gradient that is kept or saved does not hold the others'.  Bound by the copy: 28 MB at 1536 channels, 4 us.
struct UnpackParams {
  const uint16_t* stack;
  uint16_t* mat[kPackMats];   // or nullptr
  int mat_row0[kPackMats + 1];
  int n_mats, C;
};

__global__ void __launch_bounds__(256) fox_unpack_kernel(const UnpackParams p) {
  const int per_row = p.C / 8;
  const int64_t total = static_cast<int64_t>(p.mat_row0[p.n_mats]) * per_row, step = static_cast<int64_t>(gridDim.x) * 256;
  constexpr int kU = 4;
  for (int64_t e0 = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; e0 < total; e0 += kU * step) {
    uint4 v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (e0 + u * step < total) v[u] = *reinterpret_cast<const uint4*>(p.stack + (e0 + u * step) * 8);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int64_t e = e0 + u * step;
      if (e >= total) break;
      const int row = static_cast<int>(e / per_row), c = static_cast<int>(e % per_row);
      int m = 0;
      while (m + 1 < p.n_mats && row >= p.mat_row0[m + 1]) ++m;
      if (p.mat[m]) *reinterpret_cast<uint4*>(p.mat[m] + static_cast<int64_t>(row - p.mat_row0[m]) * p.C + c * 8) = v[u];
    }
  }
}

// ------------------------------------------------------------ column sums of a block's partial weight gradients
// out_i[c] = sum_r part_i[r][c] for up to six arrays in one launch (a reduction kernel and a cast each before).  A CTA
// takes 32 columns: warp w of 32 sums rows w, w + 32, ... with four loads in flight, then the warps are joined.  (Bound by
// latency: with 8 warps a CTA walked 592 rows in 19 trips; 14.1 -> 6.1 us at 768 columns, 15.8 -> 8.2 us at 1536.)
struct SumParams {
  const float* part[kPackVecs];
  int rows[kPackVecs], cols[kPackVecs], dtype[kPackVecs], block0[kPackVecs + 1];
  void* out[kPackVecs];
  int n;
};

__global__ void __launch_bounds__(1024) fox_column_sums_kernel(const SumParams p) {
  __shared__ float s[32][33];
  int i = 0;
  while (i + 1 < p.n && static_cast<int>(blockIdx.x) >= p.block0[i + 1]) ++i;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = (blockIdx.x - p.block0[i]) * 32 + lane, rows = p.rows[i], cols = p.cols[i];
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  if (col < cols) {
    const float* src = p.part[i] + col;
    for (int r = warp; r < rows; r += 128) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + 32 * u < rows) acc[u] += src[static_cast<int64_t>(r + 32 * u) * cols];
    }
  }
  s[warp][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  __syncthreads();
  if (warp == 0 && col < cols) {
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < 32; ++w) x += s[w][lane];
    if (p.dtype[i] == FOX_DTYPE_FP32) static_cast<float*>(p.out[i])[col] = x;
    else static_cast<uint16_t*>(p.out[i])[col] = static_cast<uint16_t>(
        (p.dtype[i] == FOX_DTYPE_BF16 ? pack2<true>(x, 0.f) : pack2<false>(x, 0.f)) & 0xffffu);
  }
}

static inline int blk_rc() { return cudaGetLastError() == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH; }

static int mix_params(MixParams& p, int64_t B, int64_t T, int64_t H, int64_t D, const void* y, int64_t ld, const float* wq,
                      const float* wk, const int64_t* mask, float eps) {
  if (!y || !wq || !wk || B <= 0 || T <= 0 || H <= 0) return FOX_ERR_BAD_ARG;
  if (D < 16 || D > 256 || (D & (D - 1))) return FOX_ERR_HEAD_DIM;   // (two lanes a head at least)
  if (H * D > 8 * kMixThreads || T > 2147483647LL) return FOX_ERR_TOO_LARGE;   // (8 channels a thread)
  if (reinterpret_cast<uintptr_t>(y) % 16 || ld % 8 || ld < 4 * H * D + 3 * H) return FOX_ERR_ALIGNMENT;
  p.y = (const uint16_t*)y; p.ld = ld; p.wq = wq; p.wk = wk; p.mask = mask; p.eps = eps;
  p.H = (int)H; p.D = (int)D; p.T = (int)T; p.tokens = B * T;
  return FOX_OK;
}
static int mix_threads(const MixParams& p) { return (p.H * (p.D / 8) + 31) / 32 * 32; }
// Tokens a CTA takes: 16 where that still gives every SM several CTAs (each run of tokens re-reads one row), fewer for
// short inputs so that the chip fills, at least 2.
static int mix_rows(int64_t tokens, int64_t ctas) {
  int64_t r = tokens / ctas;
  return (int)(r < 2 ? 2 : r > 16 ? 16 : r);
}

}  // namespace fox

using namespace fox;

extern "C" int fox_mix_fwd(int device, void* stream, int dtype, int64_t B, int64_t T, int64_t H, int64_t D, const void* y,
                           int64_t ld, const float* wq, const float* wk, float eps, const int64_t* mask, void* q, void* k,
                           void* v, float* rstd_q, float* rstd_k, int64_t* seq_start) {
  MixParams p{};
  int rc = mix_params(p, B, T, H, D, y, ld, wq, wk, mask, eps);
  if (rc) return rc;
  if (!q || !k || !v || (rstd_q == nullptr) != (rstd_k == nullptr)) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  p.q = (uint16_t*)q; p.k = (uint16_t*)k; p.v = (uint16_t*)v; p.rstd_q = rstd_q; p.rstd_k = rstd_k;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  p.rows = mix_rows(p.tokens, 148 * 4);
  if (seq_start && !mask) return FOX_ERR_BAD_ARG;
  p.seq_start = seq_start;
  p.mix_blocks = (int)((p.tokens + p.rows - 1) / p.rows);
  const unsigned grid = (unsigned)(p.mix_blocks + (seq_start ? B : 0));
  if (dtype == FOX_DTYPE_BF16) fox_mix_fwd_kernel<true><<<grid, mix_threads(p), 0, (cudaStream_t)stream>>>(p);
  else fox_mix_fwd_kernel<false><<<grid, mix_threads(p), 0, (cudaStream_t)stream>>>(p);
  return blk_rc();
}

extern "C" int64_t fox_mix_bwd_partials(int64_t tokens) {
  const int rows = mix_rows(tokens, 148 * 2);
  const int64_t n = (tokens + rows - 1) / rows;
  return n < 148 * 4 ? n : 148 * 4;
}

extern "C" int fox_mix_bwd(int device, void* stream, int dtype, int64_t B, int64_t T, int64_t H, int64_t D, const void* y,
                           int64_t ld, const float* wq, const float* wk, const int64_t* mask, const float* rstd_q,
                           const float* rstd_k, const void* dq, const void* dk, const void* dv, void* dy, float* dwq_partial,
                           float* dwk_partial, int64_t n_partials) {
  MixBwdParams p{};
  int rc = mix_params(p.f, B, T, H, D, y, ld, wq, wk, mask, 0.f);
  if (rc) return rc;
  if (!rstd_q || !rstd_k || !dq || !dk || !dv || !dy || !dwq_partial || !dwk_partial || n_partials <= 0) return FOX_ERR_BAD_ARG;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(dy) % 16) return FOX_ERR_ALIGNMENT;
  p.f.rstd_q = const_cast<float*>(rstd_q); p.f.rstd_k = const_cast<float*>(rstd_k);
  p.dq = (const uint16_t*)dq; p.dk = (const uint16_t*)dk; p.dv = (const uint16_t*)dv; p.dy = (uint16_t*)dy;
  p.dwq = dwq_partial; p.dwk = dwk_partial;
  p.pad0 = (int)(4 * H * D + 3 * H); p.pad1 = (int)ld;
  if (p.pad1 - p.pad0 > 32) return FOX_ERR_BAD_ARG;   // (one thread per pad column)
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  p.f.rows = mix_rows(p.f.tokens, 148 * 2);
  if (dtype == FOX_DTYPE_BF16) fox_mix_bwd_kernel<true><<<(unsigned)n_partials, mix_threads(p.f), 0, (cudaStream_t)stream>>>(p);
  else fox_mix_bwd_kernel<false><<<(unsigned)n_partials, mix_threads(p.f), 0, (cudaStream_t)stream>>>(p);
  return blk_rc();
}

extern "C" int fox_pack(int device, void* stream, int64_t n_mats, const void* const* mats, const int64_t* mat_rows, int64_t rows,
                        int64_t cols, void* stack, int64_t n_vecs, const void* const* vecs, const int64_t* vec_len,
                        const int32_t* vec_dtype, float* vecs_out, const void* bias, int64_t n_bias, int64_t bias_row,
                        void* bias_out) {
  if (n_mats < 0 || n_mats > kPackMats || n_vecs < 0 || n_vecs > kPackVecs || cols <= 0 || cols % 8) return FOX_ERR_BAD_ARG;
  PackParams p{};
  int64_t row = 0;
  for (int i = 0; i < n_mats; ++i) {
    if (!mats[i]) return FOX_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(mats[i]) % 16) return FOX_ERR_ALIGNMENT;
    p.mat[i] = (const uint16_t*)mats[i];
    p.mat_row0[i] = (int)row;
    row += mat_rows[i];
  }
  p.mat_row0[n_mats] = (int)row;
  if (row > rows || rows > 2147483647LL || (rows > 0 && (!stack || reinterpret_cast<uintptr_t>(stack) % 16))) return FOX_ERR_BAD_ARG;
  p.n_mats = (int)n_mats; p.rows = (int)rows; p.C = (int)cols; p.stack = (uint16_t*)stack;
  int64_t off = 0;
  for (int i = 0; i < n_vecs; ++i) {
    if (!vecs[i] || !vecs_out) return FOX_ERR_BAD_ARG;
    p.vec[i] = vecs[i]; p.vec_len[i] = (int)vec_len[i]; p.vec_off[i] = (int)off; p.vec_dtype[i] = vec_dtype[i];
    off += vec_len[i];
  }
  p.n_vecs = (int)n_vecs; p.vecs = vecs_out;
  if (bias_out) {
    if (!bias || n_bias <= 0 || bias_row < 0 || bias_row + n_bias > rows) return FOX_ERR_BAD_ARG;
    p.bias = (const uint16_t*)bias; p.n_bias = (int)n_bias; p.bias_row = (int)bias_row; p.bias_out = (uint16_t*)bias_out;
  }
  p.vec_blocks = n_vecs || bias_out ? 4 : 0;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  int64_t blocks = (rows * (cols / 8) + 256 * 4 - 1) / (256 * 4);
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks + p.vec_blocks == 0) return FOX_OK;
  fox_pack_kernel<<<(unsigned)(blocks + p.vec_blocks), 256, 0, (cudaStream_t)stream>>>(p);
  return blk_rc();
}

extern "C" int fox_unpack(int device, void* stream, int64_t n_mats, void* const* mats, const int64_t* mat_rows, int64_t cols,
                          const void* stack) {
  if (n_mats <= 0 || n_mats > kPackMats || cols <= 0 || cols % 8 || !stack) return FOX_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(stack) % 16) return FOX_ERR_ALIGNMENT;
  UnpackParams p{};
  int64_t row = 0;
  for (int i = 0; i < n_mats; ++i) {
    if (mat_rows[i] <= 0) return FOX_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(mats[i]) % 16) return FOX_ERR_ALIGNMENT;
    p.mat[i] = (uint16_t*)mats[i];
    p.mat_row0[i] = (int)row;
    row += mat_rows[i];
  }
  if (row > 2147483647LL) return FOX_ERR_BAD_ARG;
  p.mat_row0[n_mats] = (int)row;
  p.stack = (const uint16_t*)stack; p.n_mats = (int)n_mats; p.C = (int)cols;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  int64_t blocks = (row * (cols / 8) + 256 * 4 - 1) / (256 * 4);
  if (blocks > 148 * 8) blocks = 148 * 8;
  fox_unpack_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(p);
  return blk_rc();
}

extern "C" int fox_column_sums(int device, void* stream, int64_t n, const float* const* parts, const int64_t* rows,
                               const int64_t* cols, const int32_t* out_dtype, void* const* outs) {
  if (n <= 0 || n > kPackVecs) return FOX_ERR_BAD_ARG;
  SumParams p{};
  int64_t block = 0;
  for (int i = 0; i < n; ++i) {
    if (!parts[i] || !outs[i] || rows[i] <= 0 || cols[i] <= 0) return FOX_ERR_BAD_ARG;
    p.part[i] = parts[i]; p.rows[i] = (int)rows[i]; p.cols[i] = (int)cols[i]; p.dtype[i] = out_dtype[i]; p.out[i] = outs[i];
    p.block0[i] = (int)block;
    block += (cols[i] + 31) / 32;
  }
  p.block0[n] = (int)block;
  p.n = (int)n;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  fox_column_sums_kernel<<<(unsigned)block, 1024, 0, (cudaStream_t)stream>>>(p);
  return blk_rc();
}
