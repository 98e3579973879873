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

// eight channels as four pairs, for packed two-wide fp32 arithmetic
template <bool kBf16>
__device__ __forceinline__ void blk_unpack2(const uint4& v, float2* f) {
  f[0] = unpack2<kBf16>(v.x);
  f[1] = unpack2<kBf16>(v.y);
  f[2] = unpack2<kBf16>(v.z);
  f[3] = unpack2<kBf16>(v.w);
}
template <bool kBf16>
__device__ __forceinline__ uint4 blk_pack2(const float2* f) {
  return make_uint4(pack2<kBf16>(f[0].x, f[0].y), pack2<kBf16>(f[1].x, f[1].y), pack2<kBf16>(f[2].x, f[2].y), pack2<kBf16>(f[3].x, f[3].y));
}
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 neg2(float2 x) { return make_float2(-x.x, -x.y); }
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
// over the lanes of a head (kLanes of them, where that is known)
template <int kLanes>
__device__ __forceinline__ float head_sum(float x, int lanes) {
  if constexpr (kLanes > 0) {
#pragma unroll
    for (int o = kLanes >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  } else {
    for (int o = lanes >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  }
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
// store, so it takes one token at a time in 64 registers and has 5 CTAs per SM, where two tokens in 116 registers left 2: 16384 x 1536 bf16 96 -> 71.5 us, with
// packed arithmetic 67 (4.5 TB/s), 2048 x 768 7.5 -> 6.7 us.  (Two tokens in 80 registers: 67 and 8.1 us; one in 48 registers: 91 and 9.5 us; 4 channels a thread, which doubles
// the instructions for addresses and sums: 199 and 13 us.)
template <bool kBf16, int kLanes>
__global__ void __launch_bounds__(kMixThreads, 4) fox_mix_fwd_kernel(const MixParams p) {
  wait_for_kernel_in_front();
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
  const int lanes = kLanes ? kLanes : p.D >> 3, C = p.H * p.D;
  const int h = threadIdx.x / lanes, sub = threadIdx.x % lanes;
  const bool active = h < p.H;
  const int ch = active ? h * p.D + sub * 8 : 0;
  const float inv_d = 1.f / static_cast<float>(p.D);
  float2 wq[4], wk[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    wq[j] = active ? make_float2(p.wq[ch + 2 * j], p.wq[ch + 2 * j + 1]) : both(0.f);
    wk[j] = active ? make_float2(p.wk[ch + 2 * j], p.wk[ch + 2 * j + 1]) : both(0.f);
  }
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * p.rows, t1 = min(t0 + p.rows, p.tokens);
  uint4 kp, vp;                           // of the token before; zero where there is none
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
    pos = pos + 1 == p.T ? 0 : pos + 1;
    float2 q[4], k[4], v[4], kq[4], vq[4];
    blk_unpack2<kBf16>(qr, q);
    blk_unpack2<kBf16>(kr, k);
    blk_unpack2<kBf16>(vr, v);
    blk_unpack2<kBf16>(kp, kq);
    blk_unpack2<kBf16>(vp, vq);
    const float2 w = blk_mix_weights(mix, lanes);
    const float2 a = both(w.x), c = both(w.y), a1 = both(1.f - w.x), c1 = both(1.f - w.y);
    float2 sq = both(0.f), sk = both(0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      k[j] = __ffma2_rn(k[j], a1, __fmul2_rn(kq[j], a));
      v[j] = __ffma2_rn(v[j], c1, __fmul2_rn(vq[j], c));
      sq = __ffma2_rn(q[j], q[j], sq);
      sk = __ffma2_rn(k[j], k[j], sk);
    }
    const float rq = rsqrtf(head_sum<kLanes>(sq.x + sq.y, lanes) * inv_d + p.eps),
                rk = rsqrtf(head_sum<kLanes>(sk.x + sk.y, lanes) * inv_d + p.eps);
    if (active) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        q[j] = __fmul2_rn(q[j], __fmul2_rn(both(rq), wq[j]));
        k[j] = __fmul2_rn(k[j], __fmul2_rn(both(rk), wk[j]));
      }
      const int64_t o = t * C + ch;
      *reinterpret_cast<uint4*>(p.q + o) = blk_pack2<kBf16>(q);
      *reinterpret_cast<uint4*>(p.k + o) = blk_pack2<kBf16>(k);
      *reinterpret_cast<uint4*>(p.v + o) = blk_pack2<kBf16>(v);
      if (sub == 0 && p.rstd_q) {
        p.rstd_q[t * p.H + h] = rq;
        p.rstd_k[t * p.H + h] = rk;
      }
    }
    kp = pos == 0 ? make_uint4(0, 0, 0, 0) : kr;
    vp = pos == 0 ? make_uint4(0, 0, 0, 0) : vr;
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

// A CTA's rows: pointers to its first token, the same for every thread, and 32-bit offsets from there.
struct MixRows {
  const uint16_t *y, *dq, *dk, *dv;
  uint16_t* dy;
  const int64_t* mask;
  const float *rq, *rk;
};
__device__ __forceinline__ void mix_rows_kv(const MixRows& p, uint32_t i, uint32_t ld, uint32_t C, bool on, uint32_t ch, uint4& k, uint4& v) {
  k = v = make_uint4(0, 0, 0, 0);
  if (on && (!p.mask || p.mask[i] != 0)) {
    k = *reinterpret_cast<const uint4*>(p.y + (i * ld + C + ch));
    v = *reinterpret_cast<const uint4*>(p.y + (i * ld + 2 * C + ch));
  }
}
template <bool kBf16>
__device__ __forceinline__ void mix_rows_load(const MixRows& p, uint32_t i, uint32_t ld, uint32_t C, uint32_t H, bool on, bool before,
                                              uint32_t ch, uint32_t h, uint32_t sub, MixRow& r) {
  r.q = r.dq = r.dk = r.dv = make_uint4(0, 0, 0, 0);
  r.mix = r.rq = r.rk = 0.f;
  mix_rows_kv(p, i - 1, ld, C, on && before, ch, r.kp, r.vp);
  if (on) {
    r.q = *reinterpret_cast<const uint4*>(p.y + (i * ld + ch));
    r.dq = *reinterpret_cast<const uint4*>(p.dq + (i * C + ch));
    r.dk = *reinterpret_cast<const uint4*>(p.dk + (i * C + ch));
    r.dv = *reinterpret_cast<const uint4*>(p.dv + (i * C + ch));
    r.mix = blk_load1<kBf16>(p.y + (i * ld + 4 * C + (1 + (sub & 1)) * H + h));
    r.rq = p.rq[i * H + h];
    r.rk = p.rk[i * H + h];
  }
}

// Tokens are walked backwards: the gradient of k[t] is (1 - a[t]) dk'[t] + a[t+1] dk'[t+1], the second term carried from
// the token before in this order.  A CTA first forms the token after its range for that carry (1 / rows more reads).
// Bound by instructions and the latency of a token's chain at 12 warps per SM: what costs registers costs warps.  So a token's
// rows are not held twice (no prefetch), the norm weights are read from shared memory, addresses are 32-bit offsets, and the
// arithmetic is packed two wide (800 instructions a warp and token before).  16384 x 1536 bf16: 174 -> 123 us; 2048 x 768: 20.2
// -> 14.2 us.  (112 registers for a third CTA: 130 and 15.2 us; 96: 177; prefetching the next rows into L1: 122.)
template <bool kBf16, int kLanes>
__global__ void __launch_bounds__(kMixThreads, 2) fox_mix_bwd_kernel(const MixBwdParams p) {
  wait_for_kernel_in_front();
  const MixParams& f = p.f;
  const int lanes = kLanes ? kLanes : f.D >> 3, C = f.H * f.D;
  const int h = threadIdx.x / lanes, sub = threadIdx.x % lanes;
  const bool active = h < f.H;
  const int ch = active ? h * f.D + sub * 8 : 0;
  const float inv_d = 1.f / static_cast<float>(f.D);
  __shared__ float4 s_wq[2 * kMixThreads], s_wk[2 * kMixThreads];   // the norm weights, a thread's own
  float2 dwq[4], dwk[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    s_wq[i * kMixThreads + threadIdx.x] = active ? make_float4(f.wq[ch + 4 * i], f.wq[ch + 4 * i + 1], f.wq[ch + 4 * i + 2], f.wq[ch + 4 * i + 3]) : zero;
    s_wk[i * kMixThreads + threadIdx.x] = active ? make_float4(f.wk[ch + 4 * i], f.wk[ch + 4 * i + 1], f.wk[ch + 4 * i + 2], f.wk[ch + 4 * i + 3]) : zero;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) dwq[j] = dwk[j] = both(0.f);
  auto weights = [&](const float4* w, float2* o) {
    const float4 x = w[threadIdx.x], y = w[kMixThreads + threadIdx.x];
    o[0] = make_float2(x.x, x.y);
    o[1] = make_float2(x.z, x.w);
    o[2] = make_float2(y.x, y.y);
    o[3] = make_float2(y.z, y.w);
  };
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * f.rows; t0 < f.tokens; t0 += static_cast<int64_t>(gridDim.x) * f.rows) {
    const int64_t t1 = min(t0 + f.rows, f.tokens);
    const bool halo = t1 < f.tokens && t1 % f.T != 0;
    const int64_t last = halo ? t1 : t1 - 1;
    int pos = static_cast<int>(last % f.T);   // of the token in its sequence
    float2 ck[4], cv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ck[j] = cv[j] = both(0.f);
    const int64_t tb = t0 > 0 ? t0 - 1 : 0;   // (the row before the range is read too)
    const MixRows rows{f.y + tb * f.ld, p.dq + tb * C, p.dk + tb * C, p.dv + tb * C, p.dy + tb * f.ld, f.mask ? f.mask + tb : nullptr,
                       f.rstd_q + tb * f.H, f.rstd_k + tb * f.H};
    const uint32_t ld = static_cast<uint32_t>(f.ld), i0 = static_cast<uint32_t>(t0 - tb), i1 = static_cast<uint32_t>(t1 - tb);
    uint4 kc, vc;   // k, v of the current token
    uint32_t i = static_cast<uint32_t>(last - tb);
    mix_rows_kv(rows, i, ld, C, active, ch, kc, vc);
    for (;; --i) {
      MixRow r;
      mix_rows_load<kBf16>(rows, i, ld, C, f.H, active, i > 0, ch, h, sub, r);
      const bool first = pos == 0;   // (the row before is another sequence's)
      pos = first ? f.T - 1 : pos - 1;
      const bool own = i < i1;
      const float2 w = blk_mix_weights(r.mix, lanes);
      const bool live = !rows.mask || rows.mask[i] != 0;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      const uint32_t row = i * ld;
      float dc1;
      {   // v
        const float2 c = both(w.y), c1 = both(1.f - w.y);
        float2 v[4], vq[4], dv[4], ov[4], dc = both(0.f);
        blk_unpack2<kBf16>(vc, v);
        blk_unpack2<kBf16>(first ? zero : r.vp, vq);
        blk_unpack2<kBf16>(r.dv, dv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dc = __ffma2_rn(dv[j], __fadd2_rn(vq[j], neg2(v[j])), dc);
          ov[j] = __ffma2_rn(dv[j], c1, cv[j]);
          cv[j] = __fmul2_rn(c, dv[j]);
        }
        dc1 = dc.x + dc.y;
        if (own && active) *reinterpret_cast<uint4*>(rows.dy + (row + 2 * C + ch)) = live ? blk_pack2<kBf16>(ov) : zero;
      }
      float da1;
      {   // k
        const float2 a = both(w.x), a1 = both(1.f - w.x), rk = both(r.rk);
        float2 k[4], kq[4], dk[4], ks[4], wdy[4], s1 = both(0.f), da = both(0.f);
        blk_unpack2<kBf16>(kc, k);
        blk_unpack2<kBf16>(first ? zero : r.kp, kq);
        blk_unpack2<kBf16>(r.dk, dk);
        weights(s_wk, wdy);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ks[j] = __fmul2_rn(__ffma2_rn(k[j], a1, __fmul2_rn(kq[j], a)), rk);   // normalised k'
          wdy[j] = __fmul2_rn(wdy[j], dk[j]);
          s1 = __ffma2_rn(ks[j], wdy[j], s1);
          if (own) dwk[j] = __ffma2_rn(dk[j], ks[j], dwk[j]);
          k[j] = __fadd2_rn(kq[j], neg2(k[j]));
        }
        const float2 m1 = both(-head_sum<kLanes>(s1.x + s1.y, lanes) * inv_d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 g = __fmul2_rn(__ffma2_rn(ks[j], m1, wdy[j]), rk);   // dk'
          da = __ffma2_rn(g, k[j], da);
          ks[j] = __ffma2_rn(g, a1, ck[j]);
          ck[j] = __fmul2_rn(a, g);
        }
        da1 = da.x + da.y;
        if (own && active) *reinterpret_cast<uint4*>(rows.dy + (row + C + ch)) = live ? blk_pack2<kBf16>(ks) : zero;
      }
      if (first) {
#pragma unroll
        for (int j = 0; j < 4; ++j) ck[j] = cv[j] = both(0.f);
      }
      if (own) {   // q, and the mixing weights' logits
        float2 q[4], dq[4], wq[4], s2 = both(0.f);
        blk_unpack2<kBf16>(r.q, q);
        blk_unpack2<kBf16>(r.dq, dq);
        weights(s_wq, wq);
        const float2 rq = both(r.rq);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          q[j] = __fmul2_rn(q[j], rq);
          dwq[j] = __ffma2_rn(dq[j], q[j], dwq[j]);
          dq[j] = __fmul2_rn(dq[j], wq[j]);
          s2 = __ffma2_rn(q[j], dq[j], s2);
        }
        da1 = head_sum<kLanes>(da1, lanes);
        dc1 = head_sum<kLanes>(dc1, lanes);
        const float2 m2 = both(-head_sum<kLanes>(s2.x + s2.y, lanes) * inv_d);
        if (active) {
#pragma unroll
          for (int j = 0; j < 4; ++j) dq[j] = __fmul2_rn(__ffma2_rn(q[j], m2, dq[j]), rq);
          *reinterpret_cast<uint4*>(rows.dy + (row + ch)) = blk_pack2<kBf16>(dq);
          if (sub == 0) {
            rows.dy[row + 4 * C + f.H + h] = static_cast<uint16_t>(pack2<kBf16>(da1 * w.x * (1.f - w.x), 0.f) & 0xffffu);
            rows.dy[row + 4 * C + 2 * f.H + h] = static_cast<uint16_t>(pack2<kBf16>(dc1 * w.y * (1.f - w.y), 0.f) & 0xffffu);
          }
        }
        if (threadIdx.x < p.pad1 - p.pad0) rows.dy[row + p.pad0 + threadIdx.x] = 0;
      }
      kc = r.kp;
      vc = r.vp;
      if (i == i0) break;
    }
  }
  if (active) {
    float4* o = reinterpret_cast<float4*>(p.dwq + static_cast<int64_t>(blockIdx.x) * C + ch);
    o[0] = make_float4(dwq[0].x, dwq[0].y, dwq[1].x, dwq[1].y);
    o[1] = make_float4(dwq[2].x, dwq[2].y, dwq[3].x, dwq[3].y);
    o = reinterpret_cast<float4*>(p.dwk + static_cast<int64_t>(blockIdx.x) * C + ch);
    o[0] = make_float4(dwk[0].x, dwk[0].y, dwk[1].x, dwk[1].y);
    o[1] = make_float4(dwk[2].x, dwk[2].y, dwk[3].x, dwk[3].y);
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
  wait_for_kernel_in_front();
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
  wait_for_kernel_in_front();
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
  wait_for_kernel_in_front();
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
  const bool bf = dtype == FOX_DTYPE_BF16;
  auto kern = D == 64 ? (bf ? fox_mix_fwd_kernel<true, 8> : fox_mix_fwd_kernel<false, 8>)
              : D == 128 ? (bf ? fox_mix_fwd_kernel<true, 16> : fox_mix_fwd_kernel<false, 16>)
                         : (bf ? fox_mix_fwd_kernel<true, 0> : fox_mix_fwd_kernel<false, 0>);
  return launch_behind(kern, dim3(grid), mix_threads(p), 0, (cudaStream_t)stream, p);
}

extern "C" int64_t fox_mix_bwd_partials(int64_t tokens) {
  const int rows = mix_rows(tokens, 148 * 3);
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
  p.f.rows = mix_rows(p.f.tokens, 148 * 3);
  const bool bf = dtype == FOX_DTYPE_BF16;
  auto kern = D == 64 ? (bf ? fox_mix_bwd_kernel<true, 8> : fox_mix_bwd_kernel<false, 8>)
              : D == 128 ? (bf ? fox_mix_bwd_kernel<true, 16> : fox_mix_bwd_kernel<false, 16>)
                         : (bf ? fox_mix_bwd_kernel<true, 0> : fox_mix_bwd_kernel<false, 0>);
  return launch_behind(kern, dim3((unsigned)n_partials), mix_threads(p.f), 0, (cudaStream_t)stream, p);
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
  return launch_behind(fox_pack_kernel, dim3((unsigned)(blocks + p.vec_blocks)), 256, 0, (cudaStream_t)stream, p);
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
  return launch_behind(fox_unpack_kernel, dim3((unsigned)blocks), 256, 0, (cudaStream_t)stream, p);
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
  return launch_behind(fox_column_sums_kernel, dim3((unsigned)block), 1024, 0, (cudaStream_t)stream, p);
}
