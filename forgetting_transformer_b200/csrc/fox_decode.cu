// Single-query ("decode") forgetting attention: one new token against a cache of N keys.
//
// The path upstream's generation loop takes through the same _fwd_kernel with seqlen_q = 1
// (src/forgetting_transformer/ops/forgetting_attention.py:148-153, 591-693; the cache that feeds it is
// fgate_cache.py:77-116).  With one query row the work is a pair of matrix-vector products, bound by reading
// K and V once:
//
//   u_j = (q.k_j) sm_scale log2e + (Lambda_{N-1} - Lambda_j) log2e      (j >= seq_start, j >= start_index)
//   m = max u_j;  l = sum 2^(u_j - m);  o = sum 2^(u_j - m) v_j;   out = o / l;   L = m ln2 + ln l
//
// The keys of a (b,h) are cut into `splits` ranges, one CTA each.  D / 8 lanes share a key (16-byte loads of whole
// rows, 32 / (D/8) consecutive rows per warp instruction), four rows of K and of V are in flight per lane, and each
// group of lanes keeps a softmax stream of its own: (m, l) and eight channels of o.  (One thread per key with all of
// its channels in registers read 16 bytes of 32 different rows per instruction and reached 3.6 TB/s.)
//
// Lambda_{N-1} - Lambda_j is the sum of the log gates after j.  Without pruning nothing else needs the prefix sum, so
// the kernel forms it from the gates: a CTA scans its own range from the right, tile by tile, and a range's gate total
// shifts the maxima of the ranges left of it in the merge.  (As a kernel in front, one CTA per (b,h), the prefix sum
// took 32 us of a step against 65536 keys.)  With a pruning threshold the index scan has formed Lambda anyway.
//
// Up to 8 ranges are merged through the shared memory of their cluster; more go through a workspace and a second kernel,
// launched early (programmatic dependent launch).
#include <cooperative_groups.h>

#include <type_traits>

#include "fox_common.cuh"
#include "fox_host.h"

namespace fox {

namespace cg = cooperative_groups;

constexpr int kDecThreads = 256, kDecWarps = kDecThreads / 32;
constexpr int kDecTile = 1024;      // keys between two scans of the gates
constexpr int kDecRows = 4;         // rows of K and of V in flight per lane
constexpr int kDecMaxCluster = 8;
constexpr int kDecMaxSplits = 1024;   // taken
constexpr int kDecMostSplits = 512;   // asked for by fox_attn_decode_splits
constexpr int kDecPerSm = 3, kDecMorePerSm = 4;                                       // by the kernels' launch bounds
constexpr int64_t kDecSlots = kSms * kDecPerSm, kDecClusterSlots = 400;               // CTAs of a wave, three to an SM
constexpr int64_t kDecMoreSlots = kSms * kDecMorePerSm, kDecMoreClusterSlots = 540;   // four
constexpr int64_t kDecStartKeys = 600, kDecMergeKeys = 120, kDecLeastKeys = 128;      // (at fox_attn_decode_splits)
constexpr int64_t kDecMoreLeastKeys = 640;
constexpr int64_t kDecLongRange = 1024 * 64, kDecManyClusters = 384;   // keys times head dim; CTAs (at long_ranges)
constexpr float kDecLog2e = 1.4426950408889634f;

struct DecodeParams {
  const uint16_t *q, *k, *v;
  int64_t q_sb, q_sh, k_sb, k_sh, k_st, v_sb, v_sh, v_st;
  const float* lam;            // (B,H,N), or nullptr: from the gates
  const float* gate;           // log gates, strides g_*
  int64_t g_sb, g_sh, g_sn;
  const int64_t* seq_start;    // (B,) or nullptr
  const int64_t* start_index;  // (B,H,1) or nullptr
  float* part;                 // (B,H,splits, D + 4): o[D], m, l, gate total
  uint16_t* o;
  int64_t o_sb, o_sh;
  float* L;
  int H, N, splits;
  float qk_scale;              // sm_scale * log2(e)
  bool chained;                // between kernels of a token's chain: lets the next begin early
};

// A token's way into the attention (fox_step_mix's work, kStep below): q comes from the projections, and the CTA that has the
// last key puts it into the cache first.
struct DecodeStep {
  const float* y;              // (B, ld): [q | k | v | ogate | fgate | k mix | v mix]
  int64_t ld;
  const void *wq, *wk, *bias;  // (C), (C), (H) or nullptr
  int wq_dtype, wk_dtype, bias_dtype;
  float eps;
  const int64_t* mask;         // (B, N) or nullptr: the first valid key is N - its sum
  uint16_t *k_state, *v_state; // (B, C), replaced
  uint16_t *k_cache, *v_cache; // (B, H, cap, D)
  float* g_cache;              // (B, H, cap)
  int64_t cap;
};

__device__ __forceinline__ float dec_load_any(const void* w, int dtype, int i) {
  if (dtype == FOX_DTYPE_FP32) return static_cast<const float*>(w)[i];
  const uint32_t u = static_cast<const uint16_t*>(w)[i];
  return dtype == FOX_DTYPE_BF16 ? unpack2<true>(u).x : unpack2<false>(u).x;
}
template <bool kBf16>
__device__ __forceinline__ uint4 dec_pack(const float* f) {
  return make_uint4(pack2<kBf16>(f[0], f[1]), pack2<kBf16>(f[2], f[3]), pack2<kBf16>(f[4], f[5]), pack2<kBf16>(f[6], f[7]));
}
__device__ __forceinline__ void dec_load8(const float* p, float* f) {   // (16-byte aligned)
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <int kLanes>
__device__ __forceinline__ float dec_norm(const float* f, float inv_d, float eps) {   // over the lanes that share a row
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) ss = fmaf(f[c], f[c], ss);
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  return rsqrtf(ss * inv_d + eps);
}

template <bool kBf16>
__device__ __forceinline__ void dec_unpack(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = unpack2<kBf16>(w[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}

// (m, l) joined; a is the factor of the first stream, b of the second
__device__ __forceinline__ float dec_join(float& m, float& l, float m2, float l2, float& a, float& b) {
  const float mx = fmaxf(m, m2);
  a = m == -INFINITY ? 0.f : fast_exp2(m - mx);
  b = m2 == -INFINITY ? 0.f : fast_exp2(m2 - mx);
  l = l * a + l2 * b;
  m = mx;
  return mx;
}

// s_res of a CTA: o[D], m, l, gate total
template <bool kBf16, int D>
__device__ __forceinline__ void dec_store(const DecodeParams& p, int b, int h, int d, float o, float l) {
  const uint32_t pk = pack2<kBf16>(l > 0.f ? o / l : 0.f, 0.f);
  p.o[b * p.o_sb + h * p.o_sh + d] = static_cast<uint16_t>(pk & 0xffffu);
}

template <bool kBf16, int D, bool kCluster, int kPerSm, bool kStep = false>
__global__ void __launch_bounds__(kDecThreads, kPerSm)
fox_decode_kernel(const DecodeParams p, const std::conditional_t<kStep, DecodeStep, char> step) {
  constexpr int LPR = D / 8, RPW = 32 / LPR;
  constexpr int kBatch = kDecWarps * RPW * kDecRows;   // keys a CTA takes per step
  __shared__ float s_bias[kDecTile];                   // (sum of the gates after key j, inside the range) * log2e
  __shared__ float s_scan[kDecWarps];
  __shared__ float s_m[kDecWarps], s_l[kDecWarps];
  __shared__ float s_acc[kDecWarps][D];
  __shared__ float s_res[D + 4];
  const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = lane % LPR, grp = lane / LPR;
  const int64_t bh = static_cast<int64_t>(b) * p.H + h;
  const int N = p.N;
  int lo = 0;
  if constexpr (kStep) {
    // Before the wait for the projections: what does not come from the kernel in front.  (A kernel of the chain lets the next
    // one start after its own wait, so everything in front of the projections has ended: mask, cache and states are final.)
    if (step.mask) {
      __shared__ long long s_n[kDecWarps];
      long long n = 0;
      for (int i = tid; i < N; i += kDecThreads) n += step.mask[static_cast<int64_t>(b) * N + i];
      for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
      if (lane == 0) s_n[warp] = n;
      __syncthreads();
      n = 0;
      for (int w = 0; w < kDecWarps; ++w) n += s_n[w];
      lo = static_cast<int>(max(min(static_cast<long long>(N) - n, static_cast<long long>(N)), 0LL));
    }
  } else {
    wait_for_kernel_in_front();
    // (what follows may start, and waits for this grid's end; but not another call's kernel, whose CTAs would take their places
    // around the last ones here, on fewer SMs)
    if (p.chained || !kCluster) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.seq_start) lo = static_cast<int>(p.seq_start[b]);
    if (p.start_index) {
      const int64_t si = p.start_index[bh];
      lo = max(lo, static_cast<int>(si < N ? si : N));
    }
    lo = max(min(lo, N), 0);
  }
  const int end = kStep ? N - 1 : N;   // (the token's own key is not read from the cache)
  const int span = max(end - lo, 0);
  const int per = (span + p.splits - 1) / p.splits;
  const int j0 = min(end, lo + split * per), j1 = min(end, j0 + per);

  const uint16_t* kb = p.k + b * p.k_sb + h * p.k_sh + sub * 8;
  const uint16_t* vb = p.v + b * p.v_sb + h * p.v_sh + sub * 8;
  const float* lam = !kStep && p.lam ? p.lam + bh * N : nullptr;
  const float* gate = p.gate + b * p.g_sb + h * p.g_sh;
  const float lam_q = lam ? lam[N - 1] : 0.f;
  float carry = 0.f;   // sum of the range's gates right of the current tile
  auto bias = [&](int t0, int n) {
    __syncthreads();
    if (lam) {
      for (int i = tid; i < n; i += kDecThreads) s_bias[i] = (lam_q - lam[t0 + i]) * kDecLog2e;
    } else {
      // thread t takes keys 4t .. 4t+3 counted from the right; exclusive scan of their gates in that order
      float g[4], own = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = n - 1 - (4 * tid + c);
        g[c] = i >= 0 ? gate[static_cast<int64_t>(t0 + i) * p.g_sn] : 0.f;
        own += g[c];
      }
      float incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      if (lane == 31) s_scan[warp] = incl;
      // (a gate of minus infinity cannot be taken off the sum again)
      const float left = __shfl_up_sync(0xffffffffu, incl, 1);
      __syncthreads();
      float before = own > -INFINITY ? carry + incl - own : lane ? carry + left : carry, total = 0.f;
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        if (w < warp) before += s_scan[w];
        total += s_scan[w];
      }
      carry += total;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = n - 1 - (4 * tid + c);
        if (i >= 0) s_bias[i] = before * kDecLog2e;
        before += g[c];
      }
    }
    __syncthreads();
  };
  uint4 kr[kDecRows], vr[kDecRows];
  auto load = [&](int t0, int n, int i0) {
#pragma unroll
    for (int u = 0; u < kDecRows; ++u) {
      const int i = min(i0 + (u * kDecWarps + warp) * RPW + grp, n - 1);
      kr[u] = *reinterpret_cast<const uint4*>(kb + static_cast<int64_t>(t0 + i) * p.k_st);
    }
#pragma unroll
    for (int u = 0; u < kDecRows; ++u) {
      const int i = min(i0 + (u * kDecWarps + warp) * RPW + grp, n - 1);
      vr[u] = *reinterpret_cast<const uint4*>(vb + static_cast<int64_t>(t0 + i) * p.v_st);
    }
  };

  float qv[8];
  float g_new = 0.f;
  const bool owner = kStep && split == p.splits - 1 && warp == 0;
  // kStep: [norm weights of q, k | gate bias], the states' key and value, which the token's replace
  __shared__ __align__(16) float s_w[kStep ? 2 * D + 1 : 1];
  __shared__ uint4 s_new[2][kStep ? LPR : 1];
  if constexpr (kStep) {
    const int C = p.H * D;
    for (int i = tid; i < 2 * D; i += kDecThreads)
      s_w[i] = i < D ? dec_load_any(step.wq, step.wq_dtype, h * D + i) : dec_load_any(step.wk, step.wk_dtype, h * D + i - D);
    if (tid == 0) s_w[2 * D] = step.bias ? dec_load_any(step.bias, step.bias_dtype, h) : 0.f;
    if (tid < 2 * LPR)
      s_new[tid / LPR][tid % LPR] = *reinterpret_cast<const uint4*>((tid < LPR ? step.k_state : step.v_state) +
                                                                    static_cast<int64_t>(b) * C + h * D + (tid % LPR) * 8);
    if (j1 > j0) {   // the first tile's gates and rows, and a request for what follows them
      const int t0 = max(j0, j1 - kDecTile);
      // (32 KB of each: 444 CTAs' requests stay well inside L2)
      const uint32_t o = tid * 4096u, bytes = min(static_cast<uint32_t>(j1 - t0) * (D * 2), 32768u);
      if (o < bytes) {
        const int64_t at = (bh * step.cap + t0) * D;
        l2_request(reinterpret_cast<const char*>(step.k_cache + at) + o, min(4096u, bytes - o));
        l2_request(reinterpret_cast<const char*>(step.v_cache + at) + o, min(4096u, bytes - o));
      }
      load(t0, j1 - t0, 0);
      bias(t0, j1 - t0);
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const float inv_d = 1.f / static_cast<float>(D);
    const int ch = h * D + sub * 8;
    const float* y = step.y + b * step.ld;
    dec_load8(y + ch, qv);
    if (owner) {   // the token's key, value and gate; its projections replace the states
      const int64_t so = static_cast<int64_t>(b) * C + ch;
      float kp[8], vp[8], k_new[8], v_new[8];
      dec_load8(y + C + ch, k_new);
      dec_load8(y + 2 * C + ch, v_new);
      const float f = y[4 * C + h] + s_w[2 * D], mk = y[4 * C + p.H + h], mv = y[4 * C + 2 * p.H + h];
      dec_unpack<kBf16>(s_new[0][sub], kp);
      dec_unpack<kBf16>(s_new[1][sub], vp);
      const float ak = sigmoid_fp32(mk), av = sigmoid_fp32(mv);
      const uint4 k16 = dec_pack<kBf16>(k_new), v16 = dec_pack<kBf16>(v_new);
      dec_unpack<kBf16>(k16, k_new);
      dec_unpack<kBf16>(v16, v_new);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        k_new[c] = ak * kp[c] + (1.f - ak) * k_new[c];
        v_new[c] = av * vp[c] + (1.f - av) * v_new[c];
      }
      const float rk = dec_norm<LPR>(k_new, inv_d, step.eps);
#pragma unroll
      for (int c = 0; c < 8; ++c) k_new[c] *= rk * s_w[D + sub * 8 + c];
      const uint4 kn = dec_pack<kBf16>(k_new), vn = dec_pack<kBf16>(v_new);
      g_new = fminf(f, 0.f) - log1pf(expf(-fabsf(f)));
      if (grp == 0) {
        const int64_t row = (bh * step.cap + N - 1) * D + sub * 8;
        *reinterpret_cast<uint4*>(step.k_cache + row) = kn;
        *reinterpret_cast<uint4*>(step.v_cache + row) = vn;
        *reinterpret_cast<uint4*>(step.k_state + so) = k16;
        *reinterpret_cast<uint4*>(step.v_state + so) = v16;
      }
      if (lane == 0) step.g_cache[bh * step.cap + N - 1] = g_new;
      __syncwarp();
      if (grp == 0) {   // (read by this warp)
        s_new[0][sub] = kn;
        s_new[1][sub] = vn;
      }
    }
    const float rq = dec_norm<LPR>(qv, inv_d, step.eps);
#pragma unroll
    for (int c = 0; c < 8; ++c) qv[c] *= rq * s_w[sub * 8 + c];
    const uint4 q16 = dec_pack<kBf16>(qv);
    dec_unpack<kBf16>(q16, qv);
  } else {
    dec_unpack<kBf16>(*reinterpret_cast<const uint4*>(p.q + b * p.q_sb + h * p.q_sh + sub * 8), qv);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) qv[c] *= p.qk_scale;

  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = 0.f;
  auto use = [&](int n, int i0) {
    float s[kDecRows], mx = m;
#pragma unroll
    for (int u = 0; u < kDecRows; ++u) {
      float kv[8];
      dec_unpack<kBf16>(kr[u], kv);
      float x = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) x = fmaf(qv[c], kv[c], x);
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      const int i = i0 + (u * kDecWarps + warp) * RPW + grp;
      s[u] = i < n ? x + s_bias[min(i, n - 1)] : -INFINITY;
      mx = fmaxf(mx, s[u]);
    }
    const float ref = mx == -INFINITY ? 0.f : mx;
    const float alpha = fast_exp2(m - ref);   // 0 when m was -inf
    m = mx;
    l *= alpha;
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] *= alpha;
#pragma unroll
    for (int u = 0; u < kDecRows; ++u) {
      const float w = fast_exp2(s[u] - ref);  // 0 past the end
      float vv[8];
      dec_unpack<kBf16>(vr[u], vv);
      l += w;
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = fmaf(w, vv[c], acc[c]);
    }
  };
  if (kStep && j1 > j0) use(min(j1 - j0, kDecTile), 0);
  for (int e = j1; e > j0; e -= kDecTile) {
    const int t0 = max(j0, e - kDecTile), n = e - t0;
    const bool begun = kStep && e == j1;   // (its gates and first rows came before the wait)
    if (!begun) bias(t0, n);
    for (int i0 = begun ? kBatch : 0; i0 < n; i0 += kBatch) {
      load(t0, n, i0);
      use(n, i0);
    }
  }
  if constexpr (kStep) {
    // The token's own key.  The others' logits lack its gate, which is taken off its logit instead.
    if (owner) {
      float kv[8], vv[8], x = 0.f;
      __syncwarp();
      dec_unpack<kBf16>(s_new[0][sub], kv);
      dec_unpack<kBf16>(s_new[1][sub], vv);
#pragma unroll
      for (int c = 0; c < 8; ++c) x = fmaf(qv[c], kv[c], x);
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (grp == 0 && lo < N) {
        // (at -1e30 the others have no share left; minus infinity would make this logit infinite and its weight NaN.  Without
        // others the gate has nothing to act on.)
        const float g2 = lo < end ? g_new * kDecLog2e : 0.f;
        float f_old, f_new;
        dec_join(m, l, x - (g2 < -1e30f ? -1e30f : g2), 1.f, f_old, f_new);
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = acc[c] * f_old + vv[c] * f_new;
      }
    }
  }

  // ---- join the lane groups of a warp, then the warps ----
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
    float a, c2;
    dec_join(m, l, m2, l2, a, c2);
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = acc[c] * a + __shfl_xor_sync(0xffffffffu, acc[c], o) * c2;
  }
  if (grp == 0) {
#pragma unroll
    for (int c = 0; c < 8; ++c) s_acc[warp][sub * 8 + c] = acc[c];
    if (sub == 0) {
      s_m[warp] = m;
      s_l[warp] = l;
    }
  }
  __syncthreads();
  float mx = -INFINITY;
#pragma unroll
  for (int w = 0; w < kDecWarps; ++w) mx = fmaxf(mx, s_m[w]);
  float lt = 0.f, x = 0.f;
#pragma unroll
  for (int w = 0; w < kDecWarps; ++w) {
    const float f = s_m[w] == -INFINITY ? 0.f : fast_exp2(s_m[w] - mx);
    lt = fmaf(s_l[w], f, lt);
    if (tid < D) x = fmaf(s_acc[w][tid], f, x);
  }
  if (p.splits == 1) {
    if (tid < D) dec_store<kBf16, D>(p, b, h, tid, x, lt);
    if (tid == 0 && p.L) p.L[bh] = lt > 0.f ? mx * 0.6931471805599453f + __logf(lt) : -INFINITY;
    return;
  }
  if constexpr (kCluster) {
    cg::cluster_group cluster = cg::this_cluster();
    if (tid < D) s_res[tid] = x;
    if (tid == 0) {
      s_res[D] = mx;
      s_res[D + 1] = lt;
      s_res[D + 2] = carry * kDecLog2e;
    }
    cluster.sync();
    if (split == 0) {
      // every remote value is asked for before the first is used
      float ms[kDecMaxCluster], ls[kDecMaxCluster], gs[kDecMaxCluster], os[kDecMaxCluster];
#pragma unroll
      for (int r = 0; r < kDecMaxCluster; ++r) {
        const float* rem = cluster.map_shared_rank(s_res, r < p.splits ? r : 0);
        ms[r] = rem[D];
        ls[r] = rem[D + 1];
        gs[r] = rem[D + 2];
        os[r] = rem[tid < D ? tid : 0];
      }
      float after = 0.f, top = -INFINITY;
#pragma unroll
      for (int r = kDecMaxCluster - 1; r >= 0; --r) {
        if (r < p.splits) {
          ms[r] += after;
          after += gs[r];
          top = fmaxf(top, ms[r]);
        }
      }
      float lsum = 0.f, osum = 0.f;
#pragma unroll
      for (int r = 0; r < kDecMaxCluster; ++r) {
        if (r < p.splits && ms[r] != -INFINITY) {
          const float f = fast_exp2(ms[r] - top);
          lsum = fmaf(ls[r], f, lsum);
          osum = fmaf(os[r], f, osum);
        }
      }
      if (tid < D) dec_store<kBf16, D>(p, b, h, tid, osum, lsum);
      if (tid == 0 && p.L) p.L[bh] = lsum > 0.f ? top * 0.6931471805599453f + __logf(lsum) : -INFINITY;
    }
    cluster.sync();   // (the others' shared memory is read until here)
  } else {
    float* out = p.part + (bh * p.splits + split) * (D + 4);
    if (tid < D) out[tid] = x;
    if (tid == 0) {
      out[D] = mx;
      out[D + 1] = lt;
      out[D + 2] = carry * kDecLog2e;
    }
  }
}

// Joins the ranges of one (b,h): their (m, l, gate total) staged in shared memory, suffix sums of the totals by one warp,
// then 256 / D groups of threads each sum every (256/D)-th range.
template <bool kBf16, int D>
__global__ void __launch_bounds__(256) fox_decode_merge_kernel(const DecodeParams p) {
  __shared__ float s_w[kDecMaxSplits], s_l[kDecMaxSplits], s_g[kDecMaxSplits], s_o[256], s_top, s_sum;
  wait_for_kernel_in_front();
  if (p.chained) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int64_t bh = static_cast<int64_t>(b) * p.H + h;
  const float* base = p.part + bh * p.splits * (D + 4);
  for (int s = tid; s < p.splits; s += 256) {
    const float* r = base + s * (D + 4) + D;
    s_w[s] = r[0];
    s_l[s] = r[1];
    s_g[s] = r[2];
  }
  __syncthreads();
  if (tid < 32) {
    float after = 0.f, top = -INFINITY;
    for (int s1 = p.splits; s1 > 0; s1 -= 32) {   // ranges s1 - 1 - lane, from the right
      const int s = s1 - 1 - tid;
      const float g = s >= 0 ? s_g[s] : 0.f;
      float incl = g;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, incl, o);
        if (tid >= o) incl += x;
      }
      const float left = __shfl_up_sync(0xffffffffu, incl, 1);   // (as for the keys' biases)
      if (s >= 0) {
        const float mm = g > -INFINITY ? s_w[s] + after + incl - g : s_w[s] + after + (tid ? left : 0.f);
        s_w[s] = mm;
        top = fmaxf(top, mm);
      }
      after += __shfl_sync(0xffffffffu, incl, 31);
    }
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    float sum = 0.f;
    for (int s = tid; s < p.splits; s += 32) {
      const float w = s_w[s] == -INFINITY ? 0.f : fast_exp2(s_w[s] - top);
      s_w[s] = w;
      sum = fmaf(s_l[s], w, sum);
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (tid == 0) {
      s_top = top;
      s_sum = sum;
    }
  }
  __syncthreads();
  constexpr int kGroups = 256 / D;
  const int d = tid % D, g0 = tid / D;
  float x = 0.f;
#pragma unroll 4
  for (int s = g0; s < p.splits; s += kGroups) {
    const float w = s_w[s];
    if (w != 0.f) x = fmaf(base[s * (D + 4) + d], w, x);
  }
  s_o[tid] = x;
  __syncthreads();
  if (tid < D) {
#pragma unroll
    for (int g = 1; g < kGroups; ++g) x += s_o[g * D + tid];
    dec_store<kBf16, D>(p, b, h, tid, x, s_sum);
  }
  if (tid == 0) p.L[bh] = s_sum > 0.f ? s_top * 0.6931471805599453f + __logf(s_sum) : -INFINITY;
}

// A launch that begins while a product with much shared memory ends would find next to no L1, which its loads in flight need
// (see fox_step.cu); one with long ranges waits for SMs that it can split anew.  Short ones are over before that pays: 24 (b,h) of
// 250 keys a range 32.5 us a layer, 33.8 so; 192 of 2000 97 and 89, of 6000 178 and 148; 96 of 10000 235 and 185.  (Head dims
// 16 and 32 are bound by their instructions: 160 of 6000 keys 48 and 50.)  Clusters that need nearly every place of their wave, and
// those of eight, find them too late then: 80 x 5 of 2400 keys a range 82 and 88, 48 x 8 of 750, head dim 128, 92 and 99.  Not so the
// clusters of two that come four CTAs to an SM, 446 to 540 of them: two layers of 240 (b,h) of 4200 keys 205 us without, 187 so; of 256 of 3000 181
// and 166, of 6000 256 and 225; 512 single ranges of 4200 447 and 437.
static int long_ranges(cudaLaunchAttribute* attr, const DecodeParams& p, int64_t B, int D) {
  const int64_t ctas = B * p.H * p.splits;
  if (D < 64 || static_cast<int64_t>(p.N) * D < static_cast<int64_t>(p.splits) * kDecLongRange) return 0;
  if (p.splits > 1 && (p.splits == kDecMaxCluster || (p.splits < kDecMaxCluster && ctas > kDecManyClusters && ctas <= kDecSlots))) return 0;
  attr->id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  attr->val.sharedMemCarveout = 20;   // (of 228 KB, where four CTAs take 9 to 12 each)
  return 1;
}

template <bool kBf16, int D>
static int launch_step(const DecodeParams& p, const DecodeStep& step, int64_t B, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.splits, (unsigned)p.H, (unsigned)B);
  cfg.blockDim = dim3(kDecThreads);
  cfg.stream = st;
  cudaLaunchAttribute attrs[3] = {};
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  int n = 1 + long_ranges(&attrs[1], p, B, D);
  if (p.splits > 1) {
    attrs[n].id = cudaLaunchAttributeClusterDimension;
    attrs[n].val.clusterDim.x = (unsigned)p.splits;
    attrs[n].val.clusterDim.y = attrs[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, fox_decode_kernel<kBf16, D, true, kDecPerSm, true>, p, step) == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

// Behind another kernel without waiting for the stream: 2.1 us less a call, whatever its length (back to back, before -> now: 24 (b,h) of
// 250 keys 6.2 -> 4.5 us, 32 of 2048 x 128 13.6 -> 11.6, 24 of 65536 x 64 69.8 -> 67.7, 256 of 4099 x 128 90.4 -> 88.2, 3072 of 1500 x 64 184.3 ->
// 181.9; pruned, with its prefix sums and indices, 64 of 4096 x 128 16.5 -> 12.3).
template <bool kBf16, int D, int kPerSm>
static int launch_decode_at(const DecodeParams& p, int64_t B, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.splits, (unsigned)p.H, (unsigned)B);
  cfg.blockDim = dim3(kDecThreads);
  cfg.stream = st;
  cudaLaunchAttribute attrs[3] = {}, attr{};
  int n = 0;
  attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[n++].val.programmaticStreamSerializationAllowed = 1;
  if (p.chained) n += long_ranges(&attrs[n], p, B, D);
  cfg.attrs = attrs;
  if (p.splits <= kDecMaxCluster) {
    if (p.splits > 1) {
      attrs[n].id = cudaLaunchAttributeClusterDimension;
      attrs[n].val.clusterDim.x = (unsigned)p.splits;
      attrs[n].val.clusterDim.y = attrs[n].val.clusterDim.z = 1;
      ++n;
    }
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, fox_decode_kernel<kBf16, D, true, kPerSm>, p, '\0') == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
  }
  cfg.numAttrs = n;
  if (cudaLaunchKernelEx(&cfg, fox_decode_kernel<kBf16, D, false, kPerSm>, p, '\0') != cudaSuccess) return FOX_ERR_LAUNCH;
  cfg.gridDim = dim3((unsigned)p.H, (unsigned)B);
  cfg.blockDim = dim3(256);
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fox_decode_merge_kernel<kBf16, D>, p) == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

// Ranges per (b,h), so that the CTAs come in whole waves: 444 (three per SM) where a second kernel merges, 400 where clusters
// do (those find no room on the last SMs of a GPC: 72 x 5 CTAs 36.1 us, 72 x 6 52.1).  A (b,h) that is one range of a wave
// takes the next wave too where its shorter ranges pay for the second start, some 600 keys (256 (b,h) of 4099 keys, head dim
// 128: one range 105 us, three 94; of 1024 keys: 28.5 and 31.3).  Eight ranges need no merge kernel, which is worth some 120
// keys.  At least 128 keys a range.  Four CTAs per SM on average, as before, left a last wave nearly empty: 24 x 65536 keys of
// head dim 64 in 25 ranges 81.4 us, in 18 67.2; 48 x 8192 25.7 -> 22.6; 192 x 2048 26.2 -> 22.0; 72 x 5000 of 128 41.3 -> 36.1.
//
// Four per SM (64 registers instead of 80, no spills) share the same bandwidth, so that a range takes a third longer; they are
// taken where the waves are fewer by so much that this pays, counted in keys with 600 for a wave's start: 512 (b,h) of 4000
// keys of 128 in one wave instead of three 192 -> 162 us, of 64 102 -> 86; 256 of 4099 of 128 in one instead of two 98 -> 91, of 2048
// 54 -> 48.  With as many waves they pay where they fill one that three leave half empty (a (b,h) in two ranges instead of one) and
// the ranges are long: 256 of 1500 of 128 43 -> 37, but of 1000 of 64 17.8 and 18.5, 176 of 1200 16.4 and 17.2.  Three ranges
// instead of two in the same wave are not taken, though the one shape timed gained (144 of 2600 of 64 24.7 and 22.7).  Else they are no
// faster or slower: 384 of 8000 of 64 130 and 135, 32 of 3000 13.7 and 14.3, 4 of 30000 of 128 21.2 and 22.5, 768 of 2500 of 64 86 and 91; 24 x
// 65536 70.0 and 70.0.  (Head dim 16, whose ranges are bound by instructions, loses where they are shortest: 256 of 1300 10.4 and 11.0.)
struct DecodePlan {
  int64_t splits;
  int per_sm;
};
static int64_t waves_of(int64_t ctas, int64_t slots) { return (ctas + slots - 1) / slots; }
static int64_t fit_splits(int64_t bh, int64_t N, int64_t slots, int64_t cluster_slots) {
  auto fit = [&](int64_t waves) {
    const int64_t s = waves * slots / bh;
    return s > kDecMaxCluster ? s : waves * cluster_slots / bh > 1 ? waves * cluster_slots / bh : int64_t{1};
  };
  const int64_t waves = waves_of(bh, slots);
  int64_t s = fit(waves);
  if (s == 1) {
    const int64_t next = fit(waves + 1);
    if ((waves + 1) * (N / next + kDecStartKeys) < waves * (N + kDecStartKeys)) s = next;
  } else if (s > kDecMaxCluster && N / kDecMaxCluster < N / s + kDecMergeKeys) {
    s = kDecMaxCluster;
  }
  const int64_t most = (N + kDecLeastKeys - 1) / kDecLeastKeys;
  if (s > most) s = most;
  if (s > kDecMostSplits) s = kDecMostSplits;
  return s < 1 ? 1 : s;
}
static DecodePlan decode_plan(int64_t bh, int64_t N) {
  const int64_t s3 = fit_splits(bh, N, kDecSlots, kDecClusterSlots), s4 = fit_splits(bh, N, kDecMoreSlots, kDecMoreClusterSlots);
  auto waves = [&](int64_t s, int64_t slots, int64_t cluster_slots) { return waves_of(bh * s, s > 1 && s <= kDecMaxCluster ? cluster_slots : slots); };
  const int64_t w3 = waves(s3, kDecSlots, kDecClusterSlots), w4 = waves(s4, kDecMoreSlots, kDecMoreClusterSlots);
  const int64_t t3 = w3 * (N / s3 + kDecStartKeys), t4 = w4 * (N / s4 * kDecMorePerSm / kDecPerSm + kDecStartKeys);
  const bool more = w4 < w3 ? t4 < t3 : w4 == w3 && s3 == 1 && t4 < t3 - t3 / 20 && N / s4 >= kDecMoreLeastKeys;
  return more ? DecodePlan{s4, kDecMorePerSm} : DecodePlan{s3, kDecPerSm};
}
template <bool kBf16, int D>
static int launch_decode(const DecodeParams& p, int64_t B, cudaStream_t st) {
  const DecodePlan plan = decode_plan(B * p.H, p.N);   // (a caller may ask for other ranges than its)
  return plan.per_sm == kDecMorePerSm && plan.splits == p.splits ? launch_decode_at<kBf16, D, kDecMorePerSm>(p, B, st)
                                                                 : launch_decode_at<kBf16, D, kDecPerSm>(p, B, st);
}

}  // namespace fox

using namespace fox;

extern "C" int64_t fox_attn_decode_splits(int64_t B, int64_t H, int64_t N) {
  if (B * H <= 0) return 1;   // (fox_attn_decode refuses such a call)
  return decode_plan(B * H, N).splits;
}

extern "C" int64_t fox_attn_decode_per_sm(int64_t B, int64_t H, int64_t N) { return B * H <= 0 ? kDecPerSm : decode_plan(B * H, N).per_sm; }

// (none where the ranges are merged inside a cluster)
extern "C" int64_t fox_attn_decode_workspace_floats(int64_t B, int64_t H, int64_t D, int64_t splits) {
  return splits <= kDecMaxCluster ? 1 : B * H * splits * (D + 4);
}

static int decode(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t N, int64_t D, const fox_tensor4* q,
                  const fox_tensor4* k, const fox_tensor4* v, DecodeParams p, float sm_scale, const fox_tensor4* o, float* L,
                  float* workspace, int64_t splits) {
  if (!q || !k || !v || !o || !q->ptr || !k->ptr || !v->ptr || !o->ptr || !L || !workspace) return FOX_ERR_BAD_ARG;
  if (B <= 0 || H <= 0 || N <= 0 || N > 2147483647LL - kDecTile || H > 65535 || B > 65535 || splits <= 0 || splits > kDecMaxSplits)
    return FOX_ERR_BAD_ARG;
  if (D != 16 && D != 32 && D != 64 && D != 128) return FOX_ERR_HEAD_DIM;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  auto bad = [](const fox_tensor4* t) {
    return reinterpret_cast<uintptr_t>(t->ptr) % 16 || t->sb % 8 || t->sh % 8 || t->st % 8;
  };
  if (bad(q) || bad(k) || bad(v)) return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  p.q = (const uint16_t*)q->ptr; p.k = (const uint16_t*)k->ptr; p.v = (const uint16_t*)v->ptr;
  p.q_sb = q->sb; p.q_sh = q->sh; p.k_sb = k->sb; p.k_sh = k->sh; p.k_st = k->st;
  p.v_sb = v->sb; p.v_sh = v->sh; p.v_st = v->st;
  p.part = workspace;
  p.o = (uint16_t*)o->ptr; p.o_sb = o->sb; p.o_sh = o->sh;
  p.L = L;
  p.H = (int)H; p.N = (int)N; p.splits = (int)splits;
  p.qk_scale = sm_scale * kDecLog2e;
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == FOX_DTYPE_BF16;
  switch (D) {
    case 16: return bf ? launch_decode<true, 16>(p, B, st) : launch_decode<false, 16>(p, B, st);
    case 32: return bf ? launch_decode<true, 32>(p, B, st) : launch_decode<false, 32>(p, B, st);
    case 64: return bf ? launch_decode<true, 64>(p, B, st) : launch_decode<false, 64>(p, B, st);
    default: return bf ? launch_decode<true, 128>(p, B, st) : launch_decode<false, 128>(p, B, st);
  }
}

extern "C" int fox_attn_decode(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t N, int64_t D,
                               const fox_tensor4* q, const fox_tensor4* k, const fox_tensor4* v,
                               const float* log_lambda, const int64_t* seq_start, const int64_t* start_index,
                               float sm_scale, const fox_tensor4* o, float* L, float* workspace, int64_t splits) {
  if (!log_lambda) return FOX_ERR_BAD_ARG;
  DecodeParams p{};
  p.lam = log_lambda;
  p.seq_start = seq_start;
  p.start_index = start_index;
  return decode(device, stream, dtype, B, H, N, D, q, k, v, p, sm_scale, o, L, workspace, splits);
}

extern "C" int fox_attn_decode_gates(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t N, int64_t D,
                                     const fox_tensor4* q, const fox_tensor4* k, const fox_tensor4* v, const float* log_fgate,
                                     int64_t sb, int64_t sh, int64_t sn, const int64_t* seq_start, float sm_scale,
                                     const fox_tensor4* o, float* L, float* workspace, int64_t splits, int programmatic) {
  if (!log_fgate) return FOX_ERR_BAD_ARG;
  DecodeParams p{};
  p.gate = log_fgate;
  p.chained = programmatic != 0;
  p.g_sb = sb; p.g_sh = sh; p.g_sn = sn;
  p.seq_start = seq_start;
  return decode(device, stream, dtype, B, H, N, D, q, k, v, p, sm_scale, o, L, workspace, splits);
}

// Ranges of fox_step_attn, or 0 where fox_step_mix and fox_attn_decode_gates are the better way: more CTAs than a wave (16
// sequences x 32 heads of 8192 keys 694 us for two layers, 674 apart), or ranges so long that more than eight of them pay for
// the two launches more (24 heads of 8000 keys 105 and 101 us).
extern "C" int64_t fox_step_attn_splits(int64_t B, int64_t H, int64_t N) {
  if (B <= 0 || H <= 0) return 0;
  const int64_t s = fit_splits(B * H, N, kDecSlots, kDecClusterSlots);
  if (B * H * s > kDecSlots) return 0;
  return s <= kDecMaxCluster ? s : N <= 8 * 768 ? 8 : 0;
}

extern "C" int fox_step_attn(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t D, const float* y, int64_t ld,
                             const void* wq, int wq_dtype, const void* wk, int wk_dtype, float eps, const void* bias, int bias_dtype,
                             const int64_t* mask, void* k_state, void* v_state, void* k_cache, void* v_cache, float* g_cache,
                             int64_t capacity, int64_t pos, float sm_scale, void* o, int64_t splits) {
  if (!y || !wq || !wk || !k_state || !v_state || !k_cache || !v_cache || !g_cache || !o || B <= 0 || H <= 0 || B > 65535 || H > 65535 ||
      pos < 0 || pos >= capacity || pos >= 2147483647LL - kDecTile || splits <= 0 || splits > kDecMaxCluster)
    return FOX_ERR_BAD_ARG;
  if (D != 16 && D != 32 && D != 64 && D != 128) return FOX_ERR_HEAD_DIM;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if (ld % 4 || ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(k_state) | reinterpret_cast<uintptr_t>(v_state) |
                  reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) % 16))
    return FOX_ERR_ALIGNMENT;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  DecodeParams p{};
  p.k = (const uint16_t*)k_cache; p.v = (const uint16_t*)v_cache;
  p.k_sb = p.v_sb = H * capacity * D; p.k_sh = p.v_sh = capacity * D; p.k_st = p.v_st = D;
  p.gate = g_cache; p.g_sb = H * capacity; p.g_sh = capacity; p.g_sn = 1;
  p.o = (uint16_t*)o; p.o_sb = H * D; p.o_sh = D;
  p.H = (int)H; p.N = (int)(pos + 1); p.splits = (int)splits;
  p.qk_scale = sm_scale * kDecLog2e;
  const DecodeStep s{y, ld, wq, wk, bias, wq_dtype, wk_dtype, bias_dtype, eps, mask, (uint16_t*)k_state, (uint16_t*)v_state,
                     (uint16_t*)k_cache, (uint16_t*)v_cache, g_cache, capacity};
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == FOX_DTYPE_BF16;
  switch (D) {
    case 16: return bf ? launch_step<true, 16>(p, s, B, st) : launch_step<false, 16>(p, s, B, st);
    case 32: return bf ? launch_step<true, 32>(p, s, B, st) : launch_step<false, 32>(p, s, B, st);
    case 64: return bf ? launch_step<true, 64>(p, s, B, st) : launch_step<false, 64>(p, s, B, st);
    default: return bf ? launch_step<true, 128>(p, s, B, st) : launch_step<false, 128>(p, s, B, st);
  }
}
