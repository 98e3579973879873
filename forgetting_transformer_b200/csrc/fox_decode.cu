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
constexpr int64_t kDecSlots = 444, kDecClusterSlots = 400;                            // CTAs of a wave
constexpr int64_t kDecStartKeys = 600, kDecMergeKeys = 120, kDecLeastKeys = 128;      // (at fox_attn_decode_splits)
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
  bool pdl;                    // launched with programmatic stream serialization
};

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

template <bool kBf16, int D, bool kCluster>
__global__ void __launch_bounds__(kDecThreads, 3)
fox_decode_kernel(const DecodeParams p) {
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
  // (no effect without programmatic serialization; what follows may start, and waits for this grid's end)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int lo = p.seq_start ? static_cast<int>(p.seq_start[b]) : 0;
  if (p.start_index) {
    const int64_t si = p.start_index[bh];
    lo = max(lo, static_cast<int>(si < N ? si : N));
  }
  lo = max(min(lo, N), 0);
  const int span = N - lo;
  const int per = (span + p.splits - 1) / p.splits;
  const int j0 = min(N, lo + split * per), j1 = min(N, j0 + per);

  float qv[8];
  dec_unpack<kBf16>(*reinterpret_cast<const uint4*>(p.q + b * p.q_sb + h * p.q_sh + sub * 8), qv);
#pragma unroll
  for (int c = 0; c < 8; ++c) qv[c] *= p.qk_scale;
  const uint16_t* kb = p.k + b * p.k_sb + h * p.k_sh + sub * 8;
  const uint16_t* vb = p.v + b * p.v_sb + h * p.v_sh + sub * 8;
  const float* lam = p.lam ? p.lam + bh * N : nullptr;
  const float* gate = p.gate + b * p.g_sb + h * p.g_sh;
  const float lam_q = lam ? lam[N - 1] : 0.f;

  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) acc[c] = 0.f;
  float carry = 0.f;   // sum of the range's gates right of the current tile
  for (int e = j1; e > j0; e -= kDecTile) {
    const int t0 = max(j0, e - kDecTile), n = e - t0;
    // ---- bias of the tile's keys ----
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
      __syncthreads();
      float before = carry + incl - own, total = 0.f;
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
    // ---- the tile's keys ----
    for (int i0 = 0; i0 < n; i0 += kBatch) {
      uint4 kr[kDecRows], vr[kDecRows];
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
    if (tid == 0) p.L[bh] = lt > 0.f ? mx * 0.6931471805599453f + __logf(lt) : -INFINITY;
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
      float ms[kDecMaxCluster], after = 0.f, top = -INFINITY;
#pragma unroll
      for (int r = kDecMaxCluster - 1; r >= 0; --r) {
        ms[r] = -INFINITY;
        if (r < p.splits) {
          const float* rem = cluster.map_shared_rank(s_res, r);
          ms[r] = rem[D] + after;
          after += rem[D + 2];
          top = fmaxf(top, ms[r]);
        }
      }
      float lsum = 0.f, osum = 0.f;
#pragma unroll
      for (int r = 0; r < kDecMaxCluster; ++r) {
        if (r < p.splits && ms[r] != -INFINITY) {
          const float* rem = cluster.map_shared_rank(s_res, r);
          const float f = fast_exp2(ms[r] - top);
          lsum = fmaf(rem[D + 1], f, lsum);
          if (tid < D) osum = fmaf(rem[tid], f, osum);
        }
      }
      if (tid < D) dec_store<kBf16, D>(p, b, h, tid, osum, lsum);
      if (tid == 0) p.L[bh] = lsum > 0.f ? top * 0.6931471805599453f + __logf(lsum) : -INFINITY;
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
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
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
      if (s >= 0) {
        const float mm = s_w[s] + after + incl - g;
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

template <bool kBf16, int D>
static int launch_decode(const DecodeParams& p, int64_t B, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.splits, (unsigned)p.H, (unsigned)B);
  cfg.blockDim = dim3(kDecThreads);
  cfg.stream = st;
  cudaLaunchAttribute attrs[2] = {}, attr{};
  int n = 0;
  if (p.pdl) {
    attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attrs;
  if (p.splits <= kDecMaxCluster) {
    if (p.splits > 1) {
      attrs[n].id = cudaLaunchAttributeClusterDimension;
      attrs[n].val.clusterDim.x = (unsigned)p.splits;
      attrs[n].val.clusterDim.y = attrs[n].val.clusterDim.z = 1;
      ++n;
    }
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, fox_decode_kernel<kBf16, D, true>, p) == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
  }
  cfg.numAttrs = n;
  if (cudaLaunchKernelEx(&cfg, fox_decode_kernel<kBf16, D, false>, p) != cudaSuccess) return FOX_ERR_LAUNCH;
  cfg.gridDim = dim3((unsigned)p.H, (unsigned)B);
  cfg.blockDim = dim3(256);
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fox_decode_merge_kernel<kBf16, D>, p) == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

}  // namespace fox

using namespace fox;

// Ranges per (b,h), so that the CTAs come in whole waves: 444 (three per SM) where a second kernel merges, 400 where clusters
// do (those find no room on the last SMs of a GPC: 72 x 5 CTAs 36.1 us, 72 x 6 52.1).  A (b,h) that is one range of a wave
// takes the next wave too where its shorter ranges pay for the second start, some 600 keys (256 (b,h) of 4099 keys, head dim
// 128: one range 105 us, three 94; of 1024 keys: 28.5 and 31.3).  Eight ranges need no merge kernel, which is worth some 120
// keys.  At least 128 keys a range.  Four CTAs per SM on average, as before, left a last wave nearly empty: 24 x 65536 keys of
// head dim 64 in 25 ranges 81.4 us, in 18 67.2; 48 x 8192 25.7 -> 22.6; 192 x 2048 26.2 -> 22.0; 72 x 5000 of 128 41.3 -> 36.1.
extern "C" int64_t fox_attn_decode_splits(int64_t B, int64_t H, int64_t N) {
  const int64_t bh = B * H;
  auto fit = [&](int64_t waves) {
    const int64_t s = waves * kDecSlots / bh;
    return s > kDecMaxCluster ? s : waves * kDecClusterSlots / bh > 1 ? waves * kDecClusterSlots / bh : int64_t{1};
  };
  const int64_t waves = (bh + kDecSlots - 1) / kDecSlots;
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
  p.pdl = programmatic != 0;
  p.g_sb = sb; p.g_sh = sh; p.g_sn = sn;
  p.seq_start = seq_start;
  return decode(device, stream, dtype, B, H, N, D, q, k, v, p, sm_scale, o, L, workspace, splits);
}
