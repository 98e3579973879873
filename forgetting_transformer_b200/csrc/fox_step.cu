// One generated token through a FoX-Pro block, for up to 16 sequences: the matrix-vector products with the norms, the
// gate, SwiGLU and the residual adds folded into them, and the single-token token shift with the cache append.
//
// The modules upstream's generation loop runs for T = 1
// (src/forgetting_transformer/model/forgetting_transformer/modeling_forgetting_transformer.py:44-95, 296-430, 505-516):
//   1. h = rmsnorm(x); [q | k | v | ogate | fgate | k mix | v mix] = h W^T         fox_step_product, rmsnorm -> fp32
//   2. token shift of k, v with the kept projections, norms of q, k, cache append    fox_step_mix
//   3. attention against the cache                                                   fox_attn_decode_gates
//   4. z = x + (headnorm(o) * w * sigmoid(ogate)) Wo^T                               fox_step_product, gated norm -> + x
//   5. a = swiglu(rmsnorm(z) Wg^T)                                                   fox_step_product, rmsnorm -> swiglu
//   6. y = z + a Wd^T                                                                fox_step_product, plain -> + z
//
// Steps 2 and 3 are one kernel (fox_step_attn, fox_decode.cu) where a cluster can merge the keys' ranges.
//
// Bound by latency: a layer of hidden 1536 reads 61 MB of weights (9 us) through five kernels that wait for one another.  A CTA
// takes 8 rows of W; its 8 warps split K in interleaved blocks of 32 columns and join their sums in shared memory.
// The products are mma.sync m16n8k16 with the sequences (padded to 16) as A and the 8 weight rows as B: the matrix
// units cost nothing here, and 2 x 16 fused multiply-adds per weight on the CUDA cores would bound the kernel above 4
// sequences; tcgen05's 128-row tiles would be idle for all but a sixteenth.  The order of K inside a block of 32 is free,
// so lane (g, t) holds the 16 bytes at columns 8t .. 8t+7 of row g and feeds them to two instructions.
//
// The weights' rows come by bulk copies into shared memory (kSmem).  Through registers, as large batches still take them,
// a CTA held 64 to 128 registers a thread and the 512 and 777 CTAs of the gate and first products ran in two waves, the
// second of which began its loads where the first ended: 40 us a layer of hidden 1536 with 2000 keys, 33 now.
//
// Every kernel is launched with programmatic stream serialization.  The products behind the first request their weights
// before they wait for the kernel in front, which does not write them, so that the load latency and the launch hide behind
// it; the gate product's CTAs leave no shared memory for the next one's, so they ask for its weights in L2.  Each lets the next
// one start only after its own wait: a kernel's early reads then come after everything in front of its predecessor has
// ended.  The first product follows a kernel of someone else's, which may have written the weights, and copies them after
// the wait; what it asks for before is only brought into L2, where a later write still finds it.
#include <algorithm>

#include "fox_common.cuh"
#include "fox_host.h"

namespace fox {

constexpr int kStepThreads = 256, kStepWarps = 8;
constexpr int kStepAhead = 8;    // blocks of 32 columns a warp has in flight
constexpr int kStepMats = 7;
constexpr uint32_t kStepChunk = 4096;         // bytes of one request for what a later product reads
// The most that is asked for ahead: of more, L2 (126 MB) holds too little until it is read (2048 channels, intermediate size 16384,
// 67 MB: 82 us a layer, without 88; 24576, 100 MB: 125 and 124; 32768, 134 MB: 139 and 135).
constexpr int64_t kStepAheadMost = 96 << 20;
constexpr int kStepEarly = 2 * kSms;          // CTAs that request the first product's weights
// Input and weights of a CTA that may lie in shared memory together; more goes through registers.  (16 sequences of 1536 channels:
// the gate product would need 99 KB, and a layer takes 126 us so, 114 through registers; 2 sequences' down product, 83 KB: 59
// and 61 us a layer.)
constexpr size_t kStepSmem = 88 * 1024;
constexpr int kStepWaitSite = 91;
constexpr int64_t kSmSmem = 228 * 1024;       // of an SM
constexpr int64_t kStepStatic = 10 * 1024;    // of a CTA beside input and weights: the sums' arrays and the system's share
// A down product of so many weights, through registers behind a gate product through shared memory, waits for SMs with room for
// its loads in L1 if its inputs leave a fifth (a layer of 2048 channels, intermediate size 16384: 82 -> 64 us, two sequences 88 ->
// 71, five, whose inputs leave none, 113 -> 118; 12288: 66 -> 56; of 5632 the wait costs more than it gives: five 64.5 -> 67.8).
constexpr int64_t kStepBigWeights = 16 << 20;

enum StepInput { kInRms = 0, kInGated = 1, kInPlain = 2 };
enum StepOutput { kOutFp32 = 0, kOutAdd16 = 1, kOutSwiglu = 2, kOutAdd32 = 3 };

struct StepParams {
  const uint16_t* w[kStepMats];   // (rows[i], K) each, contiguous
  int rows[kStepMats], tile0[kStepMats + 1], n_mats;
  int B, K, D;
  int w_dtype;                    // of norm_w: FOX_DTYPE_*
  const void* x;                  // kInRms: (B,K) 16-bit or fp32 (x_fp32); kInGated: o (B,K) 16-bit; kInPlain: (B,K) 16-bit
  bool x_fp32;
  const float* gate;              // kInGated: output gate, row stride gate_ld
  int64_t gate_ld;
  const void* norm_w;             // (K)
  float eps;
  void* out;                      // kOutFp32: (B, ldo) fp32; kOutAdd16: fp32 (B, ldo); kOutSwiglu / kOutAdd32: 16-bit (B, ldo)
  int64_t ldo;
  const void* res;                // kOutAdd16: (B, ldo) 16-bit; kOutAdd32: (B, ldo) fp32
  int half;                       // kOutSwiglu: rows of each half
  const char* ahead;              // what a later product reads (16-byte aligned), or nullptr
  uint64_t ahead_bytes;           // (a multiple of 16)
  int* status;                    // where a wait that runs out is recorded; nullptr: weights through registers
};

// Where the k-th request of a thread begins in what a later product reads.  In 64 bits: 256 threads of 4096 CTAs, the grid of an
// intermediate size of 32768, ask for 2^32 bytes in one round.
__host__ __device__ __forceinline__ uint64_t step_ahead_at(uint64_t grid, uint64_t block, uint64_t thread, uint64_t k) {
  return ((k * kStepThreads + thread) * grid + block) * kStepChunk;
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint4 ldg_stream(const uint16_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <bool kBf16>
__device__ __forceinline__ void step_mma(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <bool kBf16>
__device__ __forceinline__ void unpack8s(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = unpack2<kBf16>(w[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}
template <bool kBf16>
__device__ __forceinline__ uint4 pack8s(const float* f) {
  return make_uint4(pack2<kBf16>(f[0], f[1]), pack2<kBf16>(f[2], f[3]), pack2<kBf16>(f[4], f[5]), pack2<kBf16>(f[6], f[7]));
}
// eight norm weights of any of the three types
__device__ __forceinline__ void load_w8(const void* w, int dtype, int c, float* f) {
  if (dtype == FOX_DTYPE_FP32) {
    const float4 a = static_cast<const float4*>(w)[2 * c], b = static_cast<const float4*>(w)[2 * c + 1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  } else if (dtype == FOX_DTYPE_BF16) {
    unpack8s<true>(static_cast<const uint4*>(w)[c], f);
  } else {
    unpack8s<false>(static_cast<const uint4*>(w)[c], f);
  }
}
template <bool kBf16>
__device__ __forceinline__ void load_x8(const StepParams& p, int b, int c, float* f) {
  if (p.x_fp32) {
    const float4* q = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + static_cast<int64_t>(b) * p.K) + 2 * c;
    const float4 u = q[0], v = q[1];
    f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w; f[4] = v.x; f[5] = v.y; f[6] = v.z; f[7] = v.w;
  } else {
    unpack8s<kBf16>(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.x) + static_cast<int64_t>(b) * p.K)[c], f);
  }
}

// bytes between two rows of weights in shared memory: 64 modulo 128, so that eight rows' pieces of 64 bytes meet no bank twice
__host__ __device__ __forceinline__ uint32_t step_row_bytes(int K) { return K * 2 + (K % 64 ? 0 : 64); }

template <bool kBf16, int kIn, int kOut, bool kSmem>
__global__ void __launch_bounds__(kStepThreads)
fox_step_product_kernel(const StepParams p) {
  constexpr int NT = kOut == kOutSwiglu ? 2 : 1;   // 8-row tiles of a CTA
  extern __shared__ uint4 s_x[];                   // (B, stride) chunks of 8: the normalised input in 16 bits
  __shared__ float s_red[kStepWarps][NT][128];
  __shared__ float s_ss[kStepWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int chunks = p.K / 8, stride = (chunks + 7) / 8 * 8 + 4;   // (rows 4 chunks apart modulo 8: no bank conflicts)
  const int nkb = p.K / 32;

  int mat = 0;
  while (mat + 1 < p.n_mats && static_cast<int>(blockIdx.x) >= p.tile0[mat + 1]) ++mat;
  const int row0 = (static_cast<int>(blockIdx.x) - p.tile0[mat]) * 8;
  const uint16_t* wp[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i)
    wp[i] = p.w[mat] + static_cast<int64_t>(min(row0 + g, p.rows[mat] - 1) + i * p.half) * p.K + t * 8;

  const uint32_t w_row = step_row_bytes(p.K);
  uint8_t* s_w = reinterpret_cast<uint8_t*>(s_x + p.B * stride);   // kSmem: (NT * 8 rows)
  __shared__ uint64_t bar_w;
  __shared__ int abort_flag;
  if constexpr (kSmem) {
    if (tid == 0) {
      abort_flag = 0;
      mbar_init(&bar_w, 1);
      mbar_fence_init();
      mbar_expect_tx(&bar_w, NT * 8 * p.K * 2);
    }
    __syncwarp();
  }
  auto copy = [&] {   // a lane of the first warp asks for a row
    if (warp == 0 && lane < NT * 8) {
      const int i = lane >> 3;
      const uint16_t* src = p.w[mat] + static_cast<int64_t>(min(row0 + (lane & 7), p.rows[mat] - 1) + i * p.half) * p.K;
      bulk_load(s_w + lane * w_row, src, p.K * 2, &bar_w);
    }
  };
  uint4 wr[NT][kSmem ? 1 : kStepAhead];
  auto fetch = [&](int kb0) {   // blocks kb0 + 8 j + warp
#pragma unroll
    for (int j = 0; j < kStepAhead; ++j) {
      const int kb = kb0 + j * kStepWarps + warp;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        wr[i][j] = make_uint4(0, 0, 0, 0);
        if (kb < nkb) wr[i][j] = ldg_stream(wp[i] + kb * 32);
      }
    }
  };
  constexpr bool kFirst = kIn == kInRms && kOut == kOutFp32;
  if constexpr (!kFirst) {
    if constexpr (kSmem) copy();
    else fetch(0);
  } else {
    // (a request into L2 may come before the weights are written: it is the copy that has to come after)
    const int tile = static_cast<int>(blockIdx.x) + tid * kStepEarly, tiles = static_cast<int>(gridDim.x);
    if (static_cast<int>(blockIdx.x) < kStepEarly && tile < tiles) {
      int m = 0;
      while (m + 1 < p.n_mats && tile >= p.tile0[m + 1]) ++m;
      const int row = (tile - p.tile0[m]) * 8;
      l2_request(p.w[m] + static_cast<int64_t>(row) * p.K, static_cast<uint32_t>(min(8, p.rows[m] - row)) * p.K * 2);
    }
  }
  if (p.ahead) {
    const uint64_t round = step_ahead_at(gridDim.x, 0, 0, 1);
    for (uint64_t o = step_ahead_at(gridDim.x, blockIdx.x, tid, 0); o < p.ahead_bytes; o += round)
      l2_request(p.ahead + o, static_cast<uint32_t>(min(static_cast<uint64_t>(kStepChunk), p.ahead_bytes - o)));
  }
  // one chunk of a row per lane at most: its norm weights come before the wait, its input stays in registers
  int per = 8;   // warps that share a row
  if constexpr (kIn == kInRms)
    while (per > 1 && per * p.B > 8) per >>= 1;
  const bool once = kSmem && kIn == kInRms && chunks <= per * 32;
  float nw[8];
  if (!kFirst && once && (warp % per) * 32 + lane < chunks) load_w8(p.norm_w, p.w_dtype, (warp % per) * 32 + lane, nw);
  pdl_wait();
  pdl_launch();
  if constexpr (kFirst) {
    if constexpr (kSmem) copy();
    else fetch(0);
    if (once && (warp % per) * 32 + lane < chunks) load_w8(p.norm_w, p.w_dtype, (warp % per) * 32 + lane, nw);
  }

  // ---- the input, once per CTA ----
  if constexpr (kIn == kInRms) {
    // `per` warps share a row; each row's sum of squares goes through shared memory
    const int rows_at_once = 8 / per, part = warp % per;
    for (int b0 = 0; b0 < p.B; b0 += rows_at_once) {
      const int b = b0 + warp / per;
      float ss = 0.f, x0[8];
      if (b < p.B) {
        for (int c = part * 32 + lane; c < chunks; c += per * 32) {
          load_x8<kBf16>(p, b, c, x0);
#pragma unroll
          for (int j = 0; j < 8; ++j) ss = fmaf(x0[j], x0[j], ss);
        }
      }
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (b0 > 0) __syncthreads();
      if (lane == 0) s_ss[warp] = ss;
      __syncthreads();
      ss = 0.f;
      for (int i = 0; i < per; ++i) ss += s_ss[warp - part + i];
      const float r = 1.f / sqrtf(ss / static_cast<float>(p.K) + p.eps);
      if (b < p.B && once) {
        const int c = part * 32 + lane;
        if (c < chunks) {
#pragma unroll
          for (int j = 0; j < 8; ++j) x0[j] = x0[j] * r * nw[j];
          s_x[b * stride + c] = pack8s<kBf16>(x0);
        }
      } else if (b < p.B) {
        for (int c = part * 32 + lane; c < chunks; c += per * 32) {
          float f[8], w[8];
          load_x8<kBf16>(p, b, c, f);
          load_w8(p.norm_w, p.w_dtype, c, w);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = f[j] * r * w[j];
          s_x[b * stride + c] = pack8s<kBf16>(f);
        }
      }
    }
  } else if constexpr (kIn == kInGated) {
    const int lanes = p.D / 8;   // (divides 32; K / 8 is a multiple of it, so a head's lanes are in or out together)
    const int total = p.B * chunks;
    for (int e0 = 0; e0 < total; e0 += kStepThreads) {
      const int e = e0 + tid;
      const int b = min(e, total - 1) / chunks, c = min(e, total - 1) % chunks;
      float f[8], w[8], ss = 0.f;
      load_x8<kBf16>(p, b, c, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
      for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float r = rsqrtf(ss / static_cast<float>(p.D) + p.eps);
      load_w8(p.norm_w, p.w_dtype, c, w);
      const float4* gp = reinterpret_cast<const float4*>(p.gate + b * p.gate_ld) + 2 * c;
      const float4 u = gp[0], v = gp[1];
      const float gv[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = f[j] * r * w[j] * __fdividef(1.f, 1.f + __expf(-gv[j]));
      if (e < total) s_x[b * stride + c] = pack8s<kBf16>(f);
    }
  } else {
    const uint4* x = static_cast<const uint4*>(p.x);
    for (int e = tid; e < p.B * chunks; e += kStepThreads) s_x[(e / chunks) * stride + e % chunks] = x[e];
  }
  __syncthreads();

  // ---- products ----
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const bool lo = g < p.B, hi = g + 8 < p.B;
  const uint4* xl = s_x + g * stride + t;
  if constexpr (kSmem) {
    mbar_wait(&bar_w, 0, &abort_flag, p.status, kStepWaitSite);   // (one that runs out is recorded; what follows is then discarded)
#pragma unroll 4
    for (int kb = warp; kb < nkb; kb += kStepWarps) {
      uint4 a = make_uint4(0, 0, 0, 0), a8 = a;
      if (lo) a = xl[kb * 4];
      if (hi) a8 = xl[8 * stride + kb * 4];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        const uint4 w = *reinterpret_cast<const uint4*>(s_w + (i * 8 + g) * w_row + kb * 64 + t * 16);
        step_mma<kBf16>(acc[i], a.x, a8.x, a.y, a8.y, w.x, w.y);
        step_mma<kBf16>(acc[i], a.z, a8.z, a.w, a8.w, w.z, w.w);
      }
    }
  }
  if constexpr (!kSmem) {
    for (int kb0 = 0; kb0 < nkb; kb0 += kStepAhead * kStepWarps) {
#pragma unroll
      for (int j = 0; j < kStepAhead; ++j) {
        const int kb = kb0 + j * kStepWarps + warp;
        if (kb < nkb) {
          uint4 a = make_uint4(0, 0, 0, 0), a8 = a;
          if (lo) a = xl[kb * 4];
          if (hi) a8 = xl[8 * stride + kb * 4];
#pragma unroll
          for (int i = 0; i < NT; ++i) {
            step_mma<kBf16>(acc[i], a.x, a8.x, a.y, a8.y, wr[i][j].x, wr[i][j].y);
            step_mma<kBf16>(acc[i], a.z, a8.z, a.w, a8.w, wr[i][j].z, wr[i][j].w);
          }
        }
      }
      if (kb0 + kStepAhead * kStepWarps < nkb) fetch(kb0 + kStepAhead * kStepWarps);
    }
  }
  // c0, c1: sequence g, weight rows 2t, 2t+1; c2, c3: sequence g + 8
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    float* r = s_red[warp][i];
    *reinterpret_cast<float2*>(r + g * 8 + 2 * t) = make_float2(acc[i][0], acc[i][1]);
    *reinterpret_cast<float2*>(r + (g + 8) * 8 + 2 * t) = make_float2(acc[i][2], acc[i][3]);
  }
  __syncthreads();
  if (tid < 128) {
    const int b = tid / 8, r = row0 + tid % 8;
    float v[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      v[i] = 0.f;
#pragma unroll
      for (int w = 0; w < kStepWarps; ++w) v[i] += s_red[w][i][tid];
    }
    if (b < p.B && r < p.rows[mat]) {
      int64_t col = r;
      for (int i = 0; i < mat; ++i) col += p.rows[i];
      const int64_t o = b * p.ldo + col;
      if constexpr (kOut == kOutFp32) {
        static_cast<float*>(p.out)[o] = v[0];
      } else if constexpr (kOut == kOutAdd16) {
        static_cast<float*>(p.out)[o] = v[0] + unpack2<kBf16>(static_cast<const uint16_t*>(p.res)[o]).x;
      } else {
        float y;
        if constexpr (kOut == kOutSwiglu) y = v[0] * __fdividef(1.f, 1.f + __expf(-v[0])) * v[NT - 1];
        else y = v[0] + static_cast<const float*>(p.res)[o];
        static_cast<uint16_t*>(p.out)[o] = static_cast<uint16_t>(pack2<kBf16>(y, 0.f) & 0xffffu);
      }
    }
  }
}

struct StepMixParams {
  const float* y;          // (B, ld): [q | k | v | ogate | fgate | k mix | v mix]
  int64_t ld;
  const void *wq, *wk;     // (C)
  const void* bias;        // (H) or nullptr
  int wq_dtype, wk_dtype, bias_dtype;
  float eps;
  const int64_t* mask;     // (B, N) or nullptr
  int64_t* seq_start;      // (B): N - sum of the mask
  uint16_t *k_state, *v_state;   // (B, C): the token before's projections, replaced by this one's
  uint16_t* q;             // (B, C)
  uint16_t *k_cache, *v_cache;   // (B, H, cap, D)
  float* g_cache;          // (B, H, cap)
  int64_t cap, pos;        // rows of the cache; row of this token
  int H, D;
};

__device__ __forceinline__ float load_any(const void* w, int dtype, int i) {
  if (dtype == FOX_DTYPE_FP32) return static_cast<const float*>(w)[i];
  const uint32_t u = static_cast<const uint16_t*>(w)[i];
  return dtype == FOX_DTYPE_BF16 ? unpack2<true>(u).x : unpack2<false>(u).x;
}

// CTA = one head of one sequence, thread = channel; the few values make this a matter of latency only.  With a mask there is a
// thread for four of its elements at least, up to 512, for their sum: with one a channel 6200 keys of 8 heads of 64 took 27 us a
// layer, 23 now, 12000 of 24 67 and 47, 40000 of 32 of 16 101 and 41.  (512 for 64 keys of 16 x 32 heads of 16: 34 for 32 us.)
constexpr int kMaskThreads = 512;
template <bool kBf16>
__global__ void __launch_bounds__(kMaskThreads) fox_step_mix_kernel(const StepMixParams p) {
  constexpr int kWarps = kMaskThreads / 32;
  __shared__ float s_q[kWarps], s_k[kWarps];
  __shared__ long long s_n[kWarps];
  const int h = blockIdx.x, b = blockIdx.y, d = threadIdx.x, lane = d & 31, warp = d >> 5, warps = blockDim.x >> 5;
  const int C = p.H * p.D, ch = h * p.D + d;
  const bool on = d < p.D;
  const float wq = on ? load_any(p.wq, p.wq_dtype, ch) : 0.f, wk = on ? load_any(p.wk, p.wk_dtype, ch) : 0.f;
  const float bias = p.bias ? load_any(p.bias, p.bias_dtype, h) : 0.f;
  pdl_wait();
  if (!p.mask) pdl_launch();   // (the attention's clusters would be placed around the block that still sums the mask)
  const float* y = p.y + b * p.ld;
  const float ak = sigmoid_fp32(y[4 * C + p.H + h]), av = sigmoid_fp32(y[4 * C + 2 * p.H + h]);
  float q = 0.f, k = 0.f, v = 0.f;
  if (on) {
    q = y[ch];
    const uint32_t k16 = pack2<kBf16>(y[C + ch], 0.f) & 0xffffu, v16 = pack2<kBf16>(y[2 * C + ch], 0.f) & 0xffffu;
    const int64_t so = static_cast<int64_t>(b) * C + ch;
    const float kp = unpack2<kBf16>(p.k_state[so]).x, vp = unpack2<kBf16>(p.v_state[so]).x;
    k = ak * kp + (1.f - ak) * unpack2<kBf16>(k16).x;
    v = av * vp + (1.f - av) * unpack2<kBf16>(v16).x;
    p.k_state[so] = static_cast<uint16_t>(k16);
    p.v_state[so] = static_cast<uint16_t>(v16);
  }
  float sq = q * q, sk = k * k;
  for (int o = 16; o > 0; o >>= 1) {
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
    sk += __shfl_xor_sync(0xffffffffu, sk, o);
  }
  if (lane == 0) {
    s_q[warp] = sq;
    s_k[warp] = sk;
  }
  if (p.mask && h == 0) {
    long long n = 0;
#pragma unroll 4
    for (int64_t i = d; i <= p.pos; i += blockDim.x) n += p.mask[b * (p.pos + 1) + i];
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) s_n[warp] = n;
  }
  __syncthreads();
  sq = sk = 0.f;
  for (int w = 0; w < warps; ++w) {
    sq += s_q[w];
    sk += s_k[w];
  }
  const float inv_d = 1.f / static_cast<float>(p.D);
  if (on) {
    q *= rsqrtf(sq * inv_d + p.eps) * wq;
    k *= rsqrtf(sk * inv_d + p.eps) * wk;
    const int64_t row = ((static_cast<int64_t>(b) * p.H + h) * p.cap + p.pos) * p.D + d;
    p.q[static_cast<int64_t>(b) * C + ch] = static_cast<uint16_t>(pack2<kBf16>(q, 0.f) & 0xffffu);
    p.k_cache[row] = static_cast<uint16_t>(pack2<kBf16>(k, 0.f) & 0xffffu);
    p.v_cache[row] = static_cast<uint16_t>(pack2<kBf16>(v, 0.f) & 0xffffu);
  }
  if (d == 0) {
    const float f = y[4 * C + h] + bias;
    p.g_cache[(static_cast<int64_t>(b) * p.H + h) * p.cap + p.pos] = fminf(f, 0.f) - log1pf(expf(-fabsf(f)));
    if (p.mask && h == 0) {
      long long n = 0;
      for (int w = 0; w < warps; ++w) n += s_n[w];
      p.seq_start[b] = p.pos + 1 - n;
    }
  }
}

static cudaLaunchConfig_t pdl_config(dim3 grid, int threads, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Shared memory and L1 are one array per SM, split anew only while the SM is empty; kernels that begin early keep it from
// that.  Left to itself the runtime gives these products all of it, and the attention behind them no room for its loads in flight
// (48 (b,h) of 40000 keys 114 us, 78 behind products through registers).  Long attention asks for a split of its own
// (fox_decode.cu).  The products do, all of a layer for the same, where the gate product's CTAs, as many to an SM as of the first
// product, need no more than half: 16 sequences of 512 channels 35 -> 31 us a layer, one of 768 16.5 -> 15.4.  Above that it
// takes the overlap of one product with the next: 16 of 1536 81 -> 92, one of 1024 19.8 -> 20.2.
static size_t step_x_bytes(int64_t B, int64_t K) { return static_cast<size_t>(B) * ((K / 8 + 7) / 8 * 8 + 4) * 16; }
static int step_carveout(int64_t ctas, int64_t bytes) {
  return static_cast<int>(std::min<int64_t>((ctas * bytes * 100 + kSmSmem - 1) / kSmSmem, 100));
}
static int64_t step_per_sm(int64_t grid) { return std::min<int64_t>((grid + kSms - 1) / kSms, 4); }   // (4 by registers)

template <bool kBf16, int kIn, int kOut, bool kSmem>
static int launch_product(int device, cudaStream_t st, const StepParams& p, size_t smem) {
  auto kern = fox_step_product_kernel<kBf16, kIn, kOut, kSmem>;
  static bool configured[64] = {};
  if (device < 0 || device >= 64) return FOX_ERR_DEVICE;
  if (smem > 32 * 1024 && !configured[device]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return FOX_ERR_LAUNCH;
    configured[device] = true;
  }
  cudaLaunchAttribute attrs[2] = {};
  cudaLaunchConfig_t cfg = pdl_config(dim3((unsigned)p.tile0[p.n_mats]), kStepThreads, smem, st, attrs);
  attrs[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  if (kSmem) {
    const int64_t C = kIn == kInPlain ? p.rows[0] : p.K;
    const int64_t gate = static_cast<int64_t>(step_x_bytes(p.B, C)) + 16 * step_row_bytes(static_cast<int>(C)) + kStepStatic;
    const int share = step_carveout(step_per_sm(C / 2), gate);
    attrs[1].val.sharedMemCarveout = share;
    if (share <= 50) cfg.numAttrs = 2;
  } else if (kIn == kInPlain && p.status && p.rows[0] * static_cast<int64_t>(p.K) >= kStepBigWeights) {
    const int share = step_carveout(step_per_sm(p.tile0[p.n_mats]), static_cast<int64_t>(smem) + kStepStatic);
    attrs[1].val.sharedMemCarveout = share;
    if (share <= 80) cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kern, p) == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}
template <bool kBf16, int kIn, int kOut>
static int choose_product(int device, cudaStream_t st, const StepParams& p) {
  const size_t x = step_x_bytes(p.B, p.K);
  const size_t w = static_cast<size_t>(kOut == kOutSwiglu ? 16 : 8) * step_row_bytes(p.K);
  if (x > 200 * 1024) return FOX_ERR_TOO_LARGE;
  return p.status && x + w <= kStepSmem ? launch_product<kBf16, kIn, kOut, true>(device, st, p, x + w)
                                        : launch_product<kBf16, kIn, kOut, false>(device, st, p, x);
}

}  // namespace fox

using namespace fox;

static int step_product(int device, void* stream, int dtype, int input, int output, int64_t B, int64_t K, const void* x, int x_fp32,
                        const void* norm_w, int norm_w_dtype, float eps, int64_t D, const float* gate, int64_t gate_ld, int64_t n_mats,
                        const void* const* mats, const int64_t* mat_rows, const void* residual, void* out, int64_t ldo,
                        const void* ahead, int64_t ahead_bytes, int32_t* status) {
  if (!x || !out || !mats || n_mats <= 0 || n_mats > kStepMats || B <= 0 || B > 16 || K <= 0 || ldo <= 0) return FOX_ERR_BAD_ARG;
  if (K % 32) return FOX_ERR_HEAD_DIM;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if (input != kInPlain && !norm_w) return FOX_ERR_BAD_ARG;
  if (input == kInGated && (!gate || D < 8 || D > 256 || (D & (D - 1)) || K % D || gate_ld % 4)) return FOX_ERR_BAD_ARG;
  if ((output == kOutAdd16 || output == kOutAdd32) && !residual) return FOX_ERR_BAD_ARG;
  uintptr_t align = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(gate);
  StepParams p{};
  int tile = 0;
  for (int i = 0; i < n_mats; ++i) {
    if (!mats[i] || mat_rows[i] <= 0) return FOX_ERR_BAD_ARG;
    align |= reinterpret_cast<uintptr_t>(mats[i]);
    p.w[i] = (const uint16_t*)mats[i];
    p.rows[i] = (int)mat_rows[i];
    if (output == kOutSwiglu) {   // [gate rows | value rows] of one matrix, a tile of each per CTA
      if (n_mats != 1 || mat_rows[i] % 16) return FOX_ERR_BAD_ARG;
      p.half = (int)(mat_rows[i] / 2);
      p.rows[i] = p.half;
    }
    p.tile0[i] = tile;
    tile += (p.rows[i] + 7) / 8;
  }
  p.tile0[n_mats] = tile;
  if (align % 16) return FOX_ERR_ALIGNMENT;
  if (ahead && (reinterpret_cast<uintptr_t>(ahead) % 16 || ahead_bytes < 0 || ahead_bytes % 16)) return FOX_ERR_ALIGNMENT;
  p.ahead = (const char*)ahead;
  if (ahead_bytes > kStepAheadMost) p.ahead = nullptr;
  p.ahead_bytes = (uint64_t)ahead_bytes;
  p.status = status;
  p.n_mats = (int)n_mats; p.B = (int)B; p.K = (int)K; p.D = (int)D;
  p.x = x; p.x_fp32 = x_fp32 != 0; p.norm_w = norm_w; p.w_dtype = norm_w_dtype; p.eps = eps;
  p.gate = gate; p.gate_ld = gate_ld; p.res = residual; p.out = out; p.ldo = ldo;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  cudaStream_t st = (cudaStream_t)stream;
  const bool bf = dtype == FOX_DTYPE_BF16;
#define FOX_STEP(I, O) if (input == I && output == O) return bf ? choose_product<true, I, O>(device, st, p) : choose_product<false, I, O>(device, st, p)
  FOX_STEP(kInRms, kOutFp32);
  FOX_STEP(kInGated, kOutAdd16);
  FOX_STEP(kInRms, kOutSwiglu);
  FOX_STEP(kInPlain, kOutAdd32);
#undef FOX_STEP
  return FOX_ERR_BAD_ARG;
}

extern "C" int64_t fox_step_ahead_offset(int64_t grid, int64_t block, int64_t thread, int64_t k) {
  return (int64_t)step_ahead_at((uint64_t)grid, (uint64_t)block, (uint64_t)thread, (uint64_t)k);
}

extern "C" int fox_step_product_ahead(int device, void* stream, int dtype, int input, int output, int64_t B, int64_t K,
                                      const void* x, int x_fp32, const void* norm_w, int norm_w_dtype, float eps, int64_t D,
                                      const float* gate, int64_t gate_ld, int64_t n_mats, const void* const* mats,
                                      const int64_t* mat_rows, const void* residual, void* out, int64_t ldo, const void* ahead,
                                      int64_t ahead_bytes, int32_t* status) {
  if (!status) return FOX_ERR_BAD_ARG;
  return step_product(device, stream, dtype, input, output, B, K, x, x_fp32, norm_w, norm_w_dtype, eps, D, gate, gate_ld, n_mats, mats,
                      mat_rows, residual, out, ldo, ahead, ahead_bytes, status);
}

extern "C" int fox_step_product(int device, void* stream, int dtype, int input, int output, int64_t B, int64_t K,
                                const void* x, int x_fp32, const void* norm_w, int norm_w_dtype, float eps, int64_t D,
                                const float* gate, int64_t gate_ld, int64_t n_mats, const void* const* mats,
                                const int64_t* mat_rows, const void* residual, void* out, int64_t ldo) {
  return step_product(device, stream, dtype, input, output, B, K, x, x_fp32, norm_w, norm_w_dtype, eps, D, gate, gate_ld, n_mats, mats,
                      mat_rows, residual, out, ldo, nullptr, 0, nullptr);
}

extern "C" int fox_step_mix(int device, void* stream, int dtype, int64_t B, int64_t H, int64_t D, const float* y, int64_t ld,
                            const void* wq, int wq_dtype, const void* wk, int wk_dtype, float eps, const void* bias, int bias_dtype,
                            const int64_t* mask, int64_t* seq_start, void* k_state, void* v_state, void* q, void* k_cache,
                            void* v_cache, float* g_cache, int64_t capacity, int64_t pos) {
  if (!y || !wq || !wk || !k_state || !v_state || !q || !k_cache || !v_cache || !g_cache || B <= 0 || H <= 0 || B > 65535 ||
      H > 65535 || pos < 0 || pos >= capacity || (mask && !seq_start))
    return FOX_ERR_BAD_ARG;
  if (D != 16 && D != 32 && D != 64 && D != 128) return FOX_ERR_HEAD_DIM;
  if (dtype != FOX_DTYPE_BF16 && dtype != FOX_DTYPE_FP16) return FOX_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return FOX_ERR_DEVICE;
  const StepMixParams p{y, ld, wq, wk, bias, wq_dtype, wk_dtype, bias_dtype, eps, mask, seq_start, (uint16_t*)k_state, (uint16_t*)v_state,
                        (uint16_t*)q, (uint16_t*)k_cache, (uint16_t*)v_cache, g_cache, capacity, pos, (int)H, (int)D};
  cudaLaunchAttribute attr;
  const int64_t summing = mask ? std::min<int64_t>((pos / 4 + 32) / 32 * 32, kMaskThreads) : 0;
  const int threads = (int)std::max<int64_t>(summing, D <= 32 ? 32 : D);
  const cudaLaunchConfig_t cfg = pdl_config(dim3((unsigned)H, (unsigned)B), threads, 0, (cudaStream_t)stream, &attr);
  const cudaError_t e = dtype == FOX_DTYPE_BF16 ? cudaLaunchKernelEx(&cfg, fox_step_mix_kernel<true>, p)
                                                : cudaLaunchKernelEx(&cfg, fox_step_mix_kernel<false>, p);
  return e == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}
