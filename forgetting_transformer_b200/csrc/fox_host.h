// Host-side helpers: error codes, TMA tensor-map encoding through the driver
// entry point (no link-time libcuda dependency) and a small descriptor cache.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <unordered_map>

#include "../../include/fox_b200.h"

namespace fox {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Description of a (B, H, T, D) tensor of 16-bit or 32-bit elements whose last
// dimension has unit stride; the other strides are in elements.
struct Tensor4 {
  void* ptr;
  int64_t B, H, T, D;
  int64_t sb, sh, st;
};

// Can TMA address this view?  (16-byte aligned base and byte strides.)
inline bool tma_compatible(const Tensor4& t, int elem_bytes) {
  if (reinterpret_cast<uintptr_t>(t.ptr) % 16) return false;
  const int64_t s[3] = {t.sb, t.sh, t.st};
  for (int i = 0; i < 3; ++i) {
    const int64_t bytes = s[i] * elem_bytes;
    if (bytes <= 0 || bytes % 16) return false;
  }
  return true;
}

// Tiled map with dims (D, T, H, B), box (box_d, box_t, 1, 1).  swizzle128 selects
// the 128-byte swizzle (box_d * elem_bytes must then be 128) or none.
inline int make_tmap_4d(CUtensorMap* out, const Tensor4& t, int elem_bytes, bool is_float32, bool is_bf16,
                        uint32_t box_d, uint32_t box_t, bool swizzle128) {
  EncodeTiledFn fn = get_encode_tiled();
  if (!fn) return FOX_ERR_DRIVER;
  // A dimension of extent 1 may carry any stride in a torch view; give it a legal one.
  cuuint64_t dims[4] = {(cuuint64_t)t.D, (cuuint64_t)t.T, (cuuint64_t)t.H, (cuuint64_t)t.B};
  int64_t st = t.st, sh = t.sh, sb = t.sb;
  if (t.T == 1 && (st * elem_bytes) % 16) st = t.D;
  if (t.H == 1 && (sh * elem_bytes) % 16) sh = t.D * t.T;
  if (t.B == 1 && (sb * elem_bytes) % 16) sb = t.D * t.T * t.H;
  cuuint64_t strides[3] = {(cuuint64_t)(st * elem_bytes), (cuuint64_t)(sh * elem_bytes),
                           (cuuint64_t)(sb * elem_bytes)};
  cuuint32_t box[4] = {box_d, box_t, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUtensorMapDataType dt = is_float32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                      : (is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  CUresult r = fn(out, dt, 4, t.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FOX_OK : FOX_ERR_TENSORMAP;
}

// ------------------------------------------------------------- order of items
// How many units go by length together (ItemOrder in fox_common.cuh): groups of even size whose rereads, unit_bytes a unit, stay in
// L2 (126 MB; what is written takes its part).  Forward / backward kernels in us, unit by unit -> groups of 12, 24, 48 MB, all units:
//   B2 H24 T16384 D64    2240 / 4724 -> 2151 / 4722, 2092 / 4697, 2079 / 4698, 2140 / 5191
//   B2 H16 T4096 D64     138 / 278 -> 126 / 283, 117 / 251, 114 / 253, 115 / 259
//   B4 H16 T16384 D128   4539 / 8273 + 5370 -> 16 MB 4457 / 8171 + 5316, 48 MB 4354 / 8148 + 5334, all 4788 / 8775 + 5837
//   B4 H12 T512 D64      15.1 / 24.8 -> 12.4 / 21.0 (one group from 3 MB on)
// Items that all have an SM to themselves are one group whatever they read: groups of uneven sizes are padded with CTAs that have no
// item, and those took places that the last items then shared with others (37 (b,h) of 512 x 8000, 148 items and 4 such CTAs: forward at
// D64 77 -> 107 us by two groups, 77 by one; at D128 109 -> 131, 109).  More units than an int counts stay unit by unit.
inline int64_t item_group(int64_t units, int64_t tiles, int64_t unit_bytes) {
  constexpr int64_t kGroupBytes = 48 << 20;
  if (units * tiles <= 148) return units;
  if (units > 2147483647LL - 65536) return 1;
  const int64_t fit = unit_bytes < kGroupBytes ? kGroupBytes / unit_bytes : 1;
  const int64_t groups = (units + fit - 1) / fit;
  return tiles > 65535 || groups > 65535 ? 1 : (units + groups - 1) / groups;   // (what a grid can have)
}

// ------------------------------------------------------------- tensor-map cache
struct TmapKey {
  uintptr_t ptr;
  int64_t v[7];
  uint32_t w[4];
  bool operator==(const TmapKey& o) const {
    if (ptr != o.ptr) return false;
    for (int i = 0; i < 7; ++i)
      if (v[i] != o.v[i]) return false;
    for (int i = 0; i < 4; ++i)
      if (w[i] != o.w[i]) return false;
    return true;
  }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    uint64_t h = 1469598103934665603ull ^ k.ptr;
    for (int i = 0; i < 7; ++i) h = (h ^ (uint64_t)k.v[i]) * 1099511628211ull;
    for (int i = 0; i < 4; ++i) h = (h ^ (uint64_t)k.w[i]) * 1099511628211ull;
    return (size_t)h;
  }
};

// Encoding a tensor map costs a few microseconds; training loops call with the
// same (pointer, shape, strides) over and over, so maps are memoised.
inline int cached_tmap_4d(CUtensorMap* out, const Tensor4& t, int elem_bytes, bool is_float32, bool is_bf16,
                          uint32_t box_d, uint32_t box_t, bool swizzle128) {
  static std::mutex mu;
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  TmapKey k;
  k.ptr = reinterpret_cast<uintptr_t>(t.ptr);
  k.v[0] = t.B; k.v[1] = t.H; k.v[2] = t.T; k.v[3] = t.D; k.v[4] = t.sb; k.v[5] = t.sh; k.v[6] = t.st;
  k.w[0] = box_d; k.w[1] = box_t;
  k.w[2] = (uint32_t)elem_bytes | (is_float32 ? 16u : 0u) | (is_bf16 ? 32u : 0u) | (swizzle128 ? 64u : 0u);
  k.w[3] = 0;
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(k);
    if (it != cache.end()) {
      *out = it->second;
      return FOX_OK;
    }
  }
  int rc = make_tmap_4d(out, t, elem_bytes, is_float32, is_bf16, box_d, box_t, swizzle128);
  if (rc != FOX_OK) return rc;
  std::lock_guard<std::mutex> g(mu);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(k, *out);
  return FOX_OK;
}

// Launches a kernel whose CTAs may take their SMs and set up their barriers as soon as the last CTA of the kernel in front has ended,
// before its results are written back; the kernel calls wait_for_kernel_in_front() before it reads or writes memory (its loads must
// not be __restrict__ or .nc ones, which may be done in front of the wait).  A launch behind another by stream order alone costs 1.5-2 us from
// the end of the first to the first load of the second; a pass of the attention is 5 to 7 kernels.  Forward and backward
// together, back to back, stream order -> this: B1 H2 T128 D64 30.9 -> 22.4 us, B4 H12 T512 D64 51.2 -> 41.0, B2 H16 T2048 D128
// 215 -> 203, B1 H24 T4096 D64 313 -> 301; from some 500 us a pass on within the noise.  None of the kernels lets the next begin
// earlier than that: a forward begun when its prefix sums had begun had its CTAs packed around theirs, on fewer SMs (B2 H7
// M700 N1500 D128 36.9 us by stream order, 39.5 so, 34.7 as here; B1 H4 T9000 D128 144, 157, 141).
// The kernels of a block's training pass between the products go the same way (forward and backward, all on the device: B4 T512 of 768
// channels 282 -> 265 us, B4 T1024 of 1024 593 -> 575, B1 T16384 of 1536 within the noise), but for its row norms: without
// __restrict__ their loads are issued later (backward, 16384 x 1536: 46 -> 86 us).
template <class... P, class... A>
inline int launch_behind(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
  return cudaGetLastError() == cudaSuccess ? FOX_OK : FOX_ERR_LAUNCH;
}

}  // namespace fox
