// Tensor-map (TMA) loads and mbarriers for the sm_100a kernels: the device helpers, and on the host
// the encoding of bfloat16 tensor maps of a matrix, 2-D or as runs of 64 columns (3-D), through the driver entry point (no
// link against the driver library), cached by what they describe.
//
// Alignment: a tiled TMA copy starts on a 16-byte boundary, so the innermost coordinate is always a
// multiple of 8 elements here; the other coordinates are free.  Tiles written with the 128-byte swizzle lie
// on 1024-byte boundaries of shared memory.
#pragma once
#include <cuda.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One tile of the map, starting at column x (elements) and row y, into shared memory; the bytes count
// towards `bar`.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// The same of a three-dimensional map.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// After a wait has run out the block stops issuing work; before it returns it gives the copies it still has in
// flight this long to land in its shared memory (they take microseconds when they land at all).
#define SNK_DRAIN_NS 200000ull
__device__ __forceinline__ void drain_after_abort() {
  const uint64_t start = global_ns();
  while (global_ns() - start < SNK_DRAIN_NS) {}
}

// ---------------------------------------------------------------------------------------------
// Tensor maps: bfloat16, rows of `k` elements (row pitch k * 2 bytes), box box_cols x box_rows (or rows by runs of 64
// columns, see tensor_map), 128-byte swizzle, zero fill outside.  Cached by (pointer, rows, k, box): a description, no data.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

struct MapKey {
  const void* ptr;
  long long rows, k;
  int box_rows, box_cols;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && rows == o.rows && k == o.k && box_rows == o.box_rows && box_cols == o.box_cols;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& m) const {
    return std::hash<const void*>()(m.ptr) ^ (std::hash<long long>()(m.rows) * 1315423911u) ^
           (std::hash<long long>()(m.k) * 2654435761u) ^ (size_t)m.box_rows ^ ((size_t)m.box_cols << 16);
  }
};

#define SNK_ERR_NO_ENCODER (SNK_ERR_SIZE + 100)    // the driver gave no cuTensorMapEncodeTiled
#define SNK_ERR_ENCODE 30000                       // + the CUresult of a refused encoding

// k_runs > 0: the matrix as runs of 64 columns, [k / 64][rows][64] (k a multiple of 64), a box being `box_rows` rows of
// `k_runs` runs: in shared memory every run of a box is a block of box_rows x 128 bytes of its own (swizzled alike).
static int tensor_map(const void* ptr, long long rows, long long k, int box_rows, int box_cols, CUtensorMap* out,
                      int k_runs = 0) {
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  const MapKey key{ptr, rows, k, box_rows, k_runs > 0 ? -k_runs : box_cols};
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return 0; }
  EncodeTiledFn fn = encode_fn();
  if (!fn) return SNK_ERR_NO_ENCODER;
  const bool runs = k_runs > 0;
  const cuuint64_t dims[3] = {(cuuint64_t)(runs ? 64 : k), (cuuint64_t)rows, (cuuint64_t)(k / 64)};
  const cuuint64_t strides[2] = {(cuuint64_t)k * 2, 128};
  const cuuint32_t box[3] = {(cuuint32_t)(runs ? 64 : box_cols), (cuuint32_t)box_rows, (cuuint32_t)k_runs};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap m;
  const CUresult r = fn(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, runs ? 3 : 2, const_cast<void*>(ptr), dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return SNK_ERR_ENCODE + (int)r;
  if (cache.size() > 8192) cache.clear();
  cache.emplace(key, m);
  *out = m;
  return 0;
}
