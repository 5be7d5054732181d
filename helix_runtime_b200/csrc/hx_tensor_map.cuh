// Tensor maps (what a TMA copy knows of the matrix it copies boxes of), made once per matrix.
#pragma once

#include "hx_common.cuh"

#include <cuda.h>

#include <mutex>
#include <unordered_map>

namespace {

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
  static EncodeTiled fn = [] {
    void* symbol = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &symbol, cudaEnableDefault, &result) !=
            cudaSuccess ||
        result != cudaDriverEntryPointSuccess) {
      return static_cast<EncodeTiled>(nullptr);
    }
    return reinterpret_cast<EncodeTiled>(symbol);
  }();
  return fn;
}

struct MapKey {
  const void* base;
  uint64_t rows;
  uint64_t depth;
  uint64_t ld;
  uint32_t box_rows;
  uint32_t box_columns;
  bool swizzled;
  uint64_t up_rows;      // > 0: boxes of interleaved rows
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && depth == o.depth && ld == o.ld &&
           box_rows == o.box_rows && box_columns == o.box_columns && swizzled == o.swizzled &&
           up_rows == o.up_rows;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.base);
    h = h * 1315423911u ^ k.rows;
    h = h * 1315423911u ^ k.depth;
    h = h * 1315423911u ^ k.ld;
    h = h * 1315423911u ^ k.box_rows;
    h = h * 1315423911u ^ (2 * k.box_columns + (k.swizzled ? 1 : 0));
    h = h * 1315423911u ^ k.up_rows;
    return h;
  }
};

// Maps are pure functions of (address, shape, box); encoding one costs a few microseconds, so they are
// cached for the life of the process.
int cached_tensor_map(const char* caller, const MapKey& key, CUtensorMap* out) {
  static std::mutex mutex;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  std::lock_guard<std::mutex> lock(mutex);
  auto found = cache.find(key);
  if (found != cache.end()) {
    *out = found->second;
    return HX_OK;
  }
  EncodeTiled encode = encode_tiled();
  if (encode == nullptr) {
    hx_set_error("%s: the driver does not export cuTensorMapEncodeTiled", caller);
    return HX_ERR_UNSUPPORTED;
  }
  const bool interleaved = key.up_rows > 0;
  const cuuint64_t plain_dims[2] = {key.depth, key.rows};
  const cuuint64_t plain_strides[1] = {key.ld * 2};
  const cuuint32_t plain_box[2] = {key.box_columns, key.box_rows};
  const cuuint64_t turns_dims[4] = {key.depth, 16, 2, (key.rows - key.up_rows) / 16};
  const cuuint64_t turns_strides[3] = {key.ld * 2, key.up_rows * key.ld * 2, 16 * key.ld * 2};
  const cuuint32_t turns_box[4] = {key.box_columns, 16, 2, key.box_rows / 32};
  const cuuint32_t element_strides[4] = {1, 1, 1, 1};
  CUtensorMap map;
  const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, interleaved ? 4 : 2,
                             const_cast<void*>(key.base), interleaved ? turns_dims : plain_dims,
                             interleaved ? turns_strides : plain_strides,
                             interleaved ? turns_box : plain_box, element_strides,
                             CU_TENSOR_MAP_INTERLEAVE_NONE,
                             key.swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    hx_set_error("%s: cuTensorMapEncodeTiled failed with %d (base %p rows %llu depth %llu ld %llu box "
                 "%u x %u)", caller, static_cast<int>(rc), key.base,
                 static_cast<unsigned long long>(key.rows), static_cast<unsigned long long>(key.depth),
                 static_cast<unsigned long long>(key.ld), key.box_rows, key.box_columns);
    return HX_ERR_ARGUMENT;
  }
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, map);
  *out = map;
  return HX_OK;
}

// The map of a [rows, depth] matrix of bfloat16 with row stride ld, for boxes of box_rows rows by
// box_columns columns, laid out in shared memory with the 128-byte swizzle or row behind row.
int hx_tensor_map(const char* caller, const void* base, uint64_t rows, uint64_t depth, uint64_t ld,
                  uint32_t box_rows, uint32_t box_columns, bool swizzled, CUtensorMap* out) {
  return cached_tensor_map(caller, MapKey{base, rows, depth, ld, box_rows, box_columns, swizzled, 0}, out);
}

// The map of the same matrix, whole rows, for boxes of box_rows rows (swizzled) that hold 16 rows, the 16
// that lie up_rows behind them, the next 16, and so on.  Coordinates: column, 0, 0, first row / 16; up_rows
// and rows are multiples of 16, so that nothing behind the matrix is read.
[[maybe_unused]] int hx_tensor_map_interleaved(const char* caller, const void* base, uint64_t rows,
                                               uint64_t depth, uint64_t up_rows, uint32_t box_rows,
                                               uint32_t box_columns, CUtensorMap* out) {
  return cached_tensor_map(caller, MapKey{base, rows, depth, depth, box_rows, box_columns, true, up_rows}, out);
}

}  // namespace
