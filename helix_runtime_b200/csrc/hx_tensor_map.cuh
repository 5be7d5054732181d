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
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && depth == o.depth && ld == o.ld &&
           box_rows == o.box_rows && box_columns == o.box_columns && swizzled == o.swizzled;
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
    return h;
  }
};

// The map of a [rows, depth] matrix of bfloat16 with row stride ld, for boxes of box_rows rows by
// box_columns columns, laid out in shared memory with the 128-byte swizzle or row behind row.  Maps
// are pure functions of (address, shape, box); encoding one costs a few microseconds, so they are
// cached for the life of the process.
int hx_tensor_map(const char* caller, const void* base, uint64_t rows, uint64_t depth, uint64_t ld,
                  uint32_t box_rows, uint32_t box_columns, bool swizzled, CUtensorMap* out) {
  static std::mutex mutex;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  const MapKey key{base, rows, depth, ld, box_rows, box_columns, swizzled};
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
  const cuuint64_t dims[2] = {depth, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {box_columns, box_rows};
  const cuuint32_t element_strides[2] = {1, 1};
  CUtensorMap map;
  const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
                             dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    hx_set_error("%s: cuTensorMapEncodeTiled failed with %d (base %p rows %llu depth %llu ld %llu box "
                 "%u x %u)", caller, static_cast<int>(rc), base,
                 static_cast<unsigned long long>(rows), static_cast<unsigned long long>(depth),
                 static_cast<unsigned long long>(ld), box_rows, box_columns);
    return HX_ERR_ARGUMENT;
  }
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, map);
  *out = map;
  return HX_OK;
}

}  // namespace
