// Tensor maps of the GEMM launchers, kept per thread: encoding one takes about as long as a kernel launch, a layer
// uses the same few operands at every step, and a map depends on nothing but the values it is looked up by.
#pragma once
#include <string.h>
#include "../host/driver_api.h"
#include "../host/launch.h"

namespace mep {

struct TmapKey { const void* base; int64_t rows, cols, ld; int32_t box0, box1, kind, pad; };

inline int tmap_get(CUtensorMap* m, const TmapKey& k) {
  struct Slot { TmapKey key; CUtensorMap map; bool used; };
  static thread_local Slot slots[256];
  uint64_t h = (uint64_t)(uintptr_t)k.base * 0x9E3779B97F4A7C15ull ^ (uint64_t)k.rows * 0xC2B2AE3D27D4EB4Full ^
               (uint64_t)k.ld * 0x165667B19E3779F9ull ^ (uint64_t)(k.cols + k.box0 * 131 + k.box1 * 8191 + k.kind * 65537) * 0x27D4EB2F165667C5ull;
  Slot& s = slots[(h >> 40) & 255];
  if (s.used && memcmp(&s.key, &k, sizeof(k)) == 0) { *m = s.map; return 0; }
  const DriverApi* d = driver(); if (!d) return -1;
  const int es_bytes = k.kind == 1 ? 4 : 2;
  MEP_REQUIRE(((uintptr_t)k.base & 15) == 0 && (k.ld * es_bytes) % 16 == 0 && k.ld >= k.cols, "gemm: tensor base/stride must be 16-byte aligned");
  s.used = false;                        // until the new map stands
  cuuint32_t es[3] = {1, 1, 1};
  if (k.kind == 2) {
    MEP_REQUIRE(k.cols % 64 == 0, "gemm: MN-major operand width %lld must be a multiple of 64", (long long)k.cols);
    cuuint64_t dims[3] = {64, (cuuint64_t)k.rows, (cuuint64_t)(k.cols / 64)}, strides[2] = {(cuuint64_t)k.ld * 2, 128};
    cuuint32_t box[3] = {64, (cuuint32_t)k.box1, (cuuint32_t)k.box0};
    MEP_CU_CHECK(d->TensorMapEncodeTiled(&s.map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(k.base), dims, strides, box, es,
                                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  } else {
    cuuint64_t dims[2] = {(cuuint64_t)k.cols, (cuuint64_t)k.rows}, strides[1] = {(cuuint64_t)k.ld * es_bytes};
    cuuint32_t box[2] = {(cuuint32_t)k.box0, (cuuint32_t)k.box1};
    MEP_CU_CHECK(d->TensorMapEncodeTiled(&s.map, k.kind == 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                                         const_cast<void*>(k.base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  }
  s.key = k; s.used = true; *m = s.map;
  return 0;
}
// Row-major matrix [rows, cols], pitch `ld` elements, boxes of box_rows x box_cols (128 bytes wide, 128-byte swizzle).
inline int tmap_rows(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_cols, int box_rows, bool f32 = false) {
  TmapKey k; memset(&k, 0, sizeof(k));
  k.base = base; k.rows = rows; k.cols = cols; k.ld = ld; k.box0 = box_cols; k.box1 = box_rows; k.kind = f32 ? 1 : 0;
  return tmap_get(m, k);
}
// MN-major bf16 operand [rows (k), cols (m or n)] viewed as (64 elements, rows, cols / 64): one box of `atoms` 64-wide
// atoms x `box_rows` rows lands in shared memory atom after atom.
inline int tmap_atoms(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t ld, int atoms, int box_rows = 64) {
  TmapKey k; memset(&k, 0, sizeof(k));
  k.base = base; k.rows = rows; k.cols = cols; k.ld = ld; k.box0 = atoms; k.box1 = box_rows; k.kind = 2;
  return tmap_get(m, k);
}

}  // namespace mep
