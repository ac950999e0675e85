// Encoded 2-D tensor maps, kept per (base, shape, box, type, swizzle) (moe_tc.cu).
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace xkb {

// 2-D row-major tensor [rows, cols] of `elem_bits` elements, box [box_rows, box_cols].
int make_map_2d(CUtensorMap* map, CUtensorMapDataType dt, int elem_bits, const void* base, uint64_t rows,
                uint64_t cols, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swz, const char* what);

}  // namespace xkb
