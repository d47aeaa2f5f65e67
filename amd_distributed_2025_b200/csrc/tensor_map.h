// Tensor maps of row-major 2-D arrays for tiled TMA copies.
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace b200 {

// Rows x cols elements of `elem_bytes` (1 or 2), box of box_rows x box_cols elements, whose rows are stored with a swizzle
// of 128 or 64 bytes or (0) none.  Out-of-range elements read as zero and are not written.  Encoded maps are kept in a small per-thread
// cache: a serving loop calls with the same weight (and often the same activation buffer) again and again, and the
// driver call is a visible part of a short launch.  False if the driver refuses the map.
bool make_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t elem_bytes, uint32_t box_rows,
                     uint32_t box_cols, int swizzle);

}  // namespace b200
