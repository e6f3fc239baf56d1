// The sort tiles of the density scatter's cell order (k_density_scatter): squares of
// kSortTile bins, and the shared memory of the counting pass, one count per tile.
// Plain C++, so that a host test walks every grid the library takes.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace erp {

constexpr int kGridMin = 16, kGridMax = 4096;   // bin counts of an axis (powers of two)
constexpr int kSortTile = 32;

constexpr int sort_tiles(int m, int n) { return ((m + kSortTile - 1) / kSortTile) * ((n + kSortTile - 1) / kSortTile); }
constexpr size_t sort_count_smem(int m, int n) { return sizeof(int32_t) * (size_t)sort_tiles(m, n); }
// What k_sort_count is opted in to: 64 KB at 4096 x 4096 bins, above the 48 KB a kernel
// has unasked.
constexpr size_t kSortCountSmem = sort_count_smem(kGridMax, kGridMax);
static_assert(kSortCountSmem <= 227 * 1024, "the counts of the largest grid fit a block's shared memory");

}  // namespace erp
