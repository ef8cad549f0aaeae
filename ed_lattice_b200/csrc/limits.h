// limits.h -- host-side rules that say which sectors a kernel or a table can take: sizes and
// index widths only, plain C++, so that they can be checked without a GPU.
#pragma once

#include <cstddef>
#include <cstdint>

namespace edg {

// ---- row tiles (tile.cu)
constexpr int kT16Zero = 8;  // zero slots after a tile, one per 16-byte bank group
// Shared memory of a tile kernel: the slots, `hops` down hops (value and source row) and the
// palette of `elem`-byte values, the slices' offsets.
constexpr size_t kTileSmemMax = 226 * 1024;  // leaves room for the kernels' static arrays
inline size_t tile_smem(int64_t dimup, int npal, int hops, size_t elem) {
  return size_t(dimup + kT16Zero) * 16 + size_t(hops) * ((elem + sizeof(uint32_t) + 7) / 8 * 8) + size_t(npal) * elem +
         size_t((dimup + 31) / 32) * sizeof(uint32_t);
}
// The whole product by tiles keeps a down hop as the 32-bit index of its source row's first
// element, the plain one with the value's sign in bit 31: sectors of 2^31 states and more go to
// the kernels that index in 64 bits.
inline bool tile_down_index(int64_t dim) { return dim < (int64_t(1) << 31); }

}  // namespace edg
