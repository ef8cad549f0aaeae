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


// ---- hop tables (basis.cu)
constexpr int kDwHops = 32;  // hops per row that the grouped down pass takes

// Hops of one spin's table: a directed bond acts on the configurations that have its first site
// occupied and its second one empty.
inline uint64_t hop_total(int ns, int nel, int64_t bonds) {
  if (nel < 1 || nel >= ns) return 0;
  uint64_t c = 1;  // C(ns - 2, nel - 1)
  for (int i = 1; i < nel; ++i) c = c * uint64_t(ns - 1 - i) / uint64_t(i);
  return c * uint64_t(bonds);
}
// Table offsets are 32-bit.
inline bool table_fits(uint64_t entries) { return entries < 0xffffffffull; }

// Whether a direct-form sector gets hop tables: the row tiles read them, so its rows have to fit a
// tile, and as the form is there to need no memory beside its vectors they may take 64 MB or a
// sixteenth of an FP64 vector (28 bytes a hop, complex, or 16: source and both precisions). Every
// nearest-neighbour lattice of up to 18 sites keeps within that; short rows beside very many of the other spin do not.
inline bool direct_tables(int64_t dimup, int64_t dimdw, uint64_t hops_up, uint64_t hops_dw, bool cplx) {
  if (tile_smem(dimup, 0, 0, 0) > kTileSmemMax || !table_fits(hops_up) || !table_fits(hops_dw)) return false;
  const uint64_t vec = uint64_t(dimup) * uint64_t(dimdw) * (cplx ? 16 : 8);
  const uint64_t room = vec / 16 > (uint64_t(64) << 20) ? vec / 16 : uint64_t(64) << 20;
  return (hops_up + hops_dw) * (cplx ? 28 : 16) <= room;
}

}  // namespace edg
