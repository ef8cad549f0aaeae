// limits.h -- host-side rules that say which sectors a kernel or a table can take: sizes and
// index widths only, plain C++, so that they can be checked without a GPU.
#pragma once

#include <cstddef>
#include <cstdint>

namespace edg {

constexpr size_t kSmemPerBlock = 227 * 1024;  // shared memory of one block, dynamic and static

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


// Whether the tiles beat the kernels that take an element per lane and gather (k_hxv_fused,
// k_cplx_stored); hops: mean hops per state, both spins. Stored form (the direct form's bitstring
// kernels never win). The gathers cost a read per hop; a tile costs its staging, by many blocks
// where rows are few, and lanes that idle where they are short (a slice has 32). us, tiles /
// gathers, on rings (9 to 13 hops) and square lattices (14 to 24):
//   FP64        ring 462 x 165 5.0 / 5.3, 91 x 1,001 4.4 / 4.2, 3,060 x 18 6.1 / 4.3, 15 x 5,005
//               7.8 / 5.0;  5x3 3,003 x 15 6.4 / 7.3, 6,435 x 15 7.6 / 10.7;  4x3 220 x 220 7.6 / 8.1
//   FP32        ring 495 x 495 6.5 / 6.6, 12,376 x 17 9.9 / 6.9;  5x3 3,003 x 105 9.7 / 14.8
//   complex128  ring 153 x 3,060 15.9 / 14.5, 5,005 x 15 8.0 / 6.3, 18 x 18,564 21 / 10, beyond one
//               launch 210 x 352,716 (14.8 hops) 3,520 / 2,900;  4x4 120 x 8,008 38 / 56, 4,368 x 16 7.2 / 10.4;
//               4x3 12 x 924 4.5 / 5.9;  5x4 20 x 184,756 303 / 216
//   complex64   ring 84 x 84 4.2 / 3.4, 120 x 560 4.7 / 3.8, 220 x 792 5.7 / 5.7, 18 x 18,564 16 / 8;
//               4x3 924 x 66 5.9 / 6.8;  4x4 120 x 8,008 23 / 38
// So the line lies at a number of reads, states x hops. Real sectors above 500,000 states take the
// tiles in any shape: the two passes that ran there before lose to either (18 x 48,620 FP64 39 us
// by tiles, 131 in two passes).
constexpr int64_t kFusedMaxDimC = 10000000;  // complex sectors of one launch, either precision
inline bool tile_pays(bool cplx, size_t real, int64_t dimup, int64_t dimdw, double hops) {
  const int64_t dim = dimup * dimdw;
  const double reads = double(dim) * hops;
  if (!cplx && dim > 500000) return true;
  if (dimup < 32) return cplx && real == 8 && hops >= 14.0 && dim < 32768;
  if (!cplx && real == 8) return reads >= (dimup >= 64 && dimdw >= 64 ? 6.5e5 : 1.2e6);
  if (!cplx) return reads >= 3.2e6;
  if (real == 4) return reads >= 1.2e6;
  if (dim > kFusedMaxDimC) return dimup >= 256 || hops >= 18.0;
  return dimdw >= 32 || hops >= 10.5 || dim >= 120000;
}

// ---- default H x v of a real stored sector: the single pass or two
// Single pass by gathers against two passes where the row tiles do not take the whole product (one
// |value| of up hops and several of down hops, or more than 256), us, FP64:
//   two values  3x4 (6,6), 853,776 states  61 / 41     4x4 (5,4), 7.9 M    580 / 212
//   17 sites all-to-all (5,3), 4.2 M      975 / 350    7x2 (7,3), 364 rows  64 / 58
//   two values  4x4 (7,2), 120 rows       120 / 168    5x3 (7,2), 105 rows  61 / 189
//   rows beyond the tiles  17-site ring (8,2) 106 / 201, 6x3 (9,2) 649 / 859
// So: two passes above 500,000 states, but where rows are too long for a tile, or fewer than two
// per SM, which leaves SMs idle in either pass.
constexpr int64_t kGatherMaxDim = 500000, kGatherMaxRows = 296;
inline bool single_pass_default(int64_t dimup, int64_t dimdw, int64_t most, bool tiles) {
  const int64_t dim = dimup * dimdw;
  if (dim > most) return false;
  return tiles || dim <= kGatherMaxDim || dimdw < kGatherMaxRows || tile_smem(dimup, 0, 0, 0) > kTileSmemMax;
}

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


// ---- row groups of the grouped down pass (k_dw_grp)
// Shared memory of a row of a group: its hop values (W reals each) and sources, its diagonal term,
// index, configuration and hop count.
inline size_t dw_row_smem(size_t real, int W) { return size_t(kDwHops) * (W * real + 4) + real + 12; }
inline size_t dw_group_smem(int64_t rows, size_t real, int W) { return size_t(rows) * dw_row_smem(real, W) + 16; }
// Most rows of a group: four blocks per SM stay resident.
constexpr size_t kDwGroupSmem = 52 * 1024;
inline int64_t dw_group_most(size_t real, int W) { return int64_t((kDwGroupSmem - 16) / dw_row_smem(real, W)); }
// Number of groups: one per resident block, all of them at work on the same slab of columns, or,
// where those would be larger (from 73,000 FP64 rows, 44,000 complex128), as many for each of
// several turns, with a sixteenth of room to even out their hops. ms per H x v with one group per
// resident block whatever its size (one block per SM of 200 KB at the most, a failed launch
// beyond) and now: 20-site ring (2,10), 184,756 rows, complex128 2.51 and 1.32, real FP64 1.42
// and 0.65; 5x4 lattice (3,8), 125,970 rows, complex128 13.9 and 7.3, FP32 2.01 and 1.43.
inline int64_t dw_group_count(int64_t dim, int64_t resident, size_t real, int W) {
  const int64_t rows = dw_group_most(real, W) * 15 / 16;
  if (dim <= resident) return dim < 1 ? 1 : dim;
  return resident * ((dim + resident * rows - 1) / (resident * rows));
}

}  // namespace edg
