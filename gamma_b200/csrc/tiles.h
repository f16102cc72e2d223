// The tiles of a grid-strided pass: block `block` of `blocks` takes every
// blocks-th tile of `tile` items.  Positions are 64-bit: near the largest int a
// 32-bit one would wrap when a block steps past the last tile, and never end.
#pragma once

#ifdef __CUDACC__
#define GB_TILES_HD __host__ __device__
#else
#define GB_TILES_HD
#endif

namespace gb {

// tiles of n items
GB_TILES_HD constexpr long long tile_count(long long n, int tile) { return (n + tile - 1) / tile; }

// for (Tiles t(n, tile, block, blocks); t.more(); t.next()) ... t.base ...
struct Tiles {
  long long base, step, end;  // first item of the tile; items
  GB_TILES_HD Tiles(int n, int tile, int block, int blocks)
      : base((long long)block * tile), step((long long)blocks * tile), end(n) {}
  GB_TILES_HD bool more() const { return base < end; }
  GB_TILES_HD void next() { base += step; }
};

}  // namespace gb
