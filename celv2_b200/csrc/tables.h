// tables.h: the superblock's (block, 4x4 tile) work items.
//
// Item order: blocks grouped by size class, largest first -- 64x64 (1 block x 256 tiles),
// 64x32 / 32x64 (4 x 128), 32x32 (4 x 64), 32x16 / 16x32 (16 x 32), 16x16 (16 x 16), 16x8 / 8x16
// (64 x 8), 8x8 (64 x 4), 8x4 / 4x8 (256 x 2): 3072 items, every class boundary a multiple of 32,
// so a warp's 32 consecutive items hold whole blocks (or 32 tiles of one) and a block's tile sums
// reduce with shuffles over a power-of-two segment. Intra items are the last 2304 (blocks below
// 64x64 size, kMaxBlockSize, src/gpu/intra_common.h:39). Within a block, tiles are in raster order.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace celv2cu {

constexpr int kItems = 3072;       // every block's tiles

// Item i's block b, the block's place (x, y) in the superblock and the tile's (c0, r0) in the block, in
// samples, and log2 of the block's tiles: class c covers the squares of level c / 2, whole (even c) or
// as halves (odd c); a class's items all lie in one step of 256 (or several whole ones).
__device__ __forceinline__ void item_place(int i, int& b, int& x, int& y, int& c0, int& r0, int& lwt) {
  const int st = i >> 8;  // steps per class: 1, 2, 1, 2, 1, 2, 1, 2
  const int level = st / 3, sub = st - level * 3, lgs = 6 - level;
  lwt = 2 * (4 - level) - (sub != 0);
  const int k = (sub == 2 ? 256 : 0) + (i & 255), blk = k >> lwt, t = k & ((1 << lwt) - 1);
  const int idx = sub ? blk >> 2 : blk, kind = sub ? 1 + (blk & 3) : 0;
  b = (sb_level_offset(level) + idx) * 5 + kind;
  const int lgw = lgs - (kind >= 3), lgh = lgs - (kind == 1 || kind == 2);
  x = ((idx & ((1 << level) - 1)) << lgs) + (kind == 4 ? 1 << lgw : 0);
  y = ((idx >> level) << lgs) + (kind == 2 ? 1 << lgh : 0);
  c0 = (t & ((1 << (lgw - 2)) - 1)) * 4, r0 = (t >> (lgw - 2)) * 4;
}

}  // namespace celv2cu
