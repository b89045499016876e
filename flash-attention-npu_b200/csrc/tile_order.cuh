// Order of the query tiles of ragged input, as arithmetic that the device (fwd_tc5_kernel.cuh) and a host test share.
//
// Position n -> tile: the heads are cut into chunks of chunk_heads; a chunk runs its tiles by level, highest first; a level
// holds at most one tile of every batch entry, for all heads of the chunk.  Tiles that do not exist have no position.
// Positions may be asked for in any order: the cursor only saves the walk down from the highest level when they grow,
// which is what a CTA usually sees (nothing promises it: clusterlaunchcontrol hands out whichever CTA has not started).
#pragma once

#ifdef __CUDACC__
#define FA_TILE_HD __host__ __device__ __forceinline__
#else
#define FA_TILE_HD inline
#endif

#include <stdint.h>

namespace fa {

// n / d for 0 <= n < 2^31 as a multiplication: mul = ceil(2^(31 + s) / d) with 2^s >= d exceeds 2^(31 + s) / d by less than
// 2^s / d, so the quotient is off by less than n / 2^31 / d < 1 / d and its whole part is exact.  Every role of the prefill kernel
// finds its tile by itself, four or five divisions by run-time values, of some 100 cycles each as the compiler does them.
struct FastDiv {
  uint32_t mul, shift;  // mul 0: d = 1
  void set(int d) {
    mul = shift = 0;
    if (d <= 1) return;
    const uint32_t s = 32 - (uint32_t)__builtin_clz((uint32_t)d - 1);  // (six to nine of these a call: no loop)
    mul = (uint32_t)(((1ull << (31 + s)) + (uint32_t)d - 1) / (uint32_t)d);
    shift = s - 1;
  }
  FA_TILE_HD int div(int n) const {
    return mul ? (int)(((uint64_t)(uint32_t)n * mul) >> 32 >> shift) : n;
  }
};

// Levels must offer:  int live (tiles of one head over all batch entries), int top (highest level that holds a tile),
// int count(level) (batch entries with a tile in it).
struct TileCursor {
  int chunk = 0;
  int level = -1;  // of the last position; -1: none yet
  int start = 0;   // the level's first position in the chunk
  int cnt = 0;     // tiles per head in the level
};

// False: position n has no tile.  Otherwise the tile of head `head` is that of the rank-th batch entry of cursor.level.
template <class Levels>
FA_TILE_HD bool tile_locate(TileCursor& c, const Levels& lv, int heads_all, int chunk_heads, int n, int& head, int& rank) {
  if (n >= lv.live * heads_all) return false;
  const int ck = n / (lv.live * chunk_heads);
  const int left = heads_all - ck * chunk_heads, heads = chunk_heads < left ? chunk_heads : left;
  n -= ck * lv.live * chunk_heads;
  if (c.level < 0 || ck != c.chunk || n < c.start) {  // from the top again
    c.chunk = ck;
    c.level = lv.top + 1;
    c.start = c.cnt = 0;
  }
  while (c.level > 0 && n >= c.start + c.cnt * heads) {  // the levels down to 0 hold `live` tiles per head
    c.start += c.cnt * heads;
    --c.level;
    c.cnt = lv.count(c.level);
  }
  head = ck * chunk_heads + (n - c.start) % heads;
  rank = (n - c.start) / heads;
  return true;
}

// Order of the backward's work items, shared with a host test too.  An item is a block of 128 keys or rows of a (batch entry,
// head) pair.  Items near one another should stream the same tiles (from L2), which asks for a pair's blocks to be neighbours; but under a causal mask a pair's
// blocks differ by up to the length of the sequence, and a launch that ends on the heavy blocks of its last pair leaves most
// CTAs idle meanwhile.  So the pairs are cut into chunks, and a chunk runs block 0 of all its pairs, then block 1, and so on
// (bwd_chunk in bwd.cu; a chunk of one pair is the plain order).  One pair at a time / all pairs together, forward and
// backward: 12 packed sequences of 37 - 2999 rows (16 heads of 4 groups, head dim 64) 635 / 607 us; b 2, s 1777, 8 heads, head
// dim 256 (bwd_wide_kernel) 208 / 192 us.
struct ItemPlace {
  int pair, block;
};
struct ItemOrder {
  int blocks, pairs, chunk;
  FastDiv by_chunk_items, by_chunk, by_last;  // items of a chunk, its pairs, the pairs of the last chunk (if that is short)
  void set(int blocks_, int pairs_, int chunk_) {
    blocks = blocks_;
    pairs = pairs_;
    chunk = chunk_;
    by_chunk_items.set(chunk * blocks);
    by_chunk.set(chunk);
    by_last.set(chunk > 0 ? pairs % chunk : 0);
  }
  FA_TILE_HD ItemPlace place(int t) const {
    const int ck = by_chunk_items.div(t), r = t - ck * chunk * blocks, first = ck * chunk;
    const int cnt = chunk < pairs - first ? chunk : pairs - first;  // pairs in this chunk (the last one may be short)
    const int nb = cnt == chunk ? by_chunk.div(r) : by_last.div(r);
    return {first + r - nb * cnt, nb};
  }
};

}  // namespace fa
