// Packed sequences: which rows of the token tensors a tile of a launch covers. Tiles never span sequences: a row of another
// sequence beside them, finite or not, takes no part in any sum. (With tiles cut at fixed rows a NaN reached the sequences that
// shared a tile, because zero probabilities still multiply it. They were faster, 8192 tokens, 16 heads, d = 128, forward and
// backward kernel: 5 sequences 185 + 486 us against 182 + 520, 128 sequences of 64 tokens 57 + 132 us against 132 + 203.)
#pragma once
#include "fdma_internal.h"

namespace fdma {

// Tiles of `rows` rows of one of the two token tensors (`total` rows): each sequence, and what lies before the first and after
// the last, starts a tile of its own. A launch has packed_slots() places for them, a few of which stay empty.
__host__ __device__ __forceinline__ int packed_slots(int total, int n, int rows) { return total / rows + n + 2; }

struct PackedTile {
  int seq;         // -1 and n: rows that belong to no sequence
  int begin, end;  // the rows of the sequence
  int tile;        // the tile covers [begin + tile * rows, ...) and is empty from `end` on
};

__device__ __forceinline__ int packed_bound(const int32_t* cu, int n, int total, int seq) {  // first row of a sequence
  return seq < 0 ? 0 : seq > n ? total : min(max(cu[seq], 0), total);
}

// By a whole warp. Sequence s takes the slots from first_row / rows + s + 1 on; 32-way search for the last one that starts at or
// before `slot`.
__device__ __forceinline__ PackedTile packed_tile(const int32_t* cu, int n, int total, int rows, int slot) {
  const int lane = threadIdx.x & 31;
  int lo = -1, len = n + 2;  // the sequence is in [lo, lo + len)
  while (len > 1) {
    const int step = (len + 31) / 32;
    const int s = lo + lane * step;
    const bool before = lane * step < len && packed_bound(cu, n, total, s) / rows + s + 1 <= slot;
    const int cnt = max(1, __popc(__ballot_sync(0xffffffffu, before)));
    len = min(step, len - (cnt - 1) * step);
    lo += (cnt - 1) * step;
  }
  PackedTile t;
  t.seq = lo;
  t.begin = packed_bound(cu, n, total, lo);
  t.end = max(t.begin, packed_bound(cu, n, total, lo + 1));
  t.tile = slot - (t.begin / rows + lo + 1);
  return t;
}
// The rows of the other tensor that a sequence has.
__device__ __forceinline__ int2 packed_range(const int32_t* cu, int n, int total, int seq) {
  if (seq < 0 || seq >= n) return make_int2(0, 0);
  const int begin = packed_bound(cu, n, total, seq);
  return make_int2(begin, max(begin, packed_bound(cu, n, total, seq + 1)));
}

// Rows [from, to) of a 128-byte-swizzled tile of `blocks` column blocks become zero, by a whole warp: what TMA would have filled
// in had the tensor ended there. (The swizzle moves 16-byte pieces inside their 128-byte row.) The caller makes the writes
// visible to the tensor core.
__device__ __forceinline__ void zero_tile_rows(unsigned char* tile, int blocks, int block_bytes, int from, int to) {
  const int pieces = (to - from) * 8;
  for (int b = 0; b < blocks; ++b)
    for (int i = threadIdx.x & 31; i < pieces; i += 32)
      *reinterpret_cast<uint4*>(tile + b * block_bytes + from * 128 + i * 16) = make_uint4(0, 0, 0, 0);
}

}  // namespace fdma
