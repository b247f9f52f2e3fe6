// The list of query (or key) tiles that the persistent attention kernels walk through.
#pragma once
#include "ptx.cuh"

namespace mb {

// Items are ordered by level (tile index within a sequence), last level first, then by sequence, then by `per_seq` (heads or pairs of heads),
// and dealt to the CTAs forth and back (0..G-1, G-1..0, ...): under the causal mask the last tiles are the longest, and the sums
// of unlike items stay level without atomics.  All lanes of a warp call `next` together; 32 sequences per step.
struct ItemList {
  const int* cu_seqlens;
  int batch, per_seq, levels, rows;      // rows of a level
};

struct Items {
  int level, chunk, base, round;
  uint32_t mask;                         // sequences chunk·32 + i that have rows at this level
  __device__ __forceinline__ void scan(const ItemList& l) {
    const int b = chunk * 32 + static_cast<int>(lane_id());
    int len = 0;
    if (b < l.batch) len = l.cu_seqlens[b + 1] - l.cu_seqlens[b];
    mask = __ballot_sync(0xffffffffu, len > level * l.rows);
  }
  __device__ __forceinline__ void init(const ItemList& l) {
    level = l.levels - 1;
    chunk = base = round = 0;
    scan(l);
  }
  __device__ __forceinline__ bool next(const ItemList& l, int& b, int& sub) {
    const int g = static_cast<int>(gridDim.x), i = static_cast<int>(blockIdx.x);
    const int target = round * g + ((round & 1) ? g - 1 - i : i);
    ++round;
    for (;;) {
      const int n = __popc(mask) * l.per_seq;
      if (target < base + n) {
        const int at = target - base;
        b = chunk * 32 + static_cast<int>(__fns(mask, 0, at / l.per_seq + 1));
        sub = at % l.per_seq;
        return true;
      }
      base += n;
      if (++chunk * 32 >= l.batch) {
        chunk = 0;
        if (--level < 0) return false;
      }
      scan(l);
    }
  }
};

}  // namespace mb
