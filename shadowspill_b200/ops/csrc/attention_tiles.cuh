// Which tile of which packed sequence a CTA of the attention kernels takes.
//
// A causal tile's work is proportional to its distance from one end of its sequence (queries: from the
// start, keys: from the end), and a sequence of n tiles has exactly one tile of each work 1..n. CTAs
// start in the order of their rank, so ranking by descending work starts the long tiles first and
// leaves the short ones to fill the last wave.
#pragma once
#include <cuda_runtime.h>

namespace ss {

struct TileSlot {
  int seq_start, seq_end;
  int work;          // in tiles; 0 = this rank has no tile
};

// The tile of rank `rank` in descending work, `rows` rows to a tile. Executed by ONE full warp; the
// slot is in shared memory and is read after the block's next barrier.
__device__ __forceinline__ void find_tile_by_work(const int* cu, int nseq, int rows, int rank,
                                                  TileSlot* slot) {
  const int lane = threadIdx.x & 31;
  // tiles with at least `w` work; each sequence contributes max(0, n - w + 1)
  auto at_least = [&](int w) {
    int c = 0;
    for (int s = lane; s < nseq; s += 32) c += max(0, (cu[s + 1] - cu[s] + rows - 1) / rows - w + 1);
    return __reduce_add_sync(0xffffffffu, c);
  };
  int longest = 0;
  for (int s = lane; s < nseq; s += 32) longest = max(longest, (cu[s + 1] - cu[s] + rows - 1) / rows);
  longest = __reduce_max_sync(0xffffffffu, longest);
  int lo = 0, hi = longest;               // the largest w in [1, longest] with at_least(w) > rank
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (at_least(mid) > rank) lo = mid; else hi = mid - 1;
  }
  if (lo == 0) {
    if (lane == 0) { slot->seq_start = slot->seq_end = 0; slot->work = 0; }
    return;
  }
  int skip = rank - at_least(lo + 1);     // sequences that have a tile of this work, in order
  for (int s0 = 0; s0 < nseq; s0 += 32) {
    const int s = s0 + lane;
    const bool has = s < nseq && (cu[s + 1] - cu[s] + rows - 1) / rows >= lo;
    const unsigned vote = __ballot_sync(0xffffffffu, has);
    const int before = __popc(vote & ((1u << lane) - 1));
    if (has && before == skip) { slot->seq_start = cu[s]; slot->seq_end = cu[s + 1]; slot->work = lo; }
    if (skip < __popc(vote)) return;
    skip -= __popc(vote);
  }
}

}  // namespace ss
