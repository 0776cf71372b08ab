// What the pairs of CTAs of gemm_wide.cu work on, and which of their tiles' accumulators somebody waits for.
#pragma once
#include <cuda_runtime.h>

namespace b2b {

// tile `t`, k-blocks [kb0, kb1), `split`: the other pair of the cluster has the rest of K
struct WideItem {
  int t, kb0, kb1;
  bool split;
};

struct WidePlan {
  int tiles, tok_tiles, nkb, pairs, full, rest;
  bool split;

  // `may_split`: clusters of four
  __host__ __device__ WidePlan(int tok_tiles_, int feature_tiles, int nkb_, int pairs_, bool may_split)
      : tiles(tok_tiles_ * feature_tiles), tok_tiles(tok_tiles_), nkb(nkb_), pairs(pairs_), full(tiles / pairs * pairs), rest(tiles - full),
        split(may_split && rest > 0 && rest <= pairs / 2) {}

  __host__ __device__ bool get(int i, int pair, WideItem& it) const {
    const int t = pair + i * pairs;
    if (t < full) {
      it = {t, 0, nkb, false};
      return true;
    }
    if (i != full / pairs) return false;
    if (split) {
      if ((pair >> 1) >= rest) return false;
      const int half = nkb / 2;
      it = {full + (pair >> 1), (pair & 1) ? half : 0, (pair & 1) ? nkb : half, true};
      return true;
    }
    it = {t, 0, nkb, false};
    return t < tiles;
  }

  // The products of item `i` wait until the accumulator of item i - wide_gap has been read, and nothing else waits for that: readers of an accumulator whose
  // columns are not used again say nothing.  (The odd CTA's would arrive in the even one's shared memory while that CTA, which no longer looks, may have left.)
  __host__ __device__ bool awaited(int i, int pair, int gap) const {
    WideItem it;
    return get(i + gap, pair, it);
  }
};

// accumulators that overlap: the next item waits; else the one after that
__host__ __device__ constexpr int wide_gap(bool overlap) { return overlap ? 1 : 2; }

}  // namespace b2b
