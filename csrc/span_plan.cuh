// How spans of a recurrence with a diagonal transition are run: by lin_scan (seqmix.cu), whole spans or segments of them (lin_span.cu).
//
// A call says how many sequences and how long.  One for a captured graph (`ragged`) gives the sizes of its bucket -- 2 to 8 prompts are 8 sequences,
// lengths are rounded up to a power of two, one long prompt may stand beside short ones --, so there the choice is made on the device, from
// q_len: pass 0 picks the segment length of a launch, and where lin_scan may be the faster one both kernels are launched and one of them leaves
// at once.  That costs 3 to 9 us, so calls whose sizes are true, and buckets whose sizes settle the choice, are planned on the host.
// 16 heads of 128, buckets of 8 sequences, us (lin_scan / plan for the bucket's sizes / here): 2 x 40 tokens 15 / 21 / 18, 2 x 100 32 / 44 / 34, 2 x 300
// 86 / 121 / 66, 2 x 1000 278 / 395 / 165, 2 x 2000 550 / 784 / 302, 2000 beside seven of 20 554 / 783 / 205; 8 x 40 55 / 21 / 27, 8 x 300 340 / 124 / 133.
//
// Measured times per token, ns (B200, GLA): lin_scan's blocks run side by side until about 28 heads (128 x 128) or 90 (64 x 64), then their time
// grows with the heads; a block of lin_span is one head, with one resident per SM at 128 x 128 (two at 64 x 64, at half the speed each).
// Segments: pass 0 takes 0.6 of pass 1's time, the three launches and the chain of the starts 10 us.
#pragma once
#include <cuda_runtime.h>

namespace b2b {

constexpr int SPAN_BLOCKS = 4 * 148;       // blocks of a pass over segments at most (bounds the workspace, too: 39 MB at 128 x 128)
constexpr int SPAN_MIN_SEG = 32;           // tokens
constexpr int SPAN_CHOICES = 64;           // segment lengths tried: 32, 48, .. 1040 tokens
constexpr int SPAN_SHORT_Q = 128;          // spans up to here may be left to lin_scan; three launches do not pay for them
constexpr int SPAN_MANY_HEADS = 96;        // one sequence of this many heads: segments do not pay

// Costs in ns, in whole numbers: every kernel of a launch has to come to the same choice.
typedef long long span_ns;
struct SpanWork {
  int longest, tokens;                     // of the live spans
};

// rounds of that many blocks over the machine, times 100
__host__ __device__ inline span_ns span_rounds(span_ns blocks, int dk) {
  const span_ns r = (blocks + 147) / 148;
  return dk == 128 ? 100 * r : (r > 1 ? 85 * r : 100);
}
__host__ __device__ inline int span_token_ns(int dk) { return dk == 128 ? 420 : 180; }
__host__ __device__ inline span_ns span_cost_scan(const SpanWork& w, int H, int dk) {
  const span_ns alone = static_cast<span_ns>(w.longest) * (dk == 128 ? 285 : 200), full = static_cast<span_ns>(w.tokens) * H * (dk == 128 ? 90 : 23) / 10;
  return alone > full ? alone : full;
}
__host__ __device__ inline span_ns span_cost_whole(const SpanWork& w, int H, int dk) {
  if (w.longest <= 0) return 2000;
  const span_ns blocks = (static_cast<span_ns>(w.tokens) * H + w.longest - 1) / w.longest;      // as if all were the longest
  return span_rounds(blocks, dk) * w.longest * span_token_ns(dk) / 100 + 2000;
}
__host__ __device__ inline bool span_whole_wins(const SpanWork& w, int H, int dk) { return span_cost_whole(w, H, dk) < span_cost_scan(w, H, dk); }

// `blocks` segments of L tokens over all heads, `chain` of one span
__host__ __device__ inline span_ns span_cost_cut(span_ns blocks, int chain, int L, int dk) {
  return span_rounds(blocks, dk) * L * span_token_ns(dk) * 16 / 1000 + 10000 + 300 * chain;
}
__host__ __device__ inline int span_choice(int c) { return SPAN_MIN_SEG + 16 * c; }
// (all spans are cut to the same length; more than `slots` segments in all do not fit)
__host__ __device__ inline span_ns span_cost_segments(const int* lens, int n_seqs, int longest, int L, int slots, int H, int dk) {
  constexpr span_ns never = 1LL << 60;
  if (L >= longest) return never;
  int segs = 0;
  for (int s = 0; s < n_seqs; ++s) segs += lens[s] > 0 ? (lens[s] + L - 1) / L : 0;
  if (segs > slots) return never;
  return span_cost_cut(static_cast<span_ns>(H) * segs, (longest + L - 1) / L, L, dk);
}

// workspace segments of a launch
__host__ __device__ inline int span_slots(int n_seqs, int max_q, int H) {
  const long long most = static_cast<long long>(n_seqs) * ((max_q + SPAN_MIN_SEG - 1) / SPAN_MIN_SEG);
  const int fit = SPAN_BLOCKS / H;
  return most < fit ? static_cast<int>(most) : fit;
}

#ifdef __CUDACC__
// the live spans, by a warp
__device__ inline SpanWork span_work(const int* lens, int n_seqs) {
  SpanWork w{0, 0};
  for (int s = threadIdx.x & 31; s < n_seqs; s += 32) {
    const int n = max(lens[s], 0);
    w.longest = max(w.longest, n);
    w.tokens += n;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    w.longest = max(w.longest, __shfl_xor_sync(0xffffffffu, w.longest, o));
    w.tokens += __shfl_xor_sync(0xffffffffu, w.tokens, o);
  }
  return w;
}
#endif

}  // namespace b2b
