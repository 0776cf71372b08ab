// Gated linear recurrences over spans whose transition is diagonal (lin_scan's GLA, mLSTM, HGRN2 and state-space modes), in fp32:
//
//     S <- diag(d_t) S + k_t v_t^T;   o_t = S^T q_t          (what d, k, q are per mode: see lin_scan in seqmix.cu)
//
// The arithmetic is lin_scan's, product for product (only the order of the sum over the key channels differs); what differs is the
// layout.  lin_scan gives a thread 8 x 2 state elements and one sequence heads x column blocks of parallel work: 24 shared-memory words and a
// chain of four shuffles per 48 operations, on one warp per scheduler.  Here
//
//   * a block has a whole head: 16 lanes x (dk / 16) rows, 4 columns per thread, so an operand word serves four elements; the operations are
//     packed pairs of rows (fma.rn.f32x2: the same IEEE results at half the issue slots), and the sums over the lanes are taken for
//     four tokens at once (15 shuffles per four tokens and four columns);
//   * one sequence is cut into segments that run side by side: pass 0 computes what each segment adds to a zero state and the
//     product of its decays, `lin_span_starts` chains them (S_start(g + 1) = D_g S_start(g) + local_g), pass 1 runs every segment from its
//     start.  Pass 0 takes 0.6 of pass 1's time, so it is done only where heads x sequences do not fill the machine
//     (where the sizes of the launch are a bucket's, pass 0 finds that out, and how long the segments are, from q_len: span_plan.cuh).
//
// (Retention stays with lin_scan: its constant decay rounds the same way at every step, and the products of a segment's decays drift
// further from the exact ones than the state does token by token: 3.1e-7 against 2.4e-7 over 500 tokens.)
//
// Bound (ncu, 128 x 128): shared-memory reads of the operands 65 %, fp32 pipes 57 %, 2.2 instructions per cycle of 4.  8 columns per thread
// (2 warps per scheduler, 40 % fewer reads) measured the same.  One head: 0.42 us per token at 128 x 128, 0.18 at 64 x 64.
// Measured on B200, GLA, lin_scan -> here (us): 16 heads of 128: one span of 2048 tokens 583 -> 161, 512 tokens 149 -> 56, 4 spans of 512
// 286 -> 175, 32 of 64 295 -> 119; 16 heads of 64: 2048 tokens 414 -> 69.  The error against 64 bits is that of lin_scan.
// This translation unit is compiled WITHOUT --use_fast_math.
#include "kernels.h"

#include <cstdint>

#include "fp32x2.cuh"
#include "launch.cuh"
#include "span_plan.cuh"

namespace b2b {
namespace {

enum { LS_GLA = 0, LS_MLSTM = 2, LS_HGRN2 = 3, LS_SSD = 4 };

__device__ __forceinline__ float sp_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float sp_silu(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float sp_softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sp_logsigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

struct SpanArgs {
  const float* qk;  int ld_qk, off_q, off_k;
  const float* v;   int ld_v, off_v;
  const float* z;   int ld_z, off_z;
  const float* zbias;
  const float* hparam;
  const float* beta; int ld_b, off_b;
  const float* aux;
  float qscale, inv_tau;
  float* state; float* out; int ld_out;
  const int* q_start; const int* q_len; const int* kv_len; const int* seq_slot;
  int H, G, n_seqs;
  int seg;                  // tokens per segment (0: a span is one segment), unless that is planned here (PLAN)
  int slots;                // segments in the workspace: seg: the same number per sequence; PLAN: those of the sequences behind one another
  int choose;               // PLAN: lin_scan is launched, too: leave the spans to it where it is faster
  int* plan;                // PLAN: tokens per segment as pass 0 found best, 0: spans are not cut
  float* local;             // [slots][H][dk][dv]: what a segment adds, then the state it starts from
  float* decay;             // [slots][H][dk]: product of its decays
};

constexpr int ST = 16;      // tokens per staged tile

template <int DK, int DV>
struct SpanCfg {
  static constexpr int kThreads = 4 * DV;                     // 16 lanes x DV / 4 column groups
  static constexpr int R = DK / 16;                           // state rows per thread
  static constexpr int kBuf = 3 * ST * DK + ST * 2 * DV;      // d, k, q; v with every value twice (an operand of packed pairs)
  static constexpr int kSmem = 2 * kBuf * 4;
  static constexpr int kBlocks = DK == 128 ? 1 : 2;           // per SM
};

// state rows of lane ti: ti*4 .. +3 and, for 128 rows, 64 + ti*4 .. +3
__device__ __forceinline__ int state_row(int ti, int r) { return (r >> 2) * 64 + ti * 4 + (r & 3); }

// (p + e) <- (p + e) d, e the rounding error of p: a constant decay rounds the same way every time, so a plain product drifts
__device__ __forceinline__ void chain(float& p, float& e, float d) {
  const float x = p * d;
  e = e * d + fmaf(p, d, -x);
  p = x;
}

// segments of a span
__device__ __forceinline__ int span_segments(const SpanArgs& a, int s, int L) { return s < a.n_seqs && a.q_len[s] > 0 ? (a.q_len[s] + L - 1) / L : 0; }

// sequence and segment of a workspace slot, by a warp; false behind the last one
__device__ __forceinline__ bool span_of_slot(const SpanArgs& a, int L, int slot, int& s, int& g) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int base = 0; base < a.n_seqs; base += 32) {
    const int n = span_segments(a, base + lane, L);
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, slot < before + upto);
    if (hit != 0u) {
      const int at = __ffs(hit) - 1;
      s = base + at;
      g = slot - before - __shfl_sync(0xffffffffu, upto - n, at);
      return true;
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// the cheapest segment length of this launch (0: spans are not cut), by the first SPAN_CHOICES threads of a block
__device__ __forceinline__ int span_plan(const SpanArgs& a, int dk) {
  __shared__ span_ns cost_s[SPAN_CHOICES / 32];
  __shared__ int len_s[SPAN_CHOICES / 32];
  const SpanWork w = span_work(a.q_len, a.n_seqs);
  if (threadIdx.x < SPAN_CHOICES) {
    int L = span_choice(threadIdx.x);
    span_ns cost = span_cost_segments(a.q_len, a.n_seqs, w.longest, L, a.slots, a.H, dk);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const span_ns c = __shfl_xor_sync(0xffffffffu, cost, o);
      const int l = __shfl_xor_sync(0xffffffffu, L, o);
      if (c < cost || (c == cost && l > L)) {
        cost = c;
        L = l;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      cost_s[threadIdx.x >> 5] = cost;
      len_s[threadIdx.x >> 5] = L;
    }
  }
  __syncthreads();
  span_ns best = span_cost_whole(w, a.H, dk);
  int plan = 0;
#pragma unroll
  for (int i = 0; i < SPAN_CHOICES / 32; ++i)
    if (cost_s[i] < best) {
      best = cost_s[i];
      plan = len_s[i];
    }
  return plan;
}

// Pass over segments or spans, a head of one per block.  grid (segments, heads, sequences); PLAN: (heads, slots or sequences), and the local pass, every
// block of which finds the plan first, is only as large as the machine and walks (592 blocks without work took 12 us).
template <int MODE, int DK, int DV, bool OUT, bool PLAN>
__global__ void __launch_bounds__(SpanCfg<DK, DV>::kThreads, SpanCfg<DK, DV>::kBlocks) lin_span_kernel(SpanArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  using Cfg = SpanCfg<DK, DV>;
  constexpr int NT = Cfg::kThreads, R = Cfg::R;
  constexpr bool ZC = MODE == LS_GLA || MODE == LS_HGRN2;
  static_assert(NT == 4 * DK && ST * DV == 4 * NT, "staging: a thread prepares one channel of four tokens and four values");
  extern __shared__ __align__(16) float sm[];

  constexpr bool WALK = PLAN && !OUT;
  int plan = a.seg;                                           // (all branches on the plan and the lengths are block-uniform)
  if constexpr (WALK) {
    plan = span_plan(a, DK);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.plan = plan;
    if (plan == 0) return;
  } else if constexpr (PLAN) {
    plan = a.slots > 0 ? *a.plan : 0;
    if (a.choose && !span_whole_wins(span_work(a.q_len, a.n_seqs), a.H, DK)) return;
  }
#pragma unroll 1
  for (int item = WALK ? blockIdx.x : 0;; item += gridDim.x) {
    if (!WALK && item > 0) return;
    int s, g, slot, hd;
    if constexpr (PLAN) {
      slot = WALK ? item / a.H : blockIdx.y;
      hd = WALK ? item - slot * a.H : blockIdx.x;
      s = slot;
      g = 0;
      if (plan > 0 ? !span_of_slot(a, plan, slot, s, g) : s >= a.n_seqs) return;
    } else {
      s = blockIdx.z;
      hd = blockIdx.y;
      g = blockIdx.x;
      slot = s * gridDim.x + g;
    }
    const int len = a.q_len[s];
    const int seg = plan > 0 ? plan : len;
    const int n_seg = len > 0 ? (len + seg - 1) / seg : 0;
    if (g >= n_seg || (!OUT && g == n_seg - 1)) continue;
    const int t0 = a.q_start[s] + g * seg;
    const int n = min(seg, len - g * seg);
    const int H = a.H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ti = lane & 15, cg = warp * 2 + (lane >> 4);
    const int hqk = MODE == LS_SSD ? hd / (H / a.G) : hd;
    float* S_g = a.state + (static_cast<size_t>(a.seq_slot[s]) * H + hd) * (static_cast<size_t>(DK) * DV);
    const size_t ws = static_cast<size_t>(slot) * H + hd;
    float* W_g = plan > 0 ? a.local + ws * (static_cast<size_t>(DK) * DV) : nullptr;

    pair32 S[R / 2][4];                                         // rows state_row(ti, 2 m) and the next one, columns cg*4 .. +3
    {
      const float* src = OUT ? (plan > 0 ? W_g : (a.kv_len[s] - len > 0 ? S_g : nullptr)) : nullptr;
#pragma unroll
      for (int m = 0; m < R / 2; ++m) {
        float4 x[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          x[r] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (src != nullptr) x[r] = *reinterpret_cast<const float4*>(src + static_cast<size_t>(state_row(ti, 2 * m + r)) * DV + cg * 4);
        }
        S[m][0] = pack32(x[0].x, x[1].x);
        S[m][1] = pack32(x[0].y, x[1].y);
        S[m][2] = pack32(x[0].z, x[1].z);
        S[m][3] = pack32(x[0].w, x[1].w);
      }
    }

    // ---- staging: raw rows of the next tile travel through registers; this thread has channel c of quarter `st` of a tile
    const int c = tid % DK, st = tid / DK;
    float rq[4], rk[4], rz[4], rg[4];
    float4 rv;
    const int vt = tid / (DV / 4), ve = tid % (DV / 4);
    float total = 1.f, total_e = 0.f;                           // product of the decays and its rounding error
    const float rate = MODE == LS_SSD ? expf(a.hparam[hd]) : 0.f;
    const float hconst = MODE == LS_SSD ? a.zbias[hd] : 0.f;
    const float zb = ZC ? a.zbias[hd * DK + c] : 0.f;
    const float lo = MODE == LS_HGRN2 ? a.hparam[hd * DK + c] : 0.f;
    auto fetch = [&](int tb) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool ok = tb + st * 4 + j < n;
        const size_t t = static_cast<size_t>(t0 + (ok ? tb + st * 4 + j : 0));
        const float* row = a.qk + t * a.ld_qk + hqk * DK + c;
        rq[j] = (OUT && ok) ? row[a.off_q] : 0.f;
        rk[j] = (MODE != LS_HGRN2 && ok) ? row[a.off_k] : 0.f;
        rz[j] = 0.f;
        rg[j] = 0.f;
        if (ZC) rz[j] = ok ? a.z[t * a.ld_z + a.off_z + hd * DK + c] : 0.f;
        if (MODE == LS_SSD) rz[j] = ok ? a.beta[t * a.ld_b + a.off_b + hd] : 0.f;
        if (MODE == LS_MLSTM) {
          const float4 x = ok ? *reinterpret_cast<const float4*>(a.aux + (t * H + hd) * 4) : make_float4(1.f, 0.f, 0.f, 0.f);
          rz[j] = x.x;
          rg[j] = x.y;
        }
      }
      rv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tb + vt < n) rv = *reinterpret_cast<const float4*>(a.v + static_cast<size_t>(t0 + tb + vt) * a.ld_v + a.off_v + hd * DV + 4 * ve);
    };
    auto stage = [&](int tb, float* b) {
      float *ds = b, *ks = b + ST * DK, *qs = b + 2 * ST * DK, *vs = b + 3 * ST * DK;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float q = rq[j], k = rk[j], d = 1.f;
        if (MODE == LS_GLA) d = expf(sp_logsigmoid(rz[j] + zb) * a.inv_tau);
        if (MODE == LS_MLSTM) {
          d = rz[j];
          k *= rg[j];
        }
        if (MODE == LS_SSD) {
          const float dt = sp_softplus(rz[j] + hconst);
          d = expf(-rate * dt);
          k *= dt;
        }
        if (MODE == LS_HGRN2) {
          d = lo + (1.f - lo) * sp_sigmoid(rz[j] + zb);
          k = 1.f - d;
          q = sp_silu(q);
        } else {
          q *= a.qscale;
        }
        if (tb + st * 4 + j >= n) {                             // past the end: the state stays as it is
          d = 1.f;
          k = 0.f;
        }
        const int o = (st * 4 + j) * DK + c;
        if (OUT) {
          ds[o] = d;
          ks[o] = k;
          qs[o] = q;
        } else {
          rz[j] = d;
          rk[j] = k;
        }
      }
      if constexpr (!OUT) {
        // no output wants the states inside four tokens: S <- (d1 d2 d3 d4) S + sum_t (k_t times the later decays) v_t^T
        float p = 1.f, e = 0.f;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          ks[(st * 4 + j) * DK + c] = rk[j] * (p + e);
          chain(p, e, rz[j]);
        }
        ds[st * DK + c] = p + e;
        const float before = total + total_e;                   // total <- total (p + e)
        chain(total, total_e, p);
        total_e += before * e;
      }
      float4* dst = reinterpret_cast<float4*>(vs + vt * 2 * DV + 8 * ve);
      dst[0] = make_float4(rv.x, rv.x, rv.y, rv.y);
      dst[1] = make_float4(rv.z, rv.z, rv.w, rv.w);
    };

    // ---- four tokens of a tile, from token t4 of it on
    auto four = [&](const float* b, int t4, int tb) {
      const float *ds = b, *ks = b + ST * DK, *qs = b + 2 * ST * DK, *vs = b + 3 * ST * DK;
      float o[4][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        pair32 d[R / 2], k[R / 2], q[R / 2], v[4];
#pragma unroll
        for (int r = 0; r < R; r += 4) {
          const int at = (t4 + t) * DK + state_row(ti, r);
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(ks + at);
          k[r / 2] = y.x; k[r / 2 + 1] = y.y;
          if (OUT || t == 0) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(ds + (OUT ? at : t4 / 4 * DK + state_row(ti, r)));
            d[r / 2] = x.x; d[r / 2 + 1] = x.y;
          }
          if (OUT) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(qs + at);
            q[r / 2] = w.x; q[r / 2 + 1] = w.y;
          }
        }
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(vs + (t4 + t) * 2 * DV + cg * 8 + 2 * e);
          v[e] = x.x; v[e + 1] = x.y;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          pair32 acc = 0ull;                                    // (two zeros)
#pragma unroll
          for (int m = 0; m < R / 2; ++m) {
            if (OUT || t == 0) S[m][e] = fma2(S[m][e], d[m], mul2(k[m], v[e]));        // (the larger product unrounded)
            else S[m][e] = fma2(k[m], v[e], S[m][e]);
            if (OUT) acc = m == 0 ? mul2(S[m][e], q[m]) : fma2(S[m][e], q[m], acc);
          }
          if (OUT) {
            float x, y;
            unpack32(acc, x, y);
            o[t][e] = x + y;
          }
        }
      }
      if constexpr (OUT) {
        // sums over the 16 lanes: lane ti ends with token ti >> 2, column ti & 3
#pragma unroll
        for (int sh = 8, m = 2; m >= 1; sh >>= 1, m >>= 1) {
          const bool up = (lane & sh) != 0;
#pragma unroll
          for (int j = 0; j < m; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float send = up ? o[j][e] : o[j + m][e], keep = up ? o[j + m][e] : o[j][e];
              o[j][e] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
            }
        }
#pragma unroll
        for (int sh = 2, m = 2; m >= 1; sh >>= 1, m >>= 1) {
          const bool up = (lane & sh) != 0;
#pragma unroll
          for (int e = 0; e < m; ++e) {
            const float send = up ? o[0][e] : o[0][e + m], keep = up ? o[0][e + m] : o[0][e];
            o[0][e] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
          }
        }
        const int tl = tb + t4 + (ti >> 2);
        if (tl < n) a.out[static_cast<size_t>(t0 + tl) * a.ld_out + hd * DV + cg * 4 + (ti & 3)] = o[0][0];
      }
    };

    const int tiles = (n + ST - 1) / ST;
    fetch(0);
    stage(0, sm);
    __syncthreads();
    for (int it = 0; it < tiles; ++it) {
      const float* b = sm + (it & 1) * Cfg::kBuf;
      const int tb = it * ST;
      if (it + 1 < tiles) fetch(tb + ST);
#pragma unroll
      for (int t4 = 0; t4 < ST; t4 += 4)
        if (tb + t4 < n) four(b, t4, tb);
      if (it + 1 < tiles) stage(tb + ST, sm + ((it + 1) & 1) * Cfg::kBuf);
      __syncthreads();
    }

    if (!OUT || g == n_seg - 1) {
      float* dst = OUT ? S_g : W_g;
#pragma unroll
      for (int m = 0; m < R / 2; ++m) {
        float x[2][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) unpack32(S[m][e], x[0][e], x[1][e]);
#pragma unroll
        for (int r = 0; r < 2; ++r)
          *reinterpret_cast<float4*>(dst + static_cast<size_t>(state_row(ti, 2 * m + r)) * DV + cg * 4) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
      }
    }
    if constexpr (!OUT) {                                       // product of the segment's decays: four quarters of a tile per channel
      sm[tid] = total + total_e;
      __syncthreads();
      if (tid < DK) a.decay[ws * DK + tid] = (sm[tid] * sm[DK + tid]) * (sm[2 * DK + tid] * sm[3 * DK + tid]);
      __syncthreads();                                          // (the next item is staged there)
    }
  }
}

// what every segment starts from: local[g] <- S, S <- decay[g] S + local[g], from the sequence's state on.  grid (elements / 4 / 256, H, sequences)
__global__ void __launch_bounds__(256) lin_span_starts_kernel(SpanArgs a, int dk, int dv) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int s = blockIdx.z, hd = blockIdx.y;
  const int len = a.q_len[s], L = a.plan != nullptr ? *a.plan : a.seg;
  if (len <= 0 || L <= 0) return;
  int slot = s * (a.slots / a.n_seqs);                        // of the sequence's first segment
  if (a.plan != nullptr) {
    slot = 0;
    for (int i = threadIdx.x & 31; i < s; i += 32) slot += span_segments(a, i, L);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) slot += __shfl_xor_sync(0xffffffffu, slot, o);
  }
  const int n_seg = (len + L - 1) / L;
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (e >= dk * dv) return;
  const int row = e / dv;
  float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a.kv_len[s] - len > 0)
    S = *reinterpret_cast<const float4*>(a.state + (static_cast<size_t>(a.seq_slot[s]) * a.H + hd) * (static_cast<size_t>(dk) * dv) + e);
  const size_t first = static_cast<size_t>(slot) * a.H + hd, next = a.H;
  float* w = a.local + first * (static_cast<size_t>(dk) * dv) + e;
  const float* d = a.decay + first * dk + row;
  for (int g0 = 0; g0 < n_seg; g0 += 4) {                     // four segments' loads in flight
    float4 loc[4];
    float dec[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = g0 + j < n_seg - 1;
      loc[j] = ok ? *reinterpret_cast<const float4*>(w + (g0 + j) * next * (static_cast<size_t>(dk) * dv)) : make_float4(0.f, 0.f, 0.f, 0.f);
      dec[j] = ok ? d[(g0 + j) * next * dk] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (g0 + j >= n_seg) break;
      *reinterpret_cast<float4*>(w + (g0 + j) * next * (static_cast<size_t>(dk) * dv)) = S;
      S = make_float4(dec[j] * S.x + loc[j].x, dec[j] * S.y + loc[j].y, dec[j] * S.z + loc[j].z, dec[j] * S.w + loc[j].w);
    }
  }
}

template <int MODE, int D, bool PLAN>
int launch_span(const SpanArgs& a, int n_seqs, cudaStream_t s) {
  using Cfg = SpanCfg<D, D>;
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(lin_span_kernel<MODE, D, D, true, PLAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(lin_span_kernel<MODE, D, D, false, PLAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) set[dev] = true;
  }
  const int fit = 148 * Cfg::kBlocks, items = a.H * a.slots;
  dim3 local(a.slots / n_seqs, a.H, n_seqs), outputs(a.slots > 0 ? a.slots / n_seqs : 1, a.H, n_seqs);
  if (PLAN) {
    local = dim3(items < fit ? items : fit);
    outputs = dim3(a.H, a.slots > n_seqs ? a.slots : n_seqs);
  }
  cudaError_t e = cudaSuccess;
  if (a.slots > 0) {
    e = launch_kernel(lin_span_kernel<MODE, D, D, false, PLAN>, local, dim3(Cfg::kThreads), Cfg::kSmem, s, 1u, a);
    if (e == cudaSuccess) e = launch_kernel(lin_span_starts_kernel, dim3((D * D / 4 + 255) / 256, a.H, n_seqs), dim3(256), 0, s, 1u, a, D, D);
  }
  if (e == cudaSuccess) e = launch_kernel(lin_span_kernel<MODE, D, D, true, PLAN>, outputs, dim3(Cfg::kThreads), Cfg::kSmem, s, 1u, a);
  return static_cast<int>(e);
}

template <int MODE, int D>
int launch_span_width(const SpanArgs& a, int n_seqs, bool plan, cudaStream_t s) {
  return plan ? launch_span<MODE, D, true>(a, n_seqs, s) : launch_span<MODE, D, false>(a, n_seqs, s);
}
template <int MODE>
int launch_span_mode(const SpanArgs& a, int n_seqs, int dk, bool plan, cudaStream_t s) {
  return dk == 128 ? launch_span_width<MODE, 128>(a, n_seqs, plan, s) : launch_span_width<MODE, 64>(a, n_seqs, plan, s);
}

}  // namespace

bool lin_span_supported(int mode, const float* v, int ld_v, int off_v, const float* state, const float* out, int ld_out, int max_q, int dk,
                        int dv) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return mode != 1 && mode != 5 && dk == dv && (dk == 64 || dk == 128) && max_q >= 16 && al16(v + off_v) && ld_v % 4 == 0 && al16(state) &&
         al16(out) && ld_out % 4 == 0;
}

// What to launch for n_seqs sequences of up to max_q tokens; ragged: any number of them, of any length, may be live.
SpanLaunch span_launch(int n_seqs, int max_q, int H, int dk, bool ragged) {
  SpanLaunch r{true, false, ragged, 0, 0};
  if (!ragged) {
    const SpanWork w{max_q, max_q * n_seqs};
    span_ns best = span_cost_whole(w, H, dk);
    for (int c = 0; c < SPAN_CHOICES; ++c) {
      const int L = span_choice(c), segs = (max_q + L - 1) / L;
      if (L >= max_q || static_cast<long long>(H) * n_seqs * segs > SPAN_BLOCKS) continue;
      const span_ns cost = span_cost_cut(static_cast<span_ns>(H) * n_seqs * segs, segs, L, dk);
      if (cost < best) {
        best = cost;
        r.seg = L;
        r.slots = n_seqs * segs;
      }
    }
    if (best < span_cost_scan(w, H, dk)) return r;
    return {false, true, false, 0, 0};
  }
  // Where the sizes settle it, nothing is left to the device.  Short spans at 64 x 64: whole ones are no slower than lin_scan, however few are live.
  if (dk == 64 && max_q <= SPAN_SHORT_Q) return span_launch(n_seqs, max_q, H, dk, false);
  if (n_seqs == 1) {            // the plan for the bucket's length, unless lin_scan were faster at the shortest one
    const SpanLaunch h = span_launch(1, max_q, H, dk, false);
    const int len = max_q / 2 + 1;
    const span_ns scan = span_cost_scan({len, len}, H, dk), segs = h.seg > 0 ? (len + h.seg - 1) / h.seg : 0;
    if (h.scan || (h.seg > 0 ? span_cost_cut(H * segs, static_cast<int>(segs), h.seg, dk) : span_cost_whole({len, len}, H, dk)) <= scan) return h;
  }
  if (max_q <= SPAN_SHORT_Q) {
    // the fuller the machine, the better whole spans do.  Buckets are for one sequence, for 2 to 8 and for more; lengths are more than half of theirs
    const int least = n_seqs > 8 ? 9 : (n_seqs > 1 ? 2 : 1), half = (max_q + 1) / 2;
    r.scan = !(span_whole_wins({max_q, max_q * least}, H, dk) && span_whole_wins({half, half * least}, H, dk));
    r.span = !r.scan || span_whole_wins({max_q, max_q * n_seqs}, H, dk) || span_whole_wins({half, half * n_seqs}, H, dk);
  } else if (H <= SPAN_MANY_HEADS) {
    r.slots = span_slots(n_seqs, max_q, H);
  }
  r.ragged = r.slots > 0 || (r.span && r.scan);
  return r;
}

// The choice of a ragged call for these lengths, on the host: -1 lin_scan, 0 whole spans, else tokens per segment.
int span_plan(const int* lens, int n_seqs, int max_q, int H, int dk) {
  const SpanLaunch r = span_launch(n_seqs, max_q, H, dk, true);
  if (!r.ragged) return r.span ? r.seg : -1;
  SpanWork w{0, 0};
  for (int s = 0; s < n_seqs; ++s) {
    w.longest = lens[s] > w.longest ? lens[s] : w.longest;
    w.tokens += lens[s] > 0 ? lens[s] : 0;
  }
  if (r.scan && !span_whole_wins(w, H, dk)) return -1;
  span_ns best = span_cost_whole(w, H, dk);
  int plan = 0;
  for (int c = 0; r.slots > 0 && c < SPAN_CHOICES; ++c) {
    const span_ns cost = span_cost_segments(lens, n_seqs, w.longest, span_choice(c), r.slots, H, dk);
    if (cost < best || (cost == best && plan > 0)) {          // (of equal ones the longest)
      best = cost;
      plan = span_choice(c);
    }
  }
  return plan;
}

// floats of workspace: a plan word (16 bytes), states and decays of the slots
long long span_workspace(int slots, int H, int dk) { return slots > 0 ? 4 + static_cast<long long>(slots) * H * (dk * dk + dk) : 0; }

int launch_lin_span(int mode, const float* qk, int ld_qk, int off_q, int off_k, const float* v, int ld_v, int off_v, const float* z, int ld_z,
                    int off_z, const float* zbias, const float* hparam, const float* beta, int ld_b, int off_b, const float* aux, float qscale,
                    float inv_tau, float* state, float* out, int ld_out, const int* q_start, const int* q_len, const int* kv_len,
                    const int* seq_slot, int n_seqs, int H, int G, int dk, const SpanLaunch& r, float* ws, cudaStream_t s) {
  if (n_seqs <= 0) return 0;
  if (G <= 0 || H % G != 0) return -2;
  SpanArgs a{qk, ld_qk, off_q, off_k, v, ld_v, off_v, z, ld_z, off_z, zbias, hparam, beta, ld_b, off_b, aux, qscale, inv_tau, state, out,
             ld_out, q_start, q_len, kv_len, seq_slot, H, G, n_seqs, r.seg, r.slots, r.scan ? 1 : 0, nullptr, nullptr, nullptr};
  if (r.slots > 0) {
    if (r.ragged) a.plan = reinterpret_cast<int*>(ws);
    a.local = ws + 4;
    a.decay = a.local + static_cast<size_t>(r.slots) * H * dk * dk;
  }
  switch (mode) {
    case LS_GLA: return launch_span_mode<LS_GLA>(a, n_seqs, dk, r.ragged, s);
    case LS_MLSTM: return launch_span_mode<LS_MLSTM>(a, n_seqs, dk, r.ragged, s);
    case LS_HGRN2: return launch_span_mode<LS_HGRN2>(a, n_seqs, dk, r.ragged, s);
    case LS_SSD: return launch_span_mode<LS_SSD>(a, n_seqs, dk, r.ragged, s);
    default: return -2;
  }
}

}  // namespace b2b
