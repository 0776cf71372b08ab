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
//     start.  Pass 0 takes 0.6 of pass 1's time, so it is done only where heads x sequences do not fill the machine.
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
  int H, G;
  int seg, max_segs;        // tokens per segment (0: a span is one segment), segments per sequence in the workspace
  float* local;             // [sequences][max_segs][H][dk][dv]: what a segment adds, then the state it starts from
  float* decay;             // [sequences][max_segs][H][dk]: product of its decays
};

constexpr int ST = 16;      // tokens per staged tile

template <int DK, int DV>
struct SpanCfg {
  static constexpr int kThreads = 4 * DV;                     // 16 lanes x DV / 4 column groups
  static constexpr int R = DK / 16;                           // state rows per thread
  static constexpr int kBuf = 3 * ST * DK + ST * 2 * DV;      // d, k, q; v with every value twice (an operand of packed pairs)
  static constexpr int kSmem = 2 * kBuf * 4;
};

// state rows of lane ti: ti*4 .. +3 and, for 128 rows, 64 + ti*4 .. +3
__device__ __forceinline__ int state_row(int ti, int r) { return (r >> 2) * 64 + ti * 4 + (r & 3); }

// (p + e) <- (p + e) d, e the rounding error of p: a constant decay rounds the same way every time, so a plain product drifts
__device__ __forceinline__ void chain(float& p, float& e, float d) {
  const float x = p * d;
  e = e * d + fmaf(p, d, -x);
  p = x;
}

template <int MODE, int DK, int DV, bool OUT>
__global__ void __launch_bounds__(SpanCfg<DK, DV>::kThreads, 1) lin_span_kernel(SpanArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  using Cfg = SpanCfg<DK, DV>;
  constexpr int NT = Cfg::kThreads, R = Cfg::R;
  constexpr bool ZC = MODE == LS_GLA || MODE == LS_HGRN2;
  static_assert(NT == 4 * DK && ST * DV == 4 * NT, "staging: a thread prepares one channel of four tokens and four values");
  extern __shared__ __align__(16) float sm[];

  const int s = blockIdx.z, hd = blockIdx.y, g = blockIdx.x;
  const int len = a.q_len[s];
  const int seg = a.seg > 0 ? a.seg : len;
  const int n_seg = len > 0 ? (len + seg - 1) / seg : 0;
  if (g >= n_seg || (!OUT && g == n_seg - 1)) return;         // (block-uniform)
  const int t0 = a.q_start[s] + g * seg;
  const int n = min(seg, len - g * seg);
  const int H = a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ti = lane & 15, cg = warp * 2 + (lane >> 4);
  const int hqk = MODE == LS_SSD ? hd / (H / a.G) : hd;
  float* S_g = a.state + (static_cast<size_t>(a.seq_slot[s]) * H + hd) * (static_cast<size_t>(DK) * DV);
  const size_t ws = ((static_cast<size_t>(s) * a.max_segs + g) * H + hd);
  float* W_g = a.seg > 0 ? a.local + ws * (static_cast<size_t>(DK) * DV) : nullptr;

  pair32 S[R / 2][4];                                         // rows state_row(ti, 2 m) and the next one, columns cg*4 .. +3
  {
    const float* src = OUT ? (a.seg > 0 ? W_g : (a.kv_len[s] - len > 0 ? S_g : nullptr)) : nullptr;
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
  }
}

// what every segment starts from: local[g] <- S, S <- decay[g] S + local[g], from the sequence's state on.  grid (elements / 4 / 256, H, sequences)
__global__ void __launch_bounds__(256) lin_span_starts_kernel(SpanArgs a, int dk, int dv) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int s = blockIdx.z, hd = blockIdx.y;
  const int len = a.q_len[s];
  if (len <= 0) return;
  const int n_seg = (len + a.seg - 1) / a.seg;
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (e >= dk * dv) return;
  const int row = e / dv;
  float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a.kv_len[s] - len > 0)
    S = *reinterpret_cast<const float4*>(a.state + (static_cast<size_t>(a.seq_slot[s]) * a.H + hd) * (static_cast<size_t>(dk) * dv) + e);
  const size_t first = (static_cast<size_t>(s) * a.max_segs * a.H + hd), next = a.H;
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

template <int MODE, int D>
int launch_span(const SpanArgs& a, int n_seqs, cudaStream_t s) {
  using Cfg = SpanCfg<D, D>;
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(lin_span_kernel<MODE, D, D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(lin_span_kernel<MODE, D, D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) set[dev] = true;
  }
  const dim3 grid(a.seg > 0 ? a.max_segs : 1, a.H, n_seqs);
  cudaError_t e = cudaSuccess;
  if (a.seg > 0) {
    e = launch_kernel(lin_span_kernel<MODE, D, D, false>, grid, dim3(Cfg::kThreads), Cfg::kSmem, s, 1u, a);
    if (e == cudaSuccess) e = launch_kernel(lin_span_starts_kernel, dim3((D * D / 4 + 255) / 256, a.H, n_seqs), dim3(256), 0, s, 1u, a, D, D);
  }
  if (e == cudaSuccess) e = launch_kernel(lin_span_kernel<MODE, D, D, true>, grid, dim3(Cfg::kThreads), Cfg::kSmem, s, 1u, a);
  return static_cast<int>(e);
}

template <int MODE>
int launch_span_mode(const SpanArgs& a, int n_seqs, int dk, cudaStream_t s) {
  return dk == 128 ? launch_span<MODE, 128>(a, n_seqs, s) : launch_span<MODE, 64>(a, n_seqs, s);
}

}  // namespace

bool lin_span_supported(int mode, const float* v, int ld_v, int off_v, const float* state, const float* out, int ld_out, int max_q, int dk,
                        int dv) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return mode != 1 && mode != 5 && dk == dv && (dk == 64 || dk == 128) && max_q >= 16 && al16(v + off_v) && ld_v % 4 == 0 && al16(state) &&
         al16(out) && ld_out % 4 == 0;
}

// The fastest of lin_scan (-1), whole spans (0) and segments of that many tokens, by the measured times per token (ns; B200, GLA): lin_scan's
// blocks run side by side until about 28 heads (128 x 128) or 90 (64 x 64), then their time grows with the heads; a block here is
// one head, with one resident per SM at 128 x 128 (two at 64 x 64, at half the speed each).  Segments: pass 0 takes 0.6 of pass 1's time,
// the three launches and the chain of the starts 10 us.
int span_plan(int n_seqs, int max_q, int H, int dk) {
  const double heads = static_cast<double>(H) * n_seqs, token = dk == 128 ? 420. : 180.;
  auto rounds = [&](double blocks) {
    const double r = static_cast<double>((static_cast<long long>(blocks) + 147) / 148);
    return dk == 128 ? r : (r > 1. ? 0.85 * r : 1.);
  };
  double best = (dk == 128 ? (heads * 9. > 285. ? heads * 9. : 285.) : (heads * 2.3 > 200. ? heads * 2.3 : 200.)) * max_q;
  int plan = -1;
  const double whole = rounds(heads) * max_q * token + 2000.;
  if (whole < best) {
    best = whole;
    plan = 0;
  }
  for (int L = 32; L <= 1024 && L < max_q; L += 16) {
    const int segs = (max_q + L - 1) / L;
    if (heads * segs > 4 * 148) continue;          // (bounds the workspace, too: 39 MB)
    const double cost = rounds(heads * segs) * L * token * 1.6 + 10000. + 300. * segs;
    if (cost < best) {
      best = cost;
      plan = L;
    }
  }
  return plan;
}

int launch_lin_span(int mode, const float* qk, int ld_qk, int off_q, int off_k, const float* v, int ld_v, int off_v, const float* z, int ld_z,
                    int off_z, const float* zbias, const float* hparam, const float* beta, int ld_b, int off_b, const float* aux, float qscale,
                    float inv_tau, float* state, float* out, int ld_out, const int* q_start, const int* q_len, const int* kv_len,
                    const int* seq_slot, int n_seqs, int max_q, int H, int G, int dk, int seg, float* ws, cudaStream_t s) {
  if (n_seqs <= 0) return 0;
  if (G <= 0 || H % G != 0) return -2;
  SpanArgs a{qk, ld_qk, off_q, off_k, v, ld_v, off_v, z, ld_z, off_z, zbias, hparam, beta, ld_b, off_b, aux, qscale, inv_tau, state, out,
             ld_out, q_start, q_len, kv_len, seq_slot, H, G, seg, seg > 0 ? (max_q + seg - 1) / seg : 1, nullptr, nullptr};
  if (seg > 0) {
    a.local = ws;
    a.decay = ws + static_cast<size_t>(n_seqs) * a.max_segs * H * dk * dk;
  }
  switch (mode) {
    case LS_GLA: return launch_span_mode<LS_GLA>(a, n_seqs, dk, s);
    case LS_MLSTM: return launch_span_mode<LS_MLSTM>(a, n_seqs, dk, s);
    case LS_HGRN2: return launch_span_mode<LS_HGRN2>(a, n_seqs, dk, s);
    case LS_SSD: return launch_span_mode<LS_SSD>(a, n_seqs, dk, s);
    default: return -2;
  }
}

}  // namespace b2b
