// Decode attention (one new token per sequence) over the paged KV cache on the 5th-gen tensor cores, keys as MMA rows.
//
// attention_tc.cu stacks queries into the 128 MMA rows; a decode step has only the G query heads of a key/value head, so a tile there is 128
// rows of which G count, every softmax thread walks 64 scores of one row, and 64 keys are two dependent products and two barrier round trips
// apart.  Here the operands are swapped:
//
//     S^T [keys, heads] = K Q^T        A = 128 keys (two cache pages) as they lie in the cache, B = the G heads padded to 16
//     P^T = exp2(S^T - m)              a thread has ONE key and G scores; P goes back to shared memory as [heads, keys] (4 KB)
//     O^T [channels, heads] += V^T P^T A = V read with the channels as rows (MN-major), B = P
//
// so a tile of 128 keys costs a thread G exponentials, both products are 16 columns wide, and what is left is the stream of the cache pages:
// K and V tiles share a ring of three slots (two CTAs per SM at D = 128, one at 256: 192 KB in flight per SM), consumed in the order
// K0, K1, V0, K2, V1, ..  The reference maximum of a head is kept while no score exceeds it by 2^8; one barrier with a vote per
// tile tells all threads.  The weights are summed as they are rounded for the second product.  Relative error against 64-bit sums, means of 8
// inputs, attention_tc.cu / here with unrounded sums / here: 32 x 8100 keys 0.002277 / 0.002304 / 0.002239, 32 x 500 0.00225 / 0.00217 / 0.00203,
// 8 x 3000 of 256 channels 0.00223 / 0.00220 / 0.00214 (exact running maxima: 0.0019, and 0.3 % on a decode step).
//
// Few sequences: a cluster of up to eight CTAs shares the keys of one (sequence, key/value head) and merges
// the partial sums through distributed shared memory -- no workspace and no second kernel.
//
// Bound: the cache stream.  Measured on B200 (attention_tc.cu -> here), 32 query / 8 key/value heads of 128, us: 32 sequences x 8100 keys
// 252 -> 160 (6.6 TB/s), 32 x 500 22 -> 16, 8 x 4000 50 -> 26, one x 700 18 -> 7.6, one x 8000 26 -> 13; 8 / 4 heads of 256, 32 x 4000 91 -> 80; 12 / 12 heads of 64
// (in pairs), 8 x 8000 107 -> 36, 32 x 8000 214 -> 124, 32 x 2000 56 -> 33, 8 x 400 9.8 -> 7.3, error 0.00230 -> 0.00217 (8 x 3000).
// Warp roles: 0 = TMA producer, 1 = TMEM owner + MMA issuer, 2..5 = softmax / correction / output.
#include "kernels.h"

#include <cuda.h>
#include <cuda_fp8.h>

#include <algorithm>

#include "common.cuh"
#include "launch.cuh"
#include "tmem.cuh"

namespace b2b {

int make_tmap_shared(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, int elt_bytes);

namespace {

constexpr int DPAGE = 64;
constexpr int DKEYS = 128;                         // keys per tile == MMA rows (ma_value_desc has 128 x 128 bytes between channel blocks)
constexpr int DHEADS = 16;                         // MMA columns: query heads of a key/value head, padded
constexpr int DSLOTS = 3;
constexpr int DEC_THREADS = 192;
constexpr float DEC_LOG2E = 1.4426950408889634f;

__device__ unsigned int g_decode_gave_up = 0;      // CTAs whose waits ran out since the module was loaded

struct DecodeParams {
  __nv_bfloat16* out;
  const int* block_table;
  const int* q_start;
  const int* q_len;
  const int* kv_len;
  int max_pages, n_q, n_kv, window;
  float softcap;
  uint8_t* q_out8;                                 // fused MX quantisation of the output (see attention_tc.cu), or null
  uint8_t* q_sf;
  int q_bn;
};

// PAIR: two neighbouring key/value heads of 64 channels as one of D = 128.  Their scores are products of their own (the halves of a key row, each into columns of
// its own), so nothing of one head enters the other's; of O, every column holds its head's 64 channels and 64 that nobody reads.
template <int D, bool PAIR>
struct DecCfg {
  static constexpr int kTile = DKEYS * D * 2;                      // a K or V tile
  static constexpr int kQ = DHEADS * D * 2;
  static constexpr int kP = DHEADS * DKEYS * 2;
  static constexpr int kSmem = 1024 + DSLOTS * kTile + kQ + 2 * kP + 512;
  static constexpr int kMinCtas = D == 128 ? 2 : 1;
  static constexpr uint32_t kSCols = PAIR ? 2 * DHEADS : DHEADS;
  static constexpr uint32_t kOCol = 2 * kSCols;                    // S twice, O for every 128 channels
  static constexpr uint32_t kCols = PAIR ? 128 : 64;
  static_assert(!PAIR || D == 128, "two heads of 64 channels");
};

template <int GP>
__device__ __forceinline__ void dec_ld(uint32_t taddr, float* v) {   // GP columns of this thread's lane
  uint32_t r[GP];
  if constexpr (GP == 4)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
  else if constexpr (GP == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < GP; ++i) v[i] = __uint_as_float(r[i]);
}
template <int GP>
__device__ __forceinline__ void dec_st(uint32_t taddr, const float* v) {
  if constexpr (GP == 4)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
                 "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])) : "memory");
  else if constexpr (GP == 8)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(__float_as_uint(v[0])),
                 "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])),
                 "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
                 "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
                 "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
                 "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void dec_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
__device__ __forceinline__ bool dec_vote(bool p) {                   // any of the 128 softmax threads
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred a, b;\n\t"
      "setp.ne.u32 a, %1, 0;\n\t"
      "barrier.cta.red.or.pred b, 1, 128, a;\n\t"
      "selp.u32 %0, 1, 0, b;\n\t}\n"
      : "=r"(r) : "r"(p ? 1u : 0u) : "memory");
  return r != 0;
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// GP: query heads per key/value head rounded up to 4, 8 or 16 (PAIR: to 4 or 8, twice).  grid (CTAs of the cluster, key/value heads or pairs of them, sequences)
template <int D, int GP, bool SOFTCAP, bool PAIR>
__global__ void __launch_bounds__(DEC_THREADS, (DecCfg<D, PAIR>::kMinCtas))
attn_decode_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const DecodeParams p, const int G) {
  using Cfg = DecCfg<D, PAIR>;
  constexpr int DB = D / 64, MB = D / 128;         // 64-channel blocks of a row; 128-channel blocks of O
  constexpr int GH = PAIR ? GP / 2 : GP;           // columns of a key/value head
  const int hd = PAIR ? 64 : D, heads = PAIR ? 2 * G : G;          // channels of a head, query heads of this CTA
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem + DSLOTS * Cfg::kTile;
  uint8_t* p_s = q_s + Cfg::kQ;                    // [2][16 heads x 128 keys]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(p_s + 2 * Cfg::kP);
  uint64_t* full = q_full + 1;                     // [DSLOTS]
  uint64_t* empty = full + DSLOTS;                 // [DSLOTS]
  uint64_t* s_full = empty + DSLOTS;               // [2]
  uint64_t* p_ready = s_full + 2;                  // [2]
  uint64_t* pv_done = p_ready + 2;                 // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile uint32_t* abort = tmem_slot + 1;
  __shared__ float red_s[4][DHEADS];               // per warp: maxima, then row sums

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < DSLOTS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    *abort = 0u;
    fence_barrier_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 1) tmem_alloc<Cfg::kCols>(tmem_slot);
  for (int i = threadIdx.x; i < 2 * Cfg::kP / 16; i += DEC_THREADS)        // the rows of heads that do not exist stay zero
    reinterpret_cast<uint4*>(p_s)[i] = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  const int seq = blockIdx.z, kvh = blockIdx.y, rank = blockIdx.x, parts = gridDim.x;
  const int kvlen = p.kv_len[seq];
  const bool active = p.q_len[seq] > 0 && kvlen > 0;                 // (the same for all CTAs of a cluster)
  const int kv_lo = p.window > 0 ? max(0, kvlen - p.window) : 0;
  int t_lo = kv_lo / DKEYS, t_hi = active ? (kvlen + DKEYS - 1) / DKEYS : t_lo;
  if (parts > 1) {
    const int per = (t_hi - t_lo + parts - 1) / parts;
    t_lo = min(t_hi, t_lo + rank * per);
    t_hi = min(t_hi, t_lo + per);
  }
  const int nt = t_hi - t_lo;
  bool ok = true;

  if (nt > 0 && warp == 0) {
    // -------------------------------------------------------------------------------------------------- TMA producer
    if (elect_one()) {
      mbar_arrive_expect_tx(q_full, Cfg::kQ);
#pragma unroll
      for (int c = 0; c < DB; ++c)
        tma_load_2d(q_s + c * (DHEADS * 128), &tm_q, q_full, PAIR ? 0 : c * 64, p.q_start[seq] * p.n_q + kvh * heads + (PAIR ? c * G : 0));
      const int* bt = p.block_table + static_cast<size_t>(seq) * p.max_pages;
      uint32_t i = 0;
      auto load = [&](const CUtensorMap* tm, int n) {                // K or V tile n of this CTA into the next slot
        const uint32_t s = i % DSLOTS;
        if (!(ok = ma_wait(&empty[s], (i / DSLOTS & 1u) ^ 1u, abort))) return;
        ++i;
        const int page = 2 * (t_lo + n);
        const int p0 = bt[page], p1 = (page + 1) * DPAGE < kvlen ? bt[page + 1] : p0;      // (past the end: any keys, they are masked)
        mbar_arrive_expect_tx(&full[s], Cfg::kTile);
#pragma unroll
        for (int c = 0; c < DB; ++c) {
          uint8_t* dst = smem + s * Cfg::kTile + c * (DKEYS * 128);
          tma_load_2d(dst, tm, &full[s], kvh * D + c * 64, p0 * DPAGE);
          tma_load_2d(dst + DPAGE * 128, tm, &full[s], kvh * D + c * 64, p1 * DPAGE);
        }
      };
      load(&tm_k, 0);
      for (int n = 0; ok && n < nt; ++n) {
        if (n + 1 < nt) load(&tm_k, n + 1);
        if (ok) load(&tm_v, n);
      }
    }
  } else if (nt > 0 && warp == 1) {
    // ---------------------------------------------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(DKEYS, DHEADS);
      constexpr uint32_t idesc_o = make_idesc_bf16(128, DHEADS) | (1u << 15);              // A (V) has its rows contiguous
      uint32_t i = 0;
      auto scores = [&](int n) {
        const uint32_t s = i % DSLOTS;
        if (!(ok = ma_wait(&full[s], i / DSLOTS & 1u, abort))) return;
        ++i;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t a = make_sw128_kmajor_desc(smem_u32(smem + s * Cfg::kTile + (kk / 4) * (DKEYS * 128))) + static_cast<uint64_t>((kk % 4) * 2);
          const uint64_t b = make_sw128_kmajor_desc(smem_u32(q_s + (kk / 4) * (DHEADS * 128))) + static_cast<uint64_t>((kk % 4) * 2);
          umma_bf16(tmem + static_cast<uint32_t>(n & 1) * Cfg::kSCols + (PAIR ? kk / 4 * DHEADS : 0), a, b, idesc_s, (PAIR ? kk % 4 : kk) > 0 ? 1u : 0u);
        }
        umma_commit(&empty[s]);
        umma_commit(&s_full[n & 1]);
      };
      ok = ma_wait(q_full, 0, abort);
      if (ok) scores(0);
      for (int n = 0; ok && n < nt; ++n) {
        if (n + 1 < nt) scores(n + 1);             // runs while the softmax warps work on tile n
        if (!ok) break;
        const uint32_t s = i % DSLOTS;
        if (!(ok = ma_wait(&full[s], i / DSLOTS & 1u, abort))) break;
        ++i;
        if (!(ok = ma_wait(&p_ready[n & 1], n >> 1 & 1, abort))) break;
        tc_fence_after();
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
          for (int kk = 0; kk < DKEYS / 16; ++kk) {
            const uint64_t a = ma_value_desc(smem_u32(smem + s * Cfg::kTile + m * 2 * (DKEYS * 128) + kk * (16 * 128)));
            const uint64_t b = make_sw128_kmajor_desc(smem_u32(p_s + (n & 1) * Cfg::kP + (kk / 4) * (DHEADS * 128))) + static_cast<uint64_t>((kk % 4) * 2);
            umma_bf16(tmem + Cfg::kOCol + m * DHEADS, a, b, idesc_o, (n > 0 || kk > 0) ? 1u : 0u);
          }
        umma_commit(&empty[s]);
        umma_commit(&pv_done[n & 1]);
      }
    }
  }

  float m_ref[GP], l[GP];
#pragma unroll
  for (int g = 0; g < GP; ++g) {
    m_ref[g] = -INFINITY;
    l[g] = 0.f;
  }
  const int q4 = warp & 3, row = q4 * 32 + lane;
  const uint32_t lanes = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
  float o[MB][GP];
  if (warp >= 2) {
    // ------------------------------------------------------------------------------------------------------- softmax
    const float inv_cap = SOFTCAP ? 1.f / p.softcap : 0.f;
    for (int n = 0; n < nt; ++n) {
      const int b = n & 1, key = (t_lo + n) * DKEYS + row;
      // (a wait that gave up ends the other waits through the abort word; the loop goes on, because every warp has to vote)
      ok = __all_sync(0xffffffffu, ma_wait(&s_full[b], n >> 1 & 1, abort)) && ok;
      tc_fence_after();
      float x[GP] = {};
      if (ok) {
        dec_ld<GH>(lanes + b * Cfg::kSCols, x);
        if constexpr (PAIR) dec_ld<GH>(lanes + b * Cfg::kSCols + DHEADS, x + GH);
      }
      const bool seen = key < kvlen && key >= kv_lo;
      bool up = false;
#pragma unroll
      for (int g = 0; g < GP; ++g) {
        if constexpr (SOFTCAP) x[g] = p.softcap * tanh_exp(x[g] * inv_cap);
        x[g] = seen ? x[g] * DEC_LOG2E : -INFINITY;
        up |= g % GH < G && (x[g] > m_ref[g] + 8.f || (m_ref[g] == -INFINITY && x[g] > -INFINITY));
      }
      // P(n - 2) has been read; waited for in every tile so that no parity wait lags two phases behind
      if (ok && n > 1) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[b], (n - 2) >> 1 & 1, abort));
      if (dec_vote(up)) {                          // new references: the maxima of this tile
        float alpha[GP];
#pragma unroll
        for (int g = 0; g < GP; ++g) {
          float m = x[g];
#pragma unroll
          for (int sh = 16; sh > 0; sh >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, sh));
          if (lane == 0) red_s[q4][g] = m;
        }
        dec_sync();
#pragma unroll
        for (int g = 0; g < GP; ++g) {
          const float m = fmaxf(m_ref[g], fmaxf(fmaxf(red_s[0][g], red_s[1][g]), fmaxf(red_s[2][g], red_s[3][g])));
          alpha[g] = (m_ref[g] == -INFINITY || g % GH >= G) ? 0.f : ex2(m_ref[g] - m);
          m_ref[g] = m;
          l[g] *= alpha[g];
        }
        dec_sync();                                // red_s may be written again
        if (n > 0) {
          if (ok) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[b ^ 1], (n - 1) >> 1 & 1, abort));
          tc_fence_after();
          if (ok) {
#pragma unroll
            for (int m = 0; m < MB; ++m) {
              float y[GP];
              dec_ld<GP>(lanes + Cfg::kOCol + m * DHEADS, y);
#pragma unroll
              for (int g = 0; g < GP; ++g) y[g] *= alpha[g];
              dec_st<GP>(lanes + Cfg::kOCol + m * DHEADS, y);
            }
          }
        }
      }
      uint8_t* pt = p_s + b * Cfg::kP + (row >> 6) * (DHEADS * 128) + (row & 7) * 2;
#pragma unroll
      for (int g = 0; g < GP; ++g) {
        if (g % GH < G) {
          const float e = ex2(x[g] - (m_ref[g] == -INFINITY ? 0.f : m_ref[g]));
          const __nv_bfloat16 w = __float2bfloat16_rn(e);
          l[g] += __bfloat162float(w);             // the sum of what the product sees: the rounding of a dominant weight cancels
          *reinterpret_cast<__nv_bfloat16*>(pt + g * 128 + ((((row & 63) >> 3) ^ (g & 7)) << 4)) = w;
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[b]);
    }
    if (nt > 0 && ok) {
      if (nt > 1) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[nt & 1], (nt - 2) >> 1 & 1, abort));
      if (ok) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[(nt - 1) & 1], (nt - 1) >> 1 & 1, abort));
      tc_fence_after();
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      if (nt > 0 && ok) dec_ld<GP>(lanes + Cfg::kOCol + m * DHEADS, o[m]);
      else
#pragma unroll
        for (int g = 0; g < GP; ++g) o[m][g] = 0.f;
    }
#pragma unroll
    for (int g = 0; g < GP; ++g)
#pragma unroll
      for (int sh = 16; sh > 0; sh >>= 1) l[g] += __shfl_xor_sync(0xffffffffu, l[g], sh);
    if (lane == 0)
#pragma unroll
      for (int g = 0; g < GP; ++g) red_s[q4][g] = l[g];
  }
  // ------------------------------------------------------------------- partial sums of this CTA in the (idle) ring: [heads][D], m, l
  __syncthreads();
  float* part = reinterpret_cast<float*>(smem);
  if (warp >= 2 && active) {
#pragma unroll
    for (int g = 0; g < GP; ++g) {
      if (g % GH < G) {
#pragma unroll
        for (int m = 0; m < MB; ++m) part[g * D + m * 128 + row] = o[m][g];
        if (row == 0) {
          part[DHEADS * D + g] = m_ref[g];
          part[DHEADS * D + DHEADS + g] = red_s[0][g] + red_s[1][g] + red_s[2][g] + red_s[3][g];
        }
      }
    }
  }
  if (parts > 1) {
    cluster_arrive_release();
    cluster_wait_acquire();
  } else {
    __syncthreads();
  }
  if (warp >= 2 && active) {
    // ---------------------------------------------------------------- merge: this CTA finishes every parts-th run of 128 outputs
    const uint32_t mine = smem_u32(part);
    for (int e = rank * 128 + row; e < heads * hd; e += parts * 128) {
      const int head = e / hd, g = PAIR ? head / G * GH + head % G : head;
      const uint32_t from = mine + (PAIR ? g * D + head / G * 64 + e % 64 : e) * 4;
      float m = -INFINITY;
      for (int r = 0; r < parts; ++r) m = fmaxf(m, ld_dsmem_f32(mapa_smem(mine + (DHEADS * D + g) * 4, r)));
      float num = 0.f, den = 0.f;
      for (int r = 0; r < parts; ++r) {
        const float mr = ld_dsmem_f32(mapa_smem(mine + (DHEADS * D + g) * 4, r));
        const float w = mr == -INFINITY ? 0.f : ex2(mr - m);
        den += w * ld_dsmem_f32(mapa_smem(mine + (DHEADS * D + DHEADS + g) * 4, r));
        num += w * ld_dsmem_f32(mapa_smem(from, r));
      }
      const float v = den == 0.f ? 0.f : num / den;      // (no key: zero; a NaN among the scores stays one)
      const int tok = p.q_start[seq], feat = kvh * heads * hd + e, ldq = p.n_q * hd;
      if (p.q_out8 == nullptr) {
        p.out[static_cast<size_t>(tok) * ldq + feat] = __float2bfloat16_rn(v);
      } else {                                     // e4m3 + scale of the warp's 32 features (what a separate quantiser would compute)
        const float rv = bf16_round(v);
        float amax = fabsf(rv);
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, sh));
        const int ex = mx_exponent(amax);
        p.q_out8[static_cast<size_t>(tok) * ldq + feat] = static_cast<uint8_t>(
            __nv_cvt_float_to_fp8(rv * mx_inverse(ex), __NV_SATFINITE, __NV_E4M3));
        if (lane == 0) p.q_sf[mx_sf_at(tok, feat, p.q_bn, ldq >> 7)] = static_cast<uint8_t>(ex + 127);
      }
    }
  }
  if (parts > 1) {                                 // no CTA leaves while another reads its sums (which have gone into what was stored: nothing to release)
    cluster_arrive_relaxed();
    cluster_wait_acquire();
  }
  if (*abort != 0u) __nanosleep(200000);           // copies in flight land before the shared memory is given back
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<Cfg::kCols>(tmem);
  }
  if (threadIdx.x == 0 && *abort != 0u) {          // a wait ran out: the process learns of it
    if (g_abort_word != nullptr) *g_abort_word = 1u;
    atomicAdd(&g_decode_gave_up, 1u);
  }
}

// Clusters of 4 or 8 CTAs, one per SM, that fit the device at once: fewer than 37 or 18, because GPCs have 16 to 18 SMs.
int dec_clusters(int size) {
  static int known[2][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && known[size / 8][dev] > 0) return known[size / 8][dev];
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(144);
  cfg.blockDim = dim3(DEC_THREADS);
  cfg.dynamicSmemBytes = DecCfg<256, false>::kSmem;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeClusterDimension;
  a[0].val.clusterDim.x = static_cast<unsigned>(size);
  a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
  cfg.attrs = a;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(attn_decode_kernel<256, 4, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, DecCfg<256, false>::kSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, attn_decode_kernel<256, 4, false, false>, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 112 / size;
  }
  if (dev < 64) known[size / 8][dev] = n;
  return n;
}

// CTAs of a cluster: they share the keys of a (sequence, key/value head) while that still adds resident CTAs (two per SM at 128 channels) and every CTA can have a
// tile and all clusters fit at once.  256-wide heads, 4 sequences of 8000 / 2000 keys: 16 clusters of eight ran in two rounds (37.7 / 14.6 us), in clusters of four
// 27.7 / 10.0.  With two CTAs on an SM 32 clusters of eight and 64 of four ran at once (4 and 8 sequences of 8 heads), 36 and 72 did not (6 and 12 sequences of 6 pairs, 2000
// keys: 15.0 against 10.0 us in clusters of four, 23.9 against 17.4 in clusters of two).  Those two numbers are of a B200's 148 SMs and not asked of the device:
// cudaOccupancyMaxActiveClusters counts fewer of these clusters than run at once, and by it 16 of eight became fours (2 sequences of 8000 keys 16.7 -> 21.7 us).
int dec_parts(int items, int tiles, bool one_per_sm) {
  const int slots = one_per_sm ? 148 : 296;
  int parts = 1;
  while (parts < 8 && static_cast<long long>(items) * parts * 2 <= slots && parts * 2 <= tiles) parts *= 2;
  while (parts > 2 && items > (one_per_sm ? dec_clusters(parts) : 256 / parts)) parts /= 2;
  return parts;
}

template <int D, int GP, bool SOFTCAP, bool PAIR>
int launch_dec(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const DecodeParams& p, int G, int seqs, int tiles, cudaStream_t s) {
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(attn_decode_kernel<D, GP, SOFTCAP, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, DecCfg<D, PAIR>::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) set[dev] = true;
  }
  const int kv = PAIR ? p.n_kv / 2 : p.n_kv, parts = dec_parts(seqs * kv, tiles, DecCfg<D, PAIR>::kMinCtas == 1);
  const dim3 grid(parts, kv, seqs);
  if (parts > 1)
    return static_cast<int>(launch_kernel_cx(attn_decode_kernel<D, GP, SOFTCAP, PAIR>, grid, dim3(DEC_THREADS), DecCfg<D, PAIR>::kSmem, s,
                                             static_cast<unsigned>(parts), tq, tk, tv, p, G));
  return static_cast<int>(launch_kernel(attn_decode_kernel<D, GP, SOFTCAP, PAIR>, grid, dim3(DEC_THREADS), DecCfg<D, PAIR>::kSmem, s, 1u, tq, tk, tv, p, G));
}

template <int D, bool PAIR>
int launch_dec_g(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const DecodeParams& p, int G, int seqs, int tiles,
                 cudaStream_t s) {
#define B2B_DEC(GP) \
  (p.softcap > 0.f ? launch_dec<D, GP, true, PAIR>(tq, tk, tv, p, G, seqs, tiles, s) : launch_dec<D, GP, false, PAIR>(tq, tk, tv, p, G, seqs, tiles, s))
  if constexpr (PAIR) {
    return G <= 4 ? B2B_DEC(8) : B2B_DEC(16);
  } else {
    if (G <= 4) return B2B_DEC(4);
    if (G <= 8) return B2B_DEC(8);
    return B2B_DEC(16);
  }
#undef B2B_DEC
}

}  // namespace

// 64-wide heads: the group sizes of the flash kernel (attention_tc.cu), whose weights are bf16 as well.  The others belong to attention.cu, which holds its
// weights in fp32 (4 x 3000 keys, error against 64-bit sums: 0.0015 to 0.0017 there, 0.0021 to 0.0022 here).
bool attn_decode_supported(int n_q, int n_kv, int head_dim) {
  if (n_kv <= 0 || n_q % n_kv != 0) return false;
  const int g = n_q / n_kv;
  if (head_dim == 64) return n_kv % 2 == 0 && (g == 1 || g == 2 || g == 4 || g == 8);
  return g <= DHEADS && (head_dim == 128 || head_dim == 256);
}

int launch_attn_decode(const void* q, const void* k_cache, const void* v_cache, void* out, const int* block_table, const int* q_start,
                       const int* q_len, const int* kv_len, int seqs, int max_pages, int n_tokens, int n_pages, int n_q, int n_kv,
                       int head_dim, int window, float softcap, void* q_out8, void* q_sf, int q_bn, cudaStream_t s) {
  if (!attn_decode_supported(n_q, n_kv, head_dim)) return -2;
  CUtensorMap tq, tk, tv;
  int r = make_tmap_shared(&tq, q, static_cast<uint64_t>(n_tokens) * n_q, head_dim, head_dim, DHEADS, 2);
  if (r) return r;
  const uint64_t kv_rows = static_cast<uint64_t>(n_pages) * DPAGE, kv_cols = static_cast<uint64_t>(n_kv) * head_dim;
  if ((r = make_tmap_shared(&tk, k_cache, kv_rows, kv_cols, kv_cols, DPAGE, 2))) return r;
  if ((r = make_tmap_shared(&tv, v_cache, kv_rows, kv_cols, kv_cols, DPAGE, 2))) return r;
  DecodeParams p;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.block_table = block_table; p.q_start = q_start; p.q_len = q_len; p.kv_len = kv_len;
  p.max_pages = max_pages; p.n_q = n_q; p.n_kv = n_kv; p.window = window; p.softcap = softcap;
  p.q_out8 = static_cast<uint8_t*>(q_out8);
  p.q_sf = static_cast<uint8_t*>(q_sf);
  p.q_bn = q_bn > 0 ? q_bn : 32;
  const int g = n_q / n_kv, tiles = std::max(1, max_pages / (DKEYS / DPAGE));
  if (head_dim == 64) return launch_dec_g<128, true>(tq, tk, tv, p, g, seqs, tiles, s);
  return head_dim == 128 ? launch_dec_g<128, false>(tq, tk, tv, p, g, seqs, tiles, s) : launch_dec_g<256, false>(tq, tk, tv, p, g, seqs, tiles, s);
}

int set_wait_policy_decode(uint32_t* abort_word, unsigned long long limit_ns) {
  cudaError_t e = cudaMemcpyToSymbol(g_abort_word, &abort_word, sizeof(abort_word));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_wait_limit_ns, &limit_ns, sizeof(limit_ns));
  return static_cast<int>(e);
}

unsigned attn_decode_gave_up() {
  unsigned n = 0;
  return cudaMemcpyFromSymbol(&n, g_decode_gave_up, sizeof(n)) == cudaSuccess ? n : ~0u;
}

}  // namespace b2b
