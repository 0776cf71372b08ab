// Prefill GEMM: many tokens, pairs of CTAs, persistent tiles.
//
//   out[t, n] = epilogue( sum_k X[t, k] * W[n, k] )        (the epilogues of gemm_tc.cu, bf16 or block-scaled fp8 operands, fp32 accumulators)
//
// gemm_tc.cu makes the weights the 128 MMA rows and the tokens the columns, which is what few tokens want.  With hundreds of tokens
// it is bound by shared memory (a CTA reads 128 + 256 operand rows per 128 x 256 tile) and by its epilogue (a lane owns one feature,
// so every store of a warp is 64 bytes of one token).  Here the TOKENS are the rows:
//
//   * a pair of CTAs (tcgen05 cta_group::2) owns 256 tokens x BN features: each CTA holds its 128 token rows and HALF of the
//     weight rows, the tensor cores read the other half from the neighbour's shared memory -- 128 + 128 rows per CTA for twice
//     the work of a 128 x 256 tile;
//   * one pair per two SMs walks the tiles (persistent); the accumulator is double-buffered in tensor memory, so
//     the epilogue of a tile runs under the main loop of the next one;
//   * a lane owns one token and 32 adjacent features per TMEM read: rotary pairs, gate/up pairs and residual rows are in its own
//     registers or 16-byte accesses away, and the finished 32 x 64-byte block goes through shared memory so that a warp
//     stores pieces of 64 bytes;
//   * tiles left over after the last full round may be split (clusters of four CTAs then): the two pairs of a cluster take half of K each
//     and exchange half of the columns through distributed shared memory, which halves the time of that round;
//   * the piece handoff of gemm_tc.cu is here too (wait for the upstream flag, stores into the peer, release flag), so that pieces on
//     several GPUs run the same arithmetic as one piece.
//
// Order of the tiles: token tiles first, so the pairs of a round share few weight tiles (which come from HBM once) and all of X (L2).
//
// Bound: tensor pipe (98 % active while a tile runs) and the power cap.  Measured on B200, Llama-3-8B layer shapes, us (TFLOP/s), back to
// back with cold weights, gemm_tc.cu -> here:
//   4096 tokens: QKV 218 (945) -> 129 (1598), O 157 (875) -> 94 (1462), gate/up 1041 (924) -> 573 (1679), down 404 (1191) -> 329 (1462)
//    512 tokens: QKV 39 (656) -> 21 (1246),   O 27 (633) -> 16 (1062),  gate/up 139 (866) -> 87 (1384),   down 59 (1019) -> 48 (1244)
//    160 tokens: QKV 40 -> 16, O 33 -> 13, gate/up 84 -> 52, down 60 -> 30 (the weights alone: 8, 5, 36, 18)
// These are shortest times.  For seconds on end 4096 tokens are bound by the power cap (988 W, 1.21 to 1.24 GHz): down 398 us, O 111.
//
// Block-scaled fp8 (MX): the same tiles with 128 K per stage; the scale factors come through the ring in runs of 512 bytes and are copied to tensor
// memory in front of their products.  The epilogue's lane has whole blocks of 32 features of its token, so the e4m3 copy that the next product reads
// needs no exchange between lanes.  256-wide tiles leave no columns for scale factors beside two accumulators, so these overlap by 32 columns, which
// the epilogue takes first (128-wide tiles have none of that, but twice the rounds: gate/up of 4096 tokens 384 us against 333).  gemm_tc.cu reads
// 128 + 256 operand rows per 128 x 256 tile and has no second accumulator.  Llama-3-8B layer shapes, us, back to back with cold weights, gemm_tc.cu -> here:
//   4096 tokens: QKV 223 -> 76, O 264 -> 59, gate/up 1751 -> 333 (2.9 PFLOP/s), down 461 -> 189
//    512 tokens: QKV  50 -> 17, O  44 -> 13, gate/up  286 -> 50, down 77 -> 29
//    128 tokens: QKV  28 -> 11, O  17 -> 12, gate/up   84 -> 32, down 55 -> 20
// Roles (320 threads): warp 0 = TMA producer (both CTAs), warp 1 = TMEM owner, MMA issuer in the pair's even CTA, warps 2..9 = epilogue.
#include "gemm_tc.cuh"

#include <cuda_fp8.h>

#include <type_traits>

#include "activations.cuh"
#include "common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "tmem.cuh"
#include "wide_plan.cuh"

namespace b2b {

int make_tmap_shared(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, int elt_bytes);
int make_sf_tmap(CUtensorMap* m, const void* ptr, uint64_t chunks);

namespace {

constexpr int WM = 128;                    // token rows per CTA (256 per pair)
constexpr int WK = 64;                     // K elements per stage (one 128-byte swizzled row; block-scaled fp8: 128)
constexpr int WA_BYTES = WM * 128;
constexpr int EPI_WARPS = 8;               // two per 32 token rows, each with 32 of every 64 features
constexpr int WIDE_THREADS = 64 + 32 * EPI_WARPS;
constexpr int WIDE_PAIRS = 74;             // of the 148 SMs
constexpr int EPI_PITCH = 80;              // bytes per staged row of 64: 16-byte accesses of 8 lanes fall into distinct banks
constexpr int EPI_BYTES = EPI_WARPS * 32 * EPI_PITCH;

__device__ unsigned int g_wide_gave_up = 0;        // CTAs whose waits ran out since the module was loaded

template <int BN, bool MX>
struct WideCfg {
  static constexpr int kBBytes = BN / 2 * 128;                           // this CTA's half of the weight rows
  static constexpr int kStageBytes = WA_BYTES + kBBytes;
  static constexpr int kSfBytes = MX ? 512 + BN / 128 * 512 : 0;         // scale factors: this CTA's token rows, all weight rows of the pair
  static constexpr int kStages = BN == 256 ? 6 : (BN == 192 ? 7 : 8);
  static constexpr int kLandPitch = BN / 2 + 4;                          // floats per row of the split-K landing zone
  static constexpr int kSmem = 1024 + kStages * (kStageBytes + kSfBytes) + EPI_BYTES + 512;
  static constexpr uint32_t kTmemCols = (MX || BN != 128) ? 512 : 256;
  // Accumulators: two of BN columns.  Behind two of 256 no columns are left for scale factors, so those of block-scaled tiles share 32: the
  // epilogue takes the shared columns into registers before anything else, and only then may the next tile begin.
  static constexpr bool kShared = MX && BN == 256;
  static constexpr uint32_t kAccStride = kShared ? 224 : BN;
  static constexpr uint32_t kSfCol = kAccStride + BN;                    // two sets of 16 columns
  static_assert(!MX || kSfCol + 32 <= kTmemCols, "scale factors lie behind the accumulators");
  static_assert(WM * kLandPitch * 4 <= kStages * kStageBytes, "the landing zone reuses the ring");
  static_assert(kSmem <= 232448, "shared memory of an SM");
};

template <uint32_t kCols>
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_result) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "n"(kCols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <uint32_t kCols>
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(kCols) : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// block-scaled e4m3: scale factors of both operands in tensor memory, each CTA's own token rows and all weight rows of the pair
__device__ __forceinline__ void umma2_mxf8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// scale factors of 128 rows, shared memory -> tensor memory, in both CTAs of the pair
__device__ __forceinline__ void tmem_cp2_32x128b_warpx4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// arrives on the barrier at this offset in the CTAs of `mask` once the MMAs issued so far have retired
__device__ __forceinline__ void umma2_commit(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(mask)
      : "memory");
}
// tiled load into this CTA's shared memory whose bytes are counted on a barrier of the pair's even CTA (`bar`: its cluster address)
__device__ __forceinline__ void tma_load2(void* smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

// One arrival per CTA; the last one releases the payload to the downstream piece and this piece's input slot to the upstream one -- unless a
// CTA gave up (counted in the upper half of the counter) or the process has aborted: a neighbour that waits for this payload then runs
// into its own limit and reports it, where stale rows would become tokens.
__device__ __forceinline__ void publish_handoff(const GemmParams& p, uint32_t total, bool gave_up) {
  const uint32_t mine = gave_up ? 0x10001u : 1u, done = atomicAdd(p.done_counter, mine) + mine;
  if ((done & 0xffffu) != total) return;
  __threadfence_system();
  *p.done_counter = 0;
  const volatile uint32_t* ab = g_abort_word;
  if ((done >> 16) != 0u || (ab != nullptr && *ab != 0u)) return;
  if (p.signal_flag != nullptr) {
    const uint32_t e = *reinterpret_cast<volatile uint32_t*>(p.signal_epoch) + 1;
    *reinterpret_cast<volatile uint32_t*>(p.signal_epoch) = e;
    st_release_sys(p.signal_flag, e);
  }
  if (p.bump_epoch != nullptr) {
    const uint32_t e = *reinterpret_cast<volatile uint32_t*>(p.bump_epoch) + 1;
    *reinterpret_cast<volatile uint32_t*>(p.bump_epoch) = e;
    if (p.ack_flag != nullptr) st_release_sys(p.ack_flag, e);
  }
}

// The flags of the neighbouring pieces.  Every role waits for what its own bounded waits depend on before it starts counting polls: an
// upstream or downstream piece may be late by the time limit of the process (wait_flag_ge), far longer than those waits last.
__device__ __forceinline__ void wait_upstream(const GemmParams& p) {
  if (p.wait_flag != nullptr) wait_flag_ge(p.wait_flag, *reinterpret_cast<const volatile uint32_t*>(p.wait_epoch) + 1);
}
// the consumer must have drained the previous payload of this slot
__device__ __forceinline__ void wait_downstream(const GemmParams& p) {
  if (p.free_flag != nullptr) wait_flag_ge(p.free_flag, *reinterpret_cast<const volatile uint32_t*>(p.signal_epoch) - p.free_lag);
}

struct NoMaps {};
struct SfMaps {                            // scale factors as rows of 512 bytes
  CUtensorMap w, x;
};

template <int BN, int EPI, bool MX>
__global__ void __launch_bounds__(WIDE_THREADS, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GemmParams p,
                 const int allow_split, const __grid_constant__ std::conditional_t<MX, SfMaps, NoMaps> sf_maps) {
  using Cfg = WideCfg<BN, MX>;
  constexpr int STAGES = Cfg::kStages;
  constexpr int KE = MX ? 128 : WK;                // K elements per stage
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_out = smem + STAGES * Cfg::kStageBytes;
  uint8_t* sf_s = stage_out + EPI_BYTES;           // [STAGES][kSfBytes]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(sf_s + STAGES * Cfg::kSfBytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;         // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2], of the pair's even CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort = tmem_slot + 1;
  __shared__ float freq_s[128];                    // rotary frequencies of a head (QKV epilogue)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const bool odd = (crank & 1u) != 0u;             // which half of the pair
  const uint32_t lead = crank & ~1u;
  const int pair = static_cast<int>(blockIdx.x >> 1);

  const WidePlan plan((p.m_tok + 2 * WM - 1) / (2 * WM), (p.n_out + BN - 1) / BN, p.k / KE, static_cast<int>(gridDim.x >> 1), allow_split != 0);
  constexpr int GAP = wide_gap(Cfg::kShared);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    if constexpr (MX) {
      tma_prefetch_desc(&sf_maps.w);
      tma_prefetch_desc(&sf_maps.x);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * EPI_WARPS);     // the epilogue warps of both CTAs
    }
    *abort = 0u;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc2<Cfg::kTmemCols>(tmem_slot);
  if constexpr (EPI == EPI_QKV_ROPE) {
    if (p.rope_theta > 0.f)
      for (int j = threadIdx.x; j < p.head_dim / 2; j += WIDE_THREADS)
        freq_s[j] = exp2f(-(2.f * j / static_cast<float>(p.head_dim)) * log2f(p.rope_theta));
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_relaxed();                        // the other CTAs arrive on these barriers (their initialisation is released by its own fence)
  cluster_wait_acquire();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();

  bool ok = true;
  WideItem it;
  auto fill = [&](uint32_t n, int kb, int n0, int m0, bool w, bool x) {       // stage n of this CTA
    const uint32_t s = n % STAGES;
    uint8_t* st = smem + s * Cfg::kStageBytes;
    const uint32_t bar = mapa_smem(smem_u32(&full_bar[s]), lead);
    if (w) {
      if (!odd) mbar_arrive_expect_tx(&full_bar[s], 2 * (Cfg::kStageBytes + Cfg::kSfBytes));
      tma_load2(st + WA_BYTES, &tmap_w, bar, kb * KE, n0 + (odd ? BN / 2 : 0));
      if constexpr (MX) {
#pragma unroll
        for (int j = 0; j < BN / 128; ++j)     // (rows behind the last are not there: zeros, for features that are not stored)
          tma_load2(sf_s + s * Cfg::kSfBytes + 512 + j * 512, &sf_maps.w, bar, 0, (n0 / 128 + j) * plan.nkb + kb);
      }
    }
    if (x) {
      tma_load2(st, &tmap_x, bar, kb * KE, m0 + (odd ? WM : 0));
      if constexpr (MX) {                      // runs of 128 tokens, or (sf_bn 256) of 256 whose halves lie side by side
        const int half = odd ? 1 : 0, run = p.sf_bn > 128 ? (m0 / 256 * plan.nkb + kb) * 2 + half : (m0 / 128 + half) * plan.nkb + kb;
        tma_load2(sf_s + s * Cfg::kSfBytes, &sf_maps.x, bar, 0, run);
      }
    }
  };
  if (warp == 0) {
    // ------------------------------------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t n = 0;                              // stages filled so far
      for (int i = 0; ok && plan.get(i, pair, it); ++i) {
        const int m0 = it.t % plan.tok_tiles * (2 * WM), n0 = it.t / plan.tok_tiles * BN;
        int kb = it.kb0;
        if (i == 0) {                              // the weights depend on no earlier kernel: fill the ring with them first
          const int pre = min(STAGES, it.kb1 - it.kb0);
          for (; n < static_cast<uint32_t>(pre); ++n) fill(n, kb + n, n0, m0, true, false);
          pdl_wait();                              // (the tokens' part of these stages: an epilogue warp)
          wait_upstream(p);                        // head of a piece: X is written by the upstream GPU
          if (p.wait_flag != nullptr) fence_proxy_async_all();      // peer-written (generic proxy) data -> TMA (async proxy) reads
          kb += pre;
        }
        if (i == (Cfg::kShared ? 1 : 2)) wait_downstream(p);      // (two accumulators: from here on the ring waits for the epilogue, too)
        for (; kb < it.kb1; ++kb, ++n) {
          if (!(ok = ma_wait(&empty_bar[n % STAGES], (n / STAGES & 1u) ^ 1u, abort))) break;
          fill(n, kb, n0, m0, true, true);
        }
      }
      // the odd CTA hears of its stages from the even one's products: of the last ones, too, before it leaves
      for (uint32_t j = n > STAGES ? n - STAGES : 0; ok && j < n; ++j) ok = ma_wait(&empty_bar[j % STAGES], j / STAGES & 1u, abort);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------------------------------------- MMA issuer
    if (!odd && elect_one()) {
      constexpr uint32_t idesc = MX ? make_idesc_mxf8(2 * WM, BN) : make_idesc_bf16(2 * WM, BN);
      const uint16_t both = static_cast<uint16_t>(3u << lead);
      uint32_t n = 0;
      for (int i = 0; ok && plan.get(i, pair, it); ++i) {
        const uint32_t b = i & 1;
        if (i == 0) {
          pdl_wait();                              // (no result is needed; the waits below may count once the producer's input is there)
          wait_upstream(p);
        }
        if (i == (Cfg::kShared ? 1 : 2)) wait_downstream(p);
        // (overlapping accumulators: the tile before has left the shared columns, and the one before that all of them)
        if (i >= GAP && !(ok = ma_wait(&acc_empty[(i - GAP) & 1], (i - GAP) >> 1 & 1, abort))) break;
        tc_fence_after();
        for (int kb = it.kb0; kb < it.kb1; ++kb, ++n) {
          const uint32_t s = n % STAGES;
          if (!(ok = ma_wait(&full_bar[s], n / STAGES & 1u, abort))) break;
          tc_fence_after();
          const uint64_t a = make_sw128_kmajor_desc(smem_u32(smem + s * Cfg::kStageBytes));
          const uint64_t w = make_sw128_kmajor_desc(smem_u32(smem + s * Cfg::kStageBytes + WA_BYTES));
          if constexpr (MX) {
            // two sets of columns alternate: copies and products run in the order of their issue
            const uint32_t ta = tmem + Cfg::kSfCol + (n & 1u) * 16, sf = smem_u32(sf_s + s * Cfg::kSfBytes);
            tmem_cp2_32x128b_warpx4(ta, make_sf_desc(sf));
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tmem_cp2_32x128b_warpx4(ta + 4 + 4 * j, make_sf_desc(sf + 512 + 512 * j));
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma2_mxf8(tmem + b * Cfg::kAccStride, a + 2 * k, w + 2 * k, idesc | (static_cast<uint32_t>(k) << 4) | (static_cast<uint32_t>(k) << 29),
                         (kb > it.kb0 || k > 0) ? 1u : 0u, ta, ta + 4);
          } else {
#pragma unroll
            for (int k = 0; k < WK / 16; ++k) umma2_bf16(tmem + b * BN, a + 2 * k, w + 2 * k, idesc, (kb > it.kb0 || k > 0) ? 1u : 0u);
          }
          umma2_commit(&empty_bar[s], both);
        }
        if (ok) umma2_commit(&acc_full[b], both);
      }
    }
  } else {
    // ---------------------------------------------------------------------------------------------------- epilogue
    // Two warps per 32 rows (with one, each scheduler had a single chain of reads, activations and stores): the last tile's epilogue is in nobody's shadow, and
    // with a short K all of them take longer than a main loop.  From the last product to the last store, four warps -> eight, us: 512 tokens QKV 3.1 -> 2.8,
    // O 3.8 -> 2.8, gate/up 9.5 -> 6.7, down 3.6 -> 3.1; up with GELU 768 x 3072, 240 tokens (three activations in one loop before) 9.0 -> 4.3.
    const int q = warp & 3, hw = (warp - 2) >> 2;
    const int row = q * 32 + lane;                 // TMEM lane == token row of this CTA
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q * 32) << 16);
    uint8_t* sbuf = stage_out + (warp - 2) * 32 * EPI_PITCH;
    uint8_t* srow = sbuf + lane * EPI_PITCH;       // this lane's staged row
    const int sr = lane >> 2, sc = (lane & 3) * 16;        // coalesced view: rows sr + 8 i, byte column sc
    const int q_dim = p.n_q_heads * p.head_dim, kv_dim = p.n_kv_heads * p.head_dim;
    pdl_wait();
    wait_upstream(p);
    if (warp == 2 && plan.get(0, pair, it) && elect_one()) {       // X of the first stages: the producer may still be issuing their weights
      if (p.wait_flag != nullptr) fence_proxy_async_all();
      for (int j = 0; j < min(STAGES, it.kb1 - it.kb0); ++j)
        fill(j, it.kb0 + j, it.t / plan.tok_tiles * BN, it.t % plan.tok_tiles * (2 * WM), false, true);
    }
    __syncwarp();
    wait_downstream(p);
    if constexpr (MX) {                            // sums of squares that an earlier product has read and a later one adds to
      if (p.zero_buf != nullptr && blockIdx.x == 0)
        for (int t = threadIdx.x - 64; t < p.m_tok; t += 32 * EPI_WARPS) p.zero_buf[t] = 0.f;
    }
    uint32_t hold[Cfg::kShared ? 32 : 1];          // the accumulator columns that two tiles share
    int hold_c = -1;                               // the first of them in the tile that is worked on

    // the residual values of this warp's 32 columns in the coalesced view, in flight while the accumulators are awaited or worked on
    uint4 res[EPI == EPI_RESIDUAL ? 4 : 1];
    auto fetch_res = [&](int m0, int n) {
      if constexpr (EPI == EPI_RESIDUAL) {
        const uint8_t* src = reinterpret_cast<const uint8_t*>(p.residual + n) + sc;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = m0 + q * 32 + sr + 8 * i;
          res[i] = make_uint4(0u, 0u, 0u, 0u);
          if (t < p.m_tok && n < p.n_out) res[i] = *reinterpret_cast<const uint4*>(src + static_cast<size_t>(t) * p.ld_res * 2);
        }
      }
    };
    // what belongs to this lane's token, in flight while the accumulator is awaited
    float tok_scale = 1.f, tok_pos = 0.f;
    int tok_slot = -1;
    auto fetch_token = [&](int m0) {
      const int tok = m0 + row;
      const bool live = tok < p.m_tok;
      tok_scale = (p.rstd != nullptr && live) ? p.rstd[tok] : 1.f;
      if constexpr (MX)
        if (p.sumsq != nullptr && live) tok_scale *= rsqrtf(p.sumsq[tok] / static_cast<float>(p.k) + p.eps);
      if constexpr (EPI == EPI_QKV_ROPE) {
        tok_slot = live ? p.slots[tok] : -1;
        tok_pos = (p.positions != nullptr && live) ? static_cast<float>(p.positions[tok]) : 0.f;
      }
    };
    // columns [c0, c1) of the tile at (token m0, feature n0); `land`: the other pair's partial sums of this lane's row, from column c0 on
    auto finish = [&](uint32_t acc, int m0, int n0, int c0, int c1, const float* land) {
      const int tok = m0 + row;
      const bool live = tok < p.m_tok;
      if (m0 + q * 32 >= p.m_tok) return;          // no token of this warp (warp-uniform)
      const float rs = tok_scale, pos = tok_pos;
      const int slot = tok_slot;
      float ssq = 0.f;
      auto load = [&](int c, float* v) {           // 32 accumulator columns, scaled
        uint32_t r[32];
        ma_ld32(acc + c, r);
        ma_ld_fence(r);
        if constexpr (Cfg::kShared) {              // (the next tile may be writing there)
          if (c == hold_c)
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = hold[j];
        }
        if (land != nullptr) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 o = *reinterpret_cast<const float4*>(land + (c - c0) + 4 * j);
            v[4 * j] = __uint_as_float(r[4 * j]) + o.x;
            v[4 * j + 1] = __uint_as_float(r[4 * j + 1]) + o.y;
            v[4 * j + 2] = __uint_as_float(r[4 * j + 2]) + o.z;
            v[4 * j + 3] = __uint_as_float(r[4 * j + 3]) + o.w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= rs;
        if (p.bias != nullptr) {
          const float4* b4 = reinterpret_cast<const float4*>(p.bias + n0 + c);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 bv = b4[j];
            v[4 * j] += bv.x; v[4 * j + 1] += bv.y; v[4 * j + 2] += bv.z; v[4 * j + 3] += bv.w;
          }
        }
      };
      auto put = [&](const float* v) {             // 32 values as bf16 into this lane's staged row
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(srow + j * 16) = make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]),
                                                                pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
      };
      // staged rows -> memory: `base` = address of token m0's row at this warp's first column, `ld` in bytes
      auto flush = [&](uint8_t* base, size_t ld) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = sr + 8 * i, t = q * 32 + r;
          const uint4 w = *reinterpret_cast<const uint4*>(sbuf + r * EPI_PITCH + sc);
          if (m0 + t < p.m_tok) *reinterpret_cast<uint4*>(base + static_cast<size_t>(m0 + t) * ld + sc) = w;
        }
        __syncwarp();
      };

      // Block-scaled copy of 32 finished features (this lane's staged bf16 row) for the product that reads them: e4m3, a power of two in the layout of
      // that product's operand, and the row's sum of squares.  A lane has the whole block of its token: no exchange.
      auto emit_q = [&](int feat) {
        uint32_t e8[8];
        float r[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 w = *reinterpret_cast<const uint4*>(srow + j * 16);
          const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(x[e]);
            r[8 * j + 2 * e] = f.x;
            r[8 * j + 2 * e + 1] = f.y;
          }
        }
        float most = fabsf(r[0]);                  // (of nothing but NaNs: NaN, as in the other quantisers)
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          most = fmaxf(most, fabsf(r[j]));
          ssq += r[j] * r[j];
        }
        const int ex = mx_exponent(most);
        const float inv = mx_inverse(ex);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(r[4 * j] * inv, r[4 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
          const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(r[4 * j + 2] * inv, r[4 * j + 3] * inv), __NV_SATFINITE, __NV_E4M3);
          e8[j] = lo | (hi << 16);
        }
        if (live) p.q_sf[mx_sf_at(tok, feat, p.q_bn, p.ld_q >> 7)] = static_cast<uint8_t>(ex + 127);
        __syncwarp();                              // the bf16 rows have been stored
        *reinterpret_cast<uint4*>(srow) = make_uint4(e8[0], e8[1], e8[2], e8[3]);
        *reinterpret_cast<uint4*>(srow + 16) = make_uint4(e8[4], e8[5], e8[6], e8[7]);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i) {              // 32 bytes of a row, 16 rows at a time
          const int r = (lane >> 1) + 16 * i, t = m0 + q * 32 + r;
          const uint4 w = *reinterpret_cast<const uint4*>(sbuf + r * EPI_PITCH + (lane & 1) * 16);
          if (t < p.m_tok) *reinterpret_cast<uint4*>(p.q_out8 + static_cast<size_t>(t) * p.ld_q + feat + (lane & 1) * 16) = w;
        }
        __syncwarp();
      };

      if constexpr (EPI == EPI_GLU) {              // 64 gate columns, then 64 up columns -> 64 outputs
#pragma unroll 1
        for (int c = c0 + hw * 32; c < c1 && n0 + c < p.n_out; c += 128) {
          float g[32], u[32];
          load(c, g);
          load(c + 64, u);
          if (p.act_gelu) {                        // (the branch outside: code that is not taken is not fetched either)
#pragma unroll
            for (int j = 0; j < 32; ++j) g[j] = gelu_tanh(g[j]) * u[j];
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) g[j] = silu(g[j]) * u[j];
          }
          put(g);
          const int f = (n0 + c - hw * 32) / 2 + hw * 32;
          if (!MX || p.out != nullptr) flush(reinterpret_cast<uint8_t*>(p.out) + static_cast<size_t>(f) * 2, static_cast<size_t>(p.ld_out) * 2);
          if constexpr (MX)
            if (p.q_out8 != nullptr) emit_q(f);
        }
      } else if (EPI == EPI_PLAIN && p.out_fp32) {
#pragma unroll 1
        for (int c = c0 + hw * 32; c < c1 && n0 + c < p.n_out; c += 64) {
          float v[32];
          load(c, v);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<float4*>(srow + j * 16) = make_float4(v[16 * h + 4 * j], v[16 * h + 4 * j + 1], v[16 * h + 4 * j + 2], v[16 * h + 4 * j + 3]);
            flush(reinterpret_cast<uint8_t*>(p.out) + static_cast<size_t>(n0 + c + 16 * h) * 4, static_cast<size_t>(p.ld_out) * 4);
          }
        }
      } else {
#pragma unroll 1
        for (int c = c0 + hw * 32; c < c1 && n0 + c < p.n_out; c += 64) {
          const int n = n0 + c;
          if constexpr (EPI == EPI_RESIDUAL) {     // the residual rows of this block, whole rows at a time
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(sbuf + (sr + 8 * i) * EPI_PITCH + sc) = res[i];
            if (c + 64 < c1) fetch_res(m0, n + 64);
            __syncwarp();
          }
          float v[32];
          load(c, v);
          if constexpr (EPI == EPI_RESIDUAL) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 w = *reinterpret_cast<const uint4*>(srow + j * 16);
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                v[8 * j + 2 * e] += f.x;
                v[8 * j + 2 * e + 1] += f.y;
              }
            }
          } else if constexpr (EPI == EPI_GELU) {
            if (p.act_gelu == 2) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = relu_sq(v[j]);
            } else if (p.act_gelu == 3) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = xielu(v[j], p.rope_theta, p.q_scale);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
            }
          } else if constexpr (EPI == EPI_QKV_ROPE) {
            const int sect = n < q_dim ? 0 : (n < q_dim + kv_dim ? 1 : 2);
            if (sect < 2 && p.rope_theta > 0.f) {
              const int j0 = ((n - (sect ? q_dim : 0)) % p.head_dim) >> 1;      // columns (2j, 2j+1) hold (x_j, x_{j+hd/2})
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                float sn, cs;
                sincosf(pos * freq_s[j0 + j], &sn, &cs);
                const float a = v[2 * j], b = v[2 * j + 1];
                v[2 * j] = a * cs - b * sn;
                v[2 * j + 1] = b * cs + a * sn;
              }
            }
            if (sect == 0) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] *= p.q_scale;
            }
          }
          put(v);
          if constexpr (EPI == EPI_QKV_ROPE) {
            if (n < q_dim) {
              flush(reinterpret_cast<uint8_t*>(p.q_out + n), static_cast<size_t>(q_dim) * 2);
            } else {                               // a cache row per token
              const bool key = n < q_dim + kv_dim;
              uint8_t* base = reinterpret_cast<uint8_t*>(key ? p.k_cache + (n - q_dim) : p.v_cache + (n - q_dim - kv_dim));
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int r = sr + 8 * i;
                const int sl = __shfl_sync(0xffffffffu, slot, r);
                const uint4 w = *reinterpret_cast<const uint4*>(sbuf + r * EPI_PITCH + sc);
                if (sl >= 0) *reinterpret_cast<uint4*>(base + static_cast<size_t>(sl) * kv_dim * 2 + sc) = w;
              }
              __syncwarp();
            }
          } else {
            flush(reinterpret_cast<uint8_t*>(p.out) + static_cast<size_t>(n) * 2, static_cast<size_t>(p.ld_out) * 2);
            if (EPI == EPI_RESIDUAL && p.out2 != nullptr)
              flush(reinterpret_cast<uint8_t*>(p.out2) + static_cast<size_t>(n) * 2, static_cast<size_t>(p.ld_out) * 2);
            if constexpr (MX && EPI == EPI_RESIDUAL)
              if (p.q_out8 != nullptr) emit_q(n);
          }
        }
      }
      if constexpr (MX) {
        if (p.sumsq_out != nullptr && live) {
          if (p.signal_flag != nullptr) atomicAdd_system(&p.sumsq_out[tok], ssq);          // the tail of a piece: they are the peer's
          else atomicAdd(&p.sumsq_out[tok], ssq);
        }
      }
    };

    int i = 0;
    bool tail = false;
    for (; ok && plan.get(i, pair, it); ++i) {
      const uint32_t b = i & 1;
      const int m0 = it.t % plan.tok_tiles * (2 * WM) + (odd ? WM : 0), n0 = it.t / plan.tok_tiles * BN;
      fetch_token(m0);
      fetch_res(m0, n0 + hw * 32 + (it.split && (crank >> 1) ? BN / 2 : 0));
      ok = __all_sync(0xffffffffu, ma_wait(&acc_full[b], i >> 1 & 1, abort));
      if (!ok) break;
      tc_fence_after();
      if (it.split) {                              // the last item: finished behind the exchange below
        tail = true;
        break;
      }
      if constexpr (Cfg::kShared) {
        if (hw == (b ? 0 : 1)) {                   // (columns 0.. of every 64 are the first warp's, 32.. the second's)
          hold_c = b ? 0 : static_cast<int>(Cfg::kAccStride);
          ma_ld32(lanes + Cfg::kAccStride, hold);
          ma_ld_fence(hold);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && plan.awaited(i, pair, GAP)) arrive_cluster_read(mapa_smem(smem_u32(&acc_empty[b]), lead));
        finish(lanes + b * Cfg::kAccStride, m0, n0, 0, BN, nullptr);
        hold_c = -1;
      } else {
        finish(lanes + b * BN, m0, n0, 0, BN, nullptr);
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && plan.awaited(i, pair, GAP)) arrive_cluster_read(mapa_smem(smem_u32(&acc_empty[b]), lead));
      }
    }
    if (plan.split) {
      // ------------------------------------- exchange of a split tile: pair 0 finishes columns [0, BN/2), pair 1 the others
      const uint32_t acc = lanes + (i & 1) * Cfg::kAccStride;
      const int mine = (crank >> 1) ? BN / 2 : 0, theirs = BN / 2 - mine;
      cluster_arrive_relaxed();                    // every MMA of the cluster has retired: the rings are free
      cluster_wait_acquire();
      if (tail) {
        const uint32_t zone = mapa_smem(smem_u32(smem), crank ^ 2u) + static_cast<uint32_t>(row * Cfg::kLandPitch * 4);
#pragma unroll 1
        for (int c = hw * 32; c < BN / 2; c += 64) {
          uint32_t r[32];
          ma_ld32(acc + theirs + c, r);
          ma_ld_fence(r);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            st_dsmem_v4(zone + (c + 4 * j) * 4, make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                            __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
        }
      }
      cluster_arrive_release();
      cluster_wait_acquire();
      if (tail)
        finish(acc, it.t % plan.tok_tiles * (2 * WM) + (odd ? WM : 0), it.t / plan.tok_tiles * BN, mine, mine + BN / 2,
               reinterpret_cast<const float*>(smem) + row * Cfg::kLandPitch);
      tc_fence_before();
    }
    if (p.signal_flag != nullptr || p.bump_epoch != nullptr) {        // tail of a piece: the last CTA publishes the payload
      __threadfence_system();                      // my (possibly peer-directed) stores are performed
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (threadIdx.x == 64) publish_handoff(p, gridDim.x, *abort != 0u);
    }
  }
  if (warp < 2) {
    __syncwarp();
    if (plan.split) {
      for (int k = 0; k < 2; ++k) {
        cluster_arrive_relaxed();
        cluster_wait_acquire();
      }
    }
  }
  if (*abort != 0u) __nanosleep(200000);           // copies in flight land before the shared memory is given back
  tc_fence_before();
  __syncthreads();
  // No CTA leaves while another may still read its operands (these products have retired) or arrive on its barriers.  All arrivals from another CTA are waited for:
  // acc_empty by the even CTA's products (WidePlan::awaited), stages and accumulators by the producer and the epilogue.  So there is nothing to release.
  cluster_arrive_relaxed();
  cluster_wait_acquire();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2<Cfg::kTmemCols>(tmem);
  }
  if (threadIdx.x == 0 && *abort != 0u) {          // a wait ran out: the process learns of it
    if (g_abort_word != nullptr) *g_abort_word = 1u;
    atomicAdd(&g_wide_gave_up, 1u);
  }
}

// One launch: `pairs` pairs of CTAs in clusters of 2, or (split) of 4.
template <int BN, int EPI, bool MX>
int launch_wide_one(const GemmParams& p, const CUtensorMap& tw, const CUtensorMap& tx, const SfMaps& sf, int pairs, bool split, cudaStream_t stream) {
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_wide_kernel<BN, EPI, MX>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideCfg<BN, MX>::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 64) set[dev] = true;
  }
  std::conditional_t<MX, SfMaps, NoMaps> maps;
  if constexpr (MX) maps = sf;
  return static_cast<int>(launch_kernel_cx(gemm_wide_kernel<BN, EPI, MX>, dim3(2 * pairs), dim3(WIDE_THREADS), WideCfg<BN, MX>::kSmem, stream,
                                           split ? 4u : 2u, tw, tx, p, split ? 1 : 0, maps));
}

template <int BN, bool MX>
int launch_wide_bn(const GemmParams& p, const CUtensorMap& tw, const CUtensorMap& tx, const SfMaps& sf, int pairs, bool split, cudaStream_t stream) {
  switch (p.epi) {
    case EPI_PLAIN: return launch_wide_one<BN, EPI_PLAIN, MX>(p, tw, tx, sf, pairs, split, stream);
    case EPI_RESIDUAL: return launch_wide_one<BN, EPI_RESIDUAL, MX>(p, tw, tx, sf, pairs, split, stream);
    case EPI_GLU:
      if constexpr (BN % 128 == 0) return launch_wide_one<BN, EPI_GLU, MX>(p, tw, tx, sf, pairs, split, stream);
      return -4;
    case EPI_QKV_ROPE: return launch_wide_one<BN, EPI_QKV_ROPE, MX>(p, tw, tx, sf, pairs, split, stream);
    case EPI_GELU:
      if constexpr (!MX) return launch_wide_one<BN, EPI_GELU, MX>(p, tw, tx, sf, pairs, split, stream);
      return -4;
    default: return -4;
  }
}

// Clusters of four CTAs that are resident at once: a GPC whose SM count is no multiple of four leaves some idle, so fewer than 37 (a
// persistent grid of 37 ran its last clusters in a second pass and took twice as long).
int wide_clusters4() {
  static int known[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && known[dev] > 0) return known[dev];
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(148);
  cfg.blockDim = dim3(WIDE_THREADS);
  cfg.dynamicSmemBytes = WideCfg<256, false>::kSmem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 4;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(gemm_wide_kernel<256, EPI_PLAIN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideCfg<256, false>::kSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, gemm_wide_kernel<256, EPI_PLAIN, false>, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = 1;
  }
  if (n > 37) n = 37;
  if (dev < 64) known[dev] = n;
  return n;
}

struct WideChoice {
  int bn, pairs;
  bool split;
  double cost;
};

// Rounds of a choice in units of a 256-wide tile's round (a 192-wide tile costs 0.78 of it, a 128-wide one 0.58: its token rows are reused half as often; a
// split round 0.6: half of K, and the exchange).
WideChoice wide_choice(const GemmParams& p, int bn, bool split) {
  const int tiles = ((p.m_tok + 2 * WM - 1) / (2 * WM)) * ((p.n_out + bn - 1) / bn);
  WideChoice c{bn, WIDE_PAIRS, split, 0.0};
  const double unit = bn == 256 ? 1.0 : (bn == 192 ? 0.78 : 0.58);
  if (!split) {
    c.cost = unit * ((tiles + WIDE_PAIRS - 1) / WIDE_PAIRS);
    if (tiles < WIDE_PAIRS) c.pairs = tiles;       // the next kernel of the stream may use the other SMs for its set-up
    return c;
  }
  const int clusters = wide_clusters4(), rest = tiles % (2 * clusters);
  c.pairs = tiles <= clusters ? 2 * tiles : 2 * clusters;
  c.cost = unit * (tiles / (2 * clusters) + (rest == 0 ? 0.0 : (rest <= clusters ? 0.6 : 1.0)));
  return c;
}

}  // namespace

bool gemm_wide_supported(const GemmParams& p) {
  const int elt = (p.epi == EPI_PLAIN && p.out_fp32) ? 4 : 2;
  const bool mx = p.fp8 && p.sfa != nullptr;
  if (p.norm_src || p.dbg || (p.fp8 && !mx)) return false;
  if (!mx && (p.q_out8 || p.sumsq || p.sumsq_out || p.zero_buf)) return false;
  const int ke = mx ? 128 : WK;
  if (p.n_out % 128 != 0 || p.k % ke != 0 || p.k < 2 * ke || p.m_tok <= 0) return false;
  if (mx) {
    if (p.epi == EPI_GELU || p.w_scale || p.sfb == nullptr || (p.sf_bn != 128 && p.sf_bn != 256)) return false;      // (runs of 128 tokens, alone or side by side)
    if ((reinterpret_cast<uintptr_t>(p.sfa) | reinterpret_cast<uintptr_t>(p.sfb)) & 15) return false;
    if (p.q_out8 && (((reinterpret_cast<uintptr_t>(p.q_out8) | static_cast<uintptr_t>(p.ld_q)) & 15) || (reinterpret_cast<uintptr_t>(p.q_sf) & 1))) return false;
    if (p.q_out8 && p.q_bn != 128 && p.q_bn != 256) return false;
  }
  if (p.epi == EPI_GELU && p.act_gelu == 4) return false;
  if (p.bias && (reinterpret_cast<uintptr_t>(p.bias) & 15)) return false;
  if (p.epi == EPI_QKV_ROPE) {
    if (p.head_dim > 256 || p.head_dim % 32 || (p.n_q_heads * p.head_dim) % 128 || (p.n_kv_heads * p.head_dim) % 128) return false;
    return !((reinterpret_cast<uintptr_t>(p.q_out) | reinterpret_cast<uintptr_t>(p.k_cache) | reinterpret_cast<uintptr_t>(p.v_cache)) & 15);
  }
  if (((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.out2)) & 15) || (static_cast<size_t>(p.ld_out) * elt) % 16) return false;
  if (p.epi == EPI_RESIDUAL && ((reinterpret_cast<uintptr_t>(p.residual) & 15) || (static_cast<size_t>(p.ld_res) * 2) % 16)) return false;
  return true;
}

int launch_gemm_wide(const GemmParams& p, const void* w, const void* x, int bn, int split, cudaStream_t stream) {
  if (!gemm_wide_supported(p)) return -2;
  const bool mx = p.fp8;
  // Two pairs on a tile save half of its blocks of K (0.17 us each) and exchange sums (1.6 us): 768 x 768, 240 tokens, whole 6.9 us, cut 7.4; 3072 x 768 7.4
  // and 8.2; 768 x 3072 12.4 and 10.0.  (Where the call names it, from 8 blocks on: halves of four.)
  const int blocks = p.k / (mx ? 128 : WK);
  const bool can_split = blocks >= (split == 1 ? 8 : 20);
  WideChoice best{0, 0, false, 1e30};
  for (int b = 256; b >= 128; b -= 64) {
    if (bn >= 128 && bn <= 256 && b != bn) continue;
    if (b == 192 && (p.epi == EPI_GLU || mx)) continue;                          // (gate/up pairs, and runs of scale factors, are 128 columns wide)
    for (int s = 0; s < 2; ++s) {
      if ((split == 0 || split == 1) && s != split) continue;
      if (s && (!can_split || b == 192 || (b == 128 && p.epi == EPI_GLU))) continue;     // halves are whole 64-column blocks
      const WideChoice c = wide_choice(p, b, s != 0);
      if (c.cost < best.cost) best = c;
    }
  }
  if (best.bn == 0) return -4;
  CUtensorMap tw, tx;
  SfMaps sf;
  int r = make_tmap_shared(&tw, w, p.n_out, p.k, p.k, best.bn / 2, mx ? 1 : 2);
  if (r) return r;
  if ((r = make_tmap_shared(&tx, x, p.m_tok, p.k, p.k, WM, mx ? 1 : 2))) return r;
  if (mx) {
    const uint64_t nkb = p.k / 128;
    if ((r = make_sf_tmap(&sf.w, p.sfa, p.n_out / 128 * nkb))) return r;
    if ((r = make_sf_tmap(&sf.x, p.sfb, (p.m_tok + p.sf_bn - 1) / p.sf_bn * (p.sf_bn / 128) * nkb))) return r;
    return best.bn == 128 ? launch_wide_bn<128, true>(p, tw, tx, sf, best.pairs, best.split, stream)
                          : launch_wide_bn<256, true>(p, tw, tx, sf, best.pairs, best.split, stream);
  }
  if (best.bn == 192) return launch_wide_bn<192, false>(p, tw, tx, sf, best.pairs, false, stream);
  return best.bn == 128 ? launch_wide_bn<128, false>(p, tw, tx, sf, best.pairs, best.split, stream)
                        : launch_wide_bn<256, false>(p, tw, tx, sf, best.pairs, best.split, stream);
}

int set_wait_policy_wide(uint32_t* abort_word, unsigned long long limit_ns) {
  cudaError_t e = cudaMemcpyToSymbol(g_abort_word, &abort_word, sizeof(abort_word));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_wait_limit_ns, &limit_ns, sizeof(limit_ns));
  return static_cast<int>(e);
}

unsigned gemm_wide_gave_up() {
  unsigned n = 0;
  return cudaMemcpyFromSymbol(&n, g_wide_gave_up, sizeof(n)) == cudaSuccess ? n : ~0u;
}

}  // namespace b2b
