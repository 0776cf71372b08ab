// Decode steps: all layers of a piece in ONE persistent kernel whose weight stream goes on across the ends of operations.
//
// A decode step is a chain of small dependent operations per layer (QKV, attention, O, [norm], gate/up, down, [norm]), each of which streams its
// weights or cache pages once.  As separate kernels each ends with its slowest block, starts with the latency of a launch and of its first loads, and
// has only what fits beside the kernel before it on the way.  Here 132 SMs run one CTA each for the whole step (33 clusters of four fit the device; 16 SMs
// have none), and two producer warps walk the list of weight tiles and cache pages of ALL operations: while an operation waits for the one before it, the
// next 140 to 180 KB per SM (3 to 4 us of the HBM stream) land in the ring.  132 CTAs ask for 11 to 14 TB/s with two issuing warps each, so the stream
// misses no SM; attention of few sequences, which fewer CTAs share, does (the rule in models/native.py leaves such steps to attn_decode.cu).
//
//   * operations are separated by a counter in global memory that every CTA adds to when its share of the results is stored; one warp per
//     CTA polls it.  All CTAs are resident (cooperative launch).
//   * weights are the 128 MMA rows, tokens the columns (16 / 32 / 64), as in gemm_tc.cu.  A cluster of four CTAs shares a run of rows and each takes a
//     quarter of K (reading all of X in every CTA would double the traffic from L2 at 32 tokens); the partial sums travel to the CTA that finishes a
//     quarter of the tokens with st.async, which counts its bytes on the receiver's mbarrier, and are added in the order of K.
//   * attention as in attn_decode.cu (keys as MMA rows); its cache tiles pass through the same ring, so the pages that the new token does not touch
//     are fetched while the QKV products run.  Few sequences: the CTAs of a cluster share the keys and merge through DSMEM.
//   * LayerNorm models with 64-wide heads (GPT-2): the norms are operations of a CTA per token, attention runs on CUDA cores (a warp or a CTA per
//     token and head), so prompts of up to 64 tokens take the same path.
//   * block-scaled fp8: weights, and the activations that the epilogues leave beside the bf16 ones, are e4m3 with a power of two per 32 channels; the scale
//     factors travel behind the operands' blocks and go through TMEM (tcgen05.cp) to kind::mxf8f6f4.block_scale.
//   * the sums of squares for the next norm are left by the CTAs that write the rows, one number per CTA and token, added in a fixed order.
//
// Bound: the HBM stream and, between operations, the chain of last product, exchange, store, counter, poll and first activations (3 to 4.5 us, of
// which the ring hides most).  Measured on B200, replayed back to back, two Llama-3-8B layers behind 500 keys, us (kernels one by one / here): one token 189 /
// 164, 32 tokens 220 / 185, 64 tokens 274 / 225; two Gemma-2-2B layers: one token 121 / 95, 32 tokens 146 / 122; the layers of gpt2, 16 tokens 489 / 291, 64
// tokens 622 / 430 (84 operations of 3 to 5 us); block-scaled fp8, two Llama-3-8B layers: one token 144 / 112, 16 tokens 150 / 119, 32 tokens 170 / 142.
// Roles: warps 0 and 7 = weights and pages (TMA), 1 = MMA issuer, 2..5 = epilogues and softmax, 6 = activations (TMA).
// All waits are bounded: one that runs out raises the abort word, every other wait then ends too, and the CTAs leave.
#include "kernels.h"

#include <cuda.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <cstring>

#include "activations.cuh"
#include "common.cuh"
#include "tmem.cuh"

namespace b2b {

int make_tmap_shared(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, int elt_bytes);
int make_blocks_tmap(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_blocks, int elt_bytes);

namespace {

constexpr int LC_CL = 4;                           // CTAs of a cluster == parts of K
constexpr int LC_THREADS = 256;
constexpr int LC_PAGE = 64, LC_KEYS = 128, LC_HEADS = 16;
constexpr int LC_BLOCK = 128 * 128;                // 128 rows x 64 bf16: a weight block, or 128 keys x 64 channels
constexpr int LC_XSLOTS = 6;                       // copies of activations in flight, at most
constexpr int LC_ENTRIES = 16;                     // entries of the ring in flight, at most
constexpr uint32_t LC_SPINS = 1u << 23;            // polls of a counter (0.3 us or more each) unless the plan asks for fewer
constexpr int LC_SS = 64 * 64;
constexpr float LC_LOG2E = 1.4426950408889634f;

// operations of a layer; the norms are those behind O and down and exist in some models only
enum LcOp : int { OP_QKV = 0, OP_ATT = 1, OP_O = 2, OP_NORM_A = 3, OP_GU = 4, OP_DOWN = 5, OP_NORM_F = 6, OP_COUNT = 7 };
constexpr int LC_PRODUCTS = 4;
__host__ __device__ constexpr int lc_weight(int op) { return op == OP_QKV ? 0 : (op == OP_O ? 1 : (op == OP_GU ? 2 : (op == OP_DOWN ? 3 : -1))); }

// words of the control block in front of the operations' counters
enum LcWord : int { LW_EXIT = 0, LW_ABORT = 1, LW_GAVE_UP = 2, LW_CTR = 32 };   // LW_GAVE_UP: launches that ended early, never reset

__device__ unsigned int g_chain_gave_up = 0;       // launches that ended early since the module was loaded

// what a layer needs and no call changes
struct alignas(128) LcLayer {
  CUtensorMap w[4][5];                             // weights of the four products, boxes of 8, 16, .. 128 rows
  CUtensorMap k, v;                                // cache pages: boxes of 64 keys x 64 channels
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  const __nv_bfloat16* post_attn;                  // weights of the norms behind O and down, or null
  const __nv_bfloat16* post_ffn;
  const __nv_bfloat16* post_attn_b;                // LayerNorm models: the norms in front of the MLP and of the next layer, and their biases
  const __nv_bfloat16* post_ffn_b;
  const float* bias[4];                            // of the products
  const uint8_t* sf[4];                            // block-scaled fp8: scale factors of the weights
  int window;
};

// activations come in copies of two or four blocks of K of the whole token tile: with a copy per block their issue (0.45 us per entry of the ring) was
// what a product that found its weights landed waited for (one token 177 -> 172 us, 32 tokens 201 -> 194)
struct LcMaps {                                    // activations: boxes of kXBlocks 64-channel blocks x the token tile (q: 16 heads x 64 channels)
  CUtensorMap x_in, xa, xb, attn, h, q;
};

struct LcParams {
  const LcLayer* layers;
  int n_layers, T, seqs, hidden, ffn, n_q, n_kv, head_dim, parts;
  int act, plus_one, norms, x_rows;
  float eps, rope_theta, q_scale, softcap;
  const __nv_bfloat16* x_in;
  __nv_bfloat16 *xa, *xb, *q, *attn, *h, *norm;
  const int *positions, *slots, *q_start, *q_len, *kv_len, *block_table;
  int max_pages;
  uint32_t polls;                                  // of a counter, then the launch gives up
  uint32_t* ctl;
  float* ss;                                       // [2][clusters][64 tokens] sums of squares
  uint8_t *q8_x, *q8_attn, *q8_h;                  // block-scaled fp8: the stream, the attention's output and the MLP hidden as the products read them
  uint8_t *sf_x, *sf_attn, *sf_h;                  // and their scale factors
  const uint8_t* sf_in;                            // of the piece's input
};

// what the layers are made of: RMSNorm and a gated MLP in bf16; LayerNorm, biases and no gate; the first with operands in block-scaled fp8
enum LcKind : int { KIND_RMS = 0, KIND_LN = 1, KIND_MX = 2 };

template <int BN, int KIND>
struct LcCfg {
  static constexpr int kXBlocks = BN == 16 ? 4 : 2;                // 64-channel blocks per copy of activations
  static constexpr int kX = (BN == 16 ? 24 : (BN == 32 ? 32 : 48)) * 1024;       // three copies, four at 32 tokens (six at 8 or fewer)
  static constexpr int kRing = (BN == 64 ? 190 : 207) * 1024 - kX; // weights and cache pages
  static constexpr int kCols = BN / LC_CL;                         // tokens that a CTA of a cluster finishes
  static constexpr int kZone = BN * 512 > 16384 ? BN * 512 : 16384;   // partial sums, or Q (8 KB: two of 128 channels or one of 256) and P
  static constexpr int kSmem = 1024 + kRing + kX + kZone + 640;
  static constexpr uint32_t kS = 2 * BN, kO = 2 * BN + 2 * LC_HEADS;   // TMEM columns behind the two accumulators
  static constexpr uint32_t kTmem = BN == 64 || KIND == KIND_MX ? 256 : 128;
};

__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void lc_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }     // the epilogue warps
__device__ __forceinline__ bool lc_vote(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred a, b;\n\t"
      "setp.ne.u32 a, %1, 0;\n\t"
      "barrier.cta.red.or.pred b, 1, 128, a;\n\t"
      "selp.u32 %0, 1, 0, b;\n\t}\n"
      : "=r"(r) : "r"(p ? 1u : 0u) : "memory");
  return r != 0;
}
__device__ __forceinline__ void tma_load_3d_hint(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(policy) : "memory");
}
// wait on a barrier that the CTAs of the cluster arrive at; one that gave up arrives no more, but raises the launch's abort word
__device__ __forceinline__ bool lc_wait_cluster(uint64_t* bar, uint32_t parity, volatile uint32_t* abort, uint32_t* ctl) {
  for (uint32_t spins = 0;; ++spins) {
    if (try_wait_cluster(bar, parity)) return true;
    if ((spins & 255u) == 255u) {
      if (*abort != 0u) return false;
      if (*reinterpret_cast<volatile uint32_t*>(ctl + LW_ABORT) != 0u) { *abort = 1u; return false; }
    }
    if (spins > MA_SPIN_LIMIT) {
      *abort = 1u;
      return false;
    }
  }
}
// wait until all CTAs have stored their results of an operation
__device__ __noinline__ bool lc_wait_op(const uint32_t* ctr, uint32_t target, uint32_t polls, volatile uint32_t* abort, uint32_t* ctl) {
  for (uint32_t spins = 0;; ++spins) {
    if (ld_acquire_gpu(ctr) >= target) return true;
    if ((spins & 63u) == 63u) {
      if (*abort != 0u) return false;
      if (*reinterpret_cast<volatile uint32_t*>(ctl + LW_ABORT) != 0u) { *abort = 1u; return false; }
    }
    if (spins >= polls) {
      *abort = 1u;
      return false;
    }
  }
}
// wait for copies or products in flight, also after a wait that ran out; nothing depends on the result but when this CTA's memory is given back
__device__ __noinline__ void lc_drain(uint64_t* bar, uint32_t parity) {
  for (uint32_t spins = 0; spins < (1u << 16) && !mbar_try_wait(bar, parity); ++spins) {
  }
}

// wait for an operation through the word that the CTA's polling thread keeps
__device__ __forceinline__ bool lc_wait_due(const uint32_t* due_s, int n, volatile uint32_t* abort) {
  for (uint32_t spins = 0;; ++spins) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(due_s)) : "memory");
    if (static_cast<int>(v) >= n) return true;
    if ((spins & 255u) == 255u && *abort != 0u) return false;
    if (spins > (1u << 28)) {                          // (the polling thread gives up long before)
      *abort = 1u;
      return false;
    }
  }
}

template <int N>
__device__ __forceinline__ void lc_ld(uint32_t taddr, float* v) {    // N columns of this thread's lane
  if constexpr (N == 16) {
    tmem_ld16(taddr, v);
  } else {
    uint32_t r[N];
#pragma unroll
    for (int i = 0; i < N; i += 32) ma_ld32(taddr + i, r + i);
#pragma unroll
    for (int i = 0; i < N; i += 32) ma_ld_fence(r + i);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
  }
}
template <int GP>
__device__ __forceinline__ void lc_ld_heads(uint32_t taddr, float* v) {
  uint32_t r[GP];
  if constexpr (GP == 4)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < GP; ++i) v[i] = __uint_as_float(r[i]);
}
template <int GP>
__device__ __forceinline__ void lc_st_heads(uint32_t taddr, const float* v) {
  if constexpr (GP == 4)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
                 "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])) : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(__float_as_uint(v[0])),
                 "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])),
                 "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])) : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// block-scaled copy of a value per lane, 32 consecutive features of a token: e4m3 and the power of two that brings the largest (`most`) to at most 448, in
// the layout of the product that reads it
__device__ __forceinline__ void lc_store_mx(float r, float most, int tok, int feat, int ld, uint8_t* to, uint8_t* sf, int lane) {
  const int e = mx_exponent(most);
  to[static_cast<size_t>(tok) * ld + feat] = static_cast<uint8_t>(__nv_cvt_float_to_fp8(r * mx_inverse(e), __NV_SATFINITE, __NV_E4M3));
  if (lane == 0) sf[static_cast<size_t>(feat >> 7) * 512 + (tok & 31) * 16 + (tok >> 5) * 4 + ((feat >> 5) & 3)] = static_cast<uint8_t>(e + 127);
}
// the same for tokens tok0 .. tok0 + N, `n` of them wanted, of the values as bf16 (like a separate quantiser): the N chains of shuffles run side by side
template <int N>
__device__ __forceinline__ void lc_put_mx(const float (&v)[N], int n, int tok0, int feat, int ld, uint8_t* to, uint8_t* sf, int lane) {
  float r[N], most[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    r[i] = bf16_round(v[i]);
    most[i] = fabsf(r[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) most[i] = fmaxf(most[i], __shfl_xor_sync(0xffffffffu, most[i], o));
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (i < n) {
      lc_store_mx(r[i], most[i], tok0 + i, feat, ld, to, sf, lane);
    }
}

// share of a product: units [u0, end) of the weights' rows, 64-channel blocks [kb0, kb0 + nkb) of K.  A unit is 8 rows (gate/up: 8 features).
// Shares are cut at multiples of 32 rows (gate/up: 64 or 32 features) where that makes the largest share no more than 4 % larger: a tile then takes
// one or two boxes per block of K.  With shares of single units gate/up needs up to 16, whose issue bound it at 2.3 TB/s.
struct LcShare {
  int u0, end, kb0, nkb;
};
template <bool GLU, bool MX>
__device__ LcShare lc_share(const LcParams& p, int op, int head_dim) {
  LcShare s;
  const int c = blockIdx.x / LC_CL, nc = gridDim.x / LC_CL, r = blockIdx.x % LC_CL;
  const int rows = op == OP_QKV ? (p.n_q + 2 * p.n_kv) * head_dim : p.hidden;
  const int nk = (op == OP_DOWN ? p.ffn : (op == OP_O ? p.n_q * head_dim : p.hidden)) / (MX ? 128 : 64);
  const int u = (op == OP_GU ? p.ffn : rows) / 8, most = (u + nc - 1) / nc;
  int g = GLU && op == OP_GU ? 8 : (MX ? 16 : 4);
  while (g > (MX ? (GLU && op == OP_GU ? 8 : 4) : 1) && (u % g != 0 || (u / g + nc - 1) / nc * g * 25 > most * 26)) g /= 2;
  s.u0 = u / g * c / nc * g;
  s.end = u / g * (c + 1) / nc * g;
  s.kb0 = nk * r / LC_CL;
  s.nkb = nk * (r + 1) / LC_CL - s.kb0;
  return s;
}
// units of the tile that starts at u: up to 128 rows, gate/up tiles do not cross the 64-feature blocks of their rows.  Scale factors come in runs of 128
// rows, a column of TMEM for 32 of them: block-scaled tiles do not cross the runs, and have their rows where the run has them (lc_first)
template <bool GLU, bool MX>
__device__ __forceinline__ int lc_tile(int op, int u, int end) { return min(GLU && op == OP_GU ? 8 - (u & 7) : (MX ? 16 - (u & 15) : 16), end - u); }
template <bool GLU, bool MX>
__device__ __forceinline__ int lc_first(int op, int u) { return MX && !(GLU && op == OP_GU) ? u & 15 : 0; }
template <bool GLU>
__device__ __forceinline__ int lc_rows(int op, int n) { return GLU && op == OP_GU ? n * 16 : n * 8; }

// The ring holds entries of any size back to back (slots of a fixed size would be half empty in a tile of 64 rows): all roles walk the same list and
// find the same places.
template <int BYTES>
struct LcRing {
  uint32_t pos = 0, count = 0;
  __device__ __forceinline__ uint32_t place(uint32_t bytes) {          // of the next entry
    const uint32_t at = pos + bytes > BYTES ? 0u : pos;
    pos = at + bytes;
    return at;
  }
  __device__ __forceinline__ uint32_t entry() const { return count % LC_ENTRIES; }
  __device__ __forceinline__ uint32_t parity() const { return count / LC_ENTRIES & 1u; }
};
// who fills the ring: also waits until there is room.  The two filling warps keep an account each (a word that one leaves for the other took a fence
// per entry: 5 % of a decode step)
template <int BYTES>
struct LcFill : LcRing<BYTES> {
  uint32_t tail = 0, used = 0;                     // the oldest entry in flight, bytes in flight
  __device__ __forceinline__ bool room(uint32_t bytes, uint32_t& at, uint32_t* sizes, uint64_t* empty, volatile uint32_t* abort) {
    const uint32_t before = this->pos;
    at = this->place(bytes);
    const uint32_t taken = at == before ? bytes : BYTES - before + bytes;
#pragma unroll 1
    while (used + taken > BYTES || this->count - tail >= LC_ENTRIES) {
      if (!ma_wait(&empty[tail % LC_ENTRIES], tail / LC_ENTRIES & 1u, abort)) return false;
      used -= sizes[tail % LC_ENTRIES];
      ++tail;
    }
    used += taken;
    sizes[this->entry()] = taken;
    return true;
  }
};
// weights of a tile per block of K: gate/up tiles of fewer than 64 features have their up rows at row 64 all the same
template <bool GLU>
__device__ __forceinline__ uint32_t lc_block_bytes(int op, int n) { return (GLU && op == OP_GU ? 8u + n : n) * 1024u; }

// one (sequence, key/value head): this CTA's share of its key tiles
struct LcItem {
  int seq, kvh, kvlen, kv_lo, t0, nt;
  bool active;
};
__device__ __forceinline__ LcItem lc_item(const LcParams& p, const int* kvlen_s, int window, int j, int part) {
  LcItem it;
  it.seq = j / p.n_kv;
  it.kvh = j - it.seq * p.n_kv;
  it.kvlen = kvlen_s[it.seq];                      // 0: the sequence takes no part
  it.active = it.kvlen > 0;
  it.kv_lo = window > 0 ? max(0, it.kvlen - window) : 0;
  int lo = it.kv_lo / LC_KEYS, hi = it.active ? (it.kvlen + LC_KEYS - 1) / LC_KEYS : lo;
  if (p.parts > 1) {
    const int per = (hi - lo + p.parts - 1) / p.parts;
    lo = min(hi, lo + part * per);
    hi = min(hi, lo + per);
  }
  it.t0 = lo;
  it.nt = hi - lo;
  return it;
}

// D: channels of a head, GP: query heads of a key/value head rounded up to 4 or 8.  KIND_LN: 64-wide heads, the norms are operations in
// front of the products; prompts too
template <int BN, int D, int GP, int KIND>
__global__ void __launch_bounds__(LC_THREADS, 1) layer_chain_kernel(const __grid_constant__ LcMaps maps, const LcParams p) {
  using Cfg = LcCfg<BN, KIND>;
  constexpr bool LN = KIND == KIND_LN, MX = KIND == KIND_MX;
  constexpr bool GLU = !LN;
  const int hd = LN ? p.head_dim : D;               // channels of a head
  constexpr int XB = Cfg::kXBlocks, CW = Cfg::kCols, DB = D / 64, MB = D / 128, NQ = 2 / MB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* x_s = smem + Cfg::kRing;                 // activations
  uint8_t* zone = x_s + Cfg::kX;          // partial sums of the cluster | up and gate halves | Q and P of the attention
  uint64_t* full = reinterpret_cast<uint64_t*>(zone + Cfg::kZone);   // [LC_ENTRIES]
  uint64_t* empty = full + LC_ENTRIES;             // [LC_ENTRIES]
  uint64_t* x_full = empty + LC_ENTRIES;           // [LC_XSLOTS]
  uint64_t* x_empty = x_full + LC_XSLOTS;          // [LC_XSLOTS]
  uint64_t* acc_full = x_empty + LC_XSLOTS;                 // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint64_t* zone_full = acc_empty + 2;
  uint64_t* zone_free = zone_full + 1;
  uint64_t* q_full = zone_free + 1;                // [2]
  uint64_t* q_empty = q_full + 2;                  // [2]
  uint64_t* s_full = q_empty + 2;                  // [2]
  uint64_t* p_ready = s_full + 2;                  // [2]
  uint64_t* pv_done = p_ready + 2;                 // [2]
  uint64_t* o_empty = pv_done + 2;
  uint64_t* part_full = o_empty + 1;
  uint64_t* mma_done = part_full + 1;              // all products that were asked for
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  volatile uint32_t* abort = tmem_slot + 1;
  uint32_t* due_s = tmem_slot + 2;                 // operations whose results are complete, as the activation warp has seen it
  __shared__ float rstd_s[CW];
  __shared__ int pos_s[CW], slot_s[CW], kvlen_s[BN], q_start_s[BN];
  __shared__ int fresh_s[2][LN ? 1 : BN];    // per filling warp: the first key of a sequence that this step writes, -1: not looked for
  __shared__ float red_s[4][GP];             // per warp: maxima
  __shared__ float sq_s[4][CW > GP ? CW : GP];     // per warp: sums of squares, or of a row's weights
  __shared__ float ml_s[2 * GP];             // this CTA's maxima and sums, read by the cluster
  __shared__ LcShare share_s[LC_PRODUCTS];
  __shared__ uint32_t entry_s[2][LC_ENTRIES];      // bytes of the ring's entries, with what was skipped in front of them
  __shared__ uint32_t issued_s[4];                 // copies asked for: ring entries of the two filling warps, activations, queries

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const uint32_t ctas = gridDim.x;
  if (threadIdx.x == 0) {
    for (int i = 0; i < LC_ENTRIES; ++i) {
      mbar_init(&full[i], 2);                      // the two halves
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < LC_XSLOTS; ++i) {
      mbar_init(&x_full[i], 1);
      mbar_init(&x_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 4);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    mbar_init(zone_full, 1);
    mbar_init(zone_free, 4 * LC_CL);
    mbar_init(o_empty, 4);
    mbar_init(part_full, static_cast<uint32_t>(p.parts));
    mbar_init(mma_done, 1);
    *abort = 0u;
    *due_s = 0u;
    fence_barrier_init();
  }
  if (warp == 2)
    for (int op = lane; op < OP_COUNT; op += 32)
      if (lc_weight(op) >= 0) share_s[lc_weight(op)] = lc_share<GLU, MX>(p, op, hd);
  if constexpr (LN) {                              // per token: its sequence (-1: none) and the keys that it sees
    for (int t = threadIdx.x; t < p.T; t += LC_THREADS) {
      int seq = -1, keys = 0;
      for (int i = 0; i < p.seqs; ++i) {
        const int o = t - p.q_start[i], n = p.q_len[i];
        if (o >= 0 && o < n) {
          seq = i;
          keys = max(p.kv_len[i] - n + o + 1, 0);
        }
      }
      q_start_s[t] = seq;
      kvlen_s[t] = keys;
    }
  } else if (warp > 2) {
    for (int i = threadIdx.x - 96; i < p.seqs; i += LC_THREADS - 96) {
      fresh_s[0][i] = fresh_s[1][i] = -1;
      kvlen_s[i] = p.q_len[i] > 0 ? max(p.kv_len[i], 0) : 0;
      q_start_s[i] = p.q_start[i];
    }
  }
  if (warp == 1) tmem_alloc<Cfg::kTmem>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_arrive_release();
  cluster_wait_acquire();
  const uint32_t tmem = *tmem_slot;
  const int G = p.n_q / p.n_kv;
  const bool norms = p.norms != 0;
  uint32_t* const ctr = p.ctl + LW_CTR;
  const int item0 = blockIdx.x / p.parts, part = blockIdx.x % p.parts, item_step = gridDim.x / p.parts, items = p.seqs * p.n_kv;
  const uint32_t x_bytes = static_cast<uint32_t>(p.x_rows) * 128u;     // activations per block of K
  const uint32_t x_slot = x_bytes * XB + (MX ? XB * 512u : 0u), x_slots = min(static_cast<uint32_t>(LC_XSLOTS), Cfg::kX / x_slot);
  auto skip = [&](int l, int op) {                 // (LayerNorm models: the norm in front of the next layer)
    return LN ? (op == OP_NORM_F && l == p.n_layers - 1) : (!norms && (op == OP_NORM_A || op == OP_NORM_F));
  };
  // (every role walks the operations in loops whose bodies appear once: a kernel of 250 KB of code spent microseconds per operation on
  // fetching its instructions)

  if (warp == 0 || warp == 7) {
    // ------------------------------------------------------------------------- weights and cache pages, in the order of their use
    // Two warps, each for one of the two blocks of an entry: the copies of one warp follow one another at 56 GB/s (16 KB boxes; 41 GB/s with 4 KB
    // boxes), however many are asked for, and an SM that is late then cannot use what the others leave of the stream.
    if (elect_one()) {
      const int half = warp == 7;
      uint32_t* sizes = entry_s[half];
      const uint64_t pol = l2_policy_evict_first();
      LcFill<Cfg::kRing> ring;
      uint32_t place = 0;
      bool ok = true;
      int at = 0;                                    // operations so far, over the layers
#pragma unroll 1
      for (int l = 0; ok && l < p.n_layers; ++l) {
        const LcLayer* L = p.layers + l;
        const int window = L->window;
        if (half && l + 1 < p.n_layers) {            // descriptors of the next layer
#pragma unroll 1
          for (int i = 0; i < 22; ++i) tma_prefetch_desc(&(L + 1)->w[0][0] + i);
        }
#pragma unroll 1
        for (int op = 0; ok && op < OP_COUNT; ++op) {
          if (skip(l, op)) continue;
          ++at;
          if (lc_weight(op) >= 0) {
            const LcShare sh = share_s[lc_weight(op)];
            const CUtensorMap* maps_w = L->w[lc_weight(op)];
            const int k_blocks = (op == OP_DOWN ? p.ffn : (op == OP_O ? p.n_q * hd : p.hidden)) / 128;           // (MX)
#pragma unroll 1
            for (int u = sh.u0, n; ok && u < sh.end; u += n) {
              n = lc_tile<GLU, MX>(op, u, sh.end);
              // up to five boxes per block: rows of gate/up come in blocks of [64 gate | 64 up]: gate to rows 0.., up to rows 64.. of the tile
              const bool halves = GLU && op == OP_GU && n < 8;
              const int units = (GLU && op == OP_GU && !halves) ? 16 : n, first = lc_first<GLU, MX>(op, u);
              const int row0 = GLU && op == OP_GU ? (u >> 3) * 128 + (u & 7) * 8 : u * 8;
              const uint32_t bytes = static_cast<uint32_t>(lc_rows<GLU>(op, n)) * 128u, block = lc_block_bytes<GLU>(op, first + n);
#pragma unroll 1
              for (int kb = 0; kb < sh.nkb; kb += 2) {
                const int nb = min(2, sh.nkb - kb);
                if (!(ok = ring.room(block * nb + (MX ? 1024u : 0u), place, sizes, empty, abort))) break;
                uint8_t* base = smem + place;
                uint64_t* bar = &full[ring.entry()];
                ++ring.count;
                if (half >= nb) {
                  mbar_arrive(bar);
                  continue;
                }
                mbar_arrive_expect_tx(bar, bytes + (MX && half == 0 ? nb * 512u : 0u));
                const int k = (sh.kb0 + kb + half) * (MX ? 128 : 64);
                if constexpr (MX)
                  if (half == 0)                     // scale factors of both blocks, behind them
                    bulk_load(base + nb * block, L->sf[lc_weight(op)] + (static_cast<size_t>(row0 >> 7) * k_blocks + sh.kb0 + kb) * 512, nb * 512u, bar);
                uint8_t* dst = base + half * block + first * 1024;
                if (units == 16) {
                  tma_load_2d_hint(dst, maps_w + 4, bar, k, row0, pol);
                  continue;
                }
                int row = row0;
#pragma unroll 1
                for (int i = 3; i >= 0; --i) {
                  if (!(units >> i & 1)) continue;
                  tma_load_2d_hint(dst, maps_w + i, bar, k, row, pol);
                  if (halves) tma_load_2d_hint(dst + 64 * 128, maps_w + i, bar, k, row + 64, pol);
                  dst += 1024 << i;
                  row += 8 << i;
                }
              }
            }
          } else if (!LN && op == OP_ATT) {
            bool appended = false;                   // the rows of the new tokens are in the cache
            auto pages = [&](const LcItem& it, int n) {          // of a tile
              const int page = 2 * (it.t0 + n), *bt = p.block_table + static_cast<size_t>(it.seq) * p.max_pages;
              if (n >= it.nt) return make_int2(0, 0);
              return make_int2(bt[page], bt[(page + 1) * LC_PAGE < it.kvlen ? page + 1 : page]);   // (past the end: any keys, they are masked)
            };
#pragma unroll 1
            for (int j = item0; ok && j < items; j += item_step) {
              const LcItem it = lc_item(p, kvlen_s, window, j, part);
              int2 pg = pages(it, 0), pg1 = pages(it, 1);        // fetched ahead of their use
              // K0, K1, V0, K2, V1, ..
#pragma unroll 1
              for (int i = 0; ok && i < 2 * it.nt; ++i) {
                const bool values = i == 2 * it.nt - 1 || (i > 0 && (i & 1) == 0);
                const int n = i == 0 ? 0 : (values ? (i - 1) >> 1 : (i + 1) >> 1);
                const int2 where = values || i == 0 ? pg : pg1;
                // tiles with rows of this step: the new token's, and, where tokens of one text come as sequences that share its pages, of the ones in front of
                // it (looked for once; taking the last T keys of every sequence for written delayed pages by 0.6 us per layer at 32 sequences)
                const int end = (2 * (it.t0 + n) + 2) * LC_PAGE;
                if (end > it.kvlen - p.T && !appended) {
                  int first = it.kvlen - 1;
                  if (end <= first && (first = fresh_s[half][it.seq]) < 0) {
                    first = it.kvlen - 1;
                    const int* bt = p.block_table + static_cast<size_t>(it.seq) * p.max_pages + first / LC_PAGE;
                    const int page0 = first / LC_PAGE * LC_PAGE, page = bt[0], before = bt[-1];            // (a tile lies in front of this one)
#pragma unroll 8
                    for (int t = 0; t < p.T; ++t) {
                      const int slot = p.slots[t];
                      if (slot >= 0 && slot / LC_PAGE == page) first = min(first, page0 + slot % LC_PAGE);
                      if (slot >= 0 && slot / LC_PAGE == before) first = min(first, page0 - LC_PAGE + slot % LC_PAGE);
                    }
                    fresh_s[half][it.seq] = first;
                  }
                  if (end > first) {
                    if (!(ok = lc_wait_due(due_s, at - 1, abort))) break;
                    fence_proxy_async_global();
                    appended = true;
                  }
                }
#pragma unroll 1
                for (int h = 0; h < MB; ++h) {       // 128 channels per slot
                  if (!(ok = ring.room(2 * LC_BLOCK, place, sizes, empty, abort))) break;
                  uint8_t* base = smem + place;
                  uint64_t* bar = &full[ring.entry()];
                  ++ring.count;
                  mbar_arrive_expect_tx(bar, LC_BLOCK);
                  uint8_t* dst = base + half * LC_BLOCK;
                  const CUtensorMap* m = values ? &L->v : &L->k;
                  tma_load_2d(dst, m, bar, it.kvh * D + h * 128 + half * 64, where.x * LC_PAGE);
                  tma_load_2d(dst + LC_PAGE * 128, m, bar, it.kvh * D + h * 128 + half * 64, where.y * LC_PAGE);
                }
                if (values) {
                  pg = pg1;
                  pg1 = pages(it, n + 2);
                }
              }
            }
          }
        }
      }
      issued_s[half] = ring.count;
    }
  } else if (warp == 6) {
    // --------------------------------------------------------------------------- activations, as soon as they are complete
    if (elect_one()) {
      const uint64_t pol = l2_policy_evict_last();
      uint32_t nq = 0, nx = 0, s = 0, ph = 0;
      bool ok = true;
      int at = 0;
#pragma unroll 1
      for (int l = 0; ok && l < p.n_layers; ++l) {
        const int window = p.layers[l].window;
#pragma unroll 1
        for (int op = 0; ok && op < OP_COUNT; ++op) {
          if (skip(l, op)) continue;
          if (at > 0) {                              // the operations so far are complete: this thread alone polls, the others of the CTA look at due_s
            if (!(ok = lc_wait_op(ctr + at - 1, ctas, p.polls, abort, p.ctl))) break;
            asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(due_s)), "r"(at) : "memory");
            fence_proxy_async_global();
          }
          ++at;
          if (lc_weight(op) >= 0) {
            const LcShare sh = share_s[lc_weight(op)];
            const CUtensorMap* m = op == OP_QKV ? (l == 0 ? &maps.x_in : &maps.xa) : (op == OP_O ? &maps.attn : (op == OP_GU ? &maps.xb : &maps.h));
#pragma unroll 1
            for (int u = sh.u0; ok && u < sh.end; u += lc_tile<GLU, MX>(op, u, sh.end))
#pragma unroll 1
              for (int kb = 0; kb < sh.nkb; kb += XB) {      // (whole copies, also where fewer blocks are left: they are not used)
                if (!(ok = ma_wait(&x_empty[s], ph ^ 1u, abort))) break;
                const uint32_t sf_bytes = MX ? min(XB, sh.nkb - kb) * 512u : 0u;
                mbar_arrive_expect_tx(&x_full[s], x_bytes * XB + sf_bytes);
                tma_load_3d_hint(x_s + s * x_slot, m, &x_full[s], 0, 0, sh.kb0 + kb, pol);
                if constexpr (MX)
                  bulk_load(x_s + s * x_slot + x_bytes * XB, (op == OP_QKV ? (l == 0 ? p.sf_in : p.sf_x) : op == OP_O ? p.sf_attn : op == OP_GU ? p.sf_x : p.sf_h) +
                            static_cast<size_t>(sh.kb0 + kb) * 512, sf_bytes, &x_full[s]);
                ++nx;
                if (++s == x_slots) { s = 0; ph ^= 1u; }
              }
          } else if (!LN && op == OP_ATT) {
            // Queries land where the partial sums and the exchange of gate and up lay (plain loads and stores, complete with the operations in front), which is
            // the only target of that kind: the other operations do without this fence (0.2 us each; here it hides, two layers of one token 165.3 us without
            // and with it).
            fence_proxy_async_smem();
#pragma unroll 1
            for (int j = item0; ok && j < items; j += item_step) {
              const LcItem it = lc_item(p, kvlen_s, window, j, part);
              if (it.nt <= 0) continue;
              const uint32_t b = nq % NQ;
              if (!(ok = ma_wait(&q_empty[b], ((nq / NQ) & 1u) ^ 1u, abort))) break;
              ++nq;
              mbar_arrive_expect_tx(&q_full[b], LC_HEADS * D * 2);
#pragma unroll
              for (int c = 0; c < DB; ++c)
                tma_load_2d(zone + b * (LC_HEADS * D * 2) + c * (LC_HEADS * 128), &maps.q, &q_full[b], c * 64, q_start_s[it.seq] * p.n_q + it.kvh * G);
            }
          }
        }
      }
      issued_s[2] = nx;
      issued_s[3] = nq;
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = MX ? make_idesc_mxf8(128, BN) : make_idesc_bf16(128, BN);
      constexpr uint32_t idesc_s = make_idesc_bf16(LC_KEYS, LC_HEADS);
      constexpr uint32_t idesc_o = make_idesc_bf16(128, LC_HEADS) | (1u << 15);              // A (V) has its rows contiguous
      const uint64_t desc0 = make_sw128_kmajor_desc(smem_u32(smem));         // + offset / 16 (a single thread issues: every instruction counts)
      const uint64_t desc_x = make_sw128_kmajor_desc(smem_u32(x_s));
      const uint32_t x_chunk = x_slot >> 4;
      uint32_t nblk = 0;                             // blocks of K so far (their scale factors alternate between two sets of columns)
      uint32_t xs = 0, xph = 0;
      LcRing<Cfg::kRing> ring;
      uint32_t na = 0, ns = 0, np = 0, nq = 0, no = 0;       // accumulators, score tiles, value tiles, items so far
      bool ok = true;
#pragma unroll 1
      for (int l = 0; ok && l < p.n_layers; ++l) {
        const int window = p.layers[l].window;
#pragma unroll 1
        for (int op = 0; ok && op < OP_COUNT; ++op) {
          if (lc_weight(op) >= 0) {
            const LcShare sh = share_s[lc_weight(op)];
#pragma unroll 1
            for (int u = sh.u0, n; ok && u < sh.end; u += n, ++na) {
              n = lc_tile<GLU, MX>(op, u, sh.end);
              const uint32_t block = lc_block_bytes<GLU>(op, lc_first<GLU, MX>(op, u) + n);
              if (!(ok = ma_wait(&acc_empty[na & 1u], ((na >> 1) & 1u) ^ 1u, abort))) break;
              tc_fence_after();
              const uint32_t acc = tmem + (na & 1u) * BN;
              uint32_t more = 0u;
#pragma unroll 1
              for (int kb = 0; kb < sh.nkb; kb += XB) {
                if (!(ok = ma_wait(&x_full[xs], xph, abort))) break;
                uint64_t x = desc_x + xs * x_chunk;
#pragma unroll 1
                for (int k2 = kb; k2 < min(kb + XB, sh.nkb); k2 += 2) {
                  const uint32_t nb = min(2, sh.nkb - k2);
                  // (rows that the tile does not have are read from what lies behind it, and not used)
                  const uint32_t at_w = ring.place(block * nb + (MX ? 1024u : 0u));
                  uint64_t a = desc0 + (at_w >> 4);
                  if (!(ok = ma_wait(&full[ring.entry()], ring.parity(), abort))) break;
                  tc_fence_after();
                  if constexpr (MX) {
                    // (scale factors: two sets of 16 columns behind the attention's)
                    const uint32_t sfa = smem_u32(smem) + at_w + nb * block, sfb = smem_u32(x_s) + xs * x_slot + x_bytes * XB + (k2 - kb) * 512;
#pragma unroll 1
                    for (uint32_t b = 0; b < nb; ++b, ++nblk) {
                      const uint32_t ta = tmem + Cfg::kO + 2 * LC_HEADS + (nblk & 1u) * 16, tb = ta + 4;
                      tmem_cp_32x128b_warpx4(ta, make_sf_desc(sfa + b * 512));
                      tmem_cp_32x128b_warpx4(tb, make_sf_desc(sfb + b * 512));
#pragma unroll
                      for (int k = 0; k < 4; ++k)
                        umma_mxf8(acc, a + 2 * k, x + 2 * k, idesc | (static_cast<uint32_t>(k) << 4) | (static_cast<uint32_t>(k) << 29),
                                  (more != 0u || b > 0 || k > 0) ? 1u : 0u, ta, tb);
                      a += block >> 4;
                      x += x_bytes >> 4;
                    }
                  } else {
                    umma_bf16(acc, a, x, idesc, more);
                    umma_bf16(acc, a + 2, x + 2, idesc, 1u);
                    umma_bf16(acc, a + 4, x + 4, idesc, 1u);
                    umma_bf16(acc, a + 6, x + 6, idesc, 1u);
                    if (nb == 2) {
                      a += block >> 4;
                      x += x_bytes >> 4;
                      umma_bf16(acc, a, x, idesc, 1u);
                      umma_bf16(acc, a + 2, x + 2, idesc, 1u);
                      umma_bf16(acc, a + 4, x + 4, idesc, 1u);
                      umma_bf16(acc, a + 6, x + 6, idesc, 1u);
                      x += x_bytes >> 4;
                    }
                  }
                  umma_commit(&empty[ring.entry()]);
                  ++ring.count;
                  more = 1u;
                }
                umma_commit(&x_empty[xs]);
                if (++xs == x_slots) { xs = 0; xph ^= 1u; }
              }
              umma_commit(&acc_full[na & 1u]);
            }
          } else if (!LN && op == OP_ATT) {
#pragma unroll 1
            for (int j = item0; ok && j < items; j += item_step) {
              const LcItem it = lc_item(p, kvlen_s, window, j, part);
              if (it.nt <= 0) continue;
              const uint32_t qb = nq % NQ;
              if (!(ok = ma_wait(&q_full[qb], (nq / NQ) & 1u, abort))) break;
              ++nq;
              // S(0), S(1), PV(0), S(2), PV(1), ..: scores run while the softmax warps work on the tile before
#pragma unroll 1
              for (int i = 0; ok && i < 2 * it.nt; ++i) {
                const bool values = i == 2 * it.nt - 1 || (i > 0 && (i & 1) == 0);
                if (!values) {
#pragma unroll 1
                  for (int h = 0; h < MB; ++h) {
                    const uint32_t base = smem_u32(smem) + ring.place(2 * LC_BLOCK);
                    if (!(ok = ma_wait(&full[ring.entry()], ring.parity(), abort))) break;
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                      const uint64_t a = make_sw128_kmajor_desc(base + (kk / 4) * LC_BLOCK) + static_cast<uint64_t>((kk % 4) * 2);
                      const uint64_t b = make_sw128_kmajor_desc(smem_u32(zone + qb * (LC_HEADS * D * 2) + (h * 2 + kk / 4) * (LC_HEADS * 128))) + static_cast<uint64_t>((kk % 4) * 2);
                      umma_bf16(tmem + Cfg::kS + (ns & 1u) * LC_HEADS, a, b, idesc_s, (h > 0 || kk > 0) ? 1u : 0u);
                    }
                    umma_commit(&empty[ring.entry()]);
                    ++ring.count;
                  }
                  umma_commit(&s_full[ns & 1u]);
                  ++ns;
                  if (i == max(0, 2 * it.nt - 3)) umma_commit(&q_empty[qb]);                 // the last scores: the queries have been read
                } else {
                  const bool first = i == (it.nt > 1 ? 2 : 1);
                  if (first && !(ok = ma_wait(o_empty, (no & 1u) ^ 1u, abort))) break;
                  if (!(ok = ma_wait(&p_ready[np & 1u], (np >> 1) & 1u, abort))) break;
#pragma unroll 1
                  for (int m = 0; m < MB; ++m) {
                    const uint32_t base = smem_u32(smem) + ring.place(2 * LC_BLOCK);
                    if (!(ok = ma_wait(&full[ring.entry()], ring.parity(), abort))) break;
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < LC_KEYS / 16; ++kk) {
                      const uint64_t a = ma_value_desc(base + kk * (16 * 128));
                      const uint64_t b = make_sw128_kmajor_desc(smem_u32(zone + 8192 + (np & 1u) * 4096 + (kk / 4) * (LC_HEADS * 128))) + static_cast<uint64_t>((kk % 4) * 2);
                      umma_bf16(tmem + Cfg::kO + m * LC_HEADS, a, b, idesc_o, (!first || kk > 0) ? 1u : 0u);
                    }
                    umma_commit(&empty[ring.entry()]);
                    ++ring.count;
                  }
                  umma_commit(&pv_done[np & 1u]);
                  ++np;
                }
              }
              ++no;
            }
          }
        }
      }
      umma_commit(mma_done);
    }
  } else {
    // ------------------------------------------------------------------------------------------------ epilogues and softmax
    // (a wait that gave up ends the others through the abort word; the loops go on, because every warp has to meet the others, but nothing is sent to
    // the cluster any more: its barriers count the bytes and arrivals of every exchange)
    const int et = threadIdx.x - 64, q4 = warp & 3, row = q4 * 32 + lane;
    const int col0 = rank * CW;                        // the tokens that this CTA finishes
    const uint32_t lanes = tmem + (static_cast<uint32_t>(q4 * 32) << 16);
    const int q_dim = p.n_q * hd, kv_dim = p.n_kv * hd;
    const float inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f, log_theta = p.rope_theta > 0.f ? log2f(p.rope_theta) : 0.f;
    uint32_t na = 0, nx = 0, nt_all = 0, nparts = 0;   // accumulators, exchanges, key tiles, merges so far
    int at = 0;                                        // operations so far, over the layers
    bool ok = true;
#pragma unroll 1
    for (int l = 0; l < p.n_layers; ++l) {
      const LcLayer* L = p.layers + l;
      const __nv_bfloat16* x = l == 0 ? p.x_in : p.xa;
      const int window = L->window;                    // (read here, ahead of their use)
      __nv_bfloat16 *const k_cache = L->k_cache, *const v_cache = L->v_cache;
#pragma unroll 1
      for (int op = 0; op < OP_COUNT; ++op) {
        if (skip(l, op)) continue;
        if (lc_weight(op) >= 0) {
          // ----------------------------------------------------------------------------------------------------- products
          const LcShare sh = share_s[lc_weight(op)];
          const bool work = sh.u0 < sh.end;
          // O and down: + residual, unless a norm follows; then the sums of squares of the rows are left for the norm in the next product
          const __nv_bfloat16* residual = norms ? nullptr : (op == OP_O ? x : p.xb);
          __nv_bfloat16* out = norms ? p.norm : (op == OP_O ? p.xb : p.xa);
          int ld = p.hidden;
          const float* bias = nullptr;
          if constexpr (LN) {
            bias = L->bias[lc_weight(op)];
            if (op == OP_GU) {
              residual = nullptr;
              out = p.h;
              ld = p.ffn;
            }
          }
          float sq[CW];
#pragma unroll
          for (int i = 0; i < CW; ++i) sq[i] = 0.f;
          if (ok) ok = __all_sync(0xffffffffu, lc_wait_due(due_s, at, abort));
          if (work && op == OP_QKV && et < CW) {
            const int t = col0 + et;
            pos_s[et] = (p.positions != nullptr && t < p.T) ? p.positions[t] : 0;
            slot_s[et] = t < p.T ? p.slots[t] : -1;
          }
          if (LN) {                                    // (the activations are normed)
          } else if (work && op == OP_QKV && l == 0) { // 1/rms of the rows: a warp per row
            const int k8 = p.hidden / 8;
#pragma unroll 1
            for (int t = warp - 2; t < CW; t += 4) {
              float ss = 0.f;
              const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(min(col0 + t, p.T - 1)) * p.hidden);
#pragma unroll 8
              for (int i = lane; i < k8; i += 32) {
                const uint4 v = src[i];
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 f = __bfloat1622float2(h[e]);
                  ss += f.x * f.x + f.y * f.y;
                }
              }
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
              if (lane == 0) rstd_s[t] = rsqrtf(ss / static_cast<float>(p.hidden) + p.eps);
            }
          } else if (work && (op == OP_QKV || op == OP_GU)) {      // the same from the sums of squares left by those who wrote the rows
            constexpr int TPT = 128 / CW;              // threads per token
            const float* from = p.ss + (op == OP_GU ? LC_SS : 0) + col0 + et / TPT;
            const int n = norms ? 1 : static_cast<int>(ctas) / LC_CL;
            float a = 0.f;
#pragma unroll 4
            for (int i = et % TPT; i < n; i += TPT) a += __ldcg(from + i * 64);
#pragma unroll
            for (int o = TPT / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (et % TPT == 0) rstd_s[et / TPT] = rsqrtf(a / static_cast<float>(p.hidden) + p.eps);
          }
          lc_sync();
#pragma unroll 1
          for (int u = sh.u0, n; u < sh.end; u += n) {
            n = lc_tile<GLU, MX>(op, u, sh.end);
            const int own = row - lc_first<GLU, MX>(op, u) * 8, feat = u * 8 + own;
            const bool live = GLU && op == OP_GU ? (row & 63) < n * 8 : (own >= 0 && own < n * 8);
            const float bias_v = LN && live ? bias[feat] : 0.f;
            const int sect = feat < q_dim ? 0 : (feat < q_dim + kv_dim ? 1 : 2);                  // (of QKV)
            const int fs = feat - (sect == 0 ? 0 : (sect == 1 ? q_dim : q_dim + kv_dim));
            const bool turn = !LN && sect < 2 && p.rope_theta > 0.f;
            float c1[CW], c2[CW];                      // cosines and sines | residual
            if (op == OP_QKV) {
              const float freq = turn ? exp2f(-(2.f * ((fs % D) >> 1) / static_cast<float>(D)) * log_theta) : 0.f;
#pragma unroll
              for (int i = 0; i < CW; ++i) {
                c1[i] = 1.f;
                c2[i] = 0.f;
                if (turn && col0 + i < p.T) sincosf(static_cast<float>(pos_s[i]) * freq, &c2[i], &c1[i]);
              }
            } else if (LN || op != OP_GU) {
#pragma unroll
              for (int i = 0; i < CW; ++i)
                c1[i] = (residual != nullptr && live && col0 + i < p.T) ? __bfloat162float(residual[static_cast<size_t>(col0 + i) * p.hidden + feat]) : 0.f;
            }
            if (ok) ok = __all_sync(0xffffffffu, ma_wait(&acc_full[na & 1u], (na >> 1) & 1u, abort));
            tc_fence_after();
            // partial sums of this CTA's quarter of K to the CTAs that finish the tokens; v = sums of this CTA's tokens, in the order of K
            float v[CW];
            {
              float a[BN];
              lc_ld<BN>(lanes + (na & 1u) * BN, a);
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[na & 1u]);
              ++na;
              if (nx > 0 && ok) ok = __all_sync(0xffffffffu, lc_wait_cluster(zone_free, (nx - 1) & 1u, abort, p.ctl));
              if (threadIdx.x == 64 && ok) mbar_arrive_expect_tx(zone_full, static_cast<uint32_t>(lc_rows<GLU>(op, n) * LC_CL * CW * 4));
              if (live && ok) {
#pragma unroll
                for (int d = 0; d < LC_CL; ++d) {
                  const uint32_t to = mapa_smem(smem_u32(zone), d) + static_cast<uint32_t>((rank * (CW / 4) * 128 + row) * 16);
                  const uint32_t bar = mapa_smem(smem_u32(zone_full), d);
#pragma unroll
                  for (int i = 0; i < CW / 4; ++i)
                    st_async_v4(to + i * 2048, bar, a[d * CW + 4 * i], a[d * CW + 4 * i + 1], a[d * CW + 4 * i + 2], a[d * CW + 4 * i + 3]);
                }
              }
              if (ok) ok = __all_sync(0xffffffffu, lc_wait_cluster(zone_full, nx & 1u, abort, p.ctl));
              ++nx;
#pragma unroll
              for (int i = 0; i < CW; ++i) v[i] = 0.f;
#pragma unroll
              for (int r = 0; r < LC_CL; ++r)
#pragma unroll
                for (int i = 0; i < CW / 4; ++i) {
                  const float4 f = *reinterpret_cast<const float4*>(zone + ((r * (CW / 4) + i) * 128 + row) * 16);
                  v[4 * i] += f.x; v[4 * i + 1] += f.y; v[4 * i + 2] += f.z; v[4 * i + 3] += f.w;
                }
            }
            constexpr int HB = CW / 2;
            const bool up = row >= 64;                 // gate/up: the up half finishes the second half of the tokens, the gate half the first
            if (GLU && op == OP_GU) {
              float* xch = reinterpret_cast<float*>(zone);         // [HB tokens][64] up values of the first half, then gate values of the second
              lc_sync();                               // the sums have been read
              float* to = xch + (up ? 0 : HB * 64) + (row & 63);
#pragma unroll
              for (int i = 0; i < HB; ++i) to[i * 64] = up ? v[i] : v[HB + i];
              lc_sync();
              const float* from = xch + (up ? HB * 64 : 0) + (row & 63);
#pragma unroll
              for (int i = 0; i < HB; ++i) c1[i] = from[i * 64];
            }
            __syncwarp();
            if (lane < LC_CL && ok) arrive_cluster_read(mapa_smem(smem_u32(zone_free), lane));    // the sums have been read (and the halves, stored and read back)
            if (GLU && op == OP_GU) {
              const int t0 = up ? HB : 0;
              float h[HB];
#pragma unroll
              for (int i = 0; i < HB; ++i) {
                const float rs = rstd_s[t0 + i], theirs = c1[i] * rs, mine = (up ? v[HB + i] : v[i]) * rs;
                const float g = up ? theirs : mine, w = up ? mine : theirs;
                h[i] = (p.act ? gelu_tanh(g) : silu(g)) * w;
              }
              if constexpr (MX) {                      // (whole blocks of 64 features: every lane has one)
                lc_put_mx<HB>(h, ok ? p.T - col0 - t0 : 0, col0 + t0, u * 8 + (row & 63), p.ffn, p.q8_h, p.sf_h, lane);
              } else if (live && ok) {
#pragma unroll
                for (int i = 0; i < HB; ++i)
                  if (col0 + t0 + i < p.T) p.h[static_cast<size_t>(col0 + t0 + i) * p.ffn + u * 8 + (row & 63)] = __float2bfloat16_rn(h[i]);
              }
            } else if (op == OP_QKV) {
#pragma unroll
              for (int i = 0; i < CW; ++i) {
                const int tok = col0 + i;
                if (tok >= p.T) break;                 // (the same for the warp)
                const float a = LN ? v[i] + bias_v : v[i] * rstd_s[i];
                // lanes (2j, 2j + 1) hold (x_j, x_{j + D / 2}) thanks to the row order of the weights
                const float b = __shfl_xor_sync(0xffffffffu, a, 1);
                const float o = turn ? ((lane & 1) ? (a * c1[i] + b * c2[i]) : (a * c1[i] - b * c2[i])) : a;
                if (!live || !ok) continue;
                if (sect == 0) {
                  p.q[static_cast<size_t>(tok) * q_dim + fs] = __float2bfloat16_rn(o * p.q_scale);
                } else if (slot_s[i] >= 0) {
                  (sect == 1 ? k_cache : v_cache)[static_cast<size_t>(slot_s[i]) * kv_dim + fs] = __float2bfloat16_rn(o);
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < CW; ++i) {
                v[i] += c1[i];
                if constexpr (LN) {
                  v[i] += bias_v;
                  if (op == OP_GU) v[i] = gelu_tanh(v[i]);
                }
              }
              if (live && ok)
#pragma unroll
                for (int i = 0; i < CW; ++i)
                  if (col0 + i < p.T) {
                    const __nv_bfloat16 r = __float2bfloat16_rn(v[i]);
                    out[static_cast<size_t>(col0 + i) * ld + feat] = r;
                    sq[i] += __bfloat162float(r) * __bfloat162float(r);
                  }
              if constexpr (MX) lc_put_mx<CW>(v, live && ok ? p.T - col0 : 0, col0, feat, p.hidden, p.q8_x, p.sf_x, lane);
            }
          }
          if (!LN && !norms && (op == OP_O || op == OP_DOWN)) {
#pragma unroll
            for (int i = 0; i < CW; ++i) {
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
              if (lane == 0) sq_s[q4][i] = sq[i];
            }
            lc_sync();
            if (et < CW) p.ss[(op == OP_O ? LC_SS : 0) + blockIdx.x / LC_CL * 64 + col0 + et] = sq_s[0][et] + sq_s[1][et] + sq_s[2][et] + sq_s[3][et];
          }
        } else if (LN && op == OP_ATT) {
          // ---- attention of 64-wide heads, prompts and decode: a lane per key for the scores, two channels per lane for the values.  A (token, head)
          // per warp while no token sees more than 128 keys, else per CTA, whose warps take every fourth run of 32 keys.  Bound by the latency
          // of three dependent loads (page, key, value rows), so a run's rows are all fetched before the first is used.
          float* q_s = reinterpret_cast<float*>(zone) + (warp - 2) * 64;           // per warp: the query
          float *o_s = reinterpret_cast<float*>(zone) + 256, *m_s = o_s + 256, *l_s = m_s + 4;         // the warps' sums, maxima, sums of the weights
          if (ok) ok = __all_sync(0xffffffffu, lc_wait_due(due_s, at, abort));
          int most = 0;
          for (int t = lane; t < p.T; t += 32) most = max(most, kvlen_s[t]);
          for (int i = 16; i > 0; i >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, i));
          const int w = warp - 2, parts = most > 128 ? 4 : 1, part = parts == 4 ? w : 0;
#pragma unroll 1
          for (int j = parts == 4 ? blockIdx.x : blockIdx.x * 4 + w; j < p.T * p.n_q; j += parts == 4 ? gridDim.x : gridDim.x * 4) {
            const int t = j / p.n_q, head = j - t * p.n_q, seq = q_start_s[t], keys = kvlen_s[t];
            if (seq < 0) continue;                     // (parts == 4: the same for the CTA)
            const int kvh = head / (p.n_q / p.n_kv);
            const int* bt = p.block_table + static_cast<size_t>(seq) * p.max_pages;
            const __nv_bfloat162 q2 = __ldcg(reinterpret_cast<const __nv_bfloat162*>(p.q + static_cast<size_t>(t) * q_dim + head * 64) + lane);
            float m = -INFINITY, lsum = 0.f, o0 = 0.f, o1 = 0.f;
            bool first = true;
#pragma unroll 1
            for (int k0 = part * 32; k0 < keys; k0 += parts * 32) {
              const size_t row0 = (static_cast<size_t>(bt[k0 / LC_PAGE]) * LC_PAGE + k0 % LC_PAGE) * kv_dim + kvh * 64;      // (32 keys lie in one page)
              const bool seen = k0 + lane < keys && (window <= 0 || k0 + lane >= keys - window);
              const int n = min(32, keys - k0);
              uint4 kv[8];
              __nv_bfloat162 vv[32];
              const uint4* src = reinterpret_cast<const uint4*>(k_cache + row0 + static_cast<size_t>(lane) * kv_dim);
              const __nv_bfloat162* vsrc = reinterpret_cast<const __nv_bfloat162*>(v_cache + row0) + lane;
#pragma unroll
              for (int i = 0; i < 8; ++i) kv[i] = seen ? __ldcg(src + i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
              for (int i = 0; i < 32; ++i) vv[i] = i < n ? __ldcg(vsrc + static_cast<size_t>(i) * (kv_dim / 2)) : __floats2bfloat162_rn(0.f, 0.f);
              if (first) {                             // (behind the rows' loads)
                const float2 f = __bfloat1622float2(q2);
                q_s[2 * lane] = f.x;
                q_s[2 * lane + 1] = f.y;
                __syncwarp();
                first = false;
              }
              float s = 0.f;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&kv[i]);
                const float4 qa = *reinterpret_cast<const float4*>(q_s + 8 * i), qb = *reinterpret_cast<const float4*>(q_s + 8 * i + 4);
                const float2 f0 = __bfloat1622float2(h[0]), f1 = __bfloat1622float2(h[1]), f2 = __bfloat1622float2(h[2]), f3 = __bfloat1622float2(h[3]);
                s += f0.x * qa.x + f0.y * qa.y + f1.x * qa.z + f1.y * qa.w + f2.x * qb.x + f2.y * qb.y + f3.x * qb.z + f3.y * qb.w;
              }
              s = seen ? s * LC_LOG2E : -INFINITY;
              if (!__any_sync(0xffffffffu, !(s == -INFINITY))) continue;           // (no key of this run is seen; a NaN score goes on)
              float top = s;
#pragma unroll
              for (int i = 16; i > 0; i >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, i));
              top = fmaxf(top, m);
              const float e = ex2(s - top), a = m == -INFINITY ? 0.f : ex2(m - top);
              m = top;
              lsum = lsum * a + e;
              o0 *= a;
              o1 *= a;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float2 f = __bfloat1622float2(vv[i]);
                const float pw = __shfl_sync(0xffffffffu, e, i);
                if (i < n) {
                  o0 += pw * f.x;
                  o1 += pw * f.y;
                }
              }
            }
#pragma unroll
            for (int i = 16; i > 0; i >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, i);
            __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(p.attn + static_cast<size_t>(t) * q_dim + head * 64) + lane;
            if (parts == 1) {
              if (ok) *out = lsum == 0.f ? __floats2bfloat162_rn(0.f, 0.f) : __floats2bfloat162_rn(o0 / lsum, o1 / lsum);
              __syncwarp();                            // the query has been read
              continue;
            }
            o_s[w * 64 + 2 * lane] = o0;
            o_s[w * 64 + 2 * lane + 1] = o1;
            if (lane == 0) {
              m_s[w] = m;
              l_s[w] = lsum;
            }
            lc_sync();
            if (w == 0 && ok) {
              const float top = fmaxf(fmaxf(m_s[0], m_s[1]), fmaxf(m_s[2], m_s[3]));
              float n0 = 0.f, n1 = 0.f, den = 0.f;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float a = m_s[i] == -INFINITY ? 0.f : ex2(m_s[i] - top);
                n0 += a * o_s[i * 64 + 2 * lane];
                n1 += a * o_s[i * 64 + 2 * lane + 1];
                den += a * l_s[i];
              }
              *out = den == 0.f ? __floats2bfloat162_rn(0.f, 0.f) : __floats2bfloat162_rn(n0 / den, n1 / den);
            }
            lc_sync();                                 // the sums have been read
          }
        } else if (!LN && op == OP_ATT) {
          // ---------------------------------------------------------------------------------------------------- attention
#pragma unroll 1
          for (int j = item0; j < items; j += item_step) {
            const LcItem it = lc_item(p, kvlen_s, window, j, part);
            if (!it.active) continue;                  // (the same for the CTAs that share its keys)
            float m_ref[GP], lsum[GP];
#pragma unroll
            for (int g = 0; g < GP; ++g) {
              m_ref[g] = -INFINITY;
              lsum[g] = 0.f;
            }
#pragma unroll 1
            for (int n = 0; n < it.nt; ++n, ++nt_all) {
              const uint32_t b = nt_all & 1u;
              const int key = (it.t0 + n) * LC_KEYS + row;
              if (ok) ok = __all_sync(0xffffffffu, ma_wait(&s_full[b], (nt_all >> 1) & 1u, abort));
              tc_fence_after();
              float xs[GP] = {};
              lc_ld_heads<GP>(lanes + Cfg::kS + b * LC_HEADS, xs);
              const bool seen = key < it.kvlen && key >= it.kv_lo;
              bool up = false;
#pragma unroll
              for (int g = 0; g < GP; ++g) {
                if (p.softcap > 0.f) xs[g] = p.softcap * tanh_exp(xs[g] * inv_cap);
                xs[g] = seen ? xs[g] * LC_LOG2E : -INFINITY;
                up |= g < G && (xs[g] > m_ref[g] + 8.f || (m_ref[g] == -INFINITY && xs[g] > -INFINITY));
              }
              // P(n - 2) has been read; waited for in every tile so that no parity wait lags two phases behind
              if (ok && nt_all > 1) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[b], ((nt_all - 2) >> 1) & 1u, abort));
              if (lc_vote(up)) {                       // new references: the maxima of this tile
                float alpha[GP];
#pragma unroll
                for (int g = 0; g < GP; ++g) {
                  float m = xs[g];
#pragma unroll
                  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                  if (lane == 0) red_s[q4][g] = m;
                }
                lc_sync();
#pragma unroll
                for (int g = 0; g < GP; ++g) {
                  const float m = fmaxf(m_ref[g], fmaxf(fmaxf(red_s[0][g], red_s[1][g]), fmaxf(red_s[2][g], red_s[3][g])));
                  alpha[g] = (m_ref[g] == -INFINITY || g >= G) ? 0.f : ex2(m_ref[g] - m);
                  m_ref[g] = m;
                  lsum[g] *= alpha[g];
                }
                lc_sync();                             // red_s may be written again
                if (n > 0) {
                  if (ok) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[b ^ 1u], ((nt_all - 1) >> 1) & 1u, abort));
                  tc_fence_after();
#pragma unroll
                  for (int m = 0; m < MB; ++m) {
                    float y[GP];
                    lc_ld_heads<GP>(lanes + Cfg::kO + m * LC_HEADS, y);
#pragma unroll
                    for (int g = 0; g < GP; ++g) y[g] *= alpha[g];
                    lc_st_heads<GP>(lanes + Cfg::kO + m * LC_HEADS, y);
                  }
                }
              }
              uint8_t* pt = zone + 8192 + b * 4096 + (row >> 6) * (LC_HEADS * 128) + (row & 7) * 2;
#pragma unroll
              for (int g = 0; g < GP; ++g) {
                if (g < G) {
                  const float e = ex2(xs[g] - (m_ref[g] == -INFINITY ? 0.f : m_ref[g]));
                  const __nv_bfloat16 w = __float2bfloat16_rn(e);
                  lsum[g] += __bfloat162float(w);      // the sum of what the product sees: the rounding of a dominant weight cancels
                  *reinterpret_cast<__nv_bfloat16*>(pt + g * 128 + ((((row & 63) >> 3) ^ (g & 7)) << 4)) = w;
                }
              }
              fence_proxy_async_smem();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&p_ready[b]);
            }
#pragma unroll
            for (int g = 0; g < GP; ++g)
#pragma unroll
              for (int sh = 16; sh > 0; sh >>= 1) lsum[g] += __shfl_xor_sync(0xffffffffu, lsum[g], sh);
            if (lane == 0)
#pragma unroll
              for (int g = 0; g < GP; ++g) sq_s[q4][g] = lsum[g];
            float o[MB][GP];
            if (it.nt > 0) {
              if (ok && it.nt > 1) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[nt_all & 1u], ((nt_all - 2) >> 1) & 1u, abort));
              if (ok) ok = __all_sync(0xffffffffu, ma_wait(&pv_done[(nt_all - 1) & 1u], ((nt_all - 1) >> 1) & 1u, abort));
              tc_fence_after();
#pragma unroll
              for (int m = 0; m < MB; ++m) lc_ld_heads<GP>(lanes + Cfg::kO + m * LC_HEADS, o[m]);
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(o_empty);
            } else {
#pragma unroll
              for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int g = 0; g < GP; ++g) o[m][g] = 0.f;
            }
            __nv_bfloat16* out = p.attn + static_cast<size_t>(q_start_s[it.seq]) * q_dim + it.kvh * G * D;
            if (p.parts == 1) {
              lc_sync();
              float den[GP];
#pragma unroll
              for (int g = 0; g < GP; ++g) den[g] = g < G ? sq_s[0][g] + sq_s[1][g] + sq_s[2][g] + sq_s[3][g] : 0.f;
#pragma unroll
              for (int m = 0; m < MB; ++m) {
#pragma unroll
                for (int g = 0; g < GP; ++g) o[m][g] = den[g] == 0.f ? 0.f : o[m][g] / den[g];
                if constexpr (MX) {                    // (G heads side by side: "rows" of D features)
                  float r[GP], most[GP];
#pragma unroll
                  for (int g = 0; g < GP; ++g) {
                    r[g] = bf16_round(o[m][g]);
                    most[g] = fabsf(r[g]);
                  }
#pragma unroll
                  for (int sh = 16; sh > 0; sh >>= 1)
#pragma unroll
                    for (int g = 0; g < GP; ++g) most[g] = fmaxf(most[g], __shfl_xor_sync(0xffffffffu, most[g], sh));
#pragma unroll
                  for (int g = 0; g < GP; ++g)
                    if (g < G && ok) {
                      lc_store_mx(r[g], most[g], q_start_s[it.seq], it.kvh * G * D + g * D + m * 128 + row, q_dim, p.q8_attn, p.sf_attn, lane);
                    }
                } else {
#pragma unroll
                  for (int g = 0; g < GP; ++g)
                    if (g < G && ok) out[g * D + m * 128 + row] = __float2bfloat16_rn(o[m][g]);
                }
              }
            } else {
              float* part_s = reinterpret_cast<float*>(zone + 8192);       // [G][D], over the weights of tiles that have been used
#pragma unroll
              for (int g = 0; g < GP; ++g)
                if (g < G) {
#pragma unroll
                  for (int m = 0; m < MB; ++m) part_s[g * D + m * 128 + row] = o[m][g];
                  if (row == 0) ml_s[g] = m_ref[g];
                }
              lc_sync();
              if (et < G) ml_s[GP + et] = sq_s[0][et] + sq_s[1][et] + sq_s[2][et] + sq_s[3][et];
              lc_sync();
              const int peer0 = rank - part;           // the CTAs of this item: consecutive ranks
              if (et < p.parts) arrive_cluster(mapa_smem(smem_u32(part_full), peer0 + et));
              if (ok) ok = __all_sync(0xffffffffu, lc_wait_cluster(part_full, nparts & 1u, abort, p.ctl));
              ++nparts;
#pragma unroll 1
              for (int e = part * 128 + row; e < G * D; e += p.parts * 128) {
                const int g = e / D;
                float mr[LC_CL], lr[LC_CL], nr[LC_CL], m = -INFINITY;      // (all loads in flight: each is a round trip to a neighbour)
#pragma unroll
                for (int r = 0; r < LC_CL; ++r) {
                  const uint32_t from = static_cast<uint32_t>(peer0 + min(r, p.parts - 1));
                  mr[r] = ld_cluster_f32(mapa_smem(smem_u32(&ml_s[g]), from));
                  lr[r] = ld_cluster_f32(mapa_smem(smem_u32(&ml_s[GP + g]), from));
                  nr[r] = ld_cluster_f32(mapa_smem(smem_u32(part_s + e), from));
                }
#pragma unroll
                for (int r = 0; r < LC_CL; ++r)
                  if (r < p.parts) m = fmaxf(m, mr[r]);
                float num = 0.f, den = 0.f;
#pragma unroll
                for (int r = 0; r < LC_CL; ++r) {
                  const float w = (r >= p.parts || mr[r] == -INFINITY) ? 0.f : ex2(mr[r] - m);
                  if (r < p.parts) {
                    den += w * lr[r];
                    num += w * nr[r];
                  }
                }
                const float v = den == 0.f ? 0.f : num / den;
                if (!ok) continue;
                if constexpr (MX) {
                  const float one[1] = {v};
                  lc_put_mx<1>(one, 1, q_start_s[it.seq], it.kvh * G * D + e, q_dim, p.q8_attn, p.sf_attn, lane);
                }
                else out[e] = __float2bfloat16_rn(v);
              }
            }
            lc_sync();                                 // the sums of the rows have been read
          }
        } else if (LN) {
          // ------------------------------------------------------------------------- out = LayerNorm(x): a CTA per token
          const __nv_bfloat16* w = op == OP_NORM_A ? L->post_attn : L->post_ffn;
          const __nv_bfloat16* wb = op == OP_NORM_A ? L->post_attn_b : L->post_ffn_b;
          const __nv_bfloat16* src = op == OP_NORM_A ? p.xb : p.xa;
          const int k8 = p.hidden / 8;
#pragma unroll 1
          for (int t = blockIdx.x; t < p.T; t += gridDim.x) {
            constexpr int C = 4;                       // chunks of 8 channels per thread (hidden <= 4096)
            uint4 xv[C], g[C], b[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const int i = et + 128 * c;
              xv[c] = g[c] = b[c] = make_uint4(0, 0, 0, 0);
              if (i < k8) {
                g[c] = reinterpret_cast<const uint4*>(w)[i];
                b[c] = reinterpret_cast<const uint4*>(wb)[i];
              }
            }
            if (ok) ok = __all_sync(0xffffffffu, lc_wait_due(due_s, at, abort));
            float sum = 0.f, ss = 0.f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              if (et + 128 * c < k8) xv[c] = __ldcg(reinterpret_cast<const uint4*>(src + static_cast<size_t>(t) * p.hidden) + et + 128 * c);
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&xv[c]);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                sum += f.x + f.y;
              }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) red_s[q4][0] = sum;
            lc_sync();
            const float mean = (red_s[0][0] + red_s[1][0] + red_s[2][0] + red_s[3][0]) / p.hidden;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&xv[c]);
              if (et + 128 * c < k8)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 f = __bfloat1622float2(h[j]);
                  ss += (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) sq_s[q4][0] = ss;
            lc_sync();
            const float rs = rsqrtf((sq_s[0][0] + sq_s[1][0] + sq_s[2][0] + sq_s[3][0]) / p.hidden + p.eps);
#pragma unroll
            for (int c = 0; c < C; ++c)
              if (et + 128 * c < k8 && ok) {
                uint4 o;
                const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&xv[c]);
                const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&g[c]);
                const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&b[c]);
                __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 f = __bfloat1622float2(hx[j]), fg = __bfloat1622float2(hg[j]), fb = __bfloat1622float2(hb[j]);
                  ho[j] = __floats2bfloat162_rn((f.x - mean) * rs * fg.x + fb.x, (f.y - mean) * rs * fg.y + fb.y);
                }
                reinterpret_cast<uint4*>(p.norm + static_cast<size_t>(t) * p.hidden)[et + 128 * c] = o;
              }
          }
        } else {
          // ------------------------------------------------------------- out = residual + rmsnorm(x) w: a CTA per token
          const __nv_bfloat16* w = op == OP_NORM_A ? L->post_attn : L->post_ffn;
          const __nv_bfloat16* residual = op == OP_NORM_A ? x : p.xb;
          __nv_bfloat16* out = op == OP_NORM_A ? p.xb : p.xa;
          const int k8 = p.hidden / 8;
#pragma unroll 1
          for (int t = blockIdx.x; t < p.T; t += gridDim.x) {
            const uint4* xr = reinterpret_cast<const uint4*>(p.norm + static_cast<size_t>(t) * p.hidden);
            const uint4* rr = reinterpret_cast<const uint4*>(residual + static_cast<size_t>(t) * p.hidden);
            uint4* orow = reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * p.hidden);
            constexpr int C = 4;                       // chunks of 8 channels per thread (hidden <= 4096)
            uint4 xv[C], r[C], g[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {              // (the residual is older than the operation in front)
              const int i = et + 128 * c;
              xv[c] = r[c] = g[c] = make_uint4(0, 0, 0, 0);
              if (i < k8) {
                g[c] = reinterpret_cast<const uint4*>(w)[i];
                r[c] = __ldcg(rr + i);
              }
            }
            if (ok) ok = __all_sync(0xffffffffu, lc_wait_due(due_s, at, abort));
#pragma unroll
            for (int c = 0; c < C; ++c)
              if (et + 128 * c < k8) xv[c] = __ldcg(xr + et + 128 * c);
            float ss = 0.f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&xv[c]);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                ss += f.x * f.x + f.y * f.y;
              }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) red_s[q4][0] = ss;
            lc_sync();
            const float rs = rsqrtf((red_s[0][0] + red_s[1][0] + red_s[2][0] + red_s[3][0]) / p.hidden + p.eps);
            float sq = 0.f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
              const int i = et + 128 * c;
              if (i < k8 && ok) {
                uint4 o;
                const __nv_bfloat162* hx = reinterpret_cast<const __nv_bfloat162*>(&xv[c]);
                const __nv_bfloat162* hr = reinterpret_cast<const __nv_bfloat162*>(&r[c]);
                const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&g[c]);
                __nv_bfloat162* ho = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 f = __bfloat1622float2(hx[j]), fr = __bfloat1622float2(hr[j]);
                  float2 fg = __bfloat1622float2(hg[j]);
                  if (p.plus_one) { fg.x += 1.f; fg.y += 1.f; }
                  ho[j] = __floats2bfloat162_rn(f.x * rs * fg.x + fr.x, f.y * rs * fg.y + fr.y);
                  const float2 f2 = __bfloat1622float2(ho[j]);
                  sq += f2.x * f2.x + f2.y * f2.y;
                }
                orow[i] = o;
              }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if (lane == 0) sq_s[q4][0] = sq;
            lc_sync();
            if (et == 0) p.ss[(op == OP_NORM_A ? LC_SS : 0) + t] = sq_s[0][0] + sq_s[1][0] + sq_s[2][0] + sq_s[3][0];
          }
        }
        // this CTA's results of the operation are stored
        lc_sync();
        if (threadIdx.x == 64) red_release_gpu(ctr + at, 1u);
        ++at;
      }
    }
  }

  // ------------------------------------------------------------------------------------------------------------------ leaving
  __syncwarp();
  if (*abort != 0u && lane == 0) *reinterpret_cast<volatile uint32_t*>(p.ctl + LW_ABORT) = 1u;
  tc_fence_before();
  __syncthreads();                                     // (no role waits behind this: the abort word is the same for all)
  const bool gave_up = *abort != 0u;
  if (threadIdx.x == 0) {
    lc_drain(mma_done, 0u);
    if (gave_up) {                                     // what was asked for and nobody waited for: it lands before the shared memory is given back
      const uint32_t n0 = issued_s[0], n1 = issued_s[1], n = max(n0, n1), slots = x_slots;
      for (uint32_t i = min(n0, n1); i < n; ++i) mbar_arrive(&full[i % LC_ENTRIES]);         // for the half that was not asked for
      for (uint32_t i = n - min(n, static_cast<uint32_t>(LC_ENTRIES)); i < n; ++i) lc_drain(&full[i % LC_ENTRIES], i / LC_ENTRIES & 1u);
      for (uint32_t i = issued_s[2] - min(issued_s[2], slots); i < issued_s[2]; ++i) lc_drain(&x_full[i % slots], i / slots & 1u);
      for (uint32_t i = issued_s[3] - min(issued_s[3], static_cast<uint32_t>(NQ)); i < issued_s[3]; ++i) lc_drain(&q_full[i % NQ], i / NQ & 1u);
    }
  }
  cluster_arrive_release();                            // no CTA leaves while another writes to or reads from it
  cluster_wait_acquire();
  if (gave_up && threadIdx.x == 0) {                   // sums that a neighbour sent and nobody waited for: they are on their way for a microsecond
    const unsigned long long t0 = globaltimer_ns();
    for (int i = 0; i < (1 << 20) && globaltimer_ns() - t0 < 100000ull; ++i) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<Cfg::kTmem>(tmem);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(p.ctl + LW_EXIT, 1u) == ctas - 1) {  // the last CTA: ready for the next launch
      __threadfence();
      volatile uint32_t* c = p.ctl;
      for (int i = 0; i < p.n_layers * OP_COUNT; ++i) c[LW_CTR + i] = 0u;
      if (c[LW_ABORT] != 0u) {
        c[LW_ABORT] = 0u;
        c[LW_GAVE_UP] = c[LW_GAVE_UP] + 1u;
        if (g_abort_word != nullptr) *reinterpret_cast<volatile uint32_t*>(g_abort_word) = 1u;
        atomicAdd(&g_chain_gave_up, 1u);
      }
      c[LW_EXIT] = 0u;
      __threadfence();
    }
  }
}

// clusters of four that fit the device at once with this kernel, 0 if it cannot run
template <int BN, int D, int GP, int KIND>
int chain_clusters() {
  static int known[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && known[dev] != 0) return known[dev] - 1;
  int n = 0, coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (coop && cudaFuncSetAttribute(layer_chain_kernel<BN, D, GP, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, LcCfg<BN, KIND>::kSmem) == cudaSuccess) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(LC_CL * 64);
    cfg.blockDim = dim3(LC_THREADS);
    cfg.dynamicSmemBytes = LcCfg<BN, KIND>::kSmem;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeClusterDimension;
    a[0].val.clusterDim.x = LC_CL;
    a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, layer_chain_kernel<BN, D, GP, KIND>, &cfg) != cudaSuccess) n = 0;
  }
  cudaGetLastError();
  if (dev < 64) known[dev] = n + 1;
  return n;
}

template <int BN, int D, int GP, int KIND>
int launch_chain_one(const LcMaps& maps, LcParams p, cudaStream_t s) {
  const int clusters = std::min(chain_clusters<BN, D, GP, KIND>(), 64);
  if (clusters <= 0) return -5;
  const int ctas = clusters * LC_CL, items = p.seqs * p.n_kv;
  p.parts = items * 4 <= ctas ? 4 : (items * 2 <= ctas ? 2 : 1);     // few sequences: CTAs of a cluster share the keys of one
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(LC_THREADS);
  cfg.dynamicSmemBytes = LcCfg<BN, KIND>::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute a[2];
  a[0].id = cudaLaunchAttributeClusterDimension;
  a[0].val.clusterDim.x = LC_CL;
  a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
  a[1].id = cudaLaunchAttributeCooperative;                          // the CTAs wait on one another
  a[1].val.cooperative = 1;
  cfg.attrs = a;
  cfg.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, layer_chain_kernel<BN, D, GP, KIND>, maps, p));
}

#define B2B_CHAIN64(FN, ...) B2B_CHAIN_OF(FN, 64, KIND_RMS, __VA_ARGS__)
#define B2B_CHAIN_OF(FN, BN, KIND, ...) \
  (d.layer_norm ? FN<BN, 128, 4, KIND_LN>(__VA_ARGS__) : \
   d.head_dim == 128 ? (g <= 4 ? FN<BN, 128, 4, KIND>(__VA_ARGS__) : FN<BN, 128, 8, KIND>(__VA_ARGS__)) \
                     : (g <= 4 ? FN<BN, 256, 4, KIND>(__VA_ARGS__) : FN<BN, 256, 8, KIND>(__VA_ARGS__)))
#define B2B_CHAIN(FN, BN, ...) (d.mx ? B2B_CHAIN_OF(FN, BN, KIND_MX, __VA_ARGS__) : B2B_CHAIN_OF(FN, BN, KIND_RMS, __VA_ARGS__))

}  // namespace

size_t layer_chain_table_bytes(int layers) { return static_cast<size_t>(layers) * sizeof(LcLayer); }
size_t layer_chain_control_words(int layers) { return (LW_CTR + static_cast<size_t>(layers) * 7 + 31) / 32 * 32 + 2 * LC_SS; }

bool layer_chain_supported(const ChainDims& d) {
  const int g = d.n_kv > 0 ? d.n_q / d.n_kv : 0;
  if (d.n_kv <= 0 || d.n_q % d.n_kv != 0 || d.hidden % 128 != 0 || d.hidden < 256 || d.ffn % 64 != 0 || d.ffn < 256 || d.n_q * d.head_dim < 256)
    return false;
  if (d.layer_norm) return d.head_dim == 64 && (d.n_q * 64) % 128 == 0 && (d.n_kv * 64) % 128 == 0 && d.ffn % 128 == 0 && d.hidden <= 4096;
  if (d.mx && (d.post_norms || d.ffn % 128 != 0 || d.hidden < 512 || d.ffn < 512 || d.n_q * d.head_dim < 512)) return false;
  return g <= 8 && (d.head_dim == 128 || d.head_dim == 256) && g * d.head_dim * 4 <= 8192 && (!d.post_norms || d.hidden <= 4096);
}

// tensor maps and pointers of one layer at `dst` (host memory)
int layer_chain_fill(void* dst, const ChainDims& d, const ChainLayerPtrs& w) {
  LcLayer L;
  std::memset(&L, 0, sizeof(L));
  const int q_dim = d.n_q * d.head_dim, kv_dim = d.n_kv * d.head_dim;
  const void* ptr[4] = {w.wqkv, w.wo, w.wgu, w.w_down};
  const uint64_t rows[4] = {static_cast<uint64_t>(q_dim + 2 * kv_dim), static_cast<uint64_t>(d.hidden), (d.layer_norm ? 1ull : 2ull) * d.ffn, static_cast<uint64_t>(d.hidden)};
  const uint64_t cols[4] = {static_cast<uint64_t>(d.hidden), static_cast<uint64_t>(q_dim), static_cast<uint64_t>(d.hidden), static_cast<uint64_t>(d.ffn)};
  for (int i = 0; i < 4; ++i)
    for (int b = 0; b < 5; ++b)
      if (const int r = make_tmap_shared(&L.w[i][b], ptr[i], rows[i], cols[i], cols[i], 8u << b, d.mx ? 1 : 2)) return r;
  const uint64_t keys = static_cast<uint64_t>(d.pages) * LC_PAGE;
  if (const int r = make_tmap_shared(&L.k, w.k_cache, keys, kv_dim, kv_dim, LC_PAGE, 2)) return r;
  if (const int r = make_tmap_shared(&L.v, w.v_cache, keys, kv_dim, kv_dim, LC_PAGE, 2)) return r;
  L.k_cache = static_cast<__nv_bfloat16*>(w.k_cache);
  L.v_cache = static_cast<__nv_bfloat16*>(w.v_cache);
  L.post_attn = static_cast<const __nv_bfloat16*>(w.post_attn);
  L.post_ffn = static_cast<const __nv_bfloat16*>(w.post_ffn);
  L.post_attn_b = static_cast<const __nv_bfloat16*>(w.post_attn_b);
  L.post_ffn_b = static_cast<const __nv_bfloat16*>(w.post_ffn_b);
  for (int i = 0; i < 4; ++i) {
    L.bias[i] = w.bias[i];
    L.sf[i] = static_cast<const uint8_t*>(w.sf[i]);
  }
  L.window = w.window;
  std::memcpy(dst, &L, sizeof(L));
  return 0;
}

int launch_layer_chain(const ChainDims& d, const ChainCall& c, cudaStream_t s) {
  const int g = d.n_kv > 0 ? d.n_q / d.n_kv : 0;
  if (!layer_chain_supported(d) || c.tokens < 1 || c.tokens > layer_chain_tokens(d) || c.layers < 1 || (!d.layer_norm && c.seqs > c.tokens)) return -2;
  const int bn = c.tokens <= 16 ? 16 : (c.tokens <= 32 ? 32 : 64), x_rows = c.tokens <= 8 ? 8 : bn, q_dim = d.n_q * d.head_dim;
  LcMaps m;
  auto act = [&](CUtensorMap* t, const void* ptr, uint64_t rows, int cols) {
    return make_blocks_tmap(t, ptr, rows, cols, x_rows, bn == 16 ? LcCfg<16, KIND_RMS>::kXBlocks : LcCfg<32, KIND_RMS>::kXBlocks, d.mx ? 1 : 2);
  };
  int r;
  // what the products read: LayerNorm models the normed rows, fp8 ones the copies in fp8
  const void *x_in = c.x_in, *xa = c.xa, *xb = c.xb, *attn = c.attn, *h = c.h;
  if (d.layer_norm) x_in = xa = xb = c.norm;
  if (d.mx) {
    x_in = c.q8_in;
    xa = xb = c.q8_x;
    attn = c.q8_attn;
    h = c.q8_h;
  }
  if ((r = act(&m.x_in, x_in, x_in == c.x_in ? c.tokens : c.max_tokens, d.hidden)) || (r = act(&m.xa, xa, c.max_tokens, d.hidden)) ||
      (r = act(&m.xb, xb, c.max_tokens, d.hidden)) || (r = act(&m.attn, attn, c.max_tokens, q_dim)) || (r = act(&m.h, h, c.max_tokens, d.ffn)) ||
      (r = make_tmap_shared(&m.q, c.q, static_cast<uint64_t>(c.max_tokens) * d.n_q, d.head_dim, d.head_dim, LC_HEADS, 2)))
    return r;
  LcParams p;
  p.layers = static_cast<const LcLayer*>(c.table);
  p.n_layers = c.layers; p.T = c.tokens; p.seqs = c.seqs;
  p.hidden = d.hidden; p.ffn = d.ffn; p.n_q = d.n_q; p.n_kv = d.n_kv; p.head_dim = d.head_dim; p.parts = 1;
  p.act = d.act_gelu; p.plus_one = d.plus_one; p.norms = d.post_norms; p.x_rows = x_rows;
  p.eps = d.eps; p.rope_theta = d.rope_theta; p.q_scale = d.q_scale; p.softcap = d.softcap;
  p.x_in = static_cast<const __nv_bfloat16*>(c.x_in);
  p.xa = static_cast<__nv_bfloat16*>(c.xa); p.xb = static_cast<__nv_bfloat16*>(c.xb); p.q = static_cast<__nv_bfloat16*>(c.q);
  p.attn = static_cast<__nv_bfloat16*>(c.attn); p.h = static_cast<__nv_bfloat16*>(c.h); p.norm = static_cast<__nv_bfloat16*>(c.norm);
  p.positions = c.positions; p.slots = c.slots; p.q_start = c.q_start; p.q_len = c.q_len; p.kv_len = c.kv_len; p.block_table = c.block_table;
  p.max_pages = c.max_pages;
  p.polls = c.polls > 0 ? c.polls : LC_SPINS;
  p.q8_x = static_cast<uint8_t*>(c.q8_x); p.q8_attn = static_cast<uint8_t*>(c.q8_attn); p.q8_h = static_cast<uint8_t*>(c.q8_h);
  p.sf_x = static_cast<uint8_t*>(c.sf_x); p.sf_attn = static_cast<uint8_t*>(c.sf_attn); p.sf_h = static_cast<uint8_t*>(c.sf_h);
  p.sf_in = static_cast<const uint8_t*>(c.sf_in);
  p.ctl = c.control;
  p.ss = reinterpret_cast<float*>(c.control + layer_chain_control_words(c.layers)) - 2 * LC_SS;
  if (bn == 16) return B2B_CHAIN(launch_chain_one, 16, m, p, s);
  if (bn == 32) return B2B_CHAIN(launch_chain_one, 32, m, p, s);
  return B2B_CHAIN64(launch_chain_one, m, p, s);
}

// Block-scaled fp8 steps of 33 tokens and more stay with the kernels one by one.  The line was drawn when a tile's stores held up the next one (two layers of
// Zephyr-7B, 40 tokens: 193.5 us one by one, 195.0 here) and is now too low for few keys (Llama-3-8B behind 500 keys, one by one / here: 40 tokens 211 / 194, 64
// tokens 228 / 214; but 34 tokens 193 / 192, and behind 4000 keys 335 / 373): beyond it what attention costs has not been measured.
int layer_chain_tokens(const ChainDims& d) { return d.mx ? 32 : 64; }

// clusters that are resident at once (0: the kernel cannot run here); also sets the kernels' shared memory sizes, so that a first launch may
// happen under graph capture
int layer_chain_init(const ChainDims& d) {
  const int g = d.n_kv > 0 ? d.n_q / d.n_kv : 0;
  if (!layer_chain_supported(d)) return 0;
  const int n = std::min(B2B_CHAIN(chain_clusters, 16), B2B_CHAIN(chain_clusters, 32));
  return d.mx ? n : std::min(n, B2B_CHAIN64(chain_clusters));
}

// (its own waits are counted in polls: the process's limit in time is for flags of other GPUs)
int set_wait_policy_chain(uint32_t* abort_word) { return static_cast<int>(cudaMemcpyToSymbol(g_abort_word, &abort_word, sizeof(abort_word))); }

unsigned layer_chain_gave_up() {
  unsigned n = 0;
  return cudaMemcpyFromSymbol(&n, g_chain_gave_up, sizeof(n)) == cudaSuccess ? n : ~0u;
}

}  // namespace b2b
