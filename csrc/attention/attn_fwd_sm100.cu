// Variable-length causal GQA attention forward for sm_100a: S = Q K^T and O += P V on tcgen05 with accumulators in
// TMEM, operands staged by TMA, softmax in registers, P handed to the second product through TMEM.
//
// The mask is a per-query inclusive key range [k_lo[i], k_hi[i]] (see attn_common.cuh): packed causal self-attention is
// k_lo = first token of the query's sequence, k_hi = the query itself, so tiles may straddle sequence boundaries and
// nothing is synchronised with the host; queries and keys may also be different token sets (the steps of
// context-parallel ring attention, non-causal attention).
//
// One CTA works on two 128-query tiles at once and walks the key blocks either of them can see.  The exponentials of one
// tile run while the tensor core multiplies for the other, and one K / V load serves both (two tiles in turn with P over S
// in TMEM: the scheme published as FlashAttention-4).  Online softmax; a row's accumulator is rescaled whenever its maximum
// grows.  FlashAttention-4 waits until it has grown by 2^8, which spares most of the rescales, but then the row's largest
// probabilities lie anywhere between two powers of two instead of just below 1, where the spacing of bf16 is finest
// relative to them: off from fp64 by 0.00223 instead of 0.00213 (12363 tokens; 0.00215 with the final maximum as the
// reference).
//
// Warp roles (512 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 4..7 softmax of tile 0, warps 8..11
// of tile 1 (thread = query row, a whole 128-column score row in registers: the other warps give registers up), warps
// 12..15 rescale the accumulators of both tiles.  TMEM: S0 | S1 (128 columns each, P overwrites the scores it came from as
// packed bf16) | O0 | O1.  The issuer's order is  PV_t(j), QK_t(j + 1)  for t = 0, 1: the score buffer of a tile is reused
// as soon as its P has been multiplied, MMAs of one thread complete in order, and the two tiles stay out of phase.
//
// Bound: per 128 x 128 block the two products take 1024 tensor cycles and the 16384 exponentials 1024 MUFU cycles of an
// SM; what sets the pace is the chain of a tile, load - maximum - exponentials - product - next scores.  Clock stamps of the
// form with the rescale in the softmax warps and an issuer inside `if (lane == 0)`, cycles a block and tile: wait for the
// scores 1360, load 86, maximum 430, rescale 770 (some row of 32 grows in nearly every block), exponentials 1540.  The rescale
// now runs beside the exponentials and the issuer's whole warp stays converged (umma_f16_warp).  Measured, 32 query / 8 kv
// heads of 128: 16384 tokens causal 2.19 -> 2.02 ms (1090 TFLOP/s, at the power cap: sustained, 4.28 -> 3.65 Mcycles at 1792 and
// 1717 MHz), 8192 tokens in five sequences 200 -> 183 us, 2048 tokens 58 -> 52.  Taken back: the exponentials in four parts
// instead of two (2.49 ms), a quarter of them by polynomial on the FMA pipe (2.17), two issuers (tiles drift into phase: 2.20;
// with turns for the exponentials 2.03), four softmax warps a scheduler with half a row a thread (2.22).
#include "../common/host_utils.cuh"
#include "../common/ptx.cuh"
#include "attn_common.cuh"

using namespace mcb;

namespace {

constexpr int BM = 128;  // queries per CTA
constexpr int BNK = 128; // keys per block
constexpr int ATT_THREADS = 512;

struct AttnParams {
  int T, Tk, nq, nkv, d;  // T queries, Tk keys
  float scale_log2;       // softmax scale * log2(e)
  const int* k_lo;        // [T] first visible key of each query
  const int* k_hi;        // [T] last visible key, or null: the query's own index
  const float* sinks;     // [nq] or null: a per-head logit that joins every row's softmax with a zero value vector
  __nv_bfloat16* o;       // [T, nq, d]
  float* lse;             // [nq, T] natural log of sum exp(scaled scores); -inf for a query that sees no key
  int* status;
  int pairing, per_row;   // how a CTA's two tiles are chosen; CTAs per row of tiles (set by the launcher)
};

// How the two tiles of a CTA are chosen.  PAIR_HEADS: two query heads of one kv group, same queries (the ranges are then
// equal and no block is loaded for one tile only).  PAIR_ROWS: adjacent query tiles of one head (odd GQA ratios).
// SPLIT_KEYS: one tile whose key blocks are dealt out to both softmax groups in turn, the two partial results are added at
// the end; taken up to two tiles per SM.  Two chains per SM as with pairs, but the tiles spread over twice as many CTAs; with
// more of them a pair's shared K / V loads and prologue count for more.  Forward, us, pairs and split: 72 tiles (3000 tokens, 9
// heads of 128) 75 / 45, 192 tiles (8192, 3) 159 / 90, 288 (1100, 32) 34 / 27, 448 (2048, 28) 53 / 59, 512 (2048, 32) 56 / 64.
enum { PAIR_HEADS = 0, PAIR_ROWS = 1, SPLIT_KEYS = 2 };

template <int D>
struct AttnSmem {
  static constexpr int TILE = BM * D * 2;            // one 128-row operand tile
  static constexpr int OFF_Q = 0;                     // 2 tiles
  static constexpr int OFF_K = 2 * TILE;              // 2 stages
  static constexpr int OFF_V = OFF_K + 2 * TILE;      // 2 stages
  static constexpr int OFF_BAR = OFF_V + 2 * TILE;
  static constexpr int TOTAL = OFF_BAR + 1024 + 1024;
};

// K-major operand tile [128 rows x D] stored as D/64 boxes of [128 x 64]; descriptor for the kk-th 16-wide k slice
template <int D>
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t base, int kk) {
  return make_smem_desc_sw128(base + (kk >> 2) * (BM * 128) + (kk & 3) * 32, 16, 1024);
}

__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(b_mn ? 1 : 0) << 16) | (uint32_t(n >> 3) << 17) |
         (uint32_t(m >> 4) << 24);
}

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  using L = AttnSmem<D>;
  constexpr int NBOX = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t COL_S = 0, COL_O = 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars;            // 2, per tile
  uint64_t* kv_full = bars + 2;       // 2 stages: V of block j and K of block j + ahead
  uint64_t* kv_empty = bars + 4;      // 2
  uint64_t* s_full = bars + 6;        // 2, per tile
  uint64_t* p_full = bars + 8;        // 2 x 2, per tile: halves of P (64 keys), the first with the accumulator rescaled
  uint64_t* o_done = bars + 12;       // 2, per tile: all products have completed
  uint64_t* f_full = bars + 14;       // 2 x 4, per tile and quarter of rows: the factors of a block's rescale are in s_fac
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int bx = blockIdx.x % p.per_row;
  const int mt = (gridDim.x - 1 - blockIdx.x) / p.per_row;   // long tiles of every head first: the tail gets short ones
  int head0, head1, m00, m01;
  if (p.pairing == PAIR_HEADS) {
    head0 = 2 * bx;
    head1 = head0 + 1;
    m00 = m01 = mt * BM;
  } else if (p.pairing == PAIR_ROWS) {
    head0 = head1 = bx;
    m00 = 2 * mt * BM;
    m01 = m00 + BM;
  } else {
    head0 = head1 = bx;
    m00 = m01 = mt * BM;
  }
  const bool split = p.pairing == SPLIT_KEYS;
  const int kvh = head0 / (p.nq / p.nkv);
  __shared__ int s_rng[2][8];
  __shared__ float s_fac[2][BM];                // per tile and row: what its accumulator has to be multiplied by
  __shared__ float s_part[2][2][BM];            // SPLIT_KEYS: maxima and sums of the two groups
  tile_range_partial(p.k_lo, p.k_hi, m00, p.T, s_rng[0]);
  tile_range_partial(p.k_lo, p.k_hi, m01, p.T, s_rng[1]);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&q_full[i]), 1);
      mbar_init(smem_u32(&kv_full[i]), 1);
      mbar_init(smem_u32(&kv_empty[i]), 1);
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&p_full[2 * i]), 8);     // softmax and correction warps
      mbar_init(smem_u32(&p_full[2 * i + 1]), 4);
      mbar_init(smem_u32(&o_done[i]), 1);
      for (int w = 0; w < 4; ++w) mbar_init(smem_u32(&f_full[4 * i + w]), 1);
    }
    fence_barrier_init();
    fence_proxy_async_smem();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  // key blocks [b0, b1) of each tile, and their union [jb, je)
  int b0[2], b1[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int kmin = tile_range_min(s_rng[t]), kmax = tile_range_max(s_rng[t]);
    b0[t] = warp_uniform(kmax >= kmin ? kmin / BNK : 0);
    b1[t] = warp_uniform(kmax >= kmin ? kmax / BNK + 1 : 0);
  }
  const bool any0 = b1[0] > b0[0], any1 = b1[1] > b0[1];
  const int jb = any0 ? (any1 ? min(b0[0], b0[1]) : b0[0]) : b0[1];
  const int je = max(b1[0], b1[1]);
  // the scores of a group's next block replace the P of its previous one: one block on, in split mode two
  const int ahead = split ? 2 : 1;
  // in the key range of tile t, and in split mode its turn
  auto takes = [&](int t, int j) {
    return j >= b0[t] && j < b1[t] && (!split || ((j - jb) & 1) == t);
  };

  // 512 threads x 128 registers at launch = 128 x (64 + 192 + 192 + 64)
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0 && je > jb) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!(t ? any1 && !split : any0)) continue;
        mbar_expect_tx(smem_u32(&q_full[t]), L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          tma_load_2d(smem_u32(smem + L::OFF_Q + t * L::TILE + b * BM * 128), &tm_q, (t ? head1 : head0) * D + b * 64,
                      t ? m01 : m00, smem_u32(&q_full[t]));
      }
      int n = 0;
      for (int j = jb - ahead; j < je; ++j, ++n) {
        const uint32_t st = n & 1, ph = (n >> 1) & 1;
        if (!mbar_wait(smem_u32(&kv_empty[st]), ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        const bool has_v = j >= jb, has_k = j + ahead < je;
        mbar_expect_tx(smem_u32(&kv_full[st]), (has_v + has_k) * L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          if (has_v)
            tma_load_2d(smem_u32(smem + L::OFF_V + st * L::TILE + b * BM * 128), &tm_v, kvh * D + b * 64, j * BNK,
                        smem_u32(&kv_full[st]));
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          if (has_k)
            tma_load_2d(smem_u32(smem + L::OFF_K + st * L::TILE + b * BM * 128), &tm_k, kvh * D + b * 64,
                        (j + ahead) * BNK, smem_u32(&kv_full[st]));
      }
      // drain: the last loads must land before the CTA exits
      auto drain = [](uint64_t* bar, uint32_t parity) {
        uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(smem_u32(bar), parity))
          if (globaltimer_ns() - t0 > 200000000ull) break;
      };
      for (int i = (n > 2 ? n - 2 : 0); i < n; ++i) drain(&kv_full[i & 1], (i >> 1) & 1);
      if (any0) drain(&q_full[0], 0);
      if (any1 && !split) drain(&q_full[1], 0);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer: a whole warp, see umma_f16_warp
    // Per stage and tile: P V of block j, then the scores of block j + ahead.
    if (je > jb) {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = idesc_bf16(BM, BNK, false);
      constexpr uint32_t idesc_o = idesc_bf16(BM, D, true);
      bool ok = true;
      if (any0) ok = mbar_wait_warp(smem_u32(&q_full[0]), 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      if (any1 && !split) ok = ok && mbar_wait_warp(smem_u32(&q_full[1]), 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      uint32_t np[2] = {0, 0};         // products P V issued, per tile
#pragma unroll 1
      for (int j = jb - ahead; j < je && ok; ++j) {
        const uint32_t i = j - (jb - ahead), st = i & 1;
        const uint32_t sv = smem_u32(smem + L::OFF_V + st * L::TILE), sk = smem_u32(smem + L::OFF_K + st * L::TILE);
        ok = mbar_wait_warp(smem_u32(&kv_full[st]), (i >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t ds = tmem + COL_S + t * BNK, dpv = tmem + COL_O + t * 128;
          if (ok && takes(t, j)) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              ok = ok && mbar_wait_warp(smem_u32(&p_full[2 * t + h]), np[t] & 1, abort_flag, p.status, ST_TIMEOUT_FULL);
              tc_fence_after();
              if (ok) {
#pragma unroll
                for (int kk = 4 * h; kk < 4 * h + 4; ++kk)
                  umma_f16_ts_warp(leader, dpv, ds + kk * 8, make_smem_desc_sw128(sv + kk * 2048, BM * 128, 1024), idesc_o,
                                   (np[t] | kk) ? 1u : 0u);
              }
            }
            ++np[t];
          }
          if (ok && takes(t, j + ahead)) {
            tc_fence_after();
            const uint32_t sq = smem_u32(smem + L::OFF_Q + (split ? 0 : t) * L::TILE);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk)
              umma_f16_warp(leader, ds, kmajor_desc<D>(sq, kk), kmajor_desc<D>(sk, kk), idesc_s, kk ? 1u : 0u);
            umma_commit_warp(leader, smem_u32(&s_full[t]));
          }
        }
        umma_commit_warp(leader, smem_u32(&kv_empty[st]));
      }
      umma_commit_warp(leader, smem_u32(&o_done[0]));
      umma_commit_warp(leader, smem_u32(&o_done[1]));
    }
  }
  } else if (warp >= 12) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // ------------------------------------------------------------------ correction warps: thread = query row of both tiles
    // The scores of block n exist, so every product issued before them for the tile, P V of block n - 1 included, has
    // completed; P V of block n waits for the arrival here.  Blocks are taken in the issuer's order.
    const int q = warp & 3, r = q * 32 + lane;
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    bool ok = true;
    int np[2] = {0, 0};
    for (int j = jb; j < je && ok; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!takes(t, j)) continue;
        if (np[t] && ok) {
          ok = mbar_wait_warp(smem_u32(&f_full[4 * t + q]), (np[t] & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
          const float f = s_fac[t][r];
          if (ok && __any_sync(0xffffffffu, f != 1.f)) {
            const uint32_t to = tmem + lane_addr + COL_O + t * 128;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
              uint32_t o[32];
              tmem_ld_32x32(to + c, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st_32x32(to + c, o);
            }
            tmem_st_wait();
            tc_fence_before();
          }
        }
        ++np[t];
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(smem_u32(&p_full[2 * t]));
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
    // ------------------------------------------------------------------ softmax warps: thread = query row
    const int q = warp & 3;
    const int t = (warp - 4) >> 2;
    const int r = q * 32 + lane;
    const int head = t ? head1 : head0;
    const int i = (t ? m01 : m00) + r;
    const int jfirst = (t ? b0[1] : b0[0]) + (split ? t : 0), jlast = t ? b1[1] : b1[0], jstep = split ? 2 : 1;
    const int blocks = jlast > jfirst ? (jlast - jfirst + jstep - 1) / jstep : 0;
    const bool row_ok = i < p.T;
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    const uint32_t ts = tmem + lane_addr + COL_S + t * BNK, to = tmem + lane_addr + COL_O + t * 128;
    int lo, hi;
    attn_row_range(p.k_lo, p.k_hi, i, p.T, lo, hi);
    if (lo > hi) lo = hi = 0x40000000;            // sees nothing: a range no key index reaches
    const unsigned span = (unsigned)(hi - lo);    // key k is visible iff (unsigned)(k - lo) <= span
    float mref = -INFINITY;                       // reference maximum, log2 units
    uint64_t sum2 = 0;                            // two fp32 partial row sums
    bool ok = true;
#pragma unroll 1
    for (int n = 0; n < blocks && ok; ++n) {
      const int n0 = (jfirst + n * jstep) * BNK;
      const bool full = __all_sync(0xffffffffu, lo <= n0 && n0 + BNK - 1 <= hi) && p.scale_log2 > 0.f;
      const float mul = full ? p.scale_log2 : 1.f;  // what the scores in registers still have to be multiplied by
      if (!mbar_wait_warp(smem_u32(&s_full[t]), n & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(ts + 32 * c, v[c]);
      tmem_ld_wait();
      if (!full) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int e = 0; e < 32; ++e) v[c][e] = __float_as_uint(__uint_as_float(v[c][e]) * p.scale_log2);
          if (seen_keys(lo, hi, n0 + 32 * c) == Seen::ALL) continue;
#pragma unroll
          for (int e = 0; e < 32; ++e) v[c][e] = (unsigned)(n0 + 32 * c + e - lo) <= span ? v[c][e] : 0xff800000u;
        }
      }
      float mx;
      {
        float m4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          m4[c] = __uint_as_float(v[c][0]);
#pragma unroll
          for (int e = 1; e < 32; ++e) m4[c] = fmaxf(m4[c], __uint_as_float(v[c][e]));
        }
        mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * mul;
      }
      const float mold = mref == -INFINITY ? mx : mref;   // nothing accumulated yet: sum and accumulator are zero
      mref = fmaxf(mold, mx);
      const float m2 = mref == -INFINITY ? 0.f : mref;
      const uint64_t cc = f32x2(mul, mul), mm = f32x2(-m2, -m2);
      // a block's exponentials have a sum of their own before they join the row's: with one running sum the log-sum-exp of 16384 keys is
      // off from 64 bits by 6.5e-7 (rms) instead of 5.6e-7
      uint64_t add2 = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const uint64_t x2 = fma_f32x2(f32x2(__uint_as_float(v[c][e]), __uint_as_float(v[c][e + 1])), cc, mm);
          const float2 x = f32x2_split(x2);
          const float e0 = ex2_ftz(x.x), e1 = ex2_ftz(x.y);
          add2 = add_f32x2(add2, f32x2(e0, e1));
          pk[e >> 1] = pack_bf16x2(e0, e1);
        }
        if (c == 2) {                             // the first half's stores have had the time of a quarter of the block
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&p_full[2 * t]));
        }
        tmem_st_32x16(ts + 16 * c, pk);
        if (c == 0) {                             // after the first exponentials: the correction warps have time
          const float f = mold == mref ? 1.f : ex2_ftz(mold - mref);
          if (n) {
            s_fac[t][r] = f;                      // read before P V of this block, which the next scores wait for
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&f_full[4 * t + q]));
          }
          sum2 = mul_f32x2(sum2, f32x2(f, f));
        }
      }
      sum2 = add_f32x2(sum2, add2);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[2 * t + 1]));
    }
    const float2 sp = f32x2_split(sum2);
    float sum = sp.x + sp.y, fold = 1.f, fold2 = 0.f;       // what this group's accumulator, and the other's, counts for
    int blocks2 = 0;
    float mtot = mref;
    if (split) {
      blocks2 = (b1[0] - b0[0] + t) / 2;                    // the other group's share
      s_part[0][t][r] = mref;
      s_part[1][t][r] = sum;
      asm volatile("bar.sync 1, 256;" ::: "memory");        // the eight softmax warps, also those that gave up a wait
      const float m2 = s_part[0][t ^ 1][r];
      mtot = fmaxf(mref, m2);
      fold = mref == -INFINITY ? 0.f : ex2_ftz(mref - mtot);
      fold2 = m2 == -INFINITY ? 0.f : ex2_ftz(m2 - mtot);
      sum = sum * fold + s_part[1][t ^ 1][r] * fold2;
    }
    const bool seen = blocks + blocks2 > 0;
    // learnable softmax sink: an extra logit (already in softmax units, no scale) in the row's maximum and sum
    const float sink2 = p.sinks ? p.sinks[head] * 1.4426950408889634f : -INFINITY;
    const float msum = mtot;
    mtot = fmaxf(mtot, sink2);
    const float fs = msum == -INFINITY ? 0.f : ex2_ftz(msum - mtot);
    sum = sum * fs + (p.sinks ? ex2_ftz(sink2 - mtot) : 0.f);
    const float inv = sum > 0.f ? fs / sum : 0.f;
    __nv_bfloat16* orow = p.o + ((long long)i * p.nq + head) * D;
    const int c0 = split ? t * (D / 2) : 0, c1 = split ? c0 + D / 2 : D;   // columns this group writes
    if (!seen) {
      // no row of this tile sees any key: the output is zero
      if (row_ok) {
#pragma unroll 1
        for (int c = c0; c < c1; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
      }
    } else {
      if (blocks > 0 && ok) ok = mbar_wait(smem_u32(&o_done[t]), 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      if (blocks2 > 0 && ok) ok = mbar_wait(smem_u32(&o_done[t ^ 1]), 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      const uint32_t to2 = tmem + lane_addr + COL_O + (t ^ 1) * 128;
      const float f = fold * inv, f2 = fold2 * inv;
#pragma unroll 1
      for (int c = c0; c < c1 && ok; c += 32) {
        uint32_t v[32];
        float o[32];
        if (blocks > 0) {
          tmem_ld_32x32(to + c, v);
          tmem_ld_wait();
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = blocks > 0 ? __uint_as_float(v[e]) * f : 0.f;
        if (blocks2 > 0) {
          tmem_ld_32x32(to2 + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = fmaf(__uint_as_float(v[e]), f2, o[e]);
        }
        if (row_ok) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 w;
            w.x = pack_bf16x2(o[e], o[e + 1]);
            w.y = pack_bf16x2(o[e + 2], o[e + 3]);
            w.z = pack_bf16x2(o[e + 4], o[e + 5]);
            w.w = pack_bf16x2(o[e + 6], o[e + 7]);
            *reinterpret_cast<uint4*>(orow + c + e) = w;
          }
        }
      }
    }
    if (row_ok && ok && !(split && t))
      p.lse[(long long)head * p.T + i] = sum > 0.f ? (mtot + log2f(sum)) * 0.6931471805599453f : -INFINITY;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

template <int D>
int launch_fwd(const void* q, const void* k, const void* v, AttnParams p, cudaStream_t stream) {
  CUtensorMap tq, tk, tv;
  int rc = make_tmap_2d_bf16(&tq, q, (long long)p.nq * D, p.T, (long long)p.nq * D, 64, BM);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tk, k, (long long)p.nkv * D, p.Tk, (long long)p.nkv * D, 64, BNK);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tv, v, (long long)p.nkv * D, p.Tk, (long long)p.nkv * D, 64, BNK);
  if (rc) return rc;
  static bool cfg = false;
  if (!cfg) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  const int tiles = (p.T + BM - 1) / BM, qpg = p.nq / p.nkv;
  p.pairing = tiles * p.nq <= 2 * device_sm_count() ? SPLIT_KEYS : (qpg % 2 == 0 ? PAIR_HEADS : PAIR_ROWS);
  p.per_row = p.pairing == PAIR_HEADS ? p.nq / 2 : p.nq;
  const unsigned grid = (unsigned)p.per_row * (p.pairing == PAIR_ROWS ? (tiles + 1) / 2 : tiles);
  attn_fwd_kernel<D><<<grid, ATT_THREADS, AttnSmem<D>::TOTAL, stream>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

__global__ void attn_window_starts_kernel(const int* __restrict__ seq_start, int* __restrict__ out, int T, int left) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < T) out[i] = max(seq_start[i], i - left);
}

}  // namespace

extern "C" {

// First visible key of every token of packed causal self-attention that sees at most `left` predecessors.
int mcb_attn_window_starts(const int* seq_start, int* out, int T, int left, void* stream_) {
  if (T <= 0) return 0;
  attn_window_starts_kernel<<<(unsigned)(T + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(seq_start, out, T,
                                                                                                           left);
  return (int)cudaGetLastError();
}

// General form.  q [T, nq, d], k/v [Tk, nkv, d] bf16 contiguous; k_lo / k_hi [T] int32: query i attends to the keys
// k_lo[i] .. k_hi[i] (inclusive; k_hi may be null = i, which needs Tk >= T); sinks [nq] fp32 or null; o [T, nq, d];
// lse [nq, T] fp32 (it includes the sink, which is what the backward kernels need to recompute the probabilities).
int mcb_attn_fwd_ranges(const void* q, const void* k, const void* v, const int* k_lo, const int* k_hi,
                        const float* sinks, void* o, float* lse, int T, int Tk, int nq, int nkv, int d, float scale,
                        int* status, void* stream_) {
  if (T == 0) return 0;
  if (nq % nkv || Tk <= 0 || (k_hi == nullptr && Tk < T)) return -2;
  AttnParams p{T, Tk, nq, nkv, d, scale * 1.4426950408889634f, k_lo, k_hi, sinks, (__nv_bfloat16*)o, lse, status, SPLIT_KEYS, nq};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (d == 128) return launch_fwd<128>(q, k, v, p, s);
  if (d == 64) return launch_fwd<64>(q, k, v, p, s);
  return -3;
}

}  // extern "C"
