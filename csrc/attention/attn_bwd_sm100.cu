// Variable-length causal GQA attention backward for sm_100a.  Three kernels:
//
//   delta   : delta[h, i] = sum_d O[i, h, d] * dO[i, h, d]                                  (memory bound)
//   dq      : one CTA per (128-query tile, query head), loops over 128-key blocks (and forms delta itself where that is the
//             faster way, see launch_bwd):
//               S = Q K^T, dP = dO V^T on tcgen05 -> P = exp2(S*c - lse), dS = P*(dP - delta)*scale in registers
//               -> dS (bf16) to TMEM -> dQ += dS K accumulated in TMEM
//   dk/dv   : one CTA per (128-key tile, kv head), loops over the query heads of the group and 128-query blocks:
//               S^T = K Q^T, dP^T = V dO^T -> P^T, dS^T -> dV += P^T dO, dK += dS^T Q accumulated in TMEM
//
// The softmax scale multiplies dS before it is rounded to bf16.  All operand tiles are the ones the forward kernel
// uses (row-major [tokens, heads*d] tiles fetched by TMA with the 128-byte swizzle, consumed K-major or MN-major); the
// probabilities and dS go to the second product as its A operand through TMEM, never through shared memory, and P is
// recomputed from the forward's log-sum-exp so nothing but O and lse is kept from the forward.  The mask is the
// forward's: a per-query inclusive key range [k_lo[i], k_hi[i]] (k_hi null = the query's own index, i.e. packed causal
// self-attention); queries and keys may be different token sets.  The dK/dV kernel additionally takes, per key, bounds
// [q_lo[n], q_hi[n]] on the queries that can see it (null = derived from the causal structure), which only limit its
// loop: visibility itself is always decided by the per-query ranges.
//
// Warp roles (384 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warp 2 (dk/dv) stages the per-query
// values of the next blocks, warps 4..11 element-wise: thread = TMEM lane = query row in dq, key row in dk/dv; warps
// 4..7 take columns 0..63 of every block, warps 8..11 columns 64..127, so that a block's latency is half a block's
// arithmetic.  The tensor core is kept busy by the order of the products, not by second buffers (see each kernel).
// Every wait is bounded and reports through the status buffer.  The issuer is a whole converged warp (umma_f16_warp): a block's
// 24 (dq) or 32 (dk/dv) MMAs issued by `if (lane == 0)` took longer than the tensor core needs for them.  Measured, delta to
// dK/dV, 32 query / 8 kv heads of 128, causal: one 16384-token segment 7.19 -> 6.38 ms (861 TFLOP/s counting five products), 8192
// tokens in five segments 621 -> 559 us; 3000 tokens, 9 / 3 heads 262 -> 216.
#include <climits>

#include "../common/host_utils.cuh"
#include "../common/ptx.cuh"
#include "attn_common.cuh"

using namespace mcb;

namespace {

constexpr int TM = 128;   // rows of the CTA's resident tile (TMEM lanes) and of the streamed blocks
constexpr int BWD_THREADS = 384;
constexpr int HALF = TM / 2;   // columns of a block that one element-wise warp handles
constexpr float LOG2E = 1.4426950408889634f;
// 384 threads x 168 registers at launch: 128 x (104 + 200 + 200) = 64512
#define MCB_REGS_CONTROL() asm volatile("setmaxnreg.dec.sync.aligned.u32 104;")
#define MCB_REGS_MATH() asm volatile("setmaxnreg.inc.sync.aligned.u32 200;")

struct BwdParams {
  int T, Tk, nq, nkv, d;    // T queries, Tk keys
  float scale, scale_log2;
  const int* k_lo;          // [T] first visible key of each query
  const int* k_hi;          // [T] last visible key, or null: the query's own index
  const int* q_lo;          // [Tk] bounds on the queries that see each key, or null (causal self-attention)
  const int* q_hi;
  const float* lse;         // [nq, T]
  const float* delta;       // [nq, T]
  __nv_bfloat16* dq;        // [T, nq, d]
  __nv_bfloat16* dk;        // [Tk, nkv, d]
  __nv_bfloat16* dv;        // [Tk, nkv, d]
  int* status;
  float* partial;           // head-split mode: [2 (dv, dk), splits, Tk, nkv, d] fp32 partial sums, else null
  int splits;               // CTAs per (key tile, kv head); each takes qpg / splits query heads
};

// what the dq kernel forms delta from (o null: it is given)
struct DeltaParams {
  const __nv_bfloat16 *o, *dout;   // [T, nq, d]
  float* delta;                    // [nq, T]
};

// K-major operand: tile of `rows` x D stored as D/64 boxes of [rows x 64]; kk-th 16-wide slice of the reduction dim
__device__ __forceinline__ uint64_t kdesc(uint32_t base, int kk, int rows) {
  return make_smem_desc_sw128(base + (kk >> 2) * (rows * 128) + (kk & 3) * 32, 16, 1024);
}
// MN-major B operand: tile of `rows` (reduction dim) x D (N dim) in the same box layout; kk-th 16-row slice
__device__ __forceinline__ uint64_t mndesc(uint32_t base, int kk, int rows) {
  return make_smem_desc_sw128(base + kk * 2048, rows * 128, 1024);
}

__host__ __device__ constexpr uint32_t idesc(int m, int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(b_mn ? 1 : 0) << 16) | (uint32_t(n >> 3) << 17) |
         (uint32_t(m >> 4) << 24);
}

// one TMEM lane's D accumulator columns -> a bf16 row in global memory
template <int COLS>
__device__ __forceinline__ void store_acc_row(uint32_t taddr, __nv_bfloat16* dst, bool ok) {
#pragma unroll 1
  for (int c = 0; c < COLS; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    if (ok) {
#pragma unroll
      for (int e = 0; e < 32; e += 8) {
        uint4 o;
        o.x = pack_bf16x2(__uint_as_float(v[e]), __uint_as_float(v[e + 1]));
        o.y = pack_bf16x2(__uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]));
        o.z = pack_bf16x2(__uint_as_float(v[e + 4]), __uint_as_float(v[e + 5]));
        o.w = pack_bf16x2(__uint_as_float(v[e + 6]), __uint_as_float(v[e + 7]));
        *reinterpret_cast<uint4*>(dst + c + e) = o;
      }
    }
  }
}

// one TMEM lane's accumulator columns -> an fp32 row in global memory
template <int COLS>
__device__ __forceinline__ void store_acc_row_f32(uint32_t taddr, float* dst, bool ok) {
#pragma unroll 1
  for (int c = 0; c < COLS; c += 32) {
    uint32_t v[32];
    tmem_ld_32x32(taddr + c, v);
    tmem_ld_wait();
    if (ok) {
#pragma unroll
      for (int e = 0; e < 32; e += 4)
        *reinterpret_cast<float4*>(dst + c + e) =
            make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]), __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]));
    }
  }
}

__device__ __forceinline__ void drain(uint64_t* bar, uint32_t parity) {
  uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(smem_u32(bar), parity))
    if (globaltimer_ns() - t0 > 200000000ull) break;
}

// ---------------------------------------------------------------------------------------------------- delta
// One row's delta is the sum of D / 8 terms of eight channels, each held by a lane: the kernel below and the dq kernel form and add
// them the same way, so the bits do not depend on which of them forms delta.
__device__ __forceinline__ float delta_term(const uint4& o, const uint4& dout) {
  const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&o), *y = reinterpret_cast<const __nv_bfloat162*>(&dout);
  float acc = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(x[e]), g = __bfloat1622float2(y[e]);
    acc += f.x * g.x + f.y * g.y;
  }
  return acc;
}
template <int LANES>
__device__ __forceinline__ float delta_sum(float acc) {
#pragma unroll
  for (int s = LANES / 2; s; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  return acc;
}

// D / 8 lanes per (token, head) row, 16-byte loads, 4 rows per lane group in flight: bound by reading O and dO once.
template <int D>
__global__ void __launch_bounds__(256)
attn_bwd_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                      float* __restrict__ delta, int T, int nq) {
  constexpr int LANES = D / 8, ROWS = 256 / LANES, UNROLL = 4;
  const long long rows = (long long)T * nq;
  const long long base = (long long)blockIdx.x * ROWS * UNROLL + threadIdx.x / LANES;
  const int c = (threadIdx.x % LANES) * 8;
  uint4 a[UNROLL], b[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const long long w = base + u * ROWS;
    const bool in = w < rows;
    a[u] = in ? *reinterpret_cast<const uint4*>(o + w * D + c) : make_uint4(0, 0, 0, 0);
    b[u] = in ? *reinterpret_cast<const uint4*>(dout + w * D + c) : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const long long w = base + u * ROWS;
    const float acc = delta_sum<LANES>(delta_term(a[u], b[u]));
    if (c == 0 && w < rows) delta[(w % nq) * T + w / nq] = acc;
  }
}

// ---------------------------------------------------------------------------------------------------- dQ
// Order of the products:  S0 dP0 S1 | dP(j+1) dQ(j) S(j+2) | ...  Two score buffers, one dP buffer: dP(j+1) starts as soon
// as the element-wise warps hold dP(j) in registers and runs under their arithmetic; dS(j) overwrites the scores it came
// from, so dQ(j) frees the buffer S(j+2) goes to.  K(j) is needed from S(j) to dQ(j): three stages of K, two of V.
// Bound: 3 x 512 tensor cycles and 1024 MUFU cycles per 128 x 128 block.
template <int D>
struct DqSmem {
  static constexpr int TILE = TM * D * 2;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = TILE;
  static constexpr int OFF_K = 2 * TILE;               // 3 stages
  static constexpr int OFF_V = OFF_K + 3 * TILE;       // 2 stages
  static constexpr int OFF_BAR = OFF_V + 2 * TILE;
  static constexpr int TOTAL = OFF_BAR + 1024 + 1024;
};

template <int D>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const BwdParams p, const DeltaParams dp_) {
  using L = DqSmem<D>;
  constexpr int NBOX = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t COL_S = 0, COL_DP = 256, COL_DQ = 384;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars;             // 1
  uint64_t* k_full = bars + 1;         // 3
  uint64_t* k_empty = bars + 4;        // 3
  uint64_t* v_full = bars + 7;         // 2
  uint64_t* v_empty = bars + 9;        // 2
  uint64_t* s_full = bars + 11;        // 2
  uint64_t* dp_full = bars + 13;       // 1
  uint64_t* dp_empty = bars + 14;      // 1
  uint64_t* ds_full = bars + 15;       // 2, by turns: a warp that has nothing to mask may be a block ahead of the others
  uint64_t* dq_full = bars + 17;       // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int m_tile = (gridDim.x - 1 - blockIdx.x) / p.nq;      // long tiles of every head first
  const int head = blockIdx.x % p.nq;
  const int kvh = head / (p.nq / p.nkv);
  const int m0 = m_tile * TM;
  __shared__ int s_rng[8];
  tile_range_partial(p.k_lo, p.k_hi, m0, p.T, s_rng);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(smem_u32(q_full), 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(smem_u32(&k_full[i]), 1);
      mbar_init(smem_u32(&k_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&v_full[i]), 1);
      mbar_init(smem_u32(&v_empty[i]), 1);
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&ds_full[i]), 8);
    }
    mbar_init(smem_u32(dp_full), 1);
    mbar_init(smem_u32(dp_empty), 8);
    mbar_init(smem_u32(dq_full), 1);
    fence_barrier_init();
    fence_proxy_async_smem();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_do);
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
  const int kmin = warp_uniform(tile_range_min(s_rng)), kmax = warp_uniform(tile_range_max(s_rng));
  const int kb0 = kmin / TM;
  const int nblk = kmax >= kmin ? kmax / TM - kb0 + 1 : 0;

  if (warp < 4) {
    MCB_REGS_CONTROL();
    if (warp == 0 && lane == 0 && nblk > 0) {
      // ---------------------------------------------------------------- TMA producer
      mbar_expect_tx(smem_u32(q_full), 2 * L::TILE);
#pragma unroll
      for (int b = 0; b < NBOX; ++b) {
        tma_load_2d(smem_u32(smem + L::OFF_Q + b * TM * 128), &tm_q, head * D + b * 64, m0, smem_u32(q_full));
        tma_load_2d(smem_u32(smem + L::OFF_DO + b * TM * 128), &tm_do, head * D + b * 64, m0, smem_u32(q_full));
      }
      int nk = 0, nv = 0;
      for (int j = 0; j < nblk; ++j) {
        const uint32_t ks = j % 3, kp = (j / 3) & 1, vs = j & 1, vp = (j >> 1) & 1;
        const int n0 = (kb0 + j) * TM;
        if (!mbar_wait(smem_u32(&k_empty[ks]), kp ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(smem_u32(&k_full[ks]), L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          tma_load_2d(smem_u32(smem + L::OFF_K + ks * L::TILE + b * TM * 128), &tm_k, kvh * D + b * 64, n0,
                      smem_u32(&k_full[ks]));
        ++nk;
        if (!mbar_wait(smem_u32(&v_empty[vs]), vp ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(smem_u32(&v_full[vs]), L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          tma_load_2d(smem_u32(smem + L::OFF_V + vs * L::TILE + b * TM * 128), &tm_v, kvh * D + b * 64, n0,
                      smem_u32(&v_full[vs]));
        ++nv;
      }
      // the last loads land before the CTA exits
      for (int i = (nk > 3 ? nk - 3 : 0); i < nk; ++i) drain(&k_full[i % 3], (i / 3) & 1);
      for (int i = (nv > 2 ? nv - 2 : 0); i < nv; ++i) drain(&v_full[i & 1], (i >> 1) & 1);
      drain(q_full, 0);
    } else if (warp == 1 && nblk > 0) {
      // ---------------------------------------------------------------- MMA issuer: a whole warp, see umma_f16_warp
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = idesc(TM, TM, false);
      constexpr uint32_t idesc_dq = idesc(TM, D, true);
      const uint32_t sq = smem_u32(smem + L::OFF_Q), sdo = smem_u32(smem + L::OFF_DO);
      auto issue_s = [&](int j) -> bool {
        const uint32_t ks = j % 3, kp = (j / 3) & 1;
        if (!mbar_wait_warp(smem_u32(&k_full[ks]), kp, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        const uint32_t sk = smem_u32(smem + L::OFF_K + ks * L::TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_warp(leader, tmem + COL_S + (j & 1) * TM, kdesc(sq, kk, TM), kdesc(sk, kk, TM), idesc_s, kk ? 1u : 0u);
        umma_commit_warp(leader, smem_u32(&s_full[j & 1]));
        return true;
      };
      auto issue_dp = [&](int j) -> bool {
        const uint32_t vs = j & 1, vp = (j >> 1) & 1;
        if (!mbar_wait_warp(smem_u32(&v_full[vs]), vp, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
        if (j > 0 && !mbar_wait_warp(smem_u32(dp_empty), (j & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) return false;
        tc_fence_after();
        const uint32_t sv = smem_u32(smem + L::OFF_V + vs * L::TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_warp(leader, tmem + COL_DP, kdesc(sdo, kk, TM), kdesc(sv, kk, TM), idesc_s, kk ? 1u : 0u);
        umma_commit_warp(leader, smem_u32(dp_full));
        umma_commit_warp(leader, smem_u32(&v_empty[vs]));
        return true;
      };
      bool ok = mbar_wait_warp(smem_u32(q_full), 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      if (ok) ok = issue_s(0);
      if (ok) ok = issue_dp(0);
      if (ok && nblk > 1) ok = issue_s(1);
      for (int j = 0; j < nblk && ok; ++j) {
        if (j + 1 < nblk && !issue_dp(j + 1)) { ok = false; break; }
        if (!mbar_wait_warp(smem_u32(&ds_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sk = smem_u32(smem + L::OFF_K + (j % 3) * L::TILE);
        const uint32_t ads = tmem + COL_S + (j & 1) * TM;
#pragma unroll
        for (int kk = 0; kk < TM / 16; ++kk)     // dS: 32 packed columns at the start of each 64-column half
          umma_f16_ts_warp(leader, tmem + COL_DQ, ads + (kk >> 2) * HALF + (kk & 3) * 8, mndesc(sk, kk, TM), idesc_dq,
                      (j | kk) ? 1u : 0u);
        umma_commit_warp(leader, smem_u32(&k_empty[j % 3]));
        if (j + 2 < nblk) ok = issue_s(j + 2);
      }
      if (ok) umma_commit_warp(leader, smem_u32(dq_full));
    }
  } else {
    MCB_REGS_MATH();
    const int q = warp & 3;
    const int grp = (warp - 4) >> 2;
    const int r = q * 32 + lane;
    const int i = m0 + r;
    const bool row_ok = i < p.T;
    int lo, hi;
    attn_row_range(p.k_lo, p.k_hi, i, p.T, lo, hi);
    if (lo > hi) lo = hi = 0x40000000;            // sees nothing: a range no key index reaches
    const unsigned span = (unsigned)(hi - lo);    // key k is visible iff (unsigned)(k - lo) <= span
    // a query that sees nothing has lse = -inf; its probabilities are masked below, keep the arithmetic finite
    const float lse_i = row_ok ? p.lse[(long long)head * p.T + i] : 0.f;
    const float lse2 = (lse_i == -INFINITY) ? 0.f : lse_i * LOG2E;
    float dl;
    if (dp_.o == nullptr) {
      dl = row_ok ? p.delta[(long long)head * p.T + i] : 0.f;
    } else {
      // delta of the tile's rows while the first tiles are on their way, 16 rows a warp, with the lanes of delta's own kernel
      constexpr int LANES = D / 8, ROWS = 32 / LANES;
      float* s_delta = reinterpret_cast<float*>(smem + L::OFF_BAR + 512);   // [TM], behind the barriers
      const int row0 = (warp - 4) * 16 + lane / LANES;
      uint4 a[16 / ROWS], b[16 / ROWS];
#pragma unroll
      for (int u = 0; u < 16 / ROWS; ++u) {
        const long long at = ((long long)min(m0 + row0 + u * ROWS, p.T - 1) * p.nq + head) * D + lane % LANES * 8;
        a[u] = *reinterpret_cast<const uint4*>(dp_.o + at);
        b[u] = *reinterpret_cast<const uint4*>(dp_.dout + at);
      }
#pragma unroll
      for (int u = 0; u < 16 / ROWS; ++u) {
        const float acc = delta_sum<LANES>(delta_term(a[u], b[u]));
        if (lane % LANES == 0) s_delta[row0 + u * ROWS] = acc;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");       // the eight element-wise warps, before any bounded wait
      dl = row_ok ? s_delta[r] : 0.f;
      if (row_ok && grp == 0) dp_.delta[(long long)head * p.T + i] = dl;
    }
    const uint64_t cc = f32x2(p.scale_log2, p.scale_log2), nl = f32x2(-lse2, -lse2), nd = f32x2(-dl, -dl);
    const uint64_t sc = f32x2(p.scale, p.scale);
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    bool ok = true;
    for (int j = 0; j < nblk && ok; ++j) {
      const uint32_t ts = tmem + lane_addr + COL_S + (j & 1) * TM + grp * HALF;
      const uint32_t td = tmem + lane_addr + COL_DP + grp * HALF;
      const int n0 = (kb0 + j) * TM + grp * HALF;
      const Seen seen[2] = {seen_keys(lo, hi, n0), seen_keys(lo, hi, n0 + 32)};
      uint32_t pr[HALF];
      if (!mbar_wait(smem_u32(&s_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      tmem_ld_32x32_x64(ts, pr);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (seen[c] == Seen::NONE) continue;
#pragma unroll
        for (int e = 32 * c; e < 32 * c + 32; e += 2) {
          const float2 x = f32x2_split(fma_f32x2(f32x2(__uint_as_float(pr[e]), __uint_as_float(pr[e + 1])), cc, nl));
          pr[e] = __float_as_uint(ex2_ftz(x.x));
          pr[e + 1] = __float_as_uint(ex2_ftz(x.y));
        }
      }
      if (!mbar_wait(smem_u32(dp_full), j & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t dp[HALF];
      tmem_ld_32x32_x64(td, dp);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(dp_empty));   // dP is in registers: the next dO V^T may start
      uint32_t pk[HALF / 2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (seen[c] == Seen::NONE) {
#pragma unroll
          for (int e = 16 * c; e < 16 * c + 16; ++e) pk[e] = 0;
          continue;
        }
        const bool all = seen[c] == Seen::ALL;
#pragma unroll
        for (int e = 32 * c; e < 32 * c + 32; e += 2) {
          const uint64_t d2 = add_f32x2(f32x2(__uint_as_float(dp[e]), __uint_as_float(dp[e + 1])), nd);
          float2 x = f32x2_split(mul_f32x2(mul_f32x2(d2, f32x2(__uint_as_float(pr[e]), __uint_as_float(pr[e + 1]))), sc));
          if (!all) {                             // a masked pair contributes zero whatever its P and dP are
            x.x = (unsigned)(n0 + e - lo) <= span ? x.x : 0.f;
            x.y = (unsigned)(n0 + e + 1 - lo) <= span ? x.y : 0.f;
          }
          pk[e >> 1] = pack_bf16x2(x.x, x.y);
        }
      }
      tmem_st_32x32(ts, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ds_full[j & 1]));
    }
    __nv_bfloat16* row = p.dq + ((long long)i * p.nq + head) * D + grp * (D / 2);   // each group writes half of the row
    if (nblk <= 0) {
      // no row of this tile sees any key: its queries get a zero gradient
      if (row_ok) {
#pragma unroll
        for (int c = 0; c < D / 16; ++c) reinterpret_cast<uint4*>(row)[c] = make_uint4(0, 0, 0, 0);
      }
    } else if (ok && mbar_wait(smem_u32(dq_full), 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      store_acc_row<D / 2>(tmem + lane_addr + COL_DQ + grp * (D / 2), row, row_ok);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------- dK / dV
// The accumulators take half of TMEM, one S^T and one dP^T block the other half.  Order of the products:
//   S0 | dP(j) dV(j) S(j+1) dK(j) | dP(j+1) ...
// P(j) overwrites S(j) and dS(j) overwrites dP(j); the exponentials of block j+1 run under dK(j) and dP(j+1), the dS
// arithmetic of block j under dV(j) and S(j+1), so the tensor core has work while either is computed.
// Bound: 4 x 512 tensor cycles per 128 x 128 block.
template <int D>
struct DkvSmem {
  static constexpr int TILE = TM * D * 2;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = TILE;
  static constexpr int OFF_Q = 2 * TILE;                // 2 stages
  static constexpr int OFF_DO = OFF_Q + 2 * TILE;       // 2 stages
  static constexpr int OFF_COL = OFF_DO + 2 * TILE;     // 2 buffers: per-query lse / delta / k_lo / k_hi, then of every 32
                                                        // queries the largest and smallest k_lo, smallest and largest k_hi
  static constexpr int COL_BYTES = 4 * TM * 4 + 4 * 16;
  static constexpr int OFF_BAR = OFF_COL + 2 * COL_BYTES;
  static constexpr int TOTAL = OFF_BAR + 1024 + 1024;
};

template <int D>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                    const BwdParams p) {
  using L = DkvSmem<D>;
  constexpr int NBOX = D / 64;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 384;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* kv_full = bars;            // 1
  uint64_t* q_full = bars + 1;         // 2
  uint64_t* q_empty = bars + 3;        // 2
  uint64_t* do_full = bars + 5;        // 2
  uint64_t* do_empty = bars + 7;       // 2
  uint64_t* s_full = bars + 9;         // 1
  uint64_t* p_full = bars + 10;        // 2: the first and the second 32 queries of each 64-query half
  uint64_t* dp_full = bars + 12;       // 1
  uint64_t* ds_full = bars + 13;       // 2
  uint64_t* out_full = bars + 15;      // 1
  uint64_t* col_full = bars + 16;      // 2
  uint64_t* col_empty = bars + 18;     // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* i_end_slot = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int group_cta = blockIdx.x % (p.nkv * p.splits);         // key tiles ascend slowest: long ones first when causal
  const int kvh = group_cta / p.splits, split = group_cta % p.splits;
  const int qpg = p.nq / p.nkv;
  const int n0 = blockIdx.x / (p.nkv * p.splits) * TM;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(smem_u32(kv_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&q_full[i]), 1);
      mbar_init(smem_u32(&q_empty[i]), 1);
      mbar_init(smem_u32(&do_full[i]), 1);
      mbar_init(smem_u32(&do_empty[i]), 1);
      mbar_init(smem_u32(&col_full[i]), 32);
      mbar_init(smem_u32(&col_empty[i]), 8);
      mbar_init(smem_u32(&p_full[i]), 8);
      mbar_init(smem_u32(&ds_full[i]), 8);
    }
    mbar_init(smem_u32(s_full), 1);
    mbar_init(smem_u32(dp_full), 1);
    mbar_init(smem_u32(out_full), 1);
    fence_barrier_init();
    fence_proxy_async_smem();
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_do);
  }
  __shared__ int s_rng[8];
  if (p.q_lo != nullptr) {
    tile_range_partial(p.q_lo, p.q_hi, n0, p.Tk, s_rng);
  } else if (warp == 2) {
    // causal self-attention: the last query that can see a key of this tile is the largest i with k_lo[i] <= last key (k_lo =
    // sequence starts, sorted); the first one is the tile's first key itself.  The lanes look at 32 places at a time: a step
    // waits for memory, and halving took 12 of them at 4096 tokens before the CTA's first load.
    const int n_last = min(n0 + TM - 1, p.Tk - 1);
    int lo = n_last, hi = p.T - 1;                 // the last one lies in [lo, hi]
    while (lo < hi) {
      const int step = (hi - lo + 31) / 32, i = min(lo + (lane + 1) * step, hi);
      const unsigned past = __ballot_sync(0xffffffffu, p.k_lo[i] > n_last);
      const int c = past ? __ffs(past) - 1 : 32;    // places that still see the key
      const int from = lo;
      if (c > 0) lo = min(from + c * step, hi);
      if (c < 32) hi = min(min(from + (c + 1) * step, hi) - 1, hi);
    }
    if (lane == 0) {
      i_end_slot[0] = n0;
      i_end_slot[1] = lo;
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  const int i_first = warp_uniform(p.q_lo ? tile_range_min(s_rng) : i_end_slot[0]);
  const int i_last = warp_uniform(p.q_lo ? min(tile_range_max(s_rng), p.T - 1) : i_end_slot[1]);
  const int qb0 = i_first / TM;
  const int nqb = i_last >= i_first ? i_last / TM - qb0 + 1 : 0;    // 0: no query sees a key of this tile
  const int hps = qpg / p.splits;                 // query heads handled by this CTA
  const int h_first = kvh * qpg + split * hps;
  const int iters = hps * nqb;

  if (warp < 4) {
    MCB_REGS_CONTROL();
    if (warp == 0 && lane == 0 && iters > 0) {
      // ---------------------------------------------------------------- TMA producer
      mbar_expect_tx(smem_u32(kv_full), 2 * L::TILE);
#pragma unroll
      for (int b = 0; b < NBOX; ++b) {
        tma_load_2d(smem_u32(smem + L::OFF_K + b * TM * 128), &tm_k, kvh * D + b * 64, n0, smem_u32(kv_full));
        tma_load_2d(smem_u32(smem + L::OFF_V + b * TM * 128), &tm_v, kvh * D + b * 64, n0, smem_u32(kv_full));
      }
      int nQ = 0, nD = 0, h = h_first, qb = 0;
      for (int it = 0; it < iters; ++it) {
        const uint32_t st = it & 1, ph = (it >> 1) & 1;
        const int i0 = (qb0 + qb) * TM;
        if (!mbar_wait(smem_u32(&q_empty[st]), ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(smem_u32(&q_full[st]), L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          tma_load_2d(smem_u32(smem + L::OFF_Q + st * L::TILE + b * TM * 128), &tm_q, h * D + b * 64, i0,
                      smem_u32(&q_full[st]));
        ++nQ;
        if (!mbar_wait(smem_u32(&do_empty[st]), ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        mbar_expect_tx(smem_u32(&do_full[st]), L::TILE);
#pragma unroll
        for (int b = 0; b < NBOX; ++b)
          tma_load_2d(smem_u32(smem + L::OFF_DO + st * L::TILE + b * TM * 128), &tm_do, h * D + b * 64, i0,
                      smem_u32(&do_full[st]));
        ++nD;
        if (++qb == nqb) { qb = 0; ++h; }
      }
      for (int i = (nQ > 2 ? nQ - 2 : 0); i < nQ; ++i) drain(&q_full[i & 1], (i >> 1) & 1);
      for (int i = (nD > 2 ? nD - 2 : 0); i < nD; ++i) drain(&do_full[i & 1], (i >> 1) & 1);
      drain(kv_full, 0);
    } else if (warp == 1 && iters > 0) {
      // ---------------------------------------------------------------- MMA issuer: a whole warp, see umma_f16_warp
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = idesc(TM, TM, false);
      constexpr uint32_t idesc_o = idesc(TM, D, true);
      const uint32_t sk = smem_u32(smem + L::OFF_K), sv = smem_u32(smem + L::OFF_V);
      auto issue_s = [&](int it) -> bool {
        if (!mbar_wait_warp(smem_u32(&q_full[it & 1]), (it >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
        tc_fence_after();
        const uint32_t sq = smem_u32(smem + L::OFF_Q + (it & 1) * L::TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_warp(leader, tmem + COL_S, kdesc(sk, kk, TM), kdesc(sq, kk, TM), idesc_s, kk ? 1u : 0u);
        umma_commit_warp(leader, smem_u32(s_full));
        return true;
      };
      bool ok = mbar_wait_warp(smem_u32(kv_full), 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      if (ok) ok = issue_s(0);
      for (int it = 0; it < iters && ok; ++it) {
        const uint32_t st = it & 1, ph = (it >> 1) & 1;
        const uint32_t sq = smem_u32(smem + L::OFF_Q + st * L::TILE);
        const uint32_t sdo = smem_u32(smem + L::OFF_DO + st * L::TILE);
        if (!mbar_wait_warp(smem_u32(&do_full[st]), ph, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_warp(leader, tmem + COL_DP, kdesc(sv, kk, TM), kdesc(sdo, kk, TM), idesc_s, kk ? 1u : 0u);
        umma_commit_warp(leader, smem_u32(dp_full));
        // P, dS: 32 packed columns at the start of each 64-column half; part u of them is ready first in both halves
        auto product = [&](uint32_t col_d, uint32_t col_a, uint32_t sb, uint64_t* full) -> bool {
          for (int u = 0; u < 2; ++u) {
            if (!mbar_wait_warp(smem_u32(&full[u]), it & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
            tc_fence_after();
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int kk = (v >> 1) * 4 + u * 2 + (v & 1);
              umma_f16_ts_warp(leader, tmem + col_d, tmem + col_a + (kk >> 2) * HALF + (kk & 3) * 8, mndesc(sb, kk, TM), idesc_o,
                          (it | u | v) ? 1u : 0u);
            }
          }
          return true;
        };
        if (!product(COL_DV, COL_S, sdo, p_full)) { ok = false; break; }
        umma_commit_warp(leader, smem_u32(&do_empty[st]));
        if (it + 1 < iters && !issue_s(it + 1)) { ok = false; break; }
        if (!product(COL_DK, COL_DP, sq, ds_full)) { ok = false; break; }
        umma_commit_warp(leader, smem_u32(&q_empty[st]));
      }
      if (ok) umma_commit_warp(leader, smem_u32(out_full));
    } else if (warp == 2) {
      // ---------------------------------------------------------------- per-query values of the coming blocks
      // A block's values are fetched while the block before it is laid down: their latency is longer than a block's products.
      int h = h_first, qb = 0;
      float lse[4], dl[4];
      int klo[4], khi[4];
      auto fetch = [&]() {
        const int i0 = (qb0 + qb) * TM;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * 32 + lane;
          lse[u] = i < p.T ? p.lse[(long long)h * p.T + i] : 0.f;
          dl[u] = i < p.T ? p.delta[(long long)h * p.T + i] : 0.f;
          attn_row_range(p.k_lo, p.k_hi, i, p.T, klo[u], khi[u]);
        }
        if (++qb == nqb) { qb = 0; ++h; }
      };
      if (iters > 0) fetch();
#pragma unroll 1
      for (int it = 0; it < iters; ++it) {
        const uint32_t b = it & 1, ph = (it >> 1) & 1;
        float* c_lse = reinterpret_cast<float*>(smem + L::OFF_COL + b * L::COL_BYTES);
        float* c_delta = c_lse + TM;
        int* c_lo = reinterpret_cast<int*>(c_delta + TM);
        int* c_hi = c_lo + TM;
        float x_lse[4], x_dl[4];
        int x_lo[4], x_hi[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          x_lse[u] = (lse[u] == -INFINITY) ? 0.f : -lse[u] * LOG2E;    // -inf: such a query sees nothing, masked below
          x_dl[u] = -dl[u];
          x_lo[u] = klo[u];
          x_hi[u] = khi[u];
        }
        if (it + 1 < iters) fetch();
        if (!mbar_wait(smem_u32(&col_empty[b]), ph ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = u * 32 + lane;
          c_lse[c] = x_lse[u];
          c_delta[c] = x_dl[u];
          c_lo[c] = x_lo[u];
          c_hi[c] = x_hi[u];
          const bool sees = x_lo[u] <= x_hi[u];
          const int4 edge = make_int4(__reduce_max_sync(0xffffffffu, x_lo[u]), __reduce_min_sync(0xffffffffu, sees ? x_lo[u] : INT_MAX),
                                      __reduce_min_sync(0xffffffffu, x_hi[u]), __reduce_max_sync(0xffffffffu, sees ? x_hi[u] : -1));
          if (lane == 0) reinterpret_cast<int4*>(c_hi + TM)[u] = edge;
        }
        mbar_arrive(smem_u32(&col_full[b]));
      }
    }
  } else {
    MCB_REGS_MATH();
    const int q = warp & 3;
    const int grp = (warp - 4) >> 2;
    const int r = q * 32 + lane;            // key row of this thread
    const int n = n0 + r;
    const bool row_ok = n < p.Tk;
    const uint32_t lane_addr = uint32_t(q * 32) << 16;
    const uint32_t ts = tmem + lane_addr + COL_S + grp * HALF, td = tmem + lane_addr + COL_DP + grp * HALF;
    const uint64_t cc = f32x2(p.scale_log2, p.scale_log2), sc = f32x2(p.scale, p.scale);
    bool ok = true;
    for (int it = 0; it < iters && ok; ++it) {
      const uint32_t b = it & 1;
      const float* c_lse = reinterpret_cast<const float*>(smem + L::OFF_COL + b * L::COL_BYTES) + grp * HALF;
      const float* c_delta = c_lse + TM;
      const int* c_lo = reinterpret_cast<const int*>(c_delta + TM);
      const int* c_hi = c_lo + TM;
      const int4* c_edge = reinterpret_cast<const int4*>(c_hi + TM - grp * HALF) + 2 * grp;
      if (!mbar_wait(smem_u32(&col_full[b]), (it >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
      // every query of the block sees this key: largest lower bound <= n <= smallest upper bound
      const bool full = __all_sync(0xffffffffu, row_ok && max(c_edge[0].x, c_edge[1].x) <= n && n <= min(c_edge[0].z, c_edge[1].z));
      uint32_t seen[2] = {0xffffffffu, 0xffffffffu};   // bit e: this key is visible to query e of the half block
      if (!full) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int4 x = c_edge[c];
          const Seen some = seen_of(row_ok && x.x <= n && n <= x.z, row_ok && x.y <= n && n <= x.w);
          if (some == Seen::ALL) continue;
          seen[c] = 0u;
          if (some == Seen::NONE) continue;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const int4 a = *reinterpret_cast<const int4*>(c_lo + 32 * c + e), z = *reinterpret_cast<const int4*>(c_hi + 32 * c + e);
            const int aa[4] = {a.x, a.y, a.z, a.w}, zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) seen[c] |= (row_ok && aa[u] <= n && n <= zz[u]) ? 1u << (e + u) : 0u;
          }
        }
      }
      if (!mbar_wait(smem_u32(s_full), it & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t pr[HALF];
      tmem_ld_32x32_x64(ts, pr);
      tmem_ld_wait();
#pragma unroll
      for (int u2 = 0; u2 < 2; ++u2) {
        uint32_t pk[16];
#pragma unroll
        for (int e = u2 * 32; e < u2 * 32 + 32; e += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(c_lse + e);
          const float2 x = f32x2_split(fma_f32x2(f32x2(__uint_as_float(pr[e]), __uint_as_float(pr[e + 1])), cc, f32x2(l4.x, l4.y)));
          const float2 y = f32x2_split(fma_f32x2(f32x2(__uint_as_float(pr[e + 2]), __uint_as_float(pr[e + 3])), cc, f32x2(l4.z, l4.w)));
          float v[4] = {ex2_ftz(x.x), ex2_ftz(x.y), ex2_ftz(y.x), ex2_ftz(y.y)};
          if (!full) {
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = (seen[e >> 5] >> ((e + u) & 31)) & 1u ? v[u] : 0.f;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) pr[e + u] = __float_as_uint(v[u]);
          pk[(e & 31) >> 1] = pack_bf16x2(v[0], v[1]);
          pk[((e & 31) >> 1) + 1] = pack_bf16x2(v[2], v[3]);
        }
        tmem_st_32x16(ts + u2 * 16, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&p_full[u2]));
      }
      if (!mbar_wait(smem_u32(dp_full), it & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t dp[HALF];
      tmem_ld_32x32_x64(td, dp);
      tmem_ld_wait();
#pragma unroll
      for (int u2 = 0; u2 < 2; ++u2) {
        uint32_t pk[16];
#pragma unroll
        for (int e = u2 * 32; e < u2 * 32 + 32; e += 4) {
          const float4 d4 = *reinterpret_cast<const float4*>(c_delta + e);
          const uint64_t dx = add_f32x2(f32x2(__uint_as_float(dp[e]), __uint_as_float(dp[e + 1])), f32x2(d4.x, d4.y));
          const uint64_t dy = add_f32x2(f32x2(__uint_as_float(dp[e + 2]), __uint_as_float(dp[e + 3])), f32x2(d4.z, d4.w));
          float2 x = f32x2_split(mul_f32x2(mul_f32x2(dx, f32x2(__uint_as_float(pr[e]), __uint_as_float(pr[e + 1]))), sc));
          float2 y = f32x2_split(mul_f32x2(mul_f32x2(dy, f32x2(__uint_as_float(pr[e + 2]), __uint_as_float(pr[e + 3]))), sc));
          if (!full) {                              // a masked pair contributes zero whatever its dP is
            const uint32_t m = seen[e >> 5] >> (e & 31);
            x.x = m & 1u ? x.x : 0.f;
            x.y = m & 2u ? x.y : 0.f;
            y.x = m & 4u ? y.x : 0.f;
            y.y = m & 8u ? y.y : 0.f;
          }
          pk[(e & 31) >> 1] = pack_bf16x2(x.x, x.y);
          pk[((e & 31) >> 1) + 1] = pack_bf16x2(y.x, y.y);
        }
        tmem_st_32x16(td + u2 * 16, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ds_full[u2]));
      }
      if (lane == 0) mbar_arrive(smem_u32(&col_empty[b]));
    }
    // group 0 writes dV, group 1 writes dK
    const long long row_off = ((long long)n * p.nkv + kvh) * D;
    const long long plane = (long long)p.Tk * p.nkv * D;
    if (iters == 0) {
      // no query sees this tile's keys: zero gradients (the accumulators were never written)
      if (row_ok) {
        if (p.partial == nullptr) {
          uint4* dst = reinterpret_cast<uint4*>((grp == 0 ? p.dv : p.dk) + row_off);
#pragma unroll 1
          for (int c = 0; c < D / 8; ++c) dst[c] = make_uint4(0, 0, 0, 0);
        } else {
          uint4* dst = reinterpret_cast<uint4*>(p.partial + ((long long)grp * p.splits + split) * plane + row_off);
#pragma unroll 1
          for (int c = 0; c < D / 4; ++c) dst[c] = make_uint4(0, 0, 0, 0);
        }
      }
    } else if (ok && mbar_wait(smem_u32(out_full), 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      const uint32_t acc = tmem + lane_addr + (grp == 0 ? COL_DV : COL_DK);
      if (p.partial == nullptr) store_acc_row<D>(acc, (grp == 0 ? p.dv : p.dk) + row_off, row_ok);
      else store_acc_row_f32<D>(acc, p.partial + ((long long)grp * p.splits + split) * plane + row_off, row_ok);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// sums the head-split partials: out[i] = sum_s partial[s][i] (fp32 -> bf16), 8 elements per thread
__global__ void attn_bwd_reduce_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dv,
                                       __nv_bfloat16* __restrict__ dk, long long plane, int splits) {
  const long long i8 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i8 >= plane) return;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int s2 = 0; s2 < splits; ++s2) {
      const float* src = partial + ((long long)which * splits + s2) * plane + i8;
      const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
      acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
      acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
    }
    uint4 o;
    o.x = pack_bf16x2(acc[0], acc[1]);
    o.y = pack_bf16x2(acc[2], acc[3]);
    o.z = pack_bf16x2(acc[4], acc[5]);
    o.w = pack_bf16x2(acc[6], acc[7]);
    *reinterpret_cast<uint4*>((which == 0 ? dv : dk) + i8) = o;
  }
}

template <int D>
int launch_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, float* delta, bool delta_given,
               const BwdParams& p, cudaStream_t stream) {
  // the tensor maps first: they refuse operands that are not on a 16-byte boundary, which the dq kernel would fault on
  CUtensorMap tq, tdo, tk, tv;
  const long long wq = (long long)p.nq * D, wk = (long long)p.nkv * D;
  int rc = 0;
  if ((rc = make_tmap_2d_bf16(&tq, q, wq, p.T, wq, 64, TM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tdo, dout, wq, p.T, wq, 64, TM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tk, k, wk, p.Tk, wk, 64, TM))) return rc;
  if ((rc = make_tmap_2d_bf16(&tv, v, wk, p.Tk, wk, 64, TM))) return rc;
  cudaError_t e = cudaSuccess;
  DeltaParams dp{nullptr, nullptr, nullptr};
  if (!delta_given) {
    if (reinterpret_cast<uintptr_t>(o) & 15) return -6;
    // In the dq kernel delta delays the first block, by twice as many rows of loads for heads of 128; the kernel of its own costs a
    // launch and a pass.  delta + dq + dk/dv, us, own kernel and in dq: 4095 tokens, 64 heads of 64, window 128 284 / 250, 4096,
    // 24 of 64 320 / 315, 333, 4 of 64 32 / 28; 3000, 9 of 128 203 / 186, 2048, 32 of 128 194 / 196, 8192, 32 of 128 561 / 573.
    const long long rows = (long long)p.T * p.nq;
    if (D == 64 || rows <= 32768) {
      dp = DeltaParams{(const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta};
    } else {
      constexpr int PER = 4 * 256 / (D / 8);    // rows of a block
      attn_bwd_delta_kernel<D><<<(unsigned)((rows + PER - 1) / PER), 256, 0, stream>>>(
          (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, p.T, p.nq);
      e = cudaGetLastError();
      if (e != cudaSuccess) return (int)e;
    }
  }
  static bool cfg = false;
  if (!cfg) {
    e = cudaFuncSetAttribute(attn_bwd_dq_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, DqSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(attn_bwd_dkv_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvSmem<D>::TOTAL);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  const int tiles = (p.T + TM - 1) / TM, ktiles = (p.Tk + TM - 1) / TM;
  attn_bwd_dq_kernel<D><<<(unsigned)tiles * p.nq, BWD_THREADS, DqSmem<D>::TOTAL, stream>>>(tq, tdo, tk, tv, p, dp);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  attn_bwd_dkv_kernel<D><<<(unsigned)ktiles * p.nkv * p.splits, BWD_THREADS, DkvSmem<D>::TOTAL, stream>>>(tk, tv, tq, tdo, p);
  e = cudaGetLastError();
  if (e != cudaSuccess || p.partial == nullptr) return (int)e;
  const long long plane = (long long)p.Tk * p.nkv * D;
  attn_bwd_reduce_kernel<<<(unsigned)((plane / 8 + 255) / 256), 256, 0, stream>>>(p.partial, p.dv, p.dk, plane,
                                                                                  p.splits);
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

// General form.  q/o/dout/dq [T, nq, d], k/v/dk/dv [Tk, nkv, d] bf16 contiguous; lse, delta [nq, T] fp32 (delta is
// scratch filled here, or, with `delta_given`, read as passed: ring attention computes it once from the merged
// output).  k_lo / k_hi [T]: the forward's per-query key ranges (k_hi null = the query's index).  q_lo / q_hi [Tk]:
// per key, bounds on the queries that can see it (both null for causal self-attention).  `scale` is the softmax
// scale the forward used.
//
// Head split: with few kv heads and few key tiles the dK/dV grid (tiles x nkv CTAs) cannot fill the GPU.  Passing
// `splits` > 1 (a divisor of nq / nkv) and `partial` (fp32, 2 * splits * Tk * nkv * d elements) lets `splits` CTAs
// share a (tile, kv head) pair, each over nq / nkv / splits query heads; a reduction kernel sums their partial results.
int mcb_attn_bwd_ranges(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                        float* delta, int delta_given, const int* k_lo, const int* k_hi, const int* q_lo,
                        const int* q_hi, void* dq, void* dk, void* dv, int T, int Tk, int nq, int nkv, int d,
                        float scale, float* partial, int splits, int* status, void* stream_) {
  if (T == 0 || Tk == 0) return 0;
  if (nq % nkv || (k_hi == nullptr && Tk < T) || ((q_lo == nullptr) != (q_hi == nullptr))) return -2;
  if (q_lo == nullptr && k_hi != nullptr) return -2;   // general masks need the per-key query bounds
  if (splits < 1 || (nq / nkv) % splits) return -4;
  if (splits == 1) partial = nullptr;
  else if (partial == nullptr) return -5;
  BwdParams p{T, Tk, nq, nkv, d, scale, scale * LOG2E, k_lo, k_hi, q_lo, q_hi, lse, delta,
              (__nv_bfloat16*)dq, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, status, partial, splits};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  if (d == 128) return launch_bwd<128>(q, k, v, o, dout, delta, delta_given != 0, p, s);
  if (d == 64) return launch_bwd<64>(q, k, v, o, dout, delta, delta_given != 0, p, s);
  return -3;
}

}  // extern "C"
