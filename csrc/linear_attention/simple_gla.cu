// Simple gated linear attention with a constant per-head decay a = exp(g_h), forward and backward, in chunks of 128
// tokens over packed sequences:
//
//   S_t = a S_{t-1} + k_t v_t^T,   o_t = scale * S_t^T q_t          R_t = a R_{t+1} + scale * q_t do_t^T
//   dq_t = scale * S_t do_t,   dk_t = R_t v_t,   dv_t = R_t^T k_t
//
// Chunks are the tiles of 128 tokens of the packed batch, wherever its sequences begin: a tile's outputs need the state of the
// sequence that crosses its first edge (backward, R of the one that crosses its last), for the rows of that sequence, and
// products of tokens of one sequence inside the tile.  So a batch has T / 128 tiles however many sequences it is made of.  Two
// launches: `walk` forms the states at the edges, `result` computes every tile and result independently.  States are fp32
// sums, kept as two bf16 terms (64 KB per edge and head at d = 128; 128-token tiles keep that traffic at half of the
// inputs') and enter the products as these; weights and weighted scores are split the same way: against fp64 the bf16
// results are off by 0.00166, their own rounding.  Batches of fewer than 16 tokens a sequence are evaluated token by token in fp32
// (by_token).
//
// Measured, us, inputs not in the L2, heads of 128 (64), against kernels with warp-level MMAs on chunks of one sequence each (states
// by one kernel for all chunks and a prefix sum)
//                                          forward before    now         backward before   now
//   4096 tokens, sequences of 2926 and 1170, 16 heads    87 (48)   52 (42)       183 (79)    83 (56)
//   16384 in one, 32 heads                              544 (234) 241 (161)     1318 (495)  482 (273)
//   8192 in sequences of 1024, 16 heads                 144 (62)   79 (46)       331 (130)  130 (85)
//                        128                             83 (44)   62 (40)       148 (83)   105 (71)
//                         16                            226 (101)  73 (44)       470 (194)  132 (83)
//   8192 in one, 4 heads (the chain of `walk`)           64 (44)   62 (58)       114 (62)    73 (67)
//
// Packed sequences are described by cu_seqlens on the device; nothing waits for the host.
#include <climits>

#include "../common/host_utils.cuh"
#include "warp_mma.cuh"

using namespace mcb;

namespace {

constexpr int C = 128;          // tokens of a chunk
constexpr float L2E = 1.4426950408889634f;

struct GlaParams {
  const __nv_bfloat16 *q, *k, *v, *dout;   // [T, H, D]
  __nv_bfloat16 *o, *dq, *dk, *dv;
  const float* decay;                      // [H] log-decay per step
  const int* cu;                           // [n_seq + 1]
  __nv_bfloat16 *S, *R;                    // [T / C boundaries, H, 2 terms, D, D]
  int T, n_seq, H;
  float scale;
  int* status;
};

// Log2-decay per step.  exp(-inf) = 0 is a state that forgets everything: kept finite, so that the 0 steps between a token and
// itself multiply to 0 and not to NaN.
__device__ __forceinline__ float decay2(const GlaParams& p, int h) {
  const float g2 = p.decay[h] * L2E;
  return g2 == -INFINITY ? -1e30f : g2;
}

// ---------------------------------------------------------------------------------------------------- operand tiles
// A tile of `rows` x D bf16 lies in shared memory as D / 64 boxes of [rows][64], 128-byte rows with their 16-byte chunks
// swizzled by the row: what TMA writes and tcgen05 reads.
__device__ __forceinline__ uint32_t box_addr(uint32_t box, int row, int chunk) {
  return box + row * 128 + ((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void lds16(uint32_t addr, uint32_t (&x)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(addr) : "memory");
}
// one whole 32-byte sector
__device__ __forceinline__ void stg32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// Rows [len, C) of a C-row tile that holds a sequence's last tokens belong to the next sequence, and may be infinite there:
// they meet weights of zero only as zeros.  Thread = row.
template <int D>
__device__ __forceinline__ void zero_row(uint32_t tile, int row) {
#pragma unroll
  for (int b = 0; b < D / 64; ++b)
#pragma unroll
    for (int c = 0; c < 8; ++c) sts16(box_addr(tile + b * C * 128, row, c), 0, 0, 0, 0);
}
// `rows` x D tile at row y and column x of a map whose boxes are [rows][64]
template <int D, int ROWS>
__device__ __forceinline__ void load_boxes(uint32_t leader, uint32_t tile, const CUtensorMap* map, int x, int y, uint32_t bar) {
#pragma unroll
  for (int b = 0; b < D / 64; ++b) tma_load_2d_warp(leader, tile + b * ROWS * 128, map, x + b * 64, y, bar);
}

// ---------------------------------------------------------------------------------------------------- states
// States at the edges between tiles: S behind the tokens before an edge, R of those behind it, of the sequence that crosses it,
//
//   S' = a^C S + sum_j a^(C-1-j) k_j v_j^T        R' = a^C R + scale * sum_i a^i q_i do_i^T
//
// A walk follows a sequence through its tiles for one head, one of the two and 32 columns of v (do).  Only the sums over tiles
// are a chain, and they are a multiply-add of 32 registers a thread; everything else runs ahead of it: warp 12 loads the
// rows of k (q) and the columns of v (do) by TMA; warps 4..11 (thread = token and half of the columns) multiply these by
// the decays and lay them down as two bf16 terms (columns 0..31 and 32..63 of one operand); warps 13 and 14 multiply k^T with
// both on tcgen05, tile by tile in turn; warps 0..3 (thread = row of the state) add the two halves to their rows and write
// them through shared memory and TMA as two bf16 terms, which is how they enter the results' products.  Heads of 64 use the
// same 128-row product: rows 64..127 are whatever lies behind the tile and are not read.
//
// Bound: the chain weights - issue - product - weights of a buffer (2300 cycles, three buffers) and the 600 cycles a warp takes to
// issue eight products, hence two of them: 64 tiles 50 -> 43 us against two buffers and one issuer.  Columns fetched and states
// stored by the threads themselves, a row each, kept the load / store unit busy with 32 lines an instruction: 2100 cycles a tile.
constexpr int WALK_COLS = 32;
constexpr int WALK_THREADS = 480;
constexpr int WALK_STAGES = 4;     // tiles loading or in use
constexpr int WALK_BUFS = 3;       // weighted columns and accumulators

template <int D>
struct WalkSmem {
  static constexpr int TILE = C * D * 2, W = C * 128, V = C * WALK_COLS * 2, OUT = 2 * 32 * WALK_COLS * 2;
  static constexpr int OFF_W = WALK_STAGES * TILE;      // also what a 64-wide tile's 128-row product reads behind its last stage
  static constexpr int OFF_V = OFF_W + WALK_BUFS * W;
  static constexpr int OFF_OUT = OFF_V + WALK_STAGES * V;     // per warp: 32 rows of both terms
  static constexpr int OFF_BAR = OFF_OUT + 4 * OUT;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
};

struct WalkMaps {
  CUtensorMap k, q, v, d, s, r;                 // boxes of 64 x C (k, q), WALK_COLS x C (v, do) and WALK_COLS x 32 (states)
};

// The sequences that cross an edge, by head, direction and columns, dealt out to the CTAs in turn; every warp goes through the
// same list.  Up to one sequence a tile they are taken from the list of sequences (the longest first, if there are at most 32),
// with more of them from the edges: the sequence that crosses one, at the first edge it crosses.
template <int D>
struct Walk {
  const GlaParams& p;
  const int lane, dirs, units;
  int job, nb = 0, h = 0, col0 = 0;             // nb: edges this walk crosses
  bool rev = false;
  int2 span = {0, 0};
  __device__ Walk(const GlaParams& p_, int both, int lane_)
      : p(p_), lane(lane_), dirs(both ? 2 : 1), units(min(p_.n_seq, (p_.T - 1) / C)), job((int)blockIdx.x - (int)gridDim.x) {}
  __device__ bool next() {
    constexpr int SL = D / WALK_COLS;
    const int jobs = units * dirs * p.H * SL;
    for (job += gridDim.x; job < jobs; job += gridDim.x) {
      int id = job;
      col0 = (id % SL) * WALK_COLS;
      id /= SL;
      h = id % p.H;
      id /= p.H;
      rev = dirs == 2 && (id & 1);
      id /= dirs;
      if (units == p.n_seq) {
        span = seq_span(p.cu, p.n_seq <= 32 ? longest_first(p.cu, p.n_seq, p.T, id, lane) : id, p.T);
        nb = span.y > span.x ? (span.y - 1) / C - span.x / C : 0;
      } else {
        const int e = (id + 1) * C, seq = bounds_below(p.cu, p.n_seq + 1, e, lane) - 1;
        span = seq >= 0 && seq < p.n_seq ? seq_span(p.cu, seq, p.T) : make_int2(0, 0);
        nb = span.y > e && span.x >= e - C ? (span.y - 1) / C - span.x / C : 0;
      }
      if (nb > 0) return true;
    }
    return false;
  }
  // first token of the i-th tile, and the edge the walk comes to behind it (edges counted from 0 at token C)
  __device__ int tile(int i) const { return (rev ? (span.y - 1) / C - i : span.x / C + i) * C; }
  __device__ int edge(int i) const { return rev ? (span.y - 1) / C - i - 1 : span.x / C + i; }
};

template <int D>
__global__ void __launch_bounds__(WALK_THREADS, 1)
gla_walk_kernel(const __grid_constant__ WalkMaps maps, const GlaParams p, const int both) {
  using L = WalkSmem<D>;
  constexpr int NS = WALK_STAGES, NW = WALK_BUFS;
  extern __shared__ uint8_t smem_raw[];
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  const uint32_t k_full = smem_u32(bars), k_empty = smem_u32(bars + NS);
  const uint32_t w_full = smem_u32(bars + 2 * NS), done = w_full + 8 * NW, t_empty = done + 8 * NW;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NS + 3 * NW);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < NS; ++i) {
      mbar_init(k_full + 8 * i, 1);
      mbar_init(k_empty + 8 * i, 1);
    }
    for (int i = 0; i < NW; ++i) {
      mbar_init(w_full + 8 * i, 8);             // the warps that write it
      mbar_init(done + 8 * i, 1);               // the products of a tile: weights and accumulator are released by it
      mbar_init(t_empty + 8 * i, 4);
    }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 13) {
    tmem_alloc(smem_u32(tmem_slot), 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  const uint32_t tiles = smem_u32(smem), ws = tiles + L::OFF_W;
  uint32_t it = 0;                              // tiles so far: stages and phases
  bool ok = true;

  if (warp == 12) {
    const uint32_t leader = elect_one();
    for (Walk<D> w(p, both, lane); ok && w.next(); )
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++it) {
        const uint32_t s = it % NS;
        ok = mbar_wait_warp(k_empty + 8 * s, ((it / NS) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        if (!ok) break;
        mbar_expect_tx_warp(leader, k_full + 8 * s, L::TILE + L::V);
        load_boxes<D, C>(leader, tiles + s * L::TILE, w.rev ? &maps.q : &maps.k, w.h * D, w.tile(i), k_full + 8 * s);
        tma_load_2d_warp(leader, tiles + L::OFF_V + s * L::V, w.rev ? &maps.d : &maps.v, w.h * D + w.col0, w.tile(i), k_full + 8 * s);
      }
    for (uint32_t i = it > NS ? it - NS : 0; i < it; ++i) drain(k_full + 8 * (i % NS), (i / NS) & 1);
    __syncwarp();
  } else if (warp >= 13) {
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(128, 2 * WALK_COLS, true, true);
    for (Walk<D> w(p, both, lane); ok && w.next(); )
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++it) {
        if (it % 2 != warp - 13u) continue;
        const uint32_t s = it % NW, ks = it % NS, ph = (it / NW) & 1;
        ok = mbar_wait_warp(k_full + 8 * ks, (it / NS) & 1, abort_flag, p.status, ST_TIMEOUT_FULL) &&
             mbar_wait_warp(w_full + 8 * s, ph, abort_flag, p.status, ST_TIMEOUT_FULL) &&
             mbar_wait_warp(t_empty + 8 * s, ph ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < C / 16; ++kk)
          umma_f16_warp(leader, tmem + s * 64, make_smem_desc_sw128(tiles + ks * L::TILE + kk * 2048, C * 128, 1024),
                        make_smem_desc_sw128(ws + s * L::W + kk * 2048, C * 128, 1024), idesc, kk ? 1u : 0u);
        umma_commit_warp(leader, k_empty + 8 * ks);
        umma_commit_warp(leader, done + 8 * s);
      }
  } else if (warp >= 4) {
    const int j = threadIdx.x & 127, half = (threadIdx.x >> 7) - 1;
    for (Walk<D> w(p, both, lane); ok && w.next(); ) {
      const float wgt = (w.rev ? p.scale : 1.f) * exp2f(decay2(p, w.h) * (w.rev ? j : C - 1 - j));
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++it) {
        const uint32_t s = it % NW, ks = it % NS;
        ok = mbar_wait_warp(k_full + 8 * ks, (it / NS) & 1, abort_flag, p.status, ST_TIMEOUT_FULL) &&
             mbar_wait_warp(done + 8 * s, ((it / NW) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        if (!ok) break;
        const int t = w.tile(i) + j;
        const bool in = t >= w.span.x && t < w.span.y;    // the other tokens of the first and the last tile
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = 2 * half + u;
          uint32_t x[4], hi[4], lo[4];
          // what TMA wrote: 64-byte rows, their 16-byte chunks swizzled by pairs of rows
          lds16(tiles + L::OFF_V + ks * L::V + j * 64 + ((c ^ ((j >> 1) & 3)) << 4), x);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[e]));
            split2(in ? f.x * wgt : 0.f, in ? f.y * wgt : 0.f, hi[e], lo[e]);
          }
          sts16(box_addr(ws + s * L::W, j, c), hi[0], hi[1], hi[2], hi[3]);
          sts16(box_addr(ws + s * L::W, j, 4 + c), lo[0], lo[1], lo[2], lo[3]);
        }
        if (!in && half == 0) zero_row<D>(tiles + ks * L::TILE, j);   // it may be infinite, and meets weights of zero
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(w_full + 8 * s);
      }
    }
  } else {
    const uint32_t out = tiles + L::OFF_OUT + warp * L::OUT;
    for (Walk<D> w(p, both, lane); ok && w.next(); ) {
      const CUtensorMap* map = w.rev ? &maps.r : &maps.s;
      const float full = exp2f(decay2(p, w.h) * C);       // between two edges lies a whole tile
      float st[WALK_COLS];
#pragma unroll
      for (int e = 0; e < WALK_COLS; ++e) st[e] = 0.f;
#pragma unroll 1
      for (int i = 0; i < w.nb; ++i, ++it) {
        const uint32_t s = it % NW;
        ok = mbar_wait_warp(done + 8 * s, (it / NW) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        uint32_t r[64];
        tmem_ld_32x32_x64(tmem + (uint32_t(warp * 32) << 16) + s * 64, r);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(t_empty + 8 * s);
        if (warp * 32 >= D) continue;           // heads of 64
#pragma unroll
        for (int e = 0; e < WALK_COLS; ++e)
          st[e] = fmaf(st[e], full, __uint_as_float(r[e]) + __uint_as_float(r[e + WALK_COLS]));
        tma_store_wait_read<0>();               // (lane 0's) the tile before has left the staging area
        __syncwarp();
#pragma unroll
        for (int c = 0; c < WALK_COLS / 8; ++c) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) split2(st[8 * c + 2 * u], st[8 * c + 2 * u + 1], hi[u], lo[u]);
          const uint32_t at = out + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4);
          sts16(at, hi[0], hi[1], hi[2], hi[3]);
          sts16(at + L::OUT / 2, lo[0], lo[1], lo[2], lo[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int y = (w.edge(i) * p.H + w.h) * 2 * D + warp * 32;
          tma_store_2d(map, out, w.col0, y);
          tma_store_2d(map, out + L::OUT / 2, w.col0, y + D);
          tma_store_commit();
        }
      }
    }
    tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ---------------------------------------------------------------------------------------------------- results
// One result of one tile, from the state M at its edge (S before it or R behind it) and the pairs inside it:
//   role       out_i = w_i * (X_i . M) + scale * sum_j a^|i-j| (X_i . Y_j) Z_j
//   O          o  = q S,   (q . k) v       pairs j <= i
//   DQ         dq = do S^T, (do . v) k     pairs j <= i
//   DK         dk = v R^T, (v . do) q      pairs j >= i
//   DV         dv = k R,   (k . q) do      pairs j >= i
// Persistent CTAs, two an SM, take these one after the other.  All products run on tcgen05; the state enters as two bf16 terms,
// the weighted scores X . Y_j return to TMEM as two bf16 terms, the first operand of the last product.  Shared memory holds
// three tiles: X, then in turn Y and the state's lower term, the upper term and Z.  Warp 8 loads and multiplies:
//
//   X Y^T -> scores | X M_hi -> out (loads M_lo over Y, Z over M_hi) | out += X M_lo (loads the next X, Y) | out += P Z
//
// Warp 9 finds the next tile's sequences and looks for what is not finite in Z.  Warps 0..7 (thread = row and half of its columns) weight the scores meanwhile, multiply
// the state's share by w_i before the last product, and write the result out while the next one's first products run.
//
// Bound: the waits of that chain, half of them for the state's terms, of which two CTAs overlap: about 12000 cycles a result of
// 128 x 128 with a state and 5000 without.  One CTA per result (which loaded the state in fp32 and split it itself) took 86 us
// instead of 46 for the gradients of 4096 tokens, 16 heads of 128.
enum { O, DQ, DK, DV };
constexpr int RES_THREADS = 320;

template <int D>
struct ResultSmem {
  static constexpr int TILE = C * D * 2;
  static constexpr int Y = TILE, Z = 2 * TILE;
  static constexpr int OFF_BAD = 3 * TILE;                  // per column: rows of Z that are not finite there
  static constexpr int OFF_BAR = OFF_BAD + D * 16;
  static constexpr int TOTAL = OFF_BAR + 256 + 1024;
  static_assert(D <= C, "a term of the state fits into a tile");
};

struct GlaMaps {
  CUtensorMap q, k, v, d, s, r;
};

// What the warps of a CTA need to know of one result of one tile.
struct ResultItem {
  int t, len, h, edge, role;                    // first token; tokens (0: no more items); head; the state's edge
  int state, s0, s1;                            // whether one crosses, and the rows [s0, s1) it reaches
  uint32_t starts[4];                           // bit r: a sequence starts (or the last one has ended) at row r
};

// by one warp
__device__ __forceinline__ ResultItem find_item(const GlaParams& p, int id, int roles, int lane) {
  ResultItem it{};
  it.role = roles == 1 ? O : DQ + id % roles;
  id /= roles;
  it.h = id % p.H;
  it.t = id / p.H * C;
  it.len = min(C, p.T - it.t);
  auto bound = [&](int i) { return min(max(p.cu[i], 0), p.T) - it.t; };
  const int n = p.n_seq + 1;
  bool edge_ends = it.t + C >= p.T;             // no sequence crosses the tile's last edge
  for (int i0 = bounds_below(p.cu, n, it.t, lane); i0 < n; i0 += 32) {
    const int r = i0 + lane < n ? bound(i0 + lane) : -1;
#pragma unroll
    for (int w = 0; w < 4; ++w) it.starts[w] |= __reduce_or_sync(0xffffffffu, r >= 0 && r >> 5 == w ? 1u << (r & 31) : 0u);
    edge_ends |= __any_sync(0xffffffffu, r == C);
    if (__any_sync(0xffffffffu, r >= C)) break;
  }
  int first = C, last = 0;
#pragma unroll
  for (int w = 3; w >= 0; --w)
    if (it.starts[w]) first = 32 * w + __ffs(it.starts[w]) - 1;
#pragma unroll
  for (int w = 0; w < 4; ++w)
    if (it.starts[w]) last = 32 * w + 31 - __clz(it.starts[w]);
  if (it.role >= DK) {
    it.state = !edge_ends;
    it.s0 = last;
    it.s1 = C;
    it.edge = it.t / C;
  } else {
    it.state = it.t > 0 && first > 0;
    it.s0 = 0;
    it.s1 = first;
    it.edge = it.t / C - 1;
  }
  return it;
}

// All rows meet all of Z in the last product, most of them with weights of zero: what is not finite there is taken out of Z, and
// noted, so that it stays with the rows that see it.  By warp 9, which has time: us, gradients, only where several sequences share
// the tile / by the warps of the rows / by warp 9, 16384 in one, 32 heads of 128 287 / 317 / 304, 4096 in two, 16 heads 45.6 / 47.7 /
// 46.3, 8192 in sequences of 16 88 / 67 / 69.
template <int D>
__device__ __forceinline__ bool all_finite(uint32_t z, int lane) {
  // x * 0 is zero for what is finite, and NaN is what stays in a sum
  __nv_bfloat162 sum[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) sum[e] = __float2bfloat162_rn(0.f);
  for (int b = 0; b < D / 64; ++b)
#pragma unroll 4
    for (int c = 0; c < C / 4; ++c) {           // a quarter of a warp to a row
      uint32_t x[4];
      lds16(box_addr(z + b * C * 128, 4 * c + (lane >> 3), lane & 7), x);
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[e] = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&x[e]), __float2bfloat162_rn(0.f), sum[e]);
    }
  const __nv_bfloat162 s = __hadd2(__hadd2(sum[0], sum[1]), __hadd2(sum[2], sum[3]));
  return !__any_sync(0xffffffffu, __hisnan(__low2bfloat16(s)) || __hisnan(__high2bfloat16(s)));
}
// bad[column][q]: bit r, row 32 q + r is not finite there
template <int D>
__device__ __forceinline__ void take_out(uint32_t z, uint32_t* bad, int lane) {
#pragma unroll 1
  for (int i = 0; i < 4 * (D / 8); ++i) {
    const int q = i & 3, c = i >> 2;
    const uint32_t at = box_addr(z + (c >> 3) * (C * 128), 32 * q + lane, c & 7);
    uint32_t x[4];
    lds16(at, x);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t m = 0x7f80u << (16 * (e & 1));
      const bool out = (x[e >> 1] & m) == m;
      const uint32_t rows = __ballot_sync(0xffffffffu, out);
      if (lane == 0) bad[(c * 8 + e) * 4 + q] = rows;
      if (out) x[e >> 1] &= ~(0xffffu << (16 * (e & 1)));
    }
    sts16(at, x[0], x[1], x[2], x[3]);
  }
}

template <int D, bool GRAD>
__global__ void __launch_bounds__(RES_THREADS, 2)
gla_result_kernel(const __grid_constant__ GlaMaps maps, const GlaParams p, const int items) {
  using L = ResultSmem<D>;
  constexpr int ROLES = GRAD ? 3 : 1;
  constexpr uint32_t COL_S = 0, COL_O = 128;
  extern __shared__ uint8_t smem_raw[];
  __shared__ ResultItem slots[2];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  // every barrier completes once per item: with the item's number comes its phase
  const uint32_t xy_full = smem_u32(bars), hi_full = xy_full + 8, lo_full = xy_full + 16, z_full = xy_full + 24;
  const uint32_t s_done = xy_full + 32, hi_done = xy_full + 40, m_done = xy_full + 48, o_done = xy_full + 56;
  const uint32_t p_full = xy_full + 64, o_read = xy_full + 72;
  const uint32_t item_full = xy_full + 80, item_read = xy_full + 96;         // two each, by item & 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* bad_item = abort_flag + 1;
  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    *bad_item = -1;
    for (int i = 0; i < 8; ++i) mbar_init(xy_full + 8 * i, 1);
    mbar_init(p_full, 9);
    mbar_init(o_read, 8);
    for (int i = 0; i < 2; ++i) {
      mbar_init(item_full + 8 * i, 1);
      mbar_init(item_read + 8 * i, 9);
    }
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_slot), 256);
    tmem_relinquish();
  }
  uint32_t* bad = reinterpret_cast<uint32_t*>(smem + L::OFF_BAD);
  if (!GRAD) check_bounds(p.cu, p.n_seq, p.T, p.status);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_slot);
  const uint32_t sx = smem_u32(smem), sy = sx + L::Y, sz = sx + L::Z;

  if (warp == 8) {
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(C, C, false, false), idesc_z = make_idesc_bf16(C, D, false, true);
    auto next = [&](int n) {
      ResultItem it{};
      if (mbar_wait_warp(item_full + 8 * (n & 1), (n >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) it = slots[n & 1];
      __syncwarp();
      if (leader) mbar_arrive(item_read + 8 * (n & 1));
      return it;
    };
    auto load_xy = [&](const ResultItem& it) {
      const CUtensorMap* mx = it.role == O ? &maps.q : it.role == DQ ? &maps.d : it.role == DK ? &maps.v : &maps.k;
      const CUtensorMap* my = it.role == O ? &maps.k : it.role == DQ ? &maps.v : it.role == DK ? &maps.d : &maps.q;
      mbar_expect_tx_warp(leader, xy_full, 2 * L::TILE);
      load_boxes<D, C>(leader, sx, mx, it.h * D, it.t, xy_full);
      load_boxes<D, C>(leader, sy, my, it.h * D, it.t, xy_full);
    };
    auto load_state = [&](const ResultItem& it, int term, uint32_t dst, uint32_t bar) {
      mbar_expect_tx_warp(leader, bar, D * D * 2);
      load_boxes<D, D>(leader, dst, it.role >= DK ? &maps.r : &maps.s, 0, ((it.edge * p.H + it.h) * 2 + term) * D, bar);
    };
    auto times_state = [&](bool trans, uint32_t m, bool add) {
      const uint32_t idesc = make_idesc_bf16(C, D, false, !trans);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        umma_f16_warp(leader, tmem + COL_O, make_smem_desc_sw128(sx + (kk >> 2) * (C * 128) + (kk & 3) * 32, 16, 1024),
                      trans ? make_smem_desc_sw128(m + (kk >> 2) * (D * 128) + (kk & 3) * 32, 16, 1024)
                            : make_smem_desc_sw128(m + kk * 2048, D * 128, 1024),
                      idesc, add || kk ? 1u : 0u);
    };
    auto wait = [&](uint32_t bar, uint32_t ph, int code) {
      return mbar_wait_warp(bar, ph, abort_flag, p.status, code);
    };
    ResultItem it = next(0);
    if (it.len) load_xy(it);
    int n = 0;
    bool ok = true;
    uint32_t open = it.len ? 1u : 0u, xy_ph = 0;           // loads in flight: bits xy, hi, lo, z
    for (; it.len && ok; ++n) {
      const uint32_t ph = n & 1;
      const bool trans = it.role == DQ || it.role == DK;
      if (!(ok = wait(xy_full, ph, ST_TIMEOUT_FULL))) break;
      open &= ~1u;
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (kk >> 2) * (C * 128) + (kk & 3) * 32;
        umma_f16_warp(leader, tmem + COL_S, make_smem_desc_sw128(sx + off, 16, 1024), make_smem_desc_sw128(sy + off, 16, 1024),
                      idesc_s, kk ? 1u : 0u);
      }
      umma_commit_warp(leader, s_done);
      // the last product of the item before has read Z, its result has been taken out of TMEM
      if (n && !(ok = wait(o_done, ph ^ 1, ST_TIMEOUT_EMPTY))) break;
      if (it.state) {
        load_state(it, 0, sz, hi_full);
        open |= 2u;
        if (n && !(ok = wait(o_read, ph ^ 1, ST_TIMEOUT_TMEM_EMPTY))) break;
        if (!(ok = wait(hi_full, ph, ST_TIMEOUT_FULL))) break;
        open &= ~2u;
        tc_fence_after();
        times_state(trans, sz, false);
        umma_commit_warp(leader, hi_done);
        if (!(ok = wait(hi_done, ph, ST_TIMEOUT_EMPTY))) break;
        load_state(it, 1, sy, lo_full);
        open |= 4u;
      } else {
        if (leader) {
          mbar_arrive(hi_full);
          mbar_arrive(lo_full);
        }
        __syncwarp();
        umma_commit_warp(leader, hi_done);
        if (n && !(ok = wait(o_read, ph ^ 1, ST_TIMEOUT_TMEM_EMPTY))) break;
      }
      const CUtensorMap* mz = it.role == O ? &maps.v : it.role == DQ ? &maps.k : it.role == DK ? &maps.q : &maps.d;
      mbar_expect_tx_warp(leader, z_full, L::TILE);
      load_boxes<D, C>(leader, sz, mz, it.h * D, it.t, z_full);
      open |= 8u;
      if (it.state) {
        if (!(ok = wait(lo_full, ph, ST_TIMEOUT_FULL))) break;
        open &= ~4u;
        tc_fence_after();
        times_state(trans, sy, true);
      }
      umma_commit_warp(leader, m_done);
      const bool state = it.state;
      const int steps = warp_uniform((it.len + 15) / 16);
      it = next(n + 1);
      if (!(ok = wait(m_done, ph, ST_TIMEOUT_EMPTY))) break;
      if (it.len) {
        load_xy(it);
        open |= 1u;
        xy_ph = ph ^ 1;
      }
      if (!(ok = wait(z_full, ph, ST_TIMEOUT_FULL))) break;
      open &= ~8u;
      if (!(ok = wait(p_full, ph, ST_TIMEOUT_FULL))) break;
      tc_fence_after();
#pragma unroll
      for (int term = 0; term < 2; ++term)
#pragma unroll
        for (int kk = 0; kk < C / 16; ++kk) {
          if (kk >= steps) break;
          umma_f16_ts_warp(leader, tmem + COL_O, tmem + COL_S + (kk >> 1) * 32 + term * 16 + (kk & 1) * 8,
                           make_smem_desc_sw128(sz + kk * 2048, C * 128, 1024), idesc_z, (state || term || kk) ? 1u : 0u);
        }
      umma_commit_warp(leader, o_done);
    }
    // a wait that gave up: what was loading lands before the CTA goes
    if (open & 1u) drain(xy_full, xy_ph);
    if (open & 2u) drain(hi_full, n & 1);
    if (open & 4u) drain(lo_full, n & 1);
    if (open & 8u) drain(z_full, n & 1);
    __syncwarp();
  } else if (warp == 9) {
    auto publish = [&](int n, const ResultItem& it) {
      if (!mbar_wait_warp(item_read + 8 * (n & 1), ((n >> 1) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) return false;
      if (lane == 0) {
        slots[n & 1] = it;
        mbar_arrive(item_full + 8 * (n & 1));
      }
      __syncwarp();
      return true;
    };
    int id = blockIdx.x;
    ResultItem it = find_item(p, id, ROLES, lane);
    bool ok = publish(0, it);
    for (int n = 0; ok && it.len; ++n) {
      id += gridDim.x;
      it = id < items ? find_item(p, id, ROLES, lane) : ResultItem{};
      ok = publish(n + 1, it) && mbar_wait_warp(z_full, n & 1, abort_flag, p.status, ST_TIMEOUT_FULL);
      if (!ok) break;
      if (!all_finite<D>(sz, lane)) {
        take_out<D>(sz, bad, lane);
        *bad_item = n;
        fence_proxy_async_smem();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
  } else {
    const int q = warp & 3, half = warp >> 2, row = q * 32 + lane;
    const uint32_t lanes = uint32_t(q * 32) << 16;
    const uint32_t to = tmem + lanes + COL_O + half * (D / 2), ts = tmem + lanes + COL_S + half * 64;
    const int blk = half * 2;                   // first of this warp's two blocks of 32 score columns
    auto wait = [&](uint32_t bar, uint32_t ph, int code) {
      return mbar_wait_warp(bar, ph, abort_flag, p.status, code);
    };
    for (int n = 0;; ++n) {
      const uint32_t ph = n & 1;
      if (!wait(item_full + 8 * (n & 1), (n >> 1) & 1, ST_TIMEOUT_FULL)) break;
      const ResultItem it = slots[n & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(item_read + 8 * (n & 1));
      if (it.len == 0) break;
      const bool back = GRAD && it.role >= DK;
      const float g2 = decay2(p, it.h);
      // tokens of the row's own sequence that it sees: up to `far` back, or (back) ahead
      int far;
      {
        const uint32_t upto = 0xffffffffu >> (31 - lane);
        int start = 0, end = it.len;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const uint32_t m = it.starts[w];
          const uint32_t below = w < q ? m : w == q ? m & upto : 0, above = w > q ? m : w == q ? m & ~upto : 0;
          if (below) start = 32 * w + 31 - __clz(below);
          if (above) end = min(end, 32 * w + __ffs(above) - 1);
        }
        far = back ? end - 1 - row : row - start;
      }
      if (!wait(s_done, ph, ST_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
#pragma unroll
      for (int b = 0; b < 2; ++b) {             // 32 scores -> their two terms, in the same columns
        const int j0 = (blk + b) * 32, sign = back ? 1 : -1, gap0 = sign * (j0 - row);
        uint32_t hi[16], lo[16];
        // the columns' gaps are gap0 .. gap0 + 31 or gap0 - 31 .. gap0
        if (__any_sync(0xffffffffu, back ? gap0 + 31 >= 0 && gap0 <= far : gap0 >= 0 && gap0 - 31 <= far)) {
          uint32_t r[32];
          tmem_ld_32x32(ts + b * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float x[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int gap = gap0 + sign * (e + u);
              x[u] = gap >= 0 && gap <= far ? __uint_as_float(r[e + u]) * (p.scale * exp2f(g2 * gap)) : 0.f;
            }
            split2(x[0], x[1], hi[e >> 1], lo[e >> 1]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) hi[e] = lo[e] = 0;
        }
        tmem_st_32x16(ts + b * 32, hi);
        tmem_st_32x16(ts + b * 32 + 16, lo);
      }
      if (!wait(m_done, ph, ST_TIMEOUT_TMEM_FULL)) break;
      if (it.state) {
        const bool reached = row >= it.s0 && row < it.s1;
        const float w = back ? exp2f(g2 * (C - row)) : p.scale * exp2f(g2 * (row + 1));
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < D / 2; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(to + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = reached ? __float_as_uint(__uint_as_float(r[e]) * w) : 0u;
          tmem_st_32x32(to + c, r);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (!wait(o_done, ph, ST_TIMEOUT_TMEM_FULL) || !wait(p_full, ph, ST_TIMEOUT_FULL)) break;
      const bool found = *bad_item == n;        // (p_full: warp 9 has looked)
      tc_fence_after();
      __nv_bfloat16* out = !GRAD ? p.o : it.role == DQ ? p.dq : it.role == DK ? p.dk : p.dv;
      __nv_bfloat16* dst = out + ((long long)(it.t + row) * p.H + it.h) * D + half * (D / 2);
      uint32_t r[D / 2];
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) tmem_ld_32x32(to + c, *reinterpret_cast<uint32_t(*)[32]>(r + c));
      tmem_ld_wait();
      if (found) {                              // a sum with such a term in it has no value
        const int j0 = back ? row : row - far, j1 = back ? row + far : row;
#pragma unroll
        for (int c = 0; c < D / 2; ++c) {
          bool seen = false;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            uint32_t m = bad[(half * (D / 2) + c) * 4 + w];
            if (m == 0) continue;
            for (; m; m &= m - 1) {
              const int j = 32 * w + __ffs(m) - 1;
              seen |= j >= j0 && j <= j1;
            }
          }
          if (seen) r[c] = 0x7fffffffu;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_read);       // and the notes, if any, are read: the next item's Z is loaded behind this
      if (row < it.len) {
#pragma unroll
        for (int c = 0; c < D / 2; c += 16) {
          uint32_t v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = pack_bf16x2(__uint_as_float(r[c + 2 * u]), __uint_as_float(r[c + 2 * u + 1]));
          stg32(dst + c, v);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ---------------------------------------------------------------------------------------------------- short sequences
// Token by token: one CTA of D threads per (sequence, head), thread j keeps column j of the state S [D x D] in registers.  q
// and k of the current token are staged in shared memory (double buffered) so every thread reads them as broadcasts.
template <int D>
__global__ void __launch_bounds__(D)
gla_token_fwd_kernel(const GlaParams p) {
  __shared__ float qs[2][D], ks[2][D];
  const int h = blockIdx.y, j = threadIdx.x;
  if (h == 0) check_bounds(p.cu, p.n_seq, p.T, p.status);
  const int2 span = seq_span(p.cu, blockIdx.x, p.T);
  const float a = __expf(p.decay[h]);
  const __nv_bfloat16 *__restrict__ q = p.q, *__restrict__ k = p.k, *__restrict__ v = p.v;
  __nv_bfloat16* __restrict__ o = p.o;
  float S[D];
#pragma unroll
  for (int i = 0; i < D; ++i) S[i] = 0.f;
  auto stage = [&](int t, int b) {
    const long long at = ((long long)t * p.H + h) * D + j;
    qs[b][j] = __bfloat162float(q[at]) * p.scale;
    ks[b][j] = __bfloat162float(k[at]);
  };
  if (span.x < span.y) stage(span.x, 0);
  __syncthreads();
  for (int t = span.x; t < span.y; ++t) {
    const int b = (t - span.x) & 1;
    if (t + 1 < span.y) stage(t + 1, b ^ 1);
    const long long at = ((long long)t * p.H + h) * D + j;
    const float vj = __bfloat162float(v[at]);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      S[i] = fmaf(S[i], a, ks[b][i] * vj);
      acc = fmaf(S[i], qs[b][i], acc);
    }
    o[at] = __float2bfloat16(acc);
    __syncthreads();
  }
}

// Backward in three sweeps with no stored states.  Owning rows for dq / dk and columns for dv keeps every reduction inside a
// thread:
//   forward, thread = row i of S_t :              dq_t[i] = scale * sum_c S_t[i, c] do_t[c]
//   reverse, thread = row i of R_t / scale :      dk_t[i] = scale * sum_c (R_t / scale)[i, c] v_t[c]
//   reverse, thread = column c of R_t / scale :   dv_t[c] = scale * sum_i (R_t / scale)[i, c] k_t[i]
// Every sweep is  M <- a M + x w^T,  out = scale M z  over one order of the tokens; w and z are shared, x is the thread's own.
template <int D>
__global__ void __launch_bounds__(D)
gla_token_bwd_kernel(const GlaParams p) {
  __shared__ float ws[D], zs[D];
  const int h = blockIdx.y, i = threadIdx.x;
  const int2 span = seq_span(p.cu, blockIdx.x, p.T);
  const float a = __expf(p.decay[h]);
  float M[D];
  auto sweep = [&](bool reverse, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                   const __nv_bfloat16* __restrict__ z, __nv_bfloat16* __restrict__ out) {
#pragma unroll
    for (int c = 0; c < D; ++c) M[c] = 0.f;
    for (int n = span.x; n < span.y; ++n) {
      const long long at = ((long long)(reverse ? span.x + span.y - 1 - n : n) * p.H + h) * D + i;
      const float xi = __bfloat162float(x[at]);
      ws[i] = __bfloat162float(w[at]);
      zs[i] = __bfloat162float(z[at]);
      __syncthreads();
      float acc = 0.f;
#pragma unroll
      for (int c = 0; c < D; ++c) {
        M[c] = fmaf(M[c], a, xi * ws[c]);
        acc = fmaf(M[c], zs[c], acc);
      }
      out[at] = __float2bfloat16(acc * p.scale);
      __syncthreads();
    }
  };
  sweep(false, p.k, p.v, p.dout, p.dq);
  sweep(true, p.q, p.dout, p.v, p.dk);
  sweep(true, p.dout, p.q, p.k, p.dv);
}

// Batches of fewer than 16 tokens a sequence on average: fp32 throughout, where the tiles' weights, values and states are sums of two
// bf16 terms.  A result there is a sum of a few products, and those 16 bits show: of 2048 tokens in sequences of 12, 4 heads, 0.0002 of
// the results are not the exact ones' nearest bf16 values, by tiles 0.0017 (long sequences: 0.0025 either way).
bool by_token(int T, int n_seq) { return (long long)n_seq * 16 > T; }

template <int D>
int launch_gla(const GlaParams& p, int T, bool grad, cudaStream_t s) {
  if (by_token(T, p.n_seq)) {
    const dim3 seqs(p.n_seq, p.H);
    if (grad) gla_token_bwd_kernel<D><<<seqs, D, 0, s>>>(p);
    else gla_token_fwd_kernel<D><<<seqs, D, 0, s>>>(p);
    return (int)cudaGetLastError();
  }
  constexpr int W_SMEM = WalkSmem<D>::TOTAL, R_SMEM = ResultSmem<D>::TOTAL;
  static bool cfg = false;
  cudaError_t e;
  if (!cfg) {
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute(gla_walk_kernel<D>, kAttr, W_SMEM)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gla_result_kernel<D, false>, kAttr, R_SMEM)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gla_result_kernel<D, true>, kAttr, R_SMEM)) != cudaSuccess)
      return (int)e;
    cfg = true;
  }
  const long long width = (long long)p.H * D, edges = (T - 1) / C;
  GlaMaps m;
  int rc = 0;
  if ((rc = make_tmap_2d_bf16(&m.q, p.q, width, T, width, 64, C)) || (rc = make_tmap_2d_bf16(&m.k, p.k, width, T, width, 64, C)) ||
      (rc = make_tmap_2d_bf16(&m.v, p.v, width, T, width, 64, C)))
    return rc;
  m.d = m.s = m.r = m.q;
  if (grad && (rc = make_tmap_2d_bf16(&m.d, p.dout, width, T, width, 64, C))) return rc;
  const int sms = device_sm_count();
  if (edges > 0) {
    const long long rows = edges * p.H * 2 * D;
    if ((rc = make_tmap_2d_bf16(&m.s, p.S, D, rows, D, 64, D)) || (grad && (rc = make_tmap_2d_bf16(&m.r, p.R, D, rows, D, 64, D))))
      return rc;
    constexpr auto kHalf = CU_TENSOR_MAP_SWIZZLE_64B;
    WalkMaps w{m.k, m.q, m.q, m.q, m.q, m.q};
    if ((rc = make_tmap_2d(&w.v, p.v, width, T, width, WALK_COLS, C, 2, kHalf)) ||
        (rc = make_tmap_2d(&w.s, p.S, D, rows, D, WALK_COLS, 32, 2, kHalf)) ||
        (grad && (rc = make_tmap_2d(&w.d, p.dout, width, T, width, WALK_COLS, C, 2, kHalf))) ||
        (grad && (rc = make_tmap_2d(&w.r, p.R, D, rows, D, WALK_COLS, 32, 2, kHalf))))
      return rc;
    const long long walks = (edges < p.n_seq ? edges : p.n_seq) * (D / WALK_COLS) * p.H * (grad ? 2 : 1);
    if (walks > INT_MAX / 2) return -2;
    gla_walk_kernel<D><<<(int)(walks < sms ? walks : sms), WALK_THREADS, W_SMEM, s>>>(w, p, grad);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  }
  const long long items = (edges + 1) * p.H * (grad ? 3 : 1);
  if (items > INT_MAX / 2) return -2;
  const int grid = (int)(items < 2 * sms ? items : 2 * sms);
  if (grad) gla_result_kernel<D, true><<<grid, RES_THREADS, R_SMEM, s>>>(m, p, (int)items);
  else gla_result_kernel<D, false><<<grid, RES_THREADS, R_SMEM, s>>>(m, p, (int)items);
  return (int)cudaGetLastError();
}

int run_gla(const GlaParams& p, int T, int D, bool grad, cudaStream_t s) {
  if (D == 128) return launch_gla<128>(p, T, grad, s);
  if (D == 64) return launch_gla<64>(p, T, grad, s);
  return -3;
}

}  // namespace

extern "C" {

// Rows of the state workspaces: the edges between a batch's tiles, none for short sequences.
int mcb_simple_gla_edges(int T, int n_seq) { return T <= 0 || by_token(T, n_seq) ? 0 : (T - 1) / C; }

// q, k, v, o [T, H, D]; decay [H] fp32 (log-decay per step, <= 0); cu_seqlens [n_seq + 1] int32 from 0 to T;
// states [edges, H, 2, D, D] bf16 workspace.  Boundaries outside the batch are clipped and reported through `status`.
int mcb_simple_gla_fwd(const void* q, const void* k, const void* v, const float* decay, const int* cu_seqlens, void* o,
                       void* states, int T, int n_seq, int H, int D, float scale, int* status, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GlaParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.o = (__nv_bfloat16*)o;
  p.decay = decay; p.cu = cu_seqlens; p.S = (__nv_bfloat16*)states; p.T = T; p.n_seq = n_seq; p.H = H; p.scale = scale;
  p.status = status;
  return run_gla(p, T, D, false, reinterpret_cast<cudaStream_t>(stream_));
}

// states [2, edges, H, 2, D, D] bf16 workspace
int mcb_simple_gla_bwd(const void* q, const void* k, const void* v, const void* dout, const float* decay,
                       const int* cu_seqlens, void* dq, void* dk, void* dv, void* states, int T, int n_seq, int H, int D,
                       float scale, int* status, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GlaParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.dout = (const __nv_bfloat16*)dout;
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.decay = decay; p.cu = cu_seqlens; p.S = (__nv_bfloat16*)states; p.R = p.S + (long long)((T - 1) / C) * H * 2 * D * D;
  p.T = T; p.n_seq = n_seq; p.H = H; p.scale = scale; p.status = status;
  return run_gla(p, T, D, true, reinterpret_cast<cudaStream_t>(stream_));
}

}  // extern "C"
