// Warp-level bf16 tensor-core products on swizzled shared-memory tiles, for the chunked linear-attention kernels.
//
// Those kernels multiply fp32 quantities (states, decayed weights) with bf16 inputs.  An fp32 operand is fed to the
// tensor core as a sum of bf16 terms, each the rounding error of the ones before: two terms hold 16 mantissa bits, three
// all 24.  The terms are formed in registers, which is why these products use warp-level MMAs: their operands come straight
// from the accumulators of the product before, and each is far too small to fill the tcgen05 pipe.
//
// A tile is [rows][D] bf16 with 16-byte chunks swizzled by the row: chunk c of row r is stored at chunk c ^ (r & 7), in
// tiles of 32 columns (4 chunks) at c ^ ((r / 2) & 3); eight consecutive rows of one column then lie in distinct banks.
#pragma once
#include "../common/ptx.cuh"

namespace mcb {

template <int D>
__device__ __forceinline__ uint32_t tile_addr(uint32_t base, int row, int col) {   // col: multiple of 8
  if constexpr (D == 32) return base + row * 64 + (((col >> 3) ^ ((row >> 1) & 3)) << 4);
  return base + row * (D * 2) + (((col >> 3) ^ (row & 7)) << 4);
}

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// four 8 x 8 blocks of packed accumulators, each stored transposed: the lane addresses name rows of the stored blocks
__device__ __forceinline__ void stsm4_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d) : "memory");
}
// acc (16 x 8 fp32) += a (16 x 16 bf16, row) * b (16 x 8 bf16, col)
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A operand: rows r0 .. r0+15, contraction columns k0 .. k0+15 of a row-major tile
template <int D>
__device__ __forceinline__ void load_a(uint32_t tile, int r0, int k0, int lane, uint32_t (&a)[4]) {
  ldsm4(tile_addr<D>(tile, r0 + (lane & 15), k0 + ((lane >> 4) << 3)), a);
}
// A operand taken transposed: rows = tile columns m0 .. m0+15, contraction = tile rows k0 .. k0+15
template <int D>
__device__ __forceinline__ void load_a_t(uint32_t tile, int m0, int k0, int lane, uint32_t (&a)[4]) {
  ldsm4_t(tile_addr<D>(tile, k0 + ((lane >> 4) << 3) + (lane & 7), m0 + (((lane >> 3) & 1) << 3)), a);
}
// B operand of X Y^T: two 8-wide column blocks n0, n0+8 = tile rows, contraction = tile columns k0 .. k0+15;
// b[0], b[1] belong to n0, b[2], b[3] to n0 + 8
template <int D>
__device__ __forceinline__ void load_b_nt(uint32_t tile, int n0, int k0, int lane, uint32_t (&b)[4]) {
  ldsm4(tile_addr<D>(tile, n0 + ((lane >> 4) << 3) + (lane & 7), k0 + (((lane >> 3) & 1) << 3)), b);
}
// B operand of X Y: contraction = tile rows k0 .. k0+15, two column blocks n0, n0+8 = tile columns
template <int D>
__device__ __forceinline__ void load_b_nn(uint32_t tile, int k0, int n0, int lane, uint32_t (&b)[4]) {
  ldsm4_t(tile_addr<D>(tile, k0 + (((lane >> 3) & 1) << 3) + (lane & 7), n0 + ((lane >> 4) << 3)), b);
}

// two fp32 values -> packed bf16 pair and the packed pair of rounding errors
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = pack_bf16x2(x - f.x, y - f.y);
}
// the same with NT terms
template <int NT>
__device__ __forceinline__ void split_terms(float x, float y, uint32_t (&t)[NT][4], int r) {
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    t[i][r] = *reinterpret_cast<const uint32_t*>(&h);
    const float2 f = __bfloat1622float2(h);
    x -= f.x;
    y -= f.y;
  }
}
template <int NT>
__device__ __forceinline__ void acc_to_terms(const float (&c0)[4], const float (&c1)[4], uint32_t (&t)[NT][4]) {
  split_terms<NT>(c0[0], c0[1], t, 0);
  split_terms<NT>(c0[2], c0[3], t, 1);
  split_terms<NT>(c1[0], c1[1], t, 2);
  split_terms<NT>(c1[2], c1[3], t, 3);
}
// c += a * b, b exact bf16.  The tensor core truncates each time it adds to the accumulator: the small products are summed
// in an accumulator of their own (`lo`, added once at the end), so that the sum is cut as often as a plain bf16 product's.
template <int NT>
__device__ __forceinline__ void mma_exact(float (&c)[4], float (&lo)[4], const uint32_t (&a)[NT][4], uint32_t b0, uint32_t b1) {
  mma16816(c, a[0], b0, b1);
#pragma unroll
  for (int i = 1; i < NT; ++i) mma16816(lo, a[i], b0, b1);
}
// c += a * b, both in NT terms; products of order NT and above are below the last bit.  b[.][2 u], b[.][2 u + 1]: block u
template <int NT>
__device__ __forceinline__ void mma_terms(float (&c)[4], float (&lo)[4], const uint32_t (&a)[NT][4], const uint32_t (&b)[NT][4],
                                          int u) {
  mma16816(c, a[0], b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
  for (int o = 1; o < NT; ++o)
#pragma unroll
    for (int i = 0; i <= o; ++i) mma16816(lo, a[i], b[o - i][2 * u], b[o - i][2 * u + 1]);
}

// 16-byte asynchronous copy; `bytes` 0 writes zeros instead of reading
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ROWS x D tile from rows `src + r * stride`; rows at or past `valid` become zero
template <int D, int ROWS, int THREADS>
__device__ __forceinline__ void load_tile(uint32_t tile, const __nv_bfloat16* src, long long stride, int valid) {
  constexpr int CH = D / 8;
  for (int id = threadIdx.x; id < ROWS * CH; id += THREADS) {
    const int r = id / CH, c = (id % CH) * 8;
    const bool in = r < valid;
    cp_async16(tile_addr<D>(tile, r, c), in ? src + r * stride + c : src, in ? 16 : 0);
  }
}

// Tokens [first, second) of sequence `i`, kept inside the batch whatever the boundaries say.
__device__ __forceinline__ int2 seq_span(const int* __restrict__ cu, int i, int T) {
  const int a = min(max(cu[i], 0), T), b = min(cu[i + 1], T);
  return make_int2(a, max(a, b));
}
// Boundaries that leave [0, T] are reported; the kernels stay inside their buffers all the same.  (A sequence that ends before
// it starts is an empty one.)  Called by all CTAs of one row of the grid.
__device__ __forceinline__ void check_bounds(const int* __restrict__ cu, int n_seq, int T, int* status) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_seq; i += gridDim.x * blockDim.x) {
    const int a = cu[i], b = cu[i + 1];
    if (status && (min(a, b) < 0 || max(a, b) > T)) atomicCAS(status, 0, ST_BAD_ARGUMENT);
  }
}

// How many of the first n boundaries lie below `value` (those before 0 count as 0): up to the first that does not; by one warp.
__device__ __forceinline__ int bounds_below(const int* __restrict__ cu, int n, int value, int lane) {
  int lo = 0, hi = n;                           // the answer lies in [lo, hi]
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32, i = lo + lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, i < hi && max(cu[min(i, n - 1)], 0) < value);
    const int c = ~below ? __ffs(~below) - 1 : 32;
    if (c == 0) break;
    hi = min(hi, lo + c * step);
    lo += (c - 1) * step + 1;
  }
  return lo;
}
// The sequence that comes `rank`-th when the longest are taken first (ties in the batch's order).  n_seq <= 32; by one warp.
__device__ __forceinline__ int longest_first(const int* __restrict__ cu, int n_seq, int T, int rank, int lane) {
  const int2 s = seq_span(cu, min(lane, n_seq - 1), T);
  const int len = lane < n_seq ? s.y - s.x : -1;
  int before = 0;
  for (int j = 0; j < n_seq; ++j) {
    const int other = __shfl_sync(0xffffffffu, len, j);
    before += other > len || (other == len && j < lane);
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < n_seq && before == rank)) - 1;
}

// One entry of the chunk list of a packed batch: sequence `s` contributes ceil(len / C) chunks.  Called by one warp; finds the
// sequence that holds chunk `id`.  `seq` is -1 past the end.
struct ChunkPos {
  int seq, index, t0, t1;   // index inside the sequence; token bounds of the sequence
};
// A lane reads PER sequences at a time.
template <int C, int PER>
__device__ __forceinline__ ChunkPos find_chunk_step(const int* __restrict__ cu, int n_seq, int T, int id, int lane) {
  int done = 0;
  for (int s0 = 0; s0 < n_seq; s0 += 32 * PER) {
    const int first = s0 + lane * PER;
    int edge[PER + 1];
#pragma unroll
    for (int u = 0; u <= PER; ++u) edge[u] = cu[min(first + u, n_seq)];
    int nc[PER], mine = 0;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int a = min(max(edge[u], 0), T), b = min(edge[u + 1], T);
      nc[u] = first + u < n_seq && b > a ? (b - a + C - 1) / C : 0;
      mine += nc[u];
    }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    const bool here = id >= done + incl - mine && id < done + incl;
    const unsigned m = __ballot_sync(0xffffffffu, here);
    if (m) {
      ChunkPos p{-1, id - (done + incl - mine), 0, 0};
      if (here) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
          if (p.seq >= 0) continue;
          if (p.index < nc[u]) {
            p.seq = first + u;
            p.t0 = min(max(edge[u], 0), T);
            p.t1 = min(edge[u + 1], T);
          } else {
            p.index -= nc[u];
          }
        }
      }
      const int w = __ffs(m) - 1;
      p.seq = __shfl_sync(0xffffffffu, p.seq, w);
      p.index = __shfl_sync(0xffffffffu, p.index, w);
      p.t0 = __shfl_sync(0xffffffffu, p.t0, w);
      p.t1 = __shfl_sync(0xffffffffu, p.t1, w);
      return p;
    }
    done += __shfl_sync(0xffffffffu, incl, 31);
  }
  return ChunkPos{-1, 0, 0, 0};
}
// With thousands of short sequences the search is a large part of a CTA's life, with a few it is one step either way.
template <int C>
__device__ __forceinline__ ChunkPos find_chunk(const int* __restrict__ cu, int n_seq, int T, int id, int lane) {
  return n_seq <= 64 ? find_chunk_step<C, 1>(cu, n_seq, T, id, lane) : find_chunk_step<C, 8>(cu, n_seq, T, id, lane);
}

}  // namespace mcb
