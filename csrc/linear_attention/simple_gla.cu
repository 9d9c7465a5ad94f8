// Simple gated linear attention with a constant per-head decay a = exp(g_h), forward and backward, in chunks of 128
// tokens over packed sequences:
//
//   S_t = a S_{t-1} + k_t v_t^T,   o_t = scale * S_t^T q_t          R_t = a R_{t+1} + scale * q_t do_t^T
//   dq_t = scale * S_t do_t,   dk_t = R_t v_t,   dv_t = R_t^T k_t
//
// A chunk's outputs need the state at its first token (and, backward, R behind its last one) plus products inside the
// chunk.  Three launches: `boundary` forms what each chunk adds to the state that leaves it, `scan` runs the decayed
// prefix sum over a sequence's chunk boundaries element by element, `out` computes every chunk independently.  All of
// them have chunks x heads CTAs, so a single long sequence fills the GPU; token-by-token evaluation has one CTA per
// (sequence, head).  Measured, 4096 tokens in two sequences, 16 heads of 128: forward 0.09 ms, backward 0.17 ms; token by
// token the two took 10.6 ms.  Batches of sequences of fewer than 16 tokens on average are evaluated token by token.  States
// are fp32 in memory (64 KB per chunk boundary and head at d = 128; 128-token chunks keep that traffic at half of the
// inputs') and enter the products as two bf16 terms, see warp_mma.cuh: against fp64 the bf16 results are off by 0.00166, their
// own rounding, as token by token in fp32.
//
// Packed sequences are described by cu_seqlens on the device; CTAs find their chunk from it, nothing waits for the host.
#include "../common/host_utils.cuh"
#include "warp_mma.cuh"

using namespace mcb;

namespace {

constexpr int C = 128;          // tokens of a chunk
constexpr int THREADS = 256;    // 8 warps, 16 rows each
constexpr float L2E = 1.4426950408889634f;

struct GlaParams {
  const __nv_bfloat16 *q, *k, *v, *dout;   // [T, H, D]
  __nv_bfloat16 *o, *dq, *dk, *dv;
  const float* decay;                      // [H] log-decay per step
  const int* cu;                           // [n_seq + 1]
  float *S, *R;                            // [T / C boundaries, H, D, D] fp32
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

__device__ __forceinline__ ChunkPos broadcast_pos(const ChunkPos& mine, ChunkPos* slot) {
  if (threadIdx.x == 0) *slot = mine;
  __syncthreads();
  return *slot;
}

// What the chunk before a boundary adds to S (z = 0), what the chunk behind it adds to R (z = 1):
//   sum_j a^(C-1-j) k_j v_j^T      scale * sum_i a^i q_i do_i^T          rows: warp w owns 16 of D
template <int D>
__global__ void __launch_bounds__(THREADS)
gla_boundary_kernel(const GlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  const uint32_t sx = (smem_u32(smem_raw) + 127) & ~127u, sy = sx + C * D * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y;
  ChunkPos mine{-1, 0, 0, 0, 0};
  if (warp == 0) mine = find_chunk<C, true>(p.cu, p.n_seq, p.T, blockIdx.x, lane);
  const ChunkPos pos = broadcast_pos(mine, &slot);
  if (pos.seq < 0) return;
  const bool rev = blockIdx.z != 0;
  const int t = pos.t0 + (pos.index + (rev ? 1 : 0)) * C, len = min(C, pos.t1 - t);
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  load_tile<D, C, THREADS>(sx, (rev ? p.q : p.k) + off, stride, len);
  load_tile<D, C, THREADS>(sy, (rev ? p.dout : p.v) + off, stride, len);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (warp * 16 >= D) return;
  const float g2 = decay2(p, h), f = rev ? p.scale : 1.f;
  float acc[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll 1
  for (int kk = 0; kk < C; kk += 16) {
    uint32_t a[4], hi[4], lo[4];
    load_a_t<D>(sx, warp * 16, kk, lane, a);
#pragma unroll
    for (int u = 0; u < 2; ++u) {               // registers 2u, 2u+1: tokens j, j+1
      const int j = kk + 8 * u + (lane & 3) * 2;
      const float w0 = f * exp2f(g2 * (rev ? j : C - 1 - j)), w1 = f * exp2f(g2 * (rev ? j + 1 : C - 2 - j));
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[2 * u + r]));
        split2(x.x * w0, x.y * w1, hi[2 * u + r], lo[2 * u + r]);
      }
    }
#pragma unroll
    for (int n = 0; n < D; n += 16) {
      uint32_t b[4];
      load_b_nn<D>(sy, kk, n, lane, b);
      mma16816(acc[n / 8], hi, b[0], b[1]);
      mma16816(acc[n / 8 + 1], hi, b[2], b[3]);
      mma16816(acc[n / 8], lo, b[0], b[1]);
      mma16816(acc[n / 8 + 1], lo, b[2], b[3]);
    }
  }
  float* dst = (rev ? p.R : p.S) + ((long long)blockIdx.x * p.H + h) * D * D;
  const int row = warp * 16 + (lane >> 2), col = (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    *reinterpret_cast<float2*>(dst + (long long)row * D + n * 8 + col) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2*>(dst + (long long)(row + 8) * D + n * 8 + col) = make_float2(acc[n][2], acc[n][3]);
  }
}

// Decayed prefix sums over the boundaries of a sequence, in place: S forward (z = 0), R backward (z = 1); 4 elements a
// thread, the next boundaries' contributions are loaded ahead.
template <int D>
__global__ void __launch_bounds__(256)
gla_scan_kernel(const GlaParams p) {
  constexpr int PER = D * D / (256 * 4);        // blocks per (sequence, head)
  __shared__ int first;
  const int seq = blockIdx.x / PER, part = blockIdx.x % PER, h = blockIdx.y;
  const int2 span = seq_span(p.cu, seq, p.T);
  int nb = (span.y - span.x + C - 1) / C - 1;
  if (nb <= 0) return;
  if (threadIdx.x < 32) {                       // boundaries of the sequences before this one
    int n = 0;
    for (int s = threadIdx.x; s < seq; s += 32) {
      const int2 other = seq_span(p.cu, s, p.T);
      if (other.y > other.x) n += (other.y - other.x + C - 1) / C - 1;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (threadIdx.x == 0) first = n;
  }
  __syncthreads();
  nb = min(nb, p.T / C - first);                // overlapping sequences: no more boundaries than there is room for
  if (nb <= 0) return;
  const bool rev = blockIdx.z != 0;
  const float full = exp2f(decay2(p, h) * C);   // between two boundaries lies a whole chunk
  const long long step = (long long)p.H * D * D;
  float* base = (rev ? p.R : p.S) + ((long long)first * p.H + h) * D * D + (part * 256 + threadIdx.x) * 4;
  constexpr int AHEAD = 4;
  float4 buf[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < nb) buf[i] = *reinterpret_cast<const float4*>(base + (rev ? nb - 1 - i : i) * step);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i0 = 0; i0 < nb; i0 += AHEAD) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int i = i0 + u;
      if (i >= nb) break;
      const float4 x = buf[u];
      if (i + AHEAD < nb) buf[u] = *reinterpret_cast<const float4*>(base + (rev ? nb - 1 - i - AHEAD : i + AHEAD) * step);
      acc.x = fmaf(acc.x, full, x.x);
      acc.y = fmaf(acc.y, full, x.y);
      acc.z = fmaf(acc.z, full, x.z);
      acc.w = fmaf(acc.w, full, x.w);
      *reinterpret_cast<float4*>(base + (rev ? nb - 1 - i : i) * step) = acc;
    }
  }
}

// fp32 [D, D] state -> two bf16 tiles
template <int D>
__device__ __forceinline__ void load_state(uint32_t hi, uint32_t lo, const float* __restrict__ src) {
  constexpr int AHEAD = D * D / 8 / THREADS < 4 ? D * D / 8 / THREADS : 4;      // loads in flight: 4 x 32 bytes a thread
#pragma unroll 1
  for (int id0 = threadIdx.x; id0 < D * D / 8; id0 += AHEAD * THREADS) {
    float4 x[AHEAD][2];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const float4* at = reinterpret_cast<const float4*>(src) + 2 * (id0 + u * THREADS);
      x[u][0] = at[0];
      x[u][1] = at[1];
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int r = (id0 + u * THREADS) / (D / 8), c = ((id0 + u * THREADS) % (D / 8)) * 8;
      uint32_t a[4], b[4];
      split2(x[u][0].x, x[u][0].y, a[0], b[0]);
      split2(x[u][0].z, x[u][0].w, a[1], b[1]);
      split2(x[u][1].x, x[u][1].y, a[2], b[2]);
      split2(x[u][1].z, x[u][1].w, a[3], b[3]);
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile_addr<D>(hi, r, c)), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile_addr<D>(lo, r, c)), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
    }
  }
}

// acc (16 rows x D) = X[rows r0..] * M with M [D, D] in two terms, taken as M (NT = false) or M^T (true); then every row
// is multiplied by w0 (rows of the lower half) / w1 (upper half)
template <int D, bool NT>
__device__ __forceinline__ void times_state(float (&acc)[D / 8][4], uint32_t x, uint32_t mhi, uint32_t mlo, int r0, int lane,
                                            float w0, float w1) {
#pragma unroll 1
  for (int kk = 0; kk < D; kk += 16) {
    uint32_t a[4];
    load_a<D>(x, r0, kk, lane, a);
#pragma unroll
    for (int n = 0; n < D; n += 16) {
      uint32_t b[4], c[4];
      if (NT) {
        load_b_nt<D>(mhi, n, kk, lane, b);
        load_b_nt<D>(mlo, n, kk, lane, c);
      } else {
        load_b_nn<D>(mhi, kk, n, lane, b);
        load_b_nn<D>(mlo, kk, n, lane, c);
      }
      mma16816(acc[n / 8], a, b[0], b[1]);
      mma16816(acc[n / 8 + 1], a, b[2], b[3]);
      mma16816(acc[n / 8], a, c[0], c[1]);
      mma16816(acc[n / 8 + 1], a, c[2], c[3]);
    }
  }
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    acc[n][0] *= w0;
    acc[n][1] *= w0;
    acc[n][2] *= w1;
    acc[n][3] *= w1;
  }
}

// acc += (f * a^|i - j| * (X_i . Y_j)) Z_j over the column blocks jb in [jb0, jb1): rows i = r0.. of X, visible pairs
// j <= i (LOWER) or j >= i
template <int D, bool LOWER>
__device__ __forceinline__ void inside_chunk(float (&acc)[D / 8][4], uint32_t x, uint32_t y, uint32_t z, int r0, int jb0,
                                             int jb1, int lane, float g2, float f) {
  uint32_t xa[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) load_a<D>(x, r0, kk * 16, lane, xa[kk]);
  const int i = r0 + (lane >> 2);
#pragma unroll 1
  for (int jb = jb0; jb < jb1; ++jb) {
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t b[4];
      load_b_nt<D>(y, jb * 16, kk * 16, lane, b);
      mma16816(s[0], xa[kk], b[0], b[1]);
      mma16816(s[1], xa[kk], b[2], b[3]);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = jb * 16 + n * 8 + (lane & 3) * 2 + (e & 1);
        const int gap = LOWER ? i + (e >> 1) * 8 - j : j - i - (e >> 1) * 8;
        s[n][e] = gap >= 0 ? s[n][e] * (f * exp2f(g2 * gap)) : 0.f;
      }
    }
    uint32_t hi[4], lo[4];
    acc_to_a(s[0], s[1], hi, lo);
#pragma unroll
    for (int n = 0; n < D; n += 16) {
      uint32_t b[4];
      load_b_nn<D>(z, jb * 16, n, lane, b);
      mma16816(acc[n / 8], hi, b[0], b[1]);
      mma16816(acc[n / 8 + 1], hi, b[2], b[3]);
      mma16816(acc[n / 8], lo, b[0], b[1]);
      mma16816(acc[n / 8 + 1], lo, b[2], b[3]);
    }
  }
}

template <int D>
__device__ __forceinline__ void zero_acc(float (&acc)[D / 8][4]) {
#pragma unroll
  for (int n = 0; n < D / 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
}

// rows r0.. of the result, those below `len`
template <int D>
__device__ __forceinline__ void store_rows(const float (&acc)[D / 8][4], __nv_bfloat16* dst, long long stride, int r0, int len,
                                           int lane) {
  const int row = r0 + (lane >> 2), col = (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    if (row < len) *reinterpret_cast<uint32_t*>(dst + row * stride + n * 8 + col) = pack_bf16x2(acc[n][0], acc[n][1]);
    if (row + 8 < len) *reinterpret_cast<uint32_t*>(dst + (row + 8) * stride + n * 8 + col) = pack_bf16x2(acc[n][2], acc[n][3]);
  }
}

// Bound: shared-memory operand reads of the 128-row products (two per MMA term); one CTA per (chunk, head).
template <int D>
__global__ void __launch_bounds__(THREADS)
gla_out_kernel(const GlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  constexpr int TILE = C * D * 2;
  const uint32_t sq = (smem_u32(smem_raw) + 127) & ~127u, sk = sq + TILE, sv = sk + TILE, shi = sv + TILE, slo = shi + D * D * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y;
  ChunkPos mine{-1, 0, 0, 0, 0};
  if (warp == 0) mine = find_chunk<C, false>(p.cu, p.n_seq, p.T, blockIdx.x, lane);
  const ChunkPos pos = broadcast_pos(mine, &slot);
  if (pos.seq < 0 || pos.boundary0 + pos.index > p.T / C) return;
  const int t = pos.t0 + pos.index * C, len = min(C, pos.t1 - t);
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  load_tile<D, C, THREADS>(sq, p.q + off, stride, len);
  load_tile<D, C, THREADS>(sk, p.k + off, stride, len);
  load_tile<D, C, THREADS>(sv, p.v + off, stride, len);
  cp_async_commit();
  if (h == 0) check_bounds(p.cu, p.n_seq, p.T, p.status);
  if (pos.index > 0) load_state<D>(shi, slo, p.S + ((long long)(pos.boundary0 + pos.index - 1) * p.H + h) * D * D);
  cp_async_wait<0>();
  __syncthreads();
  const int r0 = warp * 16;
  if (r0 >= len) return;
  const float g2 = decay2(p, h);
  const int i = r0 + (lane >> 2);
  float acc[D / 8][4];
  zero_acc<D>(acc);
  if (pos.index > 0)
    times_state<D, false>(acc, sq, shi, slo, r0, lane, p.scale * exp2f(g2 * (i + 1)), p.scale * exp2f(g2 * (i + 9)));
  inside_chunk<D, true>(acc, sq, sk, sv, r0, 0, warp + 1, lane, g2, p.scale);
  store_rows<D>(acc, p.o + off, stride, r0, len, lane);
}

template <int D>
__global__ void __launch_bounds__(THREADS)
gla_grad_kernel(const GlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  constexpr int TILE = C * D * 2;
  const uint32_t sq = (smem_u32(smem_raw) + 127) & ~127u, sk = sq + TILE, sv = sk + TILE, sd = sv + TILE;
  const uint32_t shi = sd + TILE, slo = shi + D * D * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y;
  ChunkPos mine{-1, 0, 0, 0, 0};
  if (warp == 0) mine = find_chunk<C, false>(p.cu, p.n_seq, p.T, blockIdx.x, lane);
  const ChunkPos pos = broadcast_pos(mine, &slot);
  if (pos.seq < 0 || pos.boundary0 + pos.index > p.T / C) return;
  const int t = pos.t0 + pos.index * C, len = min(C, pos.t1 - t);
  const bool first = pos.index == 0;
  const bool last = t + len >= pos.t1 || pos.boundary0 + pos.index >= p.T / C;   // (the latter: overlapping sequences)
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  load_tile<D, C, THREADS>(sq, p.q + off, stride, len);
  load_tile<D, C, THREADS>(sk, p.k + off, stride, len);
  load_tile<D, C, THREADS>(sv, p.v + off, stride, len);
  load_tile<D, C, THREADS>(sd, p.dout + off, stride, len);
  cp_async_commit();
  const long long bnd = ((long long)(pos.boundary0 + pos.index) * p.H + h) * D * D, prev = bnd - (long long)p.H * D * D;
  if (!first) load_state<D>(shi, slo, p.S + prev);
  cp_async_wait<0>();
  __syncthreads();
  const int r0 = warp * 16, i = r0 + (lane >> 2);
  const int nblk = (len + 15) / 16;
  const float g2 = decay2(p, h);
  float acc[D / 8][4];
  if (r0 < len) {
    zero_acc<D>(acc);
    if (!first)
      times_state<D, true>(acc, sd, shi, slo, r0, lane, p.scale * exp2f(g2 * (i + 1)), p.scale * exp2f(g2 * (i + 9)));
    inside_chunk<D, true>(acc, sd, sv, sk, r0, 0, warp + 1, lane, g2, p.scale);
    store_rows<D>(acc, p.dq + off, stride, r0, len, lane);
  }
  if (!last) {
    __syncthreads();
    load_state<D>(shi, slo, p.R + bnd);
    __syncthreads();
  }
  if (r0 >= len) return;
  // a chunk that is not its sequence's last one is full: R decays by a^(C - j) to token j
  const float w0 = exp2f(g2 * (C - i)), w1 = exp2f(g2 * (C - i - 8));
  zero_acc<D>(acc);
  if (!last) times_state<D, true>(acc, sv, shi, slo, r0, lane, w0, w1);
  inside_chunk<D, false>(acc, sv, sd, sq, r0, warp, nblk, lane, g2, p.scale);
  store_rows<D>(acc, p.dk + off, stride, r0, len, lane);
  zero_acc<D>(acc);
  if (!last) times_state<D, false>(acc, sk, shi, slo, r0, lane, w0, w1);
  inside_chunk<D, false>(acc, sk, sq, sd, r0, warp, nblk, lane, g2, p.scale);
  store_rows<D>(acc, p.dv + off, stride, r0, len, lane);
}

// One chunk of one result, from the state M at its edge (S before it or R behind it) and the pairs inside it:
//   ROLE       out_i = w_i * (X_i . M) + scale * sum_j a^|i-j| (X_i . Y_j) Z_j
//   O          o  = q S,   (q . k) v       pairs j <= i
//   DQ         dq = do S^T, (do . v) k     pairs j <= i
//   DK         dk = v R^T, (v . do) q      pairs j >= i
//   DV         dv = k R,   (k . q) do      pairs j >= i
// The state's two terms lie where Y and Z go afterwards, so that three tiles are all a CTA holds and two CTAs share an SM
// (D = 128: 96 KB each against 160 and 192 above): one computes while the other waits for its tiles.  See `two_per_sm`.
enum { O, DQ, DK, DV };

template <int D, int ROLE>
__device__ __forceinline__ void chunk_result(const GlaParams& p, uint32_t sx, const ChunkPos& pos, int h) {
  constexpr int TILE = C * D * 2;
  constexpr bool BACK = ROLE >= DK;
  const uint32_t sy = sx + TILE, sz = sy + TILE;
  const __nv_bfloat16* X = ROLE == O ? p.q : ROLE == DQ ? p.dout : ROLE == DK ? p.v : p.k;
  const __nv_bfloat16* Y = ROLE == O ? p.k : ROLE == DQ ? p.v : ROLE == DK ? p.dout : p.q;
  const __nv_bfloat16* Z = ROLE == O ? p.v : ROLE == DQ ? p.k : ROLE == DK ? p.q : p.dout;
  __nv_bfloat16* out = ROLE == O ? p.o : ROLE == DQ ? p.dq : ROLE == DK ? p.dk : p.dv;
  const int t = pos.t0 + pos.index * C, len = min(C, pos.t1 - t);
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  const int bnd = pos.boundary0 + pos.index;
  // last chunk of a sequence, or (overlapping sequences) no boundary behind it
  const bool state = BACK ? t + len < pos.t1 && bnd < p.T / C : pos.index > 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = warp * 16, i = r0 + (lane >> 2);
  const float g2 = decay2(p, h);
  float acc[D / 8][4];
  zero_acc<D>(acc);
  load_tile<D, C, THREADS>(sx, X + off, stride, len);
  cp_async_commit();
  if (state) {
    load_state<D>(sy, sz, (BACK ? p.R : p.S) + ((long long)(BACK ? bnd : bnd - 1) * p.H + h) * D * D);
    cp_async_wait<0>();
    __syncthreads();
    // a chunk that is not its sequence's last one is full: R decays by a^(C - i) to token i
    const float w0 = BACK ? exp2f(g2 * (C - i)) : p.scale * exp2f(g2 * (i + 1));
    const float w1 = BACK ? exp2f(g2 * (C - i - 8)) : p.scale * exp2f(g2 * (i + 9));
    if (r0 < len) times_state<D, ROLE == DQ || ROLE == DK>(acc, sx, sy, sz, r0, lane, w0, w1);
    __syncthreads();
  }
  load_tile<D, C, THREADS>(sy, Y + off, stride, len);
  load_tile<D, C, THREADS>(sz, Z + off, stride, len);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (r0 >= len) return;
  inside_chunk<D, !BACK>(acc, sx, sy, sz, r0, BACK ? warp : 0, BACK ? (len + 15) / 16 : warp + 1, lane, g2, p.scale);
  store_rows<D>(acc, out + off, stride, r0, len, lane);
}

// z (gradients): dq, dk, dv
template <int D, bool GRAD>
__global__ void __launch_bounds__(THREADS, 2)
gla_result_kernel(const GlaParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  static_assert(D <= C, "a term of the state fits into a tile");
  const uint32_t sx = (smem_u32(smem_raw) + 127) & ~127u;
  const int h = blockIdx.y;
  ChunkPos mine{-1, 0, 0, 0, 0};
  if (threadIdx.x < 32) mine = find_chunk<C, false>(p.cu, p.n_seq, p.T, blockIdx.x, threadIdx.x);
  const ChunkPos pos = broadcast_pos(mine, &slot);
  if (pos.seq < 0 || pos.boundary0 + pos.index > p.T / C) return;
  if (!GRAD) {
    if (h == 0) check_bounds(p.cu, p.n_seq, p.T, p.status);
    chunk_result<D, O>(p, sx, pos, h);
  } else if (blockIdx.z == 0) {
    chunk_result<D, DQ>(p, sx, pos, h);
  } else if (blockIdx.z == 1) {
    chunk_result<D, DK>(p, sx, pos, h);
  } else {
    chunk_result<D, DV>(p, sx, pos, h);
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

// A chunk costs about the same however few of its 128 rows a sequence fills, the token kernels cost the same per token.
// Measured, 8192 tokens, 16 heads, sequences of 8 / 12 / 16 / 32 tokens, us:
//   heads of 128, forward    chunked 574 / 377 / 283 / 158      token by token 442 / 436 / 430 / 441
//                            (226 and 134 at 16 and 32 since two CTAs share an SM)
//                 + backward        1509 / 1004 / 753 / 423                    1520 / 1519 / 1524 / 1571
//   heads of 64,  forward           183 / 123 / 94 / 57                        93 / 93 / 93 / 95
//                 + backward        552 / 370 / 283 / 171                      368 / 372 / 375 / 382
bool by_token(int T, int n_seq) { return (long long)n_seq * 16 > T; }

// One result a CTA and two CTAs an SM, or all results in one CTA.  Heads of 128 only: with 64 several CTAs of either kind share
// an SM.  There have to be CTAs to share SMs, and the gradients read 9 tiles instead of 4, which pays where the states' products
// and loads are most of the work, not in sequences of one chunk.  Measured, us, all in one / one a CTA:
//   heads of 128, 16384 tokens x 32 heads      forward 679 / 548    backward 1482 / 1316
//   8192 x 16, sequences of 1024                       165 / 144              359 / 332
//                           200                        157 / 138              331 / 321
//                           128                         85 / 83               151 / 185
//                            32                        161 / 134              269 / 327
//   1000 x 16, one sequence                             34 / 38                58 / 64
//   heads of 64, 16384 x 32                            241 / 247              505 / 529
bool two_per_sm(int D, int T, int n_seq, int H, bool grad) {
  return D == 128 && (long long)(T / C) * H > device_sm_count() && (!grad || (long long)n_seq * C < T);
}

template <int D>
int launch_gla(const GlaParams& p, int T, bool grad, cudaStream_t s) {
  if (by_token(T, p.n_seq)) {
    const dim3 seqs(p.n_seq, p.H);
    if (grad) gla_token_bwd_kernel<D><<<seqs, D, 0, s>>>(p);
    else gla_token_fwd_kernel<D><<<seqs, D, 0, s>>>(p);
    return (int)cudaGetLastError();
  }
  constexpr int B_SMEM = 2 * C * D * 2 + 128, R_SMEM = 3 * C * D * 2 + 128;
  constexpr int O_SMEM = R_SMEM + 2 * D * D * 2, G_SMEM = O_SMEM + C * D * 2;
  static bool cfg = false;
  cudaError_t e;
  if (!cfg) {
    constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute(gla_boundary_kernel<D>, kAttr, B_SMEM)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gla_out_kernel<D>, kAttr, O_SMEM)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gla_grad_kernel<D>, kAttr, G_SMEM)) != cudaSuccess)
      return (int)e;
    if constexpr (D == 128)
      if ((e = cudaFuncSetAttribute(gla_result_kernel<D, false>, kAttr, R_SMEM)) != cudaSuccess ||
          (e = cudaFuncSetAttribute(gla_result_kernel<D, true>, kAttr, R_SMEM)) != cudaSuccess)
        return (int)e;
    cfg = true;
  }
  const int bounds = T / C;                      // a sequence has at most (len - 1) / C boundaries
  if (bounds > 0) {
    gla_boundary_kernel<D><<<dim3(bounds, p.H, grad ? 2 : 1), THREADS, B_SMEM, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    gla_scan_kernel<D><<<dim3(p.n_seq * (D * D / 1024), p.H, grad ? 2 : 1), 256, 0, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  }
  dim3 grid((T + C - 1) / C + p.n_seq, p.H);   // at least the number of chunks of any packing of T tokens
  if constexpr (D == 128)
    if (two_per_sm(D, T, p.n_seq, p.H, grad)) {
      grid.z = grad ? 3 : 1;
      if (grad) gla_result_kernel<D, true><<<grid, THREADS, R_SMEM, s>>>(p);
      else gla_result_kernel<D, false><<<grid, THREADS, R_SMEM, s>>>(p);
      return (int)cudaGetLastError();
    }
  if (grad) gla_grad_kernel<D><<<grid, THREADS, G_SMEM, s>>>(p);
  else gla_out_kernel<D><<<grid, THREADS, O_SMEM, s>>>(p);
  return (int)cudaGetLastError();
}

int run_gla(const GlaParams& p, int T, int D, bool grad, cudaStream_t s) {
  if (D == 128) return launch_gla<128>(p, T, grad, s);
  if (D == 64) return launch_gla<64>(p, T, grad, s);
  return -3;
}

}  // namespace

extern "C" {

// Rows of the state workspaces: the chunk boundaries a packed batch of T tokens can have at most, none for short sequences.
int mcb_simple_gla_boundaries(int T, int n_seq) { return by_token(T, n_seq) ? 0 : T / C; }

// q, k, v, o [T, H, D]; decay [H] fp32 (log-decay per step, <= 0); cu_seqlens [n_seq + 1] int32 from 0 to T;
// states [boundaries, H, D, D] fp32 workspace.  Boundaries outside the batch are clipped and reported through `status`.
int mcb_simple_gla_fwd(const void* q, const void* k, const void* v, const float* decay, const int* cu_seqlens, void* o,
                       float* states, int T, int n_seq, int H, int D, float scale, int* status, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GlaParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.o = (__nv_bfloat16*)o;
  p.decay = decay; p.cu = cu_seqlens; p.S = states; p.T = T; p.n_seq = n_seq; p.H = H; p.scale = scale;
  p.status = status;
  return run_gla(p, T, D, false, reinterpret_cast<cudaStream_t>(stream_));
}

// states [2, boundaries, H, D, D] fp32 workspace
int mcb_simple_gla_bwd(const void* q, const void* k, const void* v, const void* dout, const float* decay,
                       const int* cu_seqlens, void* dq, void* dk, void* dv, float* states, int T, int n_seq, int H, int D,
                       float scale, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GlaParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.dout = (const __nv_bfloat16*)dout;
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.decay = decay; p.cu = cu_seqlens; p.S = states; p.R = states + (long long)(T / C) * H * D * D;
  p.T = T; p.n_seq = n_seq; p.H = H; p.scale = scale;
  return run_gla(p, T, D, true, reinterpret_cast<cudaStream_t>(stream_));
}

}  // extern "C"
