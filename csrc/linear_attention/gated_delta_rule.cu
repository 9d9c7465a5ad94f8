// Gated delta rule in chunks of 64 tokens over packed sequences, forward and backward (d = 64 or 128, dk = dv).
//
//   S <- exp(g_t) S;   S <- S + beta_t k_t (v_t - S^T k_t)^T;   o_t = scale * S^T q_t
//
// With G the running sum of g inside a chunk, D_ij = exp(G_i - G_j), L_ij = (k_i . k_j) D_ij below the diagonal,
// I + M = (I + L beta)^-1 (the WY form), P = scale (q k^T) D below the diagonal, p = scale (q . k) on it, and S the state
// the chunk starts from:
//
//   E = exp(G) (k S) - M (v - exp(G) (k S))    V = beta (v - E)
//   O = scale exp(G) (q S) + P V               o = O + p V        S' = exp(G_last) S + (exp(G_last - G) k)^T V
//
// (E is what the state and the chunk's earlier tokens predict for v) and backward, dS' given:
//
//   F = P^T do + exp(G_last - G) (k dS')       N = F + beta^-1 M^T (beta (F + p do))      Y = N + p do      B = beta Y
//
//   dv = B    dS = exp(G_last) dS' + (scale exp(G) q)^T do - (exp(G) k)^T B    dP = do V^T    dL = -(B V^T)
//
//   dbeta_i = Y_i . (v_i - E_i)      dG_i = do_i . O_i - V_i . N_i - B_i . E_i,  plus <S', dS'> at the last token
//
// with dq, dk following from the products (gdr_grad_kernel).  dG needs no product of its own: reads leave with exp(G_i),
// writes enter with exp(-G_j), so it is what a token reads less what is read of it.  A pair (i, i) does both; M, P and
// with them O, E, N leave it out, so that the terms are as small as the decays make them and nothing cancels.  A beta below
// 2^-40 enters M and the quotient by beta as 2^-40, which changes results by less than their last bit.
//
// Launches: `prep` forms M and P of every chunk independently (kept for the backward pass); `scan` walks the chunks of a
// (sequence, head, 64 columns of v) in order; backward, `scan` runs again and keeps S, V and E, `scan_bwd` walks in reverse and
// keeps dS' and B, `grad` finishes every chunk independently.
//
// Precision: every value and accumulation is fp32, decays come from a 48-bit running sum.  Operands of a product that are not
// bf16 inputs enter the tensor core as sums of bf16 terms (warp_mma.cuh): two of them (16 bits) in products that only feed
// bf16 results (o, dq, dk), three (24 bits) in the backward scans, which also feed the fp32 results dg and dbeta.
// Against fp64, seven mixes of decays (none .. 500 a token), keys of length 1 and 1.35, up to 4096 tokens: the bf16 results are
// as far off as those of an fp32 torch evaluation (0.0017, their own rounding), dg and dbeta by 1.4e-7 .. 5.4e-7, torch by
// 2.8e-7 .. 3.8e-5.  Two terms throughout and decays from an fp32 sum gave 4.5e-6 .. 7.8e-5.
//
// In the scans four warps own 16 columns of v, with S^T (16 x d) in their accumulators: the accumulators of every product are the
// first operand of the next one.  Bound: the latency of what a chunk does one after the other (a warp issues every tenth cycle, the
// MMAs, forward about 500 a strip, backward 900 and 800, take 40 to 48 % of the time); the next chunk's tiles are copied
// meanwhile.  With one warp for a strip, which passes nothing on and forms every term itself, us, before / now, scan, the
// backward pass's scan and scan_bwd: 4096 tokens in three sequences, 32 heads of 128 171, 297, 358 / 133, 213, 233; in 64
// sequences 176, 308, 431 / 159, 257, 289; 8192 in one, 16 heads 636, 1120, 1338 / 504, 809, 897.  Two warps a strip: 173, 276,
// 307 (of the first).  No change from starting the strips apart, slower with the operands of M and P fetched before the
// strip's barrier (162, 335, 367: registers) and with 8 + 8 tokens a warp, for which M and P have as many blocks in each (145,
// 231, 274: more instructions).
// Measured, 4096 tokens in three sequences, 32 heads of 128: forward 0.19 ms (prep 0.06), backward 0.72 ms (grad 0.28).  The batched
// torch evaluation of the rule was most of a 29.5 ms block.
#include "../common/host_utils.cuh"
#include "warp_mma.cuh"

using namespace mcb;

namespace {

constexpr int C = 64;           // tokens of a chunk
constexpr int THREADS = 128;    // 4 warps, 16 tokens each
constexpr int ST = 512;         // scans: 4 strips of 16 columns of v, 4 warps each
constexpr int SQ = C * C * 2;   // bytes of one bf16 term of a chunk's square matrices
constexpr int MP = 3;           // terms kept of M and P

// rows of `gb`: G as a sum of two floats, beta, exp(G), exp(G_last - G), the diagonal p
enum { G_HI, G_LO, G_BETA, G_EXP, G_REST, G_DIAG, G_ROWS };

// M and P are kept as the ten 16 x 16 blocks on and below the diagonal, 512 bytes each; the two halves of a row change places every
// four rows, so that in shared memory, where they are copied as they are, eight rows of a half lie in distinct banks.
constexpr int SQB = 10 * 512;   // bytes of one term
constexpr int MPE = MP * SQB / 2;   // elements of all terms of M, or of P
__device__ __forceinline__ int block_off(int bi, int bj, int r, int half) {
  return (bi * (bi + 1) / 2 + bj) * 512 + r * 32 + ((half ^ ((r >> 2) & 1)) << 4);
}

struct GdrParams {
  const __nv_bfloat16 *q, *k, *v, *dout;   // [T, H, D]
  const float *g, *beta;                   // [T, H]
  const int* cu;                           // [n_seq + 1]
  __nv_bfloat16 *o, *dq, *dk, *dv;
  float *dg, *dbeta;                       // [T, H]
  // per chunk and head, chunks numbered through the packed batch:
  __nv_bfloat16* mp;                       // [2, MP, 10, 16, 16]: blocks of M and P
  float* gb;                               // [G_ROWS, 64] (beta 0 past the end of the sequence)
  float *S, *dS;                           // [D, D]: S^T and dS'^T
  __nv_bfloat16 *V, *B;                    // [2, D, 64]: V^T and B^T, two terms, as tiles in shared memory
  float* E;                                // [D / 16, 8, 32, 4]: E^T as the accumulators of the scans hold it
  float *oo, *nn, *yy;                     // [D / 16, 64]: do . O, V . N + B . E and dbeta over 16 columns of v
  int T, n_seq, H;
  float scale;
  int* status;
};

__device__ __forceinline__ ChunkPos locate(const GdrParams& p, ChunkPos* slot) {
  ChunkPos mine{-1, 0, 0, 0};
  if (threadIdx.x < 32) mine = find_chunk<C>(p.cu, p.n_seq, p.T, blockIdx.x, threadIdx.x);
  if (threadIdx.x == 0) *slot = mine;
  __syncthreads();
  return *slot;
}

// exp of a sum of two floats, the second far smaller
__device__ __forceinline__ float exp_pair(float hi, float lo) {
  const float e = expf(hi);
  return fmaf(e, lo, e);
}
// the beta that M is built from
__device__ __forceinline__ float nonzero(float b) { return fabsf(b) < 0x1p-40f ? copysignf(0x1p-40f, b) : b; }

// ---------------------------------------------------------------------------------------------------- prep
template <int D>
constexpr int PREP_TILES = 2 * C * D * 2 > C * (C + 4) * 4 ? 2 * C * D * 2 : C * (C + 4) * 4;   // q and k, later I + M

template <int D>
__global__ void __launch_bounds__(THREADS)
gdr_prep_kernel(const GdrParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  __shared__ float s_gh[C], s_gl[C], s_b[C];
  constexpr int LDA = C + 4;
  const uint32_t sq = (smem_u32(smem_raw) + 127) & ~127u, sk = sq + C * D * 2;
  float* sA = reinterpret_cast<float*>(smem_raw + (sq + PREP_TILES<D> - smem_u32(smem_raw)));  // [64][LDA]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y;
  const ChunkPos pos = locate(p, &slot);
  if (pos.seq < 0) return;
  const int t = pos.t0 + pos.index * C, len = min(C, pos.t1 - t);
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  const long long ch = (long long)blockIdx.x * p.H + h;
  load_tile<D, C, THREADS>(sq, p.q + off, stride, len);
  load_tile<D, C, THREADS>(sk, p.k + off, stride, len);
  cp_async_commit();
  if (h == 0) check_bounds(p.cu, p.n_seq, p.T, p.status);
  if (warp == 0) {                              // running sum of g: two tokens a lane
    const long long a = (long long)(t + 2 * lane) * p.H + h;
    const bool in0 = 2 * lane < len, in1 = 2 * lane + 1 < len;
    const double g0 = in0 ? p.g[a] : 0.f, g1 = in1 ? p.g[a + p.H] : 0.f;
    double run = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += x;
    }
    const double last = __shfl_sync(0xffffffffu, run, 31);
    const double G[2] = {run - g1, run};
    const float b[2] = {in0 ? p.beta[a] : 0.f, in1 ? p.beta[a + p.H] : 0.f};
    float* gb = p.gb + ch * G_ROWS * C;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = 2 * lane + u;
      const float hi = (float)G[u], lo = isfinite(hi) ? (float)(G[u] - hi) : 0.f;
      const float rh = (float)(last - G[u]), rl = isfinite(rh) ? (float)((last - G[u]) - rh) : 0.f;
      s_gh[j] = gb[G_HI * C + j] = hi;
      s_gl[j] = gb[G_LO * C + j] = lo;
      gb[G_BETA * C + j] = b[u];
      gb[G_EXP * C + j] = exp_pair(hi, lo);
      gb[G_REST * C + j] = exp_pair(rh, rl);
      s_b[j] = nonzero(b[u]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  const int r0 = warp * 16, i = r0 + (lane >> 2);
  __nv_bfloat16* mp = p.mp + ch * 2 * MPE;
  const float gh[2] = {s_gh[i], s_gh[i + 8]}, gl[2] = {s_gl[i], s_gl[i + 8]};
  for (int jb = 0; jb < 4; ++jb) {
    float kk2[2][4] = {}, qk2[2][4] = {};
    if (jb <= warp) {
#pragma unroll
      for (int kk = 0; kk < D; kk += 16) {
        uint32_t a[4], c[4], b[4];
        load_a<D>(sk, r0, kk, lane, a);
        load_a<D>(sq, r0, kk, lane, c);
        load_b_nt<D>(sk, jb * 16, kk, lane, b);
        mma16816(kk2[0], a, b[0], b[1]);
        mma16816(kk2[1], a, b[2], b[3]);
        mma16816(qk2[0], c, b[0], b[1]);
        mma16816(qk2[1], c, b[2], b[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int j = jb * 16 + n * 8 + (lane & 3) * 2;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float pv[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int ii = i + 8 * r, jj = j + u;
          const float d = jj < ii ? expf((gh[r] - s_gh[jj]) + (gl[r] - s_gl[jj])) : 0.f;
          const float qk = p.scale * qk2[n][2 * r + u];
          sA[ii * LDA + jj] = jj < ii ? s_b[jj] * kk2[n][2 * r + u] * d : 0.f;
          pv[u] = jj < ii ? qk * d : 0.f;
          if (jj == ii) p.gb[(ch * G_ROWS + G_DIAG) * C + ii] = qk;
        }
        uint32_t t[MP][4];
        split_terms<MP>(pv[0], pv[1], t, 0);
#pragma unroll
        for (int m = 0; m < MP; ++m)
          if (jb <= warp)
            *reinterpret_cast<uint32_t*>(mp + MPE + (m * SQB + block_off(warp, jb, (lane >> 2) + 8 * r, n)) / 2 +
                                         (lane & 3) * 2) = t[m][0];
      }
    }
  }
  __syncthreads();
  // I + M = (I + A)^-1 in blocks of 16: X_ii by forward substitution, a block to a warp, then X_ij = -X_ii sum_k A_ik X_kj row block by
  // row block.  A warp has four columns of every block column, so that nothing but its own results goes into its next ones.
  // X takes the place of the q / k tiles, which nothing reads any more.  A column to a thread, 64 rows one after the other, was 25000 of
  // the kernel's 43000 cycles: 4096 tokens, 32 heads of 128 84 -> 61 us, of 64 75 -> 47, 200 tokens, 4 heads 16 -> 11.
  float* sX = reinterpret_cast<float*>(smem_raw + (sq - smem_u32(smem_raw)));  // [64][LDA]
  if (lane < 16) {
    const float* A = sA + r0 * LDA + r0;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float s0 = r == lane ? 1.f : 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
      for (int c = 0; c < r; c += 4) {
        const float4 a = *reinterpret_cast<const float4*>(A + r * LDA + c);
        s0 = fmaf(-a.x, x[c], s0);
        if (c + 1 < r) s1 = fmaf(-a.y, x[c + 1], s1);
        if (c + 2 < r) s2 = fmaf(-a.z, x[c + 2], s2);
        if (c + 3 < r) s3 = fmaf(-a.w, x[c + 3], s3);
      }
      x[r] = (s0 + s1) + (s2 + s3);
      sX[(r0 + r) * LDA + r0 + lane] = x[r];
    }
  }
  __syncthreads();
  {
    const int row = lane >> 1, col = warp * 4 + (lane & 1) * 2;
    // out += a[row][0 .. 15] x[0 .. 15][col, col + 1]
    auto block = [&](float2& out, const float* a, const float* x) {
#pragma unroll
      for (int t = 0; t < 16; t += 4) {
        const float4 f = *reinterpret_cast<const float4*>(a + row * LDA + t);
        const float w[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 g = *reinterpret_cast<const float2*>(x + (t + u) * LDA + col);
          out.x = fmaf(w[u], g.x, out.x);
          out.y = fmaf(w[u], g.y, out.y);
        }
      }
    };
#pragma unroll
    for (int ib = 1; ib < 4; ++ib) {
      float2 y[3];
#pragma unroll
      for (int jb = 0; jb < ib; ++jb) {
        float2 sum = make_float2(0.f, 0.f);
#pragma unroll
        for (int kb = jb; kb < ib; ++kb) block(sum, sA + ib * 16 * LDA + kb * 16, sX + kb * 16 * LDA + jb * 16);
        *reinterpret_cast<float2*>(sX + (ib * 16 + row) * LDA + jb * 16 + col) = sum;
      }
      __syncwarp();
#pragma unroll
      for (int jb = 0; jb < ib; ++jb) {
        y[jb] = make_float2(0.f, 0.f);
        block(y[jb], sX + ib * 16 * LDA + ib * 16, sX + ib * 16 * LDA + jb * 16);
      }
      __syncwarp();
#pragma unroll
      for (int jb = 0; jb < ib; ++jb)
        *reinterpret_cast<float2*>(sX + (ib * 16 + row) * LDA + jb * 16 + col) = make_float2(-y[jb].x, -y[jb].y);
      __syncwarp();
    }
  }
  __syncthreads();
  for (int id = threadIdx.x; id < C * 8; id += THREADS) {
    const int r = id >> 3, c = (id & 7) * 8;
    if ((c >> 4) > (r >> 4)) continue;
    const float4 u = *reinterpret_cast<const float4*>(sX + r * LDA + c), v = *reinterpret_cast<const float4*>(sX + r * LDA + c + 4);
    float rest[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (c + e == r) rest[e] = 0.f;
#pragma unroll
    for (int m = 0; m < MP; ++m) {
      uint32_t t[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 h2 = __floats2bfloat162_rn(rest[2 * e], rest[2 * e + 1]);
        t[e] = *reinterpret_cast<const uint32_t*>(&h2);
        const float2 f = __bfloat1622float2(h2);
        rest[2 * e] -= f.x;
        rest[2 * e + 1] -= f.y;
      }
      *reinterpret_cast<uint4*>(mp + (m * SQB + block_off(r >> 4, c >> 4, r & 15, (c >> 3) & 1)) / 2) = make_uint4(t[0], t[1], t[2], t[3]);
    }
  }
}

// ---------------------------------------------------------------------------------------------------- scans
// Shared memory of a scan: two stages of k, q, 64-column slices of v and of do (X / Z), the last rows of gb and NT terms of M and P;
// what the four warps of a strip pass on to each other.
template <int D, int NT, bool WITH_DO>
struct ScanSmem {
  static constexpr int K = 0, Q = C * D * 2, X = 2 * C * D * 2, Z = X + SQ, G = Z + (WITH_DO ? SQ : 0);
  static constexpr int M = G + 4 * C * 4, P = M + NT * SQB, STAGE = P + NT * SQB;
  static constexpr int SHARE = 2 * STAGE;
  static constexpr int PART = 4 * NT * 512, STRIP = 2 * PART;        // 16 x 64 as second operands; S^T takes both parts
  static constexpr int BARS = SHARE + 4 * STRIP;
  static constexpr int TOTAL = BARS + 64 + 128;
  static_assert(D / 16 * NT * 512 <= 2 * PART && TOTAL + 64 <= 232448, "shared memory");
};

// arrives when this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
// A thread's part of the copies of a chunk, found once: with the addresses formed for each chunk they took 1400 of the 8000 cycles
// a chunk spends on its way through a warp.
template <int D, int NT, bool WITH_DO>
struct StageLoad {
  using L = ScanSmem<D, NT, WITH_DO>;
  static constexpr int N = D * C / 8 / ST;      // 16-byte pieces of q or k
  static constexpr int ROWS = ST / (D / 8);     // rows between two of them
  uint32_t off, at, xoff, xat;                  // of the first piece: elements from the chunk's first, bytes in the tile
  int row, xrow;
  __device__ __forceinline__ StageLoad(const GdrParams& p) {
    const uint32_t stride = p.H * D;
    row = threadIdx.x / (D / 8);
    off = row * stride + threadIdx.x % (D / 8) * 8;
    at = tile_addr<D>(0, row, threadIdx.x % (D / 8) * 8);
    xrow = threadIdx.x >> 3;
    xoff = xrow * stride + (threadIdx.x & 7) * 8;
    xat = tile_addr<64>(0, xrow, (threadIdx.x & 7) * 8);
  }
  // by all threads; the mbarriers `full` (tiles, gb) and full + 16 (M and P) have counts of ST + 1 and 1
  __device__ __forceinline__ void operator()(uint32_t st, uint32_t full, const GdrParams& p, int t, int len, int h, int col0,
                                             long long ch) const {
    static_assert(ROWS % 8 == 0, "the same place in the swizzle");
    if (threadIdx.x == 0) {
      mbar_expect_tx(full, 4 * C * 4);
      bulk_load_1d(st + L::G, p.gb + (ch * G_ROWS + G_BETA) * C, 4 * C * 4, full);
      mbar_expect_tx(full + 16, 2 * NT * SQB);
      bulk_load_1d(st + L::M, p.mp + ch * 2 * MPE, NT * SQB, full + 16);
      bulk_load_1d(st + L::P, p.mp + (ch * 2 + 1) * MPE, NT * SQB, full + 16);
    }
    const long long first = ((long long)t * p.H + h) * D;
    const __nv_bfloat16 *k = p.k + first, *q = p.q + first;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const bool in = row + i * ROWS < len;
      const uint32_t o = in ? off + i * ROWS * (uint32_t)(p.H * D) : 0;
      cp_async16(st + L::K + at + i * ROWS * D * 2, k + o, in ? 16 : 0);
      cp_async16(st + L::Q + at + i * ROWS * D * 2, q + o, in ? 16 : 0);
    }
    const bool in = xrow < len;
    const uint32_t o = (in ? xoff : 0) + col0;
    cp_async16(st + L::X + xat, p.v + first + o, in ? 16 : 0);
    if (WITH_DO) cp_async16(st + L::Z + xat, p.dout + first + o, in ? 16 : 0);
    cp_async_arrive(full);
  }
};

struct ScanPos {
  int t0, len, chunk0, n, h, col0;   // the sequence; its first chunk and their number; head; first column of v
};
__device__ __forceinline__ int seq_len(const GdrParams& p, int i) {
  const int2 s = seq_span(p.cu, i, p.T);
  return s.y - s.x;
}
template <int D>
__device__ __forceinline__ ScanPos scan_pos(const GdrParams& p, int* slot) {
  constexpr int SL = D / 64;
  ScanPos s;
  int seq = blockIdx.x / (p.H * SL);
  const int rest = blockIdx.x % (p.H * SL);
  // Few sequences: the longest ones are walked first, or the last to start would set the time (sequences of 1463, 585 and
  // 2048 tokens, 64 walks each: 194 -> 151 us).  With more than 32 of them one walk is a small share of the launch and the
  // order of the batch does.
  if (p.n_seq <= 32) {
    if (threadIdx.x < 32) {
      const int i = longest_first(p.cu, p.n_seq, p.T, seq, threadIdx.x);
      if (threadIdx.x == 0) *slot = i;
    }
    __syncthreads();
    seq = *slot;
    __syncthreads();
  }
  s.h = rest / SL;
  s.col0 = (rest % SL) * 64;
  const int2 span = seq_span(p.cu, seq, p.T);
  s.t0 = span.x;
  s.len = span.y - span.x;
  s.n = (s.len + C - 1) / C;
  if (threadIdx.x < 32) {
    int n = 0;
    for (int i = threadIdx.x; i < seq; i += 32) {
      n += (seq_len(p, i) + C - 1) / C;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (threadIdx.x == 0) *slot = n;
  }
  __syncthreads();
  s.chunk0 = *slot;
  s.n = max(0, min(s.n, p.T / C + p.n_seq - s.chunk0));   // overlapping sequences: no more chunks than there is room for
  s.len = min(s.len, s.n * C);
  return s;
}

__device__ __forceinline__ float2 lds2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float lds1(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// accumulators (16 rows x 8 N columns) -> fp32 rows of `ld` columns
template <int N>
__device__ __forceinline__ void store_f32(const float (&a)[N][4], float* dst, int ld, int row, int lane) {
  dst += (long long)row * ld + (lane & 3) * 2;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    *reinterpret_cast<float2*>(dst + n * 8) = make_float2(a[n][0], a[n][1]);
    *reinterpret_cast<float2*>(dst + 8 * ld + n * 8) = make_float2(a[n][2], a[n][3]);
  }
}
template <int N>
__device__ __forceinline__ void zero(float (&a)[N][4]) {
#pragma unroll
  for (int n = 0; n < N; ++n) a[n][0] = a[n][1] = a[n][2] = a[n][3] = 0.f;
}
// the accumulator of the small products joins the other one
template <int N>
__device__ __forceinline__ void join(float (&a)[N][4], const float (&b)[N][4]) {
#pragma unroll
  for (int n = 0; n < N; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) a[n][e] += b[n][e];
}
// NT terms of block (bi, bj) of M or P, as the B operand of X M^T (TRANS) or X M
template <int NT, bool TRANS>
__device__ __forceinline__ void load_square_b(uint32_t tile, int bi, int bj, int lane, uint32_t (&b)[NT][4]) {
#pragma unroll
  for (int m = 0; m < NT; ++m) {
    if (TRANS) ldsm4(tile + m * SQB + block_off(bi, bj, ((lane >> 4) << 3) + (lane & 7), (lane >> 3) & 1), b[m]);
    else ldsm4_t(tile + m * SQB + block_off(bi, bj, (((lane >> 3) & 1) << 3) + (lane & 7), lane >> 4), b[m]);
  }
}

// The four strips of a CTA do not wait for each other: their chunks are shifted against each other by up to half a chunk, so that the
// tensor-core products of one strip meet the arithmetic and the waits of others on each scheduler (a warp of every strip).  A stage
// is loaded by all threads, in the middle of the chunk before it and once all strips are done with the chunk that was in it.
struct ScanRing {
  uint32_t full, empty;                         // mbarriers of the first stage; + 8 of the second; + 16 (full) of M and P
  volatile int* abort_flag;
  int* status;
  int loads = 0;                                // of chunks, by this warp
  bool ok = true;                               // of this warp's waits so far
  __device__ __forceinline__ void init(uint32_t bars, volatile int* flag, int* st) {
    full = bars;
    empty = bars + 32;
    abort_flag = flag;
    status = st;
    if (threadIdx.x == 0) {
      *flag = 0;
      for (int i = 0; i < 2; ++i) {
        mbar_init(full + 8 * i, ST + 1);
        mbar_init(full + 16 + 8 * i, 1);
        mbar_init(empty + 8 * i, ST / 32);
      }
      fence_barrier_init();
    }
    __syncthreads();
  }
  // A wait that gives up reports it and the walk goes on to its end, with what is there, so that the barriers of a strip stay whole;
  // the warp waits for nothing and loads nothing any more.
  __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity, int code) {
    if (ok) ok = mbar_wait_warp(bar, parity, abort_flag, status, code);
  }
  __device__ __forceinline__ void wait_full(int i) { wait(full + 8 * (i & 1), (i >> 1) & 1, ST_TIMEOUT_FULL); }
  __device__ __forceinline__ void wait_squares(int i) { wait(full + 16 + 8 * (i & 1), (i >> 1) & 1, ST_TIMEOUT_FULL); }
  __device__ __forceinline__ bool wait_empty(int i) {          // until stage i & 1 is free for the i-th chunk
    if (i >= 2) wait(empty + 8 * (i & 1), ((i >> 1) & 1) ^ 1, ST_TIMEOUT_EMPTY);
    loads += ok;
    return ok;
  }
  // At the end of the walk.  A warp that has seen everything land has nothing to wait for; nothing lands in a CTA that is gone.
  __device__ __forceinline__ void finish() {
    if (ok) return;
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (threadIdx.x >= 32) return;              // the first warp issues the bulk copies
    for (int i = max(loads - 2, 0); i < loads; ++i) {
      drain(full + 8 * (i & 1), (i >> 1) & 1);
      drain(full + 16 + 8 * (i & 1), (i >> 1) & 1);
    }
  }
  __device__ __forceinline__ void done(int i, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * (i & 1));
  }
};

// Four warps share a strip of 16 columns of v: each has 16 of a chunk's tokens as columns of the token products and a quarter of
// the d columns of the state.  What all of them need as the second operand of the next product goes through shared memory as the
// terms it enters in, formed once; a lane reads what the same lane of another warp wrote.
__device__ __forceinline__ void strip_sync(int strip) { asm volatile("bar.sync %0, 128;" ::"r"(1 + strip) : "memory"); }
template <int NT>
__device__ __forceinline__ void share(uint32_t at, int kk, const uint32_t (&a)[NT][4]) {          // `at` includes the lane
#pragma unroll
  for (int m = 0; m < NT; ++m)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + (kk * NT + m) * 512), "r"(a[m][0]), "r"(a[m][1]), "r"(a[m][2]),
                 "r"(a[m][3]) : "memory");
}
template <int NT>
__device__ __forceinline__ void shared_terms(uint32_t at, int kk, uint32_t (&a)[NT][4]) {
#pragma unroll
  for (int m = 0; m < NT; ++m)
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a[m][0]), "=r"(a[m][1]), "=r"(a[m][2]), "=r"(a[m][3])
                 : "r"(at + (kk * NT + m) * 512) : "memory");
}
template <int NT, int N>
__device__ __forceinline__ void share_state(uint32_t at, int quarter, const float (&S)[N][4]) {
#pragma unroll
  for (int n = 0; n < N; n += 2) {
    uint32_t a[NT][4];
    acc_to_terms<NT>(S[n], S[n + 1], a);
    share<NT>(at, (quarter * N + n) / 2, a);
  }
}

// x [2][4] holds (16 columns of v) x (16 tokens), `tile` bf16 rows of the same tokens and columns: the dot product of every token
// over these columns -> dst[64]
__device__ __forceinline__ void token_dots(const float (&x)[2][4], uint32_t tile, float* dst, int strip, int tok0, int lane) {
  uint32_t a[4];
  load_a_t<64>(tile, strip * 16, tok0, lane, a);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[2 * u]));
    const float2 y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[2 * u + 1]));
    float d0 = fmaf(x[u][0], y0.x, x[u][2] * y1.x), d1 = fmaf(x[u][1], y0.y, x[u][3] * y1.y);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      d0 += __shfl_xor_sync(0xffffffffu, d0, o);
      d1 += __shfl_xor_sync(0xffffffffu, d1, o);
    }
    if (lane < 4) *reinterpret_cast<float2*>(dst + tok0 + u * 8 + lane * 2) = make_float2(d0, d1);
  }
}

// accumulators (16 rows x 16 tokens) -> two bf16 planes with 64 columns, 16-byte chunks where tile_addr<64> has them
__device__ __forceinline__ void store_terms(const float (&a)[2][4], __nv_bfloat16* dst, long long plane, int row, int tok0, int lane) {
#pragma unroll
  for (int n = 0; n < 2; ++n) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      uint32_t hi, lo;
      split2(a[n][2 * r], a[n][2 * r + 1], hi, lo);
      __nv_bfloat16* at = dst + tile_addr<64>(0, row + 8 * r, tok0 + n * 8) / 2 + (lane & 3) * 2;
      *reinterpret_cast<uint32_t*>(at) = hi;
      *reinterpret_cast<uint32_t*>(at + plane) = lo;
    }
  }
}

// x [2][4] holds (16 columns of v) x (16 tokens): written as bf16 rows of tokens through the warp's part of `tile`
__device__ __forceinline__ void store_transposed(const float (&x)[2][4], uint32_t tile, __nv_bfloat16* dst, long long stride, int len,
                                                 int strip, int tok0, int lane) {
  __syncwarp();
  stsm4_t(tile_addr<64>(tile, tok0 + ((lane >> 4) << 3) + (lane & 7), strip * 16 + (((lane >> 3) & 1) << 3)),
          pack_bf16x2(x[0][0], x[0][1]), pack_bf16x2(x[0][2], x[0][3]), pack_bf16x2(x[1][0], x[1][1]), pack_bf16x2(x[1][2], x[1][3]));
  __syncwarp();
  const int tok = tok0 + (lane >> 1), col = strip * 16 + (lane & 1) * 8;
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(tile_addr<64>(tile, tok, col)) : "memory");
  if (tok < len) *reinterpret_cast<uint4*>(dst + (long long)tok * stride + col) = v;
}

// SAVE: keep S, V and E of every chunk for the backward pass and form do . O of every token; else the outputs
template <int D, bool SAVE>
__global__ void __launch_bounds__(ST, 1)
gdr_scan_kernel(const GdrParams p) {
  constexpr int NT = SAVE ? 3 : 2, NB = D / 32;  // NB: 8-column blocks of a quarter of the state
  using L = ScanSmem<D, NT, SAVE>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int slot, flag;
  const uint32_t base = (smem_u32(smem_raw) + 127) & ~127u;
  const int lane = threadIdx.x & 31, strip = warp_uniform(threadIdx.x >> 7), quarter = (warp_uniform(threadIdx.x >> 5) + strip) & 3;
  const ScanPos s = scan_pos<D>(p, &slot);
  if (s.n == 0) return;
  const long long stride = (long long)p.H * D;
  const int row = s.col0 + strip * 16 + (lane >> 2), tok0 = quarter * 16;
  const uint32_t part0 = base + L::SHARE + strip * L::STRIP + lane * 16, part1 = part0 + L::PART;   // S in both; X, what V adds to S; V
  float St[NB][4];
  zero(St);
  ScanRing ring;
  ring.init(base + L::BARS, &flag, p.status);
  const StageLoad<D, NT, SAVE> copy(p);
  auto load = [&](int c) {
    if (c >= s.n || !ring.wait_empty(c)) return;
    copy(base + (c & 1) * L::STAGE, ring.full + 8 * (c & 1), p, s.t0 + c * C, min(C, s.len - c * C), s.h, s.col0,
                            (long long)(s.chunk0 + c) * p.H + s.h);
  };
  load(0);
  for (int c = 0; c < s.n; ++c) {
    const uint32_t st = base + (c & 1) * L::STAGE;
    const int t = s.t0 + c * C, len = min(C, s.len - c * C);
    const long long ch = (long long)(s.chunk0 + c) * p.H + s.h;
    ring.wait_full(c);
    if (c > 0) strip_sync(strip);               // S
    if (SAVE) store_f32(St, p.S + ch * D * D + quarter * (D / 4), D, row, lane);
    float X[2][4] = {}, O[2][4] = {}, Xl[2][4] = {}, Ol[2][4] = {};
    if (c > 0) {                                // the state is zero before the first chunk
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        uint32_t a[NT][4], b[4], d[4];
        shared_terms<NT>(part0, kk, a);
        load_b_nt<D>(st + L::K, tok0, kk * 16, lane, b);
        load_b_nt<D>(st + L::Q, tok0, kk * 16, lane, d);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma_exact<NT>(X[u], Xl[u], a, b[2 * u], b[2 * u + 1]);
          mma_exact<NT>(O[u], Ol[u], a, d[2 * u], d[2 * u + 1]);
        }
      }
      join(X, Xl);
      join(O, Ol);
    }
    // V (as -E so far) = -exp(G) k S, X = v - exp(G) k S; columns = tokens
    const uint32_t sb = st + L::G + (tok0 + (lane & 3) * 2) * 4, se = sb + C * 4, sr = se + C * 4, sp = sr + C * 4;   // rows of gb
    const float el = lds1(st + L::G + (2 * C - 1) * 4);
    float V[2][4], Vl[2][4] = {};
    float2 vv[2][2];
    {
      uint32_t a[4];
      load_a_t<64>(st + L::X, strip * 16, tok0, lane, a);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 e = lds2(se + u * 32);
        vv[u][0] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[2 * u]));
        vv[u][1] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[2 * u + 1]));
        float (&x)[4] = X[u], (&o)[4] = O[u], (&y)[4] = V[u];
        y[0] = -e.x * x[0];
        y[1] = -e.y * x[1];
        y[2] = -e.x * x[2];
        y[3] = -e.y * x[3];
        x[0] = vv[u][0].x + y[0];
        x[1] = vv[u][0].y + y[1];
        x[2] = vv[u][1].x + y[2];
        x[3] = vv[u][1].y + y[3];
        o[0] *= p.scale * e.x;
        o[1] *= p.scale * e.y;
        o[2] *= p.scale * e.x;
        o[3] *= p.scale * e.y;
      }
    }
    strip_sync(strip);                          // all have read S
    {
      uint32_t a[NT][4];
      acc_to_terms<NT>(X[0], X[1], a);
      share<NT>(part0, quarter, a);
    }
    strip_sync(strip);
    ring.wait_squares(c);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk > quarter) break;                  // M is lower triangular
      uint32_t a[NT][4], b[NT][4];
      shared_terms<NT>(part0, kk, a);
      load_square_b<NT, true>(st + L::M, quarter, kk, lane, b);
      mma_terms<NT>(V[0], Vl[0], a, b, 0);
      mma_terms<NT>(V[1], Vl[1], a, b, 1);
    }
    join(V, Vl);
    load(c + 1);
    if (SAVE) {
      float4* e = reinterpret_cast<float4*>(p.E + (ch * (D / 16) + (s.col0 >> 4) + strip) * (16 * C)) + lane;
#pragma unroll
      for (int n = 0; n < 2; ++n) e[(2 * quarter + n) * 32] = make_float4(-V[n][0], -V[n][1], -V[n][2], -V[n][3]);
    }
    {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 b = lds2(sb + u * 32);
        float (&x)[4] = V[u];
        x[0] = b.x * (vv[u][0].x + x[0]);
        x[1] = b.y * (vv[u][0].y + x[1]);
        x[2] = b.x * (vv[u][1].x + x[2]);
        x[3] = b.y * (vv[u][1].y + x[3]);
      }
      uint32_t a[NT][4];
      acc_to_terms<NT>(V[0], V[1], a);
      share<NT>(part1, quarter, a);
    }
    strip_sync(strip);                          // V; and all have read X
    if (c + 1 < s.n) {
      float W[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 w = lds2(sr + u * 32);
        W[u][0] = V[u][0] * w.x;
        W[u][1] = V[u][1] * w.y;
        W[u][2] = V[u][2] * w.x;
        W[u][3] = V[u][3] * w.y;
      }
      uint32_t a[NT][4];
      acc_to_terms<NT>(W[0], W[1], a);
      share<NT>(part0, quarter, a);
    }
    if (SAVE) store_terms(V, p.V + ch * 2 * D * C, (long long)D * C, row, tok0, lane);
    zero(Ol);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk > quarter) break;                  // P is lower triangular
      uint32_t a[NT][4], b[NT][4];
      shared_terms<NT>(part1, kk, a);
      load_square_b<NT, true>(st + L::P, quarter, kk, lane, b);
      mma_terms<NT>(O[0], Ol[0], a, b, 0);
      mma_terms<NT>(O[1], Ol[1], a, b, 1);
    }
    join(O, Ol);
    if (SAVE) {
      token_dots(O, st + L::Z, p.oo + (ch * (D / 16) + (s.col0 >> 4) + strip) * C, strip, tok0, lane);
    } else {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float2 d = lds2(sp + n * 32);
        O[n][0] = fmaf(d.x, V[n][0], O[n][0]);
        O[n][1] = fmaf(d.y, V[n][1], O[n][1]);
        O[n][2] = fmaf(d.x, V[n][2], O[n][2]);
        O[n][3] = fmaf(d.y, V[n][3], O[n][3]);
      }
      store_transposed(O, st + L::X, p.o + ((long long)t * p.H + s.h) * D + s.col0, stride, len, strip, tok0, lane);
    }
    if (c + 1 < s.n) {
      strip_sync(strip);
      float U[NB][4] = {}, Ul[NB][4] = {};      // what the chunk adds is summed apart: many chunks meet in the state
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t a[NT][4];
        shared_terms<NT>(part0, kk, a);
#pragma unroll
        for (int n = 0; n < NB; n += 2) {
          uint32_t b[4];
          load_b_nn<D>(st + L::K, kk * 16, quarter * (D / 4) + n * 8, lane, b);
          mma_exact<NT>(U[n], Ul[n], a, b[0], b[1]);
          mma_exact<NT>(U[n + 1], Ul[n + 1], a, b[2], b[3]);
        }
      }
      join(U, Ul);
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) St[n][e] = fmaf(St[n][e], el, U[n][e]);
      ring.done(c, lane);
      strip_sync(strip);                        // all have read V and what it adds
      share_state<NT>(part0, quarter, St);
    }
  }
  ring.finish();
}

template <int D>
__global__ void __launch_bounds__(ST, 1)
gdr_scan_bwd_kernel(const GdrParams p) {
  constexpr int NT = 3, NB = D / 32;
  using L = ScanSmem<D, NT, true>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ int slot, flag;
  const uint32_t base = (smem_u32(smem_raw) + 127) & ~127u;
  const int lane = threadIdx.x & 31, strip = warp_uniform(threadIdx.x >> 7), quarter = (warp_uniform(threadIdx.x >> 5) + strip) & 3;
  const ScanPos s = scan_pos<D>(p, &slot);
  if (s.n == 0) return;
  const long long stride = (long long)p.H * D;
  const int row = s.col0 + strip * 16 + (lane >> 2), tok0 = quarter * 16;
  const uint32_t part0 = base + L::SHARE + strip * L::STRIP + lane * 16, part1 = part0 + L::PART;   // dS in both; beta (F + p do), do; B
  float dSt[NB][4];
  zero(dSt);
  const int lastc = s.n - 1;
  ScanRing ring;
  ring.init(base + L::BARS, &flag, p.status);
  const StageLoad<D, NT, true> copy(p);
  auto load = [&](int it) {
    const int c = lastc - it;
    if (c < 0 || !ring.wait_empty(it)) return;
    copy(base + (it & 1) * L::STAGE, ring.full + 8 * (it & 1), p, s.t0 + c * C, min(C, s.len - c * C), s.h, s.col0,
                            (long long)(s.chunk0 + c) * p.H + s.h);
  };
  load(0);
  for (int it = 0; it < s.n; ++it) {
    const int c = lastc - it;
    const uint32_t st = base + (it & 1) * L::STAGE;
    const int t = s.t0 + c * C, len = min(C, s.len - c * C);
    const long long ch = (long long)(s.chunk0 + c) * p.H + s.h;
    const long long part = ch * (D / 16) + (s.col0 >> 4) + strip;
    float4 Ev[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) Ev[n] = reinterpret_cast<const float4*>(p.E + part * (16 * C))[(2 * quarter + n) * 32 + lane];
    ring.wait_full(it);
    if (it > 0) strip_sync(strip);              // dS
    store_f32(dSt, p.dS + ch * D * D + quarter * (D / 4), D, row, lane);
    const uint32_t sb = st + L::G + (tok0 + (lane & 3) * 2) * 4, se = sb + C * 4, sr = se + C * 4, sp = sr + C * 4;   // rows of gb
    const float el = lds1(st + L::G + (2 * C - 1) * 4);
    float dV[2][4] = {}, lo[2][4] = {};
    if (it > 0) {                               // nothing flows into the sequence's last state
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        uint32_t a[NT][4], b[4];
        shared_terms<NT>(part0, kk, a);
        load_b_nt<D>(st + L::K, tok0, kk * 16, lane, b);
        mma_exact<NT>(dV[0], lo[0], a, b[0], b[1]);
        mma_exact<NT>(dV[1], lo[1], a, b[2], b[3]);
      }
      join(dV, lo);
      zero(lo);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float2 w = lds2(sr + n * 32);
        dV[n][0] *= w.x;
        dV[n][1] *= w.y;
        dV[n][2] *= w.x;
        dV[n][3] *= w.y;
      }
    }
    strip_sync(strip);                          // all have read dS
    ring.wait_squares(it);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk < quarter) continue;               // rows i of P from column block j <= i
      uint32_t da[4], b[NT][4];                 // do^T: rows = columns of v, contraction = tokens
      load_a_t<64>(st + L::Z, strip * 16, kk * 16, lane, da);
      load_square_b<NT, false>(st + L::P, kk, quarter, lane, b);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mma16816(dV[u], da, b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
        for (int m = 1; m < NT; ++m) mma16816(lo[u], da, b[m][2 * u], b[m][2 * u + 1]);
      }
    }
    join(dV, lo);
    zero(lo);
    uint32_t da[4];
    load_a_t<64>(st + L::Z, strip * 16, tok0, lane, da);
    {
      uint32_t a[NT][4];                        // beta (F + p do); registers 2u, 2u + 1: tokens of the lower / upper half of the slice
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 b = lds2(sb + u * 32), d = lds2(sp + u * 32);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&da[2 * u + r]));
          split_terms<NT>(nonzero(b.x) * fmaf(d.x, x.x, dV[u][2 * r]), nonzero(b.y) * fmaf(d.y, x.y, dV[u][2 * r + 1]), a, 2 * u + r);
        }
      }
      share<NT>(part0, quarter, a);
    }
    strip_sync(strip);
    float B[2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {            // M^T (beta (F + p do))
      if (kk < quarter) continue;
      uint32_t a[NT][4], b[NT][4];
      shared_terms<NT>(part0, kk, a);
      load_square_b<NT, false>(st + L::M, kk, quarter, lane, b);
      mma_terms<NT>(B[0], lo[0], a, b, 0);
      mma_terms<NT>(B[1], lo[1], a, b, 1);
    }
    join(B, lo);
    load(it + 1);
    float *nn = p.nn + part * C, *yy = p.yy + part * C;
    uint32_t va[4], ab[NT][4];                  // ab: -exp(G) B
    load_a_t<64>(st + L::X, strip * 16, tok0, lane, va);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float2 b = lds2(sb + u * 32), d = lds2(sp + u * 32), eg = lds2(se + u * 32);
      const float E[4] = {Ev[u].x, Ev[u].y, Ev[u].z, Ev[u].w};
      float dn[2] = {0.f, 0.f}, dy[2] = {0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 x2 = *reinterpret_cast<const __nv_bfloat162*>(&da[2 * u + (e >> 1)]);
        const __nv_bfloat162 v2 = *reinterpret_cast<const __nv_bfloat162*>(&va[2 * u + (e >> 1)]);
        const float x = e & 1 ? __high2float(x2) : __low2float(x2), v = e & 1 ? __high2float(v2) : __low2float(v2);
        const float be = e & 1 ? b.y : b.x, W = v - E[e];
        const float N = dV[u][e] + B[u][e] / nonzero(be), Y = fmaf(e & 1 ? d.y : d.x, x, N);
        dn[e & 1] += be * fmaf(W, N, Y * E[e]);
        dy[e & 1] = fmaf(Y, W, dy[e & 1]);
        B[u][e] = be * Y;
      }
      split_terms<NT>(-eg.x * B[u][0], -eg.y * B[u][1], ab, 2 * u);
      split_terms<NT>(-eg.x * B[u][2], -eg.y * B[u][3], ab, 2 * u + 1);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          dn[r] += __shfl_xor_sync(0xffffffffu, dn[r], o);
          dy[r] += __shfl_xor_sync(0xffffffffu, dy[r], o);
        }
      }
      if (lane < 4) {
        *reinterpret_cast<float2*>(nn + tok0 + u * 8 + lane * 2) = make_float2(dn[0], dn[1]);
        *reinterpret_cast<float2*>(yy + tok0 + u * 8 + lane * 2) = make_float2(dy[0], dy[1]);
      }
    }
    share<NT>(part1, quarter, ab);
    store_terms(B, p.B + ch * 2 * D * C, (long long)D * C, row, tok0, lane);
    store_transposed(B, st + L::X, p.dv + ((long long)t * p.H + s.h) * D + s.col0, stride, len, strip, tok0, lane);
    if (c > 0) {
      strip_sync(strip);                        // all have read beta (F + p do)
      {
        uint32_t q[NT][4];                      // scale exp(G) do
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float2 e = lds2(se + u * 32);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&da[2 * u + r]));
            split_terms<NT>(x.x * (p.scale * e.x), x.y * (p.scale * e.y), q, 2 * u + r);
          }
        }
        share<NT>(part0, quarter, q);
      }
      strip_sync(strip);
      float U[NB][4] = {}, Ul[NB][4] = {};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t aq[NT][4], ak[NT][4];
        shared_terms<NT>(part0, kk, aq);
        shared_terms<NT>(part1, kk, ak);
#pragma unroll
        for (int n = 0; n < NB; n += 2) {
          uint32_t b[4], d[4];
          load_b_nn<D>(st + L::Q, kk * 16, quarter * (D / 4) + n * 8, lane, b);
          load_b_nn<D>(st + L::K, kk * 16, quarter * (D / 4) + n * 8, lane, d);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma_exact<NT>(U[n + u], Ul[n + u], aq, b[2 * u], b[2 * u + 1]);
            mma_exact<NT>(U[n + u], Ul[n + u], ak, d[2 * u], d[2 * u + 1]);
          }
        }
      }
      join(U, Ul);
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) dSt[n][e] = fmaf(dSt[n][e], el, U[n][e]);
      ring.done(it, lane);
      strip_sync(strip);                        // all have read both parts
      share_state<NT>(part0, quarter, dSt);
    }
  }
  ring.finish();
}

// ---------------------------------------------------------------------------------------------------- grad
// dq, dk, dg, dbeta of one chunk.  Rows = tokens, 16 to a warp:
//
//   F = do S^T   E = B S^T   H = V dS'^T   dP = scale (do V^T) D   dA = -(B V^T) D  (on and below / below the diagonal)
//   dq = scale exp(G) F + dP k      dk = exp(G_last - G) H - exp(G) E + dA k + dP^T q + dA^T k
//
// dP and dA are formed first, each 16 x 16 block once, and kept as two terms in shared memory, where they are read as they are and
// transposed.  Then four warps share 16 tokens: two halves of the d columns, 32 columns at a time, and for each one warp for
// F, E and dq and one for H and dk, which takes E from the other.  S^T and dS'^T are read 32 columns per half at a time,
// the first while dP and dA are formed; everything else the chunk needs is resident.  V, B and the states enter as two bf16 terms: dq
// and dk are rounded to bf16.  dg and dbeta are put together from the scans' dot products and <S', dS'>, in fp32.
// Bound: 6200 warp-level MMAs a chunk (6.6 us) and 320 KB.
// With two warps to 16 tokens, each forming the blocks of dP and dA it needs in both orientations (8600 MMAs), us, before / now: 4096
// tokens, 32 heads of 128 381 / 275, in 64 sequences 500 / 362; of 64 134 / 128.  What is left is the phases of a lone CTA
// (the MMAs take a third of the time): states on their way to the L2 a wave of CTAs ahead gave 1 to 4 %, and cost 2 % at 64.
constexpr int GT = 512;

template <int D>
struct GradSmem {
  static constexpr int TILE = C * D * 2;
  static constexpr int Q = 0, K = TILE, DO = 2 * TILE;                      // token tiles
  static constexpr int VT = 3 * TILE, YT = 5 * TILE;                        // V^T, B^T: two terms of [D][64] each
  static constexpr int ST = 7 * TILE;                                       // per half: S^T, dS'^T, two terms of [D][32] each
  static constexpr int STRIP = D * 32 * 2;
  static constexpr int DP = ST + 2 * 4 * STRIP, DA = DP + 2 * SQ;           // two terms of [64][64] each
  static constexpr int E = DA + 2 * SQ;                                     // 8 warps: 16 x 32 fp32
  static constexpr int TOTAL = E + 8 * 2048 + 128;
  static_assert(TOTAL + 1024 <= 232448, "shared memory");
};

// four neighbouring columns of a tile, as two bf16 terms
template <int D>
__device__ __forceinline__ void put4(uint32_t hi, uint32_t lo, int r, int c, const float4& x) {
  uint32_t a[2], b[2];
  split2(x.x, x.y, a[0], b[0]);
  split2(x.z, x.w, a[1], b[1]);
  const int off = (c & 7) * 2;
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(tile_addr<D>(hi, r, c & ~7) + off), "r"(a[0]), "r"(a[1]) : "memory");
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(tile_addr<D>(lo, r, c & ~7) + off), "r"(b[0]), "r"(b[1]) : "memory");
}

// 32 columns per half of S and dS' of this chunk, and of S' (null behind the sequence's last chunk, whose dS' is zero)
template <int D>
struct Strips {
  static constexpr int N = D * 16 / GT;
  float4 x[N], y[N], z[N];
  __device__ __forceinline__ void at(int i, int& half, int& r, int& c) const {
    const int id = threadIdx.x + i * GT;
    half = id / (D * 8);
    r = (id >> 3) % D;
    c = (id & 7) * 4;
  }
  __device__ __forceinline__ void fetch(const float* S, const float* dS, const float* next, int w) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      int half, r, c;
      at(i, half, r, c);
      const long long o = (long long)r * D + half * (D / 2) + w * 32 + c;
      x[i] = *reinterpret_cast<const float4*>(S + o);
      y[i] = *reinterpret_cast<const float4*>(dS + o);
      z[i] = next ? *reinterpret_cast<const float4*>(next + o) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  // -> tiles; returns this thread's share of <S', dS'>
  __device__ __forceinline__ float put(uint32_t tiles) const {
    constexpr int STRIP = GradSmem<D>::STRIP;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      int half, r, c;
      at(i, half, r, c);
      const uint32_t st = tiles + half * 4 * STRIP;
      put4<32>(st, st + STRIP, r, c, x[i]);
      put4<32>(st + 2 * STRIP, st + 3 * STRIP, r, c, y[i]);
      dot += (y[i].x * z[i].x + y[i].y * z[i].y) + (y[i].z * z[i].z + y[i].w * z[i].w);
    }
    return dot;
  }
};

// block (rb, cb) of dP (B false) or dA -> two terms of its tile
template <int D, bool B>
__device__ __forceinline__ void pair_block(uint32_t base, int rb, int cb, const float* s_gh, const float* s_gl, float scale, int lane) {
  using L = GradSmem<D>;
  float d[2][4] = {};
#pragma unroll
  for (int kk = 0; kk < D; kk += 16) {
    uint32_t vh[4], vl[4];
    load_b_nn<64>(base + L::VT, kk, cb * 16, lane, vh);
    load_b_nn<64>(base + L::VT + L::TILE, kk, cb * 16, lane, vl);
    if (B) {
      uint32_t yh[4], yl[4];
      load_a_t<64>(base + L::YT, rb * 16, kk, lane, yh);
      load_a_t<64>(base + L::YT + L::TILE, rb * 16, kk, lane, yl);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mma16816(d[u], yh, vh[2 * u], vh[2 * u + 1]);
        mma16816(d[u], yl, vh[2 * u], vh[2 * u + 1]);
        mma16816(d[u], yh, vl[2 * u], vl[2 * u + 1]);
      }
    } else {
      uint32_t a[4];
      load_a<D>(base + L::DO, rb * 16, kk, lane, a);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mma16816(d[u], a, vh[2 * u], vh[2 * u + 1]);
        mma16816(d[u], a, vl[2 * u], vl[2 * u + 1]);
      }
    }
  }
  const uint32_t tile = base + (B ? L::DA : L::DP);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = rb * 16 + (lane >> 2) + 8 * r, j = cb * 16 + n * 8 + (lane & 3) * 2;
      float x[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const bool in = B ? j + e < i : j + e <= i;
        const float D_ = in ? expf((s_gh[i] - s_gh[j + e]) + (s_gl[i] - s_gl[j + e])) : 0.f;
        x[e] = B ? (in ? -d[n][2 * r + e] * D_ : 0.f) : d[n][2 * r + e] * (scale * D_);
      }
      uint32_t hi, lo;
      split2(x[0], x[1], hi, lo);
      const uint32_t at = tile_addr<64>(tile, i, j & ~7) + (lane & 3) * 4;
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(hi) : "memory");
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + SQ), "r"(lo) : "memory");
    }
}

// out += X Y for 16 rows r0 of X (two terms of [64][64], TRANS: its transpose) and 32 columns c0 of the token tile Y, over the
// 16 x 16 blocks k0 .. k1 - 1
template <int D, bool TRANS>
__device__ __forceinline__ void add_pairs(float (&out)[4][4], uint32_t x, uint32_t y, int r0, int c0, int k0, int k1, int lane) {
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    uint32_t xh[4], xl[4];
    if (TRANS) {
      load_a_t<64>(x, r0, k * 16, lane, xh);
      load_a_t<64>(x + SQ, r0, k * 16, lane, xl);
    } else {
      load_a<64>(x, r0, k * 16, lane, xh);
      load_a<64>(x + SQ, r0, k * 16, lane, xl);
    }
#pragma unroll
    for (int n = 0; n < 4; n += 2) {
      uint32_t b[4];
      load_b_nn<D>(y, k * 16, c0 + n * 8, lane, b);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mma16816(out[n + u], xh, b[2 * u], b[2 * u + 1]);
        mma16816(out[n + u], xl, b[2 * u], b[2 * u + 1]);
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(GT, 1)
gdr_grad_kernel(const GdrParams p) {
  using L = GradSmem<D>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ ChunkPos slot;
  __shared__ float s_gh[C], s_gl[C], s_red[GT / 32];
  __shared__ __align__(8) uint64_t vb_full;
  __shared__ int flag;
  constexpr int NW = D / 64;                   // strips of a half
  const uint32_t base = (smem_u32(smem_raw) + 127) & ~127u;
  const int lane = threadIdx.x & 31, id = warp_uniform(threadIdx.x >> 5), warp = id & 3, half = (id >> 2) & 1, h = blockIdx.y;
  const ChunkPos pos = locate(p, &slot);
  if (pos.seq < 0) return;
  const int t = pos.t0 + pos.index * C, len = min(C, pos.t1 - t);
  const long long stride = (long long)p.H * D, off = ((long long)t * p.H + h) * D;
  const long long ch = (long long)blockIdx.x * p.H + h;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&vb_full), 1);
    fence_barrier_init();
    mbar_expect_tx(smem_u32(&vb_full), 4 * L::TILE);
    bulk_load_1d(base + L::VT, p.V + ch * 2 * D * C, 2 * L::TILE, smem_u32(&vb_full));
    bulk_load_1d(base + L::YT, p.B + ch * 2 * D * C, 2 * L::TILE, smem_u32(&vb_full));
  }
  {
    constexpr int PIECES = D / 8, ROWS = GT / PIECES;
    const int row = threadIdx.x / PIECES, c = threadIdx.x % PIECES * 8;
    const uint32_t to = tile_addr<D>(base, row, c), from = row * (uint32_t)stride + c;
    static_assert(ROWS % 8 == 0, "the same place in the swizzle");
#pragma unroll
    for (int u = 0; u < C / ROWS; ++u) {
      const bool in = row + u * ROWS < len;
      const uint32_t o = in ? from + u * ROWS * (uint32_t)stride : 0;
      cp_async16(to + L::Q + u * ROWS * D * 2, p.q + off + o, in ? 16 : 0);
      cp_async16(to + L::K + u * ROWS * D * 2, p.k + off + o, in ? 16 : 0);
      cp_async16(to + L::DO + u * ROWS * D * 2, p.dout + off + o, in ? 16 : 0);
    }
  }
  cp_async_commit();
  const float* gb = p.gb + ch * G_ROWS * C;
  if (threadIdx.x < C) {
    s_gh[threadIdx.x] = gb[G_HI * C + threadIdx.x];
    s_gl[threadIdx.x] = gb[G_LO * C + threadIdx.x];
  }
  const float *S = p.S + ch * D * D, *dS = p.dS + ch * D * D;
  const bool more = t + C < pos.t1 && blockIdx.x + 1 < gridDim.x;   // (the latter: overlapping sequences)
  const float* next = more ? S + (long long)p.H * D * D : nullptr;
  Strips<D> strips;
  strips.fetch(S, dS, next, 0);
  const int r0 = warp * 16, i = r0 + (lane >> 2), c2 = (lane & 3) * 2;
  const float eg[2] = {gb[G_EXP * C + i], gb[G_EXP * C + i + 8]}, el[2] = {gb[G_REST * C + i], gb[G_REST * C + i + 8]};
  if (threadIdx.x == 0) flag = 0;
  cp_async_wait<0>();
  __syncthreads();                             // (the mbarrier too)
  const bool landed = mbar_wait_warp(smem_u32(&vb_full), 0, &flag, p.status, ST_TIMEOUT_FULL);   // if not, it is reported
  {
    // ten blocks of dA (48 MMAs) and ten of dP (32): one of dA, or one or two of dP to a warp
    auto row_of = [](int b) { return b >= 6 ? 3 : b >= 3 ? 2 : b >= 1 ? 1 : 0; };
    if (id < 10) {
      const int rb = row_of(id);
      pair_block<D, true>(base, rb, id - rb * (rb + 1) / 2, s_gh, s_gl, p.scale, lane);
    } else {
#pragma unroll 1
      for (int b = id - 10; b < 10; b += 6) {
        const int rb = row_of(b);
        pair_block<D, false>(base, rb, b - rb * (rb + 1) / 2, s_gh, s_gl, p.scale, lane);
      }
    }
  }
  float tot = strips.put(base + L::ST);
  __syncthreads();
  const uint32_t st = base + L::ST + half * 4 * L::STRIP, ex = base + L::E + (id & 7) * 2048 + lane * 16;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    if (w + 1 < NW) strips.fetch(S, dS, next, w + 1);
    const int c0 = half * (D / 2) + w * 32;
    float out[4][4] = {};
    __nv_bfloat16* dst;
    if (id < 8) {
      float E[4][4] = {};
#pragma unroll 1
      for (int kk = 0; kk < D; kk += 16) {      // contraction over the columns of v
        uint32_t a[4], yh[4], yl[4];
        load_a<D>(base + L::DO, r0, kk, lane, a);
        load_a_t<64>(base + L::YT, r0, kk, lane, yh);
        load_a_t<64>(base + L::YT + L::TILE, r0, kk, lane, yl);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t b[4], d[4];
          load_b_nn<32>(st, kk, n * 8, lane, b);
          load_b_nn<32>(st + L::STRIP, kk, n * 8, lane, d);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma16816(out[n + u], a, b[2 * u], b[2 * u + 1]);
            mma16816(E[n + u], yh, b[2 * u], b[2 * u + 1]);
            mma16816(out[n + u], a, d[2 * u], d[2 * u + 1]);
            mma16816(E[n + u], yl, b[2 * u], b[2 * u + 1]);
            mma16816(E[n + u], yh, d[2 * u], d[2 * u + 1]);
          }
        }
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ex + n * 512), "f"(E[n][0]), "f"(E[n][1]), "f"(E[n][2]),
                     "f"(E[n][3]) : "memory");
#pragma unroll
        for (int e = 0; e < 4; ++e) out[n][e] *= p.scale * eg[e >> 1];
      }
      add_pairs<D, false>(out, base + L::DP, base + L::K, r0, c0, 0, warp + 1, lane);
      dst = p.dq;
    } else {
#pragma unroll 1
      for (int kk = 0; kk < D; kk += 16) {
        uint32_t vh[4], vl[4];
        load_a_t<64>(base + L::VT, r0, kk, lane, vh);
        load_a_t<64>(base + L::VT + L::TILE, r0, kk, lane, vl);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
          uint32_t b[4], d[4];
          load_b_nn<32>(st + 2 * L::STRIP, kk, n * 8, lane, b);
          load_b_nn<32>(st + 3 * L::STRIP, kk, n * 8, lane, d);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma16816(out[n + u], vh, b[2 * u], b[2 * u + 1]);
            mma16816(out[n + u], vl, b[2 * u], b[2 * u + 1]);
            mma16816(out[n + u], vh, d[2 * u], d[2 * u + 1]);
          }
        }
      }
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) out[n][e] *= el[e >> 1];
      add_pairs<D, false>(out, base + L::DA, base + L::K, r0, c0, 0, warp + 1, lane);
      add_pairs<D, true>(out, base + L::DP, base + L::Q, r0, c0, warp, 4, lane);
      add_pairs<D, true>(out, base + L::DA, base + L::K, r0, c0, warp, 4, lane);
      dst = p.dk;
    }
    __syncthreads();                            // E is there; the strips have been read
    if (id >= 8) {
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        float E[4];
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(E[0]), "=f"(E[1]), "=f"(E[2]), "=f"(E[3])
                     : "r"(ex + n * 512) : "memory");
#pragma unroll
        for (int e = 0; e < 4; ++e) out[n][e] = fmaf(-eg[e >> 1], E[e], out[n][e]);
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (i + 8 * r < len)
          *reinterpret_cast<uint32_t*>(dst + off + (i + 8 * r) * stride + c0 + n * 8 + c2) = pack_bf16x2(out[n][2 * r], out[n][2 * r + 1]);
    if (w + 1 < NW) {
      tot += strips.put(base + L::ST);
      __syncthreads();
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (lane == 0) s_red[threadIdx.x >> 5] = tot;
  __syncthreads();
  if (threadIdx.x >= 32 && threadIdx.x < 32 + C) {
    const int r = threadIdx.x - 32;
    float b = 0.f;
#pragma unroll
    for (int w = 0; w < D / 16; ++w) b += p.yy[(ch * (D / 16) + w) * C + r];
    if (r < len) p.dbeta[(long long)(t + r) * p.H + h] = b;
  }
  if (threadIdx.x < 32) {                        // gradient of G -> gradient of g (suffix sums)
    double x[2] = {0., 0.};
#pragma unroll
    for (int w = 0; w < D / 16; ++w) {
      const long long at = (ch * (D / 16) + w) * C + 2 * lane;
      const float2 a = *reinterpret_cast<const float2*>(p.oo + at), b = *reinterpret_cast<const float2*>(p.nn + at);
      x[0] += (double)a.x - b.x;
      x[1] += (double)a.y - b.y;
    }
    if (lane == 31) {
#pragma unroll
      for (int w = 0; w < GT / 32; ++w) x[1] += s_red[w];
    }
    double run = x[0] + x[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_down_sync(0xffffffffu, run, o);
      if (lane + o < 32) run += y;
    }
    const long long at = (long long)(t + 2 * lane) * p.H + h;
    if (2 * lane < len) p.dg[at] = (float)run;
    if (2 * lane + 1 < len) p.dg[at + p.H] = (float)(run - x[0]);
    if (!landed) drain(smem_u32(&vb_full), 0);
  }
}

template <int D>
int launch_gdr(const GdrParams& p, int T, bool grad, cudaStream_t s) {
  constexpr int PREP = PREP_TILES<D> + C * (C + 4) * 4 + 128;
  constexpr int FWD = ScanSmem<D, 2, false>::TOTAL, SAVE = ScanSmem<D, 3, true>::TOTAL;
  static bool cfg = false;
  cudaError_t e;
  if (!cfg) {
    if ((e = cudaFuncSetAttribute(gdr_prep_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gdr_scan_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gdr_scan_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAVE)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gdr_scan_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAVE)) != cudaSuccess ||
        (e = cudaFuncSetAttribute(gdr_grad_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, GradSmem<D>::TOTAL)) != cudaSuccess)
      return (int)e;
    cfg = true;
  }
  const dim3 chunks(T / C + p.n_seq, p.H);       // at least the number of chunks of any packing of T tokens
  const unsigned scans = (unsigned)p.n_seq * p.H * (D / 64);
  if (!grad) {
    gdr_prep_kernel<D><<<chunks, THREADS, PREP, s>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
    gdr_scan_kernel<D, false><<<scans, ST, FWD, s>>>(p);
    return (int)cudaGetLastError();
  }
  gdr_scan_kernel<D, true><<<scans, ST, SAVE, s>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  gdr_scan_bwd_kernel<D><<<scans, ST, SAVE, s>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  gdr_grad_kernel<D><<<chunks, GT, GradSmem<D>::TOTAL, s>>>(p);
  return (int)cudaGetLastError();
}

int run_gdr(const GdrParams& p, int T, int D, bool grad, cudaStream_t s) {
  if (D == 128) return launch_gdr<128>(p, T, grad, s);
  if (D == 64) return launch_gdr<64>(p, T, grad, s);
  return -3;
}

GdrParams common(const void* q, const void* k, const void* v, const float* g, const float* beta, const int* cu, void* mp, float* gb,
                 int T, int n_seq, int H, float scale) {
  GdrParams p{};
  p.q = (const __nv_bfloat16*)q; p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
  p.g = g; p.beta = beta; p.cu = cu; p.mp = (__nv_bfloat16*)mp; p.gb = gb; p.T = T; p.n_seq = n_seq; p.H = H; p.scale = scale;
  return p;
}

}  // namespace

extern "C" {

// Chunks a packed batch of T tokens in n_seq sequences can have at most: rows of the workspaces.
int mcb_gdr_chunks(int T, int n_seq) { return T / C + n_seq; }

// q, k, v, o [T, H, D] bf16; g, beta [T, H] fp32; cu_seqlens [n_seq + 1] int32 from 0 to T.  Workspaces, per chunk and
// head: mp [2, 3, 10, 16, 16] bf16, gb [6, 64] fp32; the backward pass reads them again.  Boundaries outside the batch are clipped
// and reported through `status`.
int mcb_gdr_fwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const int* cu_seqlens, void* o,
                void* mp, float* gb, int T, int n_seq, int H, int D, float scale, int* status, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GdrParams p = common(q, k, v, g, beta, cu_seqlens, mp, gb, T, n_seq, H, scale);
  p.o = (__nv_bfloat16*)o;
  p.status = status;
  return run_gdr(p, T, D, false, reinterpret_cast<cudaStream_t>(stream_));
}

// mp and gb as the forward pass left them.  Further workspaces, per chunk and head: states [2, D, D] fp32 (all S first, then
// all dS), values [2, 2, D, 64] bf16 (all V, then all B), predictions [D, 64] fp32, dots [3, D / 16, 64] fp32.
int mcb_gdr_bwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const int* cu_seqlens,
                const void* dout, void* dq, void* dk, void* dv, float* dg, float* dbeta, void* mp, float* gb,
                float* states, void* values, float* predictions, float* dots, int T, int n_seq, int H, int D, float scale,
                int* status, void* stream_) {
  if (n_seq <= 0 || T <= 0) return 0;
  GdrParams p = common(q, k, v, g, beta, cu_seqlens, mp, gb, T, n_seq, H, scale);
  const long long n = (long long)mcb_gdr_chunks(T, n_seq) * H;
  p.dout = (const __nv_bfloat16*)dout;
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv; p.dg = dg; p.dbeta = dbeta;
  p.S = states; p.dS = p.S + n * D * D;
  p.V = (__nv_bfloat16*)values; p.B = p.V + n * 2 * D * C;
  p.E = predictions;
  p.oo = dots; p.nn = p.oo + n * (D / 16) * C; p.yy = p.nn + n * (D / 16) * C;
  p.status = status;
  return run_gdr(p, T, D, true, reinterpret_cast<cudaStream_t>(stream_));
}

}  // extern "C"
