// Everything between the input projection of a gated-DeltaNet block and its delta rule, one pass each way.
//
// The projection row of a token holds, per key-head group, [q (d) | k (d) | v (R d) | z (R d) | b (R) | a (R)].  Forward:
// causal depthwise conv (4 taps) + SiLU over q | k | v, L2 normalisation of q and k, q and k repeated for the R value heads
// of the group, z copied out, beta = sigmoid(b), g = -exp(A_log) softplus(a + dt_bias).  Backward: the gradient of the
// whole projection row, of the taps and of the two per-head vectors; everything in between is recomputed from the
// projection, which is all that is kept.
//
// A warp owns one slice of a group (q, k, one of the R times v, or z and the gates) and walks consecutive tokens with the last
// rows in registers, so every projection element is read once (plus 3 rows of overlap per walk) instead of once per slice,
// copy, norm and tap.
//
// Bound: the latency of the rows.  Four rows are in flight per warp, kept as they lie in memory, and a row's registers are
// loaded again as soon as it is widened; loading four rows, using them up and loading the next four left the schedulers idle
// for 68 % of the cycles, half of the stalls waiting for these loads.  Measured, 4096 tokens, 16 groups, R = 2, d = 128, that
// way / this way: forward 94 / 67 us, backward 280 / 146 (the copy rate would take 36 and 70); 300 tokens 32 / 16 and 83 / 36;
// R = 1 66 / 52 and 210 / 118; d = 64 66 / 45 and 165 / 89.
//
// Values are rounded to bf16 where the separate operators store them (convolution output, normalised q / k).
#include "../common/host_utils.cuh"
#include "../common/partials.cuh"
#include "../common/ptx.cuh"

#include <type_traits>

using namespace mcb;

namespace {

constexpr int KW = 4;            // taps
constexpr int WARPS = 4;
constexpr int TOK_F = 16;        // tokens a warp walks, forward / backward (which repeats 3 tokens of the next walk):
constexpr int TOK_B = 32;        // enough warps at a few thousand tokens

struct InParams {
  const __nv_bfloat16* proj;               // [T, ld]
  const __nv_bfloat16 *w, *A_log, *dt;     // [G * (2 + R) d, 4], [G * R], [G * R]
  const int* seq_start;                    // [T]
  __nv_bfloat16 *q, *k, *v, *z;            // [T, G * R, d]
  float *g, *beta;                         // [T, G * R]
  const __nv_bfloat16 *dq, *dk, *dv, *dz;
  const float *dg, *dbeta;
  __nv_bfloat16* dproj;                    // [T, ld_d]
  float* wpart;                            // [blocks along T, G * (2 + R) d * 4]
  float* hpart;                            // [blocks along T, 2 * G * R]: dA_log, ddt_bias
  long long ld, ld_d;
  int T, G;
};

__device__ __forceinline__ float wsum(float x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// SiLU's sigmoid: fast exponential and division, as in the stand-alone convolution (its result is rounded to bf16)
__device__ __forceinline__ float sigmoid_(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
__device__ __forceinline__ float bf_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

// The gates, as torch evaluates them: results fp32, infinite arguments included (an infinite gate is open or shut, A_log =
// -inf never decays).  The decays are summed over hundreds of tokens before they are exponentiated, so these functions are
// the full-precision ones: this file is compiled without --use_fast_math (build_ext.py).
__device__ __forceinline__ float gate_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float softplus_(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// N consecutive bf16 (N even) at a 4-byte aligned address: as they are, and as floats
template <int N>
__device__ __forceinline__ void ldn(const __nv_bfloat16* p, uint32_t (&x)[N / 2]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) x[i] = reinterpret_cast<const uint32_t*>(p)[i];
}
template <int N>
__device__ __forceinline__ void widen(const uint32_t (&x)[N / 2], float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
template <int N>
__device__ __forceinline__ void ldn(const __nv_bfloat16* p, float (&f)[N]) {
  uint32_t x[N / 2];
  ldn<N>(p, x);
  widen<N>(x, f);
}
template <int N>
__device__ __forceinline__ void stn(__nv_bfloat16* p, const uint32_t (&x)[N / 2]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) reinterpret_cast<uint32_t*>(p)[i] = x[i];
}
template <int N>
__device__ __forceinline__ void stn(__nv_bfloat16* p, const float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) *reinterpret_cast<uint32_t*>(p + i) = pack_bf16x2(f[i], f[i + 1]);
}

// The projection row of a group has S = 2 + R convolved slices of d channels (q, k, R times v), then z and the gates.  A
// block's z index names one slice, or (index S) z and the gates; a lane owns PER = d / 32 consecutive channels.
template <int D, int R>
__global__ void __launch_bounds__(WARPS * 32)
gdn_inputs_fwd_kernel(const InParams p) {
  constexpr int PER = D / 32, S = 2 + R;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = blockIdx.y, s = blockIdx.z;
  const int t0 = (blockIdx.x * WARPS + warp) * TOK_F, t1 = min(t0 + TOK_F, p.T);
  if (t0 >= p.T) return;
  const __nv_bfloat16* src = p.proj + (long long)grp * (2 * D + 2 * R * D + 2 * R) + s * D + lane * PER;
  auto out_row = [&](int t) { return ((long long)t * p.G + grp) * R * D + lane * PER; };
  if (s == S) {                                  // z and the gates
    const int hv = lane < R ? grp * R + lane : 0;
    const float neg_a = lane < R ? -expf(__bfloat162float(p.A_log[hv])) : 0.f;
    const float dtb = lane < R ? __bfloat162float(p.dt[hv]) : 0.f;
    for (int tb = t0; tb < t1; tb += KW) {
      uint32_t z[KW][R][PER / 2];                // four rows in flight
      __nv_bfloat16 b[KW], a[KW];
#pragma unroll
      for (int u = 0; u < KW; ++u) {
        const __nv_bfloat16* row = src + (tb + u) * p.ld;
        if (tb + u >= t1) break;
#pragma unroll
        for (int r = 0; r < R; ++r) ldn<PER>(row + r * D, z[u][r]);
        if (lane < R) {
          b[u] = row[R * D + lane - lane * PER];
          a[u] = row[R * D + R + lane - lane * PER];
        }
      }
#pragma unroll
      for (int u = 0; u < KW; ++u) {
        const int t = tb + u;
        if (t >= t1) break;
#pragma unroll
        for (int r = 0; r < R; ++r) stn<PER>(p.z + out_row(t) + r * D, z[u][r]);
        if (lane < R) {
          const long long at = (long long)t * p.G * R + hv;
          p.beta[at] = gate_sigmoid(__bfloat162float(b[u]));
          p.g[at] = neg_a * softplus_(__bfloat162float(a[u]) + dtb);
        }
      }
    }
    return;
  }
  float w[PER][KW], x[KW][PER];                  // row t is slot t & 3
#pragma unroll
  for (int c = 0; c < PER; ++c)
#pragma unroll
    for (int j = 0; j < KW; ++j)
      w[c][j] = __bfloat162float(p.w[(((long long)grp * S + s) * D + lane * PER + c) * KW + j]);
#pragma unroll
  for (int u = 0; u < KW; ++u)
#pragma unroll
    for (int c = 0; c < PER; ++c) x[u][c] = 0.f;
#pragma unroll
  for (int b = 1; b < KW; ++b)
    if (t0 - b >= 0) ldn<PER>(src + (t0 - b) * p.ld, x[KW - b]);    // t0 is a multiple of 4
  uint32_t nx[KW][PER / 2];                      // the next four rows, in flight: a row's slot is loaded again once it is read
  int first[KW];
  auto fetch = [&](int t, int u) {
    if (t < t1) {
      ldn<PER>(src + t * p.ld, nx[u]);
      first[u] = p.seq_start[t];
    }
  };
#pragma unroll
  for (int u = 0; u < KW; ++u) fetch(t0 + u, u);
  for (int tb = t0; tb < t1; tb += KW) {
#pragma unroll
    for (int u = 0; u < KW; ++u) {
      const int t = tb + u;
      if (t >= t1) break;
      widen<PER>(nx[u], x[u]);
      const int back = t - first[u];             // rows of the same sequence before this one
      fetch(t + KW, u);
      float y[PER];
#pragma unroll
      for (int c = 0; c < PER; ++c) {
        float a = 0.f;
        if (back >= KW - 1) {                    // the whole window lies in the sequence (the same for all lanes)
#pragma unroll
          for (int j = 0; j < KW; ++j) a = fmaf(w[c][j], x[(u + 1 + j) & 3][c], a);
        } else {
#pragma unroll
          for (int j = 0; j < KW; ++j) a = fmaf(w[c][j], (KW - 1 - j) <= back ? x[(u + 1 + j) & 3][c] : 0.f, a);
        }
        y[c] = bf_round(a * sigmoid_(a));
      }
      if (s >= 2) {
        stn<PER>(p.v + out_row(t) + (s - 2) * D, y);
      } else {
        float ss = 0.f;
#pragma unroll
        for (int c = 0; c < PER; ++c) ss += y[c] * y[c];
        const float r = rsqrtf(wsum(ss) + 1e-6f);
#pragma unroll
        for (int c = 0; c < PER; ++c) y[c] *= r;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) stn<PER>((s == 0 ? p.q : p.k) + out_row(t) + rr * D, y);
      }
    }
  }
}

// Backward.  Four rows whose windows lie in one sequence go through straight-line code, in which they overlap.  That takes 154 ..
// 168 registers at d = 128 (96 at 64) and spills at 128 (80), so three (five) CTAs share an SM instead of four (six).  us, row by
// row with four (six) / straight with four (six) / straight with three (five), 4096 tokens: d = 128, R = 2, 16 groups 194 / 196 / 146,
// R = 1 118 / 138 / 118, R = 4, 8 groups 181 / 169 / 118; d = 64, R = 1 97 / 93 / 73, R = 2 105 / 87 / 89, R = 4 97 / 101 / 77.
template <int D, int R>
__global__ void __launch_bounds__(WARPS * 32, D == 128 ? 3 : 5)
gdn_inputs_bwd_kernel(const InParams p) {
  constexpr int PER = D / 32, S = 2 + R;
  __shared__ float s_w[WARPS][D * KW];
  __shared__ float s_h[WARPS][2][R];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = blockIdx.y, s = blockIdx.z;
  const int t0 = (blockIdx.x * WARPS + warp) * TOK_B, t1 = min(t0 + TOK_B, p.T);
  const int width = 2 * D + 2 * R * D + 2 * R;
  const __nv_bfloat16* src = p.proj + (long long)grp * width + s * D + lane * PER;
  __nv_bfloat16* dst = p.dproj + (long long)grp * width + s * D + lane * PER;
  auto grad_row = [&](int t) { return ((long long)t * p.G + grp) * R * D + lane * PER; };
  if (s == S) {                                  // z and the gates
    const int hv = lane < R ? grp * R + lane : 0;
    const float neg_a = lane < R ? -expf(__bfloat162float(p.A_log[hv])) : 0.f;
    const float dtb = lane < R ? __bfloat162float(p.dt[hv]) : 0.f;
    float dA = 0.f, ddt = 0.f;
    for (int tb = t0; tb < t1; tb += KW) {
      uint32_t z[KW][R][PER / 2];                // four rows in flight
      __nv_bfloat16 b[KW], a[KW];
      float db[KW], dgs[KW];
#pragma unroll
      for (int u = 0; u < KW; ++u) {
        const int t = tb + u;
        if (t >= t1) break;
#pragma unroll
        for (int r = 0; r < R; ++r) ldn<PER>(p.dz + grad_row(t) + r * D, z[u][r]);
        if (lane < R) {
          const __nv_bfloat16* ba = src - lane * PER + t * p.ld + R * D + lane;
          const long long at = (long long)t * p.G * R + hv;
          b[u] = ba[0];
          a[u] = ba[R];
          db[u] = p.dbeta[at];
          dgs[u] = p.dg[at];
        }
      }
#pragma unroll
      for (int u = 0; u < KW; ++u) {
        const int t = tb + u;
        if (t >= t1) break;
#pragma unroll
        for (int r = 0; r < R; ++r) stn<PER>(dst + t * p.ld_d + r * D, z[u][r]);
        if (lane < R) {
          __nv_bfloat16* dba = dst - lane * PER + t * p.ld_d + R * D + lane;
          const float beta = gate_sigmoid(__bfloat162float(b[u]));
          dba[0] = __float2bfloat16(db[u] * beta * (1.f - beta));
          const float xx = __bfloat162float(a[u]) + dtb, dg = dgs[u];
          const float da = dg * neg_a * gate_sigmoid(xx);
          dba[R] = __float2bfloat16(da);
          dA += dg * neg_a * softplus_(xx);
          ddt += da;
        }
      }
    }
    if (lane < R) {
      s_h[warp][0][lane] = dA;
      s_h[warp][1][lane] = ddt;
    }
    __syncthreads();
    if (threadIdx.x < 2 * R) {                   // the block's sums, in a fixed order
      const int which = threadIdx.x / R, r = threadIdx.x % R;
      p.hpart[(long long)blockIdx.x * 2 * p.G * R + which * p.G * R + grp * R + r] =
          (s_h[0][which][r] + s_h[1][which][r]) + (s_h[2][which][r] + s_h[3][which][r]);
    }
    return;
  }
  float dw[PER][KW];
#pragma unroll
  for (int c = 0; c < PER; ++c)
#pragma unroll
    for (int j = 0; j < KW; ++j) dw[c][j] = 0.f;
  if (t0 < t1) {
    float w[PER][KW], x[KW][PER], dp[KW][PER];   // row t and its dpre in slot t & 3
#pragma unroll
    for (int c = 0; c < PER; ++c)
#pragma unroll
      for (int j = 0; j < KW; ++j)
        w[c][j] = __bfloat162float(p.w[(((long long)grp * S + s) * D + lane * PER + c) * KW + j]);
#pragma unroll
    for (int u = 0; u < KW; ++u)
#pragma unroll
      for (int c = 0; c < PER; ++c) x[u][c] = dp[u][c] = 0.f;
    int start[KW];                               // first token of the sequence of row t, in slot t & 3
#pragma unroll
    for (int u = 0; u < KW; ++u) start[u] = 0x7fffffff;
#pragma unroll
    for (int b = 1; b < KW; ++b)
      if (t0 - b >= 0) ldn<PER>(src + (t0 - b) * p.ld, x[KW - b]);
    const int last = t1 + KW - 1;                // dpre of the KW - 1 tokens behind the walk reaches into it
    const int te = min(last, p.T);
    // four rows and their gradients in flight: a row's slot is loaded again once it is read
    const __nv_bfloat16* dn = (s == 0 ? p.dq : s == 1 ? p.dk : p.dv) + (s < 2 ? 0 : s - 2) * D;
    uint32_t nx[KW][PER / 2], nd[KW][R][PER / 2];
    int nf[KW];                                  // of four rows, loaded four rows ahead
    auto fetch = [&](int t, int u) {
      ldn<PER>(src + t * p.ld, nx[u]);
      ldn<PER>(dn + grad_row(t), nd[u][0]);
      if (s < 2) {
#pragma unroll
        for (int r = 1; r < R; ++r) ldn<PER>(dn + grad_row(t) + r * D, nd[u][r]);
      }
    };
    auto row = [&](auto whole, int t, int u) {
      constexpr bool W = decltype(whole)::value;
      if (!W) {
#pragma unroll
        for (int c = 0; c < PER; ++c) dp[u][c] = 0.f;
      }
      if (W || t < te) {
        const int back = t - start[u];
        float pre[PER], sg[PER], y[PER], d[PER];
        widen<PER>(nx[u], x[u]);
        widen<PER>(nd[u][0], d);
        if (s < 2) {
#pragma unroll
          for (int r = 1; r < R; ++r) {
            float e[PER];
            widen<PER>(nd[u][r], e);
#pragma unroll
            for (int c = 0; c < PER; ++c) d[c] += e[c];
          }
        }
        if (W || t + KW < te) fetch(t + KW, u);
#pragma unroll
        for (int c = 0; c < PER; ++c) {
          float a = 0.f;
          if (W || back >= KW - 1) {
#pragma unroll
            for (int j = 0; j < KW; ++j) a = fmaf(w[c][j], x[(u + 1 + j) & 3][c], a);
          } else {
#pragma unroll
            for (int j = 0; j < KW; ++j) a = fmaf(w[c][j], (KW - 1 - j) <= back ? x[(u + 1 + j) & 3][c] : 0.f, a);
          }
          pre[c] = a;
          sg[c] = sigmoid_(a);
          y[c] = bf_round(a * sg[c]);
        }
        if (s < 2) {                             // through y * rsqrt(sum y^2 + eps)
          float ss = 0.f, dot = 0.f;
#pragma unroll
          for (int c = 0; c < PER; ++c) {
            ss += y[c] * y[c];
            dot += y[c] * d[c];
          }
          const float r = rsqrtf(wsum(ss) + 1e-6f);
          dot = wsum(dot) * r * r;
#pragma unroll
          for (int c = 0; c < PER; ++c) d[c] = r * (d[c] - y[c] * dot);
        }
#pragma unroll
        for (int c = 0; c < PER; ++c) {
          dp[u][c] = d[c] * sg[c] * (1.f + pre[c] * (1.f - sg[c]));
          if (W || t < t1) {                     // every token's tap gradients are added once, by its own walk
            if (W || back >= KW - 1) {
#pragma unroll
              for (int j = 0; j < KW; ++j) dw[c][j] = fmaf(dp[u][c], x[(u + 1 + j) & 3][c], dw[c][j]);
            } else {
#pragma unroll
              for (int j = 0; j < KW; ++j)
                dw[c][j] = fmaf(dp[u][c], (KW - 1 - j) <= back ? x[(u + 1 + j) & 3][c] : 0.f, dw[c][j]);
            }
          }
        }
      }
      // dpre of the rows t-3 .. t is complete for the projection row t - 3, as far as they share its sequence
      const int tr = t - (KW - 1);
      if (W || (tr >= t0 && tr < t1)) {
        float dx[PER];
#pragma unroll
        for (int c = 0; c < PER; ++c) dx[c] = 0.f;
#pragma unroll
        for (int j = 0; j < KW; ++j) {           // tap j of row t - j
          if (W || start[(u + 4 - j) & 3] <= tr) {
#pragma unroll
            for (int c = 0; c < PER; ++c) dx[c] = fmaf(w[c][j], dp[(u + 4 - j) & 3][c], dx[c]);
          }
        }
        stn<PER>(dst + tr * p.ld_d, dx);
      }
    };
    auto first_token = [&](int t) { return t < te ? p.seq_start[t] : 0x7fffffff; };   // past the batch: in no sequence
#pragma unroll
    for (int u = 0; u < KW; ++u) {
      nf[u] = first_token(t0 + u);
      if (t0 + u < te) fetch(t0 + u, u);
    }
    for (int tb = t0; tb < last; tb += KW) {
      // four rows and those loaded meanwhile inside the walk, each row's window inside its sequence: straight-line code, in
      // which the rows overlap
      bool whole = tb > t0 && tb + KW <= t1 && tb + 2 * KW <= te;
#pragma unroll
      for (int u = 0; u < KW; ++u) whole &= tb + u - nf[u] >= KW - 1;
      if (whole) {
#pragma unroll
        for (int u = 0; u < KW; ++u) {
          start[u] = nf[u];
          nf[u] = p.seq_start[tb + KW + u];
        }
#pragma unroll
        for (int u = 0; u < KW; ++u) row(std::true_type{}, tb + u, u);
        continue;
      }
#pragma unroll
      for (int u = 0; u < KW; ++u) {
        if (tb + u >= last) break;
        start[u] = nf[u];
        nf[u] = first_token(tb + KW + u);
        row(std::false_type{}, tb + u, u);
      }
    }
  }
  // the block's sums, in a fixed order
#pragma unroll
  for (int c = 0; c < PER; ++c)
#pragma unroll
    for (int j = 0; j < KW; ++j) s_w[warp][(lane * PER + c) * KW + j] = dw[c][j];
  __syncthreads();
  for (int id = threadIdx.x; id < D * KW; id += WARPS * 32)
    p.wpart[((long long)blockIdx.x * p.G * S + (long long)grp * S + s) * D * KW + id] =
        (s_w[0][id] + s_w[1][id]) + (s_w[2][id] + s_w[3][id]);
}

int blocks_t(int T, int tok) { return (T + WARPS * tok - 1) / (WARPS * tok); }

template <int D, int R>
int launch_inputs(const InParams& p, bool grad, float* dw, float* dA, float* ddt, cudaStream_t s) {
  if (!grad) {
    gdn_inputs_fwd_kernel<D, R><<<dim3(blocks_t(p.T, TOK_F), p.G, 3 + R), WARPS * 32, 0, s>>>(p);
    return (int)cudaGetLastError();
  }
  const int nb = blocks_t(p.T, TOK_B);
  gdn_inputs_bwd_kernel<D, R><<<dim3(nb, p.G, 3 + R), WARPS * 32, 0, s>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  launch_reduce_partials<float>(p.wpart, nb, p.G * (2 + R) * D * KW, dw, nullptr, p.G * (2 + R) * D * KW, s);
  if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  launch_reduce_partials<float>(p.hpart, nb, 2 * p.G * R, dA, ddt, p.G * R, s);
  return (int)cudaGetLastError();
}

int run_inputs(const InParams& p, int D, int R, bool grad, float* dw, float* dA, float* ddt, cudaStream_t s) {
  if ((p.ld & 1) || (p.ld_d & 1)) return -2;     // rows start on 4-byte boundaries
  if (D == 128 && R == 1) return launch_inputs<128, 1>(p, grad, dw, dA, ddt, s);
  if (D == 128 && R == 2) return launch_inputs<128, 2>(p, grad, dw, dA, ddt, s);
  if (D == 128 && R == 4) return launch_inputs<128, 4>(p, grad, dw, dA, ddt, s);
  if (D == 64 && R == 1) return launch_inputs<64, 1>(p, grad, dw, dA, ddt, s);
  if (D == 64 && R == 2) return launch_inputs<64, 2>(p, grad, dw, dA, ddt, s);
  if (D == 64 && R == 4) return launch_inputs<64, 4>(p, grad, dw, dA, ddt, s);
  return -3;
}

}  // namespace

extern "C" {

// Rows of the two partial-sum workspaces of the backward pass.
int mcb_gdn_inputs_partials(int T) { return blocks_t(T, TOK_B); }

// proj [T, ld] bf16 with G groups of [q d | k d | v R d | z R d | b R | a R]; w [G (2 + R) d, 4]; A_log, dt_bias [G R] bf16;
// seq_start [T] int32.  Out: q, k, v, z [T, G R, d] bf16, g, beta [T, G R] fp32.
int mcb_gdn_inputs_fwd(const void* proj, long long ld, const void* w, const void* A_log, const void* dt, const int* seq_start,
                       void* q, void* k, void* v, void* z, float* g, float* beta, int T, int G, int R, int D, void* stream_) {
  if (T <= 0) return 0;
  InParams p{};
  p.proj = (const __nv_bfloat16*)proj; p.ld = ld; p.w = (const __nv_bfloat16*)w; p.A_log = (const __nv_bfloat16*)A_log;
  p.dt = (const __nv_bfloat16*)dt; p.seq_start = seq_start;
  p.q = (__nv_bfloat16*)q; p.k = (__nv_bfloat16*)k; p.v = (__nv_bfloat16*)v; p.z = (__nv_bfloat16*)z; p.g = g; p.beta = beta;
  p.T = T; p.G = G;
  return run_inputs(p, D, R, false, nullptr, nullptr, nullptr, reinterpret_cast<cudaStream_t>(stream_));
}

// dproj [T, G (2 d + 2 R d + 2 R)] contiguous; dw, dA, ddt fp32, zero on entry; wpart [partials, G (2 + R) d 4],
// hpart [partials, 2 G R] fp32 workspaces.
int mcb_gdn_inputs_bwd(const void* proj, long long ld, const void* w, const void* A_log, const void* dt, const int* seq_start,
                       const void* dq, const void* dk, const void* dv, const void* dz, const float* dg, const float* dbeta,
                       void* dproj, float* dw, float* dA, float* ddt, float* wpart, float* hpart, int T, int G, int R, int D,
                       void* stream_) {
  if (T <= 0) return 0;
  InParams p{};
  p.proj = (const __nv_bfloat16*)proj; p.ld = ld; p.w = (const __nv_bfloat16*)w; p.A_log = (const __nv_bfloat16*)A_log;
  p.dt = (const __nv_bfloat16*)dt; p.seq_start = seq_start;
  p.dq = (const __nv_bfloat16*)dq; p.dk = (const __nv_bfloat16*)dk; p.dv = (const __nv_bfloat16*)dv;
  p.dz = (const __nv_bfloat16*)dz; p.dg = dg; p.dbeta = dbeta;
  p.dproj = (__nv_bfloat16*)dproj; p.ld_d = (long long)G * (2 * D + 2 * R * D + 2 * R);
  p.wpart = wpart; p.hpart = hpart; p.T = T; p.G = G;
  return run_inputs(p, D, R, true, dw, dA, ddt, reinterpret_cast<cudaStream_t>(stream_));
}

}  // extern "C"
