// Element-wise kernels of the linear-attention blocks (gated DeltaNet, lightning attention).
//
//   causal depthwise conv1d (+SiLU) forward / backward over packed sequences          (memory bound)
//   gated RMSNorm  y = rmsnorm(x) * w * silu(z)  forward / backward                  (memory bound)
//   (the operators themselves: gated_delta_rule.cu with gdn_inputs.cu, simple_gla.cu)
//
// Packed sequences are described by `seq_start[t]` (index of the first token of t's sequence), as in the attention
// kernels: no host synchronisation, histories never cross a sequence boundary.
#include <initializer_list>
#include "../common/host_utils.cuh"
#include "../common/ptx.cuh"

using namespace mcb;

namespace {

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]);
  o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]);
  o.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = o;
}

// the KW taps of 8 consecutive channels are 8 * KW contiguous bf16 (w is [C, KW]): fetched with 16-byte loads when the
// span is a multiple of 16 bytes, which it is for KW = 2 and 4
template <int KW>
__device__ __forceinline__ void load_taps(const __nv_bfloat16* __restrict__ w, int c0, float (&wt)[8][KW]) {
  if constexpr ((8 * KW * 2) % 16 == 0) {
    const uint4* src = reinterpret_cast<const uint4*>(w + (long long)c0 * KW);
    float flat[8 * KW];
#pragma unroll
    for (int v = 0; v < 8 * KW / 8; ++v) {
      const uint4 raw = src[v];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(h[i]);
        flat[v * 8 + 2 * i] = t.x;
        flat[v * 8 + 2 * i + 1] = t.y;
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int j = 0; j < KW; ++j) wt[c][j] = flat[c * KW + j];
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
      for (int j = 0; j < KW; ++j) wt[c][j] = __bfloat162float(w[(c0 + c) * KW + j]);
  }
}

// ------------------------------------------------------------------------------------------ causal conv1d + SiLU
// x, y [T, C] bf16; w [C, KW] bf16 (KW <= 4); thread = (token, 8 channels)
template <int KW>
__global__ void conv1d_silu_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                       const int* __restrict__ seq_start, __nv_bfloat16* __restrict__ y, int T, int C,
                                       int act) {
  const int cv = C / 8;
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= (long long)T * cv) return;
  const int t = int(id / cv), c0 = int(id % cv) * 8;
  const int s0 = seq_start[t];
  float wt[8][KW];
  load_taps<KW>(w, c0, wt);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < KW; ++j) {
    const int tt = t - (KW - 1) + j;
    if (tt >= s0) {
      float f[8];
      load8(x + (long long)tt * C + c0, f);
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[c] = fmaf(wt[c][j], f[c], acc[c]);
    }
  }
  if (act) {
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = acc[c] * sigmoidf_(acc[c]);
  }
  store8(y + (long long)t * C + c0, acc);
}

// dx [T, C] bf16, dw [C, KW] fp32 (accumulated with atomics; zeroed by the caller).  Block = 32 tokens x 8-channel
// groups: each thread walks 32 consecutive tokens of its channels so the dw partial sums stay in registers.
template <int KW>
__global__ void conv1d_silu_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                       const __nv_bfloat16* __restrict__ dy, const int* __restrict__ seq_start,
                                       __nv_bfloat16* __restrict__ dx, float* __restrict__ dw, int T, int C, int act) {
  constexpr int TOK = 32;
  const int cv = C / 8;
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nchunk = (T + TOK - 1) / TOK;
  if (id >= (long long)nchunk * cv) return;
  const int chunk = int(id / cv), c0 = int(id % cv) * 8;
  const int t_lo = chunk * TOK, t_hi = min(T, t_lo + TOK);
  float wt[8][KW], dwa[8][KW];
  load_taps<KW>(w, c0, wt);
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int j = 0; j < KW; ++j) dwa[c][j] = 0.f;
  // dpre of tokens t .. t+KW-1 is needed for dx[t]; walk tokens and keep a window of dpre values
  // dpre[u] = dy[u] * d silu(pre[u]),  pre[u] = sum_j w[j] x[u-(KW-1)+j]
  auto dpre_at = [&](int u, bool own, float (&out)[8]) {
    const int s0 = seq_start[u];
    float pre[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float xs[KW][8];
#pragma unroll
    for (int j = 0; j < KW; ++j) {
      const int tt = u - (KW - 1) + j;
      if (tt >= s0) {
        load8(x + (long long)tt * C + c0, xs[j]);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) xs[j][c] = 0.f;
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) pre[c] = fmaf(wt[c][j], xs[j][c], pre[c]);
    }
    float g[8];
    load8(dy + (long long)u * C + c0, g);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float d = g[c];
      if (act) {
        const float s = sigmoidf_(pre[c]);
        d *= s * (1.f + pre[c] * (1.f - s));
      }
      out[c] = d;
      if (own) {   // every token's weight-gradient term is added exactly once, by the thread that owns the token
#pragma unroll
        for (int j = 0; j < KW; ++j) dwa[c][j] = fmaf(d, xs[j][c], dwa[c][j]);
      }
    }
  };
  for (int t = t_lo; t < t_hi; ++t) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int s0 = seq_start[t];
    // dx[t] = sum_j w[j] * dpre[t + (KW-1) - j]  for targets in the same sequence
#pragma unroll
    for (int j = 0; j < KW; ++j) {
      const int u = t + (KW - 1) - j;
      if (u < T && seq_start[u] == s0) {
        float d[8];
        dpre_at(u, u == t, d);
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = fmaf(wt[c][j], d[c], acc[c]);
      }
    }
    store8(dx + (long long)t * C + c0, acc);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int j = 0; j < KW; ++j) atomicAdd(&dw[(c0 + c) * KW + j], dwa[c][j]);
}

// ------------------------------------------------------------------------------------------ gated RMSNorm
// rows x D (D = 64, 128 or 256), D / 8 lanes to a row, eight columns a lane; the warp's next rows are loaded while it works on these.
// y = x * rstd * w * silu(z).  WIDE: all tensors start on 16-byte boundaries.  us, a warp to a row, two bytes a lane / now, forward and
// backward: 131072 x 128 31, 47 / 25, 39, x 64 22, 35 / 16, 23; 65536 x 256 31, 47 / 25, 39.
template <bool WIDE>
__device__ __forceinline__ uint4 row8(const __nv_bfloat16* p) {
  if (WIDE) return *reinterpret_cast<const uint4*>(p);
  uint32_t v[4];
  const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = h[2 * i] | (uint32_t)h[2 * i + 1] << 16;
  return make_uint4(v[0], v[1], v[2], v[3]);
}
template <bool WIDE>
__device__ __forceinline__ void put_row8(__nv_bfloat16* p, const float (&f)[8]) {
  if (WIDE) {
    store8(p, f);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = __float2bfloat16(f[i]);
  }
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[i]));
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
template <int LANES>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LANES / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int D, bool WIDE>
__global__ void __launch_bounds__(256, 5)
gated_rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ w,
                         __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, long long rows, float eps) {
  constexpr int LANES = D / 8, PER = 32 / LANES;            // rows of a warp
  const int lane = threadIdx.x & 31, c0 = lane % LANES * 8;
  const long long step = (((long long)gridDim.x * blockDim.x) >> 5) * PER;
  long long first = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * PER;   // of the warp
  float wv[8];
  unpack8(row8<WIDE>(w + c0), wv);
  uint4 xr, zr;
  auto fetch = [&](long long row) {
    xr = zr = make_uint4(0, 0, 0, 0);
    if (row >= rows) return;
    xr = row8<WIDE>(x + row * D + c0);
    zr = row8<WIDE>(z + row * D + c0);
  };
  fetch(first + lane / LANES);
  for (; first < rows; first += step) {
    const long long row = first + lane / LANES;
    float xv[8], zv[8], o[8], ss = 0.f;
    unpack8(xr, xv);
    unpack8(zr, zv);
    fetch(row + step);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += xv[i] * xv[i];
    const float r = rsqrtf(group_sum<LANES>(ss) / D + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // the normalised value is rounded to bf16 before the weight multiply, as the module it replaces does
      const float n = __bfloat162float(__float2bfloat16(xv[i] * r));
      o[i] = wv[i] * n * zv[i] * sigmoidf_(zv[i]);
    }
    if (row < rows) {
      put_row8<WIDE>(y + row * D + c0, o);
      if (c0 == 0) rstd[row] = r;
    }
  }
}

template <int D, bool WIDE>
__global__ void __launch_bounds__(256)
gated_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ w,
                         const __nv_bfloat16* __restrict__ dy, const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx,
                         __nv_bfloat16* __restrict__ dz, float* __restrict__ dw, long long rows) {
  constexpr int LANES = D / 8, PER = 32 / LANES;
  __shared__ float dws[D];
  for (int i = threadIdx.x; i < D; i += blockDim.x) dws[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, c0 = lane % LANES * 8;
  const long long step = (((long long)gridDim.x * blockDim.x) >> 5) * PER;
  long long first = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * PER;
  float wv[8], dwl[8] = {};
  unpack8(row8<WIDE>(w + c0), wv);
  uint4 xr, zr, gr;
  float rr = 0.f;
  auto fetch = [&](long long row) {
    xr = zr = gr = make_uint4(0, 0, 0, 0);
    if (row >= rows) return;
    xr = row8<WIDE>(x + row * D + c0);
    zr = row8<WIDE>(z + row * D + c0);
    gr = row8<WIDE>(dy + row * D + c0);
    rr = rstd[row];
  };
  fetch(first + lane / LANES);
  for (; first < rows; first += step) {
    const long long row = first + lane / LANES;
    const float r = rr;
    float xv[8], zv[8], gv[8], gz[8], dn[8], dot = 0.f;
    unpack8(xr, xv);
    unpack8(zr, zv);
    unpack8(gr, gv);
    fetch(row + step);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = sigmoidf_(zv[i]);
      const float n = xv[i] * r;
      gz[i] = gv[i] * wv[i] * n * s * (1.f + zv[i] * (1.f - s));     // d/dz of silu(z)
      dn[i] = gv[i] * wv[i] * zv[i] * s;                             // gradient w.r.t. the normalised value
      dwl[i] += gv[i] * n * zv[i] * s;
      dot += dn[i] * xv[i];
    }
    const float k = group_sum<LANES>(dot) * r * r * r / D;
    if (row < rows) {
#pragma unroll
      for (int i = 0; i < 8; ++i) dn[i] = dn[i] * r - xv[i] * k;
      put_row8<WIDE>(dx + row * D + c0, dn);
      put_row8<WIDE>(dz + row * D + c0, gz);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int o = LANES; o < 32; o <<= 1) dwl[i] += __shfl_xor_sync(0xffffffffu, dwl[i], o);
    if (lane < LANES) atomicAdd(&dws[c0 + i], dwl[i]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(&dw[i], dws[i]);
}

bool on_16_bytes(std::initializer_list<const void*> ps) {
  uintptr_t bits = 0;
  for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
  return bits % 16 == 0;
}
// CTAs for warps of `rows_of_warp` rows, no more than what an SM holds
unsigned row_grid(long long rows, int rows_of_warp, int ctas_per_sm) {
  const long long want = (rows + 8 * rows_of_warp - 1) / (8 * rows_of_warp), cap = (long long)ctas_per_sm * device_sm_count();
  return (unsigned)(want < cap ? want : cap);
}

}  // namespace

extern "C" {

int mcb_conv1d_silu_fwd(const void* x, const void* w, const int* seq_start, void* y, int T, int C, int KW, int act,
                        void* stream_) {
  if (T == 0) return 0;
  if (C % 8) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const long long n = (long long)T * (C / 8);
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (KW == 4)
    conv1d_silu_fwd_kernel<4><<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, seq_start,
                                                   (__nv_bfloat16*)y, T, C, act);
  else if (KW == 2)
    conv1d_silu_fwd_kernel<2><<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, seq_start,
                                                   (__nv_bfloat16*)y, T, C, act);
  else if (KW == 3)
    conv1d_silu_fwd_kernel<3><<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w, seq_start,
                                                   (__nv_bfloat16*)y, T, C, act);
  else
    return -3;
  return (int)cudaGetLastError();
}

// dw [C, KW] fp32 must be zero on entry
int mcb_conv1d_silu_bwd(const void* x, const void* w, const void* dy, const int* seq_start, void* dx, float* dw, int T,
                        int C, int KW, int act, void* stream_) {
  if (T == 0) return 0;
  if (C % 8) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const long long n = (long long)((T + 31) / 32) * (C / 8);
  const unsigned grid = (unsigned)((n + 127) / 128);
#define MCB_CONV_BWD(K_)                                                                                              \
  conv1d_silu_bwd_kernel<K_><<<grid, 128, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w,                    \
                                                  (const __nv_bfloat16*)dy, seq_start, (__nv_bfloat16*)dx, dw, T, C, act)
  if (KW == 4) MCB_CONV_BWD(4);
  else if (KW == 3) MCB_CONV_BWD(3);
  else if (KW == 2) MCB_CONV_BWD(2);
  else return -3;
#undef MCB_CONV_BWD
  return (int)cudaGetLastError();
}

int mcb_gated_rmsnorm_fwd(const void* x, const void* z, const void* w, void* y, float* rstd, long long rows, int D,
                          float eps, void* stream_) {
  if (rows == 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const bool wide = on_16_bytes({x, z, w, y});
#define MCB_GN_FWD(D_)                                                                                               \
  (wide ? gated_rmsnorm_fwd_kernel<D_, true> : gated_rmsnorm_fwd_kernel<D_, false>)                                  \
      <<<row_grid(rows, 256 / D_, 5), 256, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)z, (const __nv_bfloat16*)w,   \
                                                   (__nv_bfloat16*)y, rstd, rows, eps)
  if (D == 128) MCB_GN_FWD(128);
  else if (D == 64) MCB_GN_FWD(64);
  else if (D == 256) MCB_GN_FWD(256);
  else return -3;
#undef MCB_GN_FWD
  return (int)cudaGetLastError();
}

// dw [D] fp32 must be zero on entry
int mcb_gated_rmsnorm_bwd(const void* x, const void* z, const void* w, const void* dy, const float* rstd, void* dx,
                          void* dz, float* dw, long long rows, int D, void* stream_) {
  if (rows == 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  const bool wide = on_16_bytes({x, z, w, dy, dx, dz});
#define MCB_GN_BWD(D_)                                                                                               \
  (wide ? gated_rmsnorm_bwd_kernel<D_, true> : gated_rmsnorm_bwd_kernel<D_, false>)                                  \
      <<<row_grid(rows, 256 / D_, 3), 256, 0, s>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)z, (const __nv_bfloat16*)w,   \
                                                   (const __nv_bfloat16*)dy, rstd, (__nv_bfloat16*)dx, (__nv_bfloat16*)dz, dw, rows)
  if (D == 128) MCB_GN_BWD(128);
  else if (D == 64) MCB_GN_BWD(64);
  else if (D == 256) MCB_GN_BWD(256);
  else return -3;
#undef MCB_GN_BWD
  return (int)cudaGetLastError();
}

}  // extern "C"
