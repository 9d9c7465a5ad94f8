// Fused post-processing of a packed QKV projection: split per query group, per-head RMSNorm on q/k
// (optional), rotary embedding on the first `rot` dims (rotate-half or interleaved pairs), and the
// transposition-free scatter into separate q / k / v (/ gate) tensors the attention kernel reads.
// One pass over the data instead of split + 2 norms + 2 ropes + copies.  Backward is the exact
// transpose (inverse rotation, norm backward, per-head weight gradients).
//
// Packed layout per token (the layout the bridge produces for `linear_qkv`):
//   for each of `ng` groups: [ qpg query heads (each optionally followed by its gate head) | k | v ], head size d.
// cos/sin are per-token tables [T, rot/2] fp32, so positions, packing, context-parallel chunking,
// MRoPE sections and attention scaling are all decided by whoever builds the table.
#include <initializer_list>
#include "../common/partials.cuh"
#include "../common/host_utils.cuh"
#include "../common/ptx.cuh"

using namespace mcb;

namespace {

constexpr int MAX_D = 256;
constexpr int WARPS = 8;
constexpr int FWD_CTAS = 4, BWD_CTAS = 3;   // CTAs an SM holds of the fast kernels

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct QkvLayout {
  int ng, qpg, d, gate;  // gate: 1 -> q heads are interleaved with gate heads
  int rot;               // rotary dims (0 = none)
  int interleaved;       // 1 -> pairs (2i, 2i+1); 0 -> pairs (i, i + rot/2)
  int norm;              // 1 -> per-head RMSNorm on q and k
  int zero_centered;
  float eps;
  long long ld;          // row stride of the packed tensor
};

// slot -> kind: 0 q, 1 gate, 2 k, 3 v ; head index within its output tensor
__device__ __forceinline__ void decode_slot(const QkvLayout& L, int slot, int& kind, int& head) {
  const int per_group = L.qpg * (1 + L.gate) + 2;
  const int g = slot / per_group, r = slot - g * per_group;
  const int nqslots = L.qpg * (1 + L.gate);
  if (r < nqslots) {
    if (L.gate) {
      kind = (r & 1) ? 1 : 0;
      head = g * L.qpg + (r >> 1);
    } else {
      kind = 0;
      head = g * L.qpg + r;
    }
  } else if (r == nqslots) {
    kind = 2;
    head = g;
  } else {
    kind = 3;
    head = g;
  }
}

__global__ void __launch_bounds__(WARPS * 32)
qkv_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
               const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cosb, const float* __restrict__ sinb,
               __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ v,
               __nv_bfloat16* __restrict__ gate, long long T, QkvLayout L) {
  __shared__ float sm[WARPS][MAX_D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slots = L.ng * (L.qpg * (1 + L.gate) + 2);
  const int nq = L.ng * L.qpg, d = L.d, half = L.rot / 2;
  // a block walks tokens, its warps walk the heads of the token: no 64-bit division on the hot path
  for (long long t = blockIdx.x; t < T; t += gridDim.x)
  for (int slot = warp; slot < slots; slot += WARPS) {
    int kind, head;
    decode_slot(L, slot, kind, head);
    const __nv_bfloat16* src = qkv + t * L.ld + (long long)slot * d;
    __nv_bfloat16* dst = kind == 0 ? q + (t * nq + head) * d
                         : kind == 1 ? gate + (t * nq + head) * d
                         : kind == 2 ? k + (t * L.ng + head) * d
                                     : v + (t * L.ng + head) * d;
    if (kind == 1 || kind == 3 || (!L.norm && L.rot == 0)) {
      for (int i = lane * 8; i < d; i += 256) *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(src + i);
      continue;
    }
    float ss = 0.f;
    for (int i = lane * 2; i < d; i += 64) {
      float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + i));
      sm[warp][i] = f.x;
      sm[warp][i + 1] = f.y;
      ss += f.x * f.x + f.y * f.y;
    }
    float rstd = 1.f;
    const __nv_bfloat16* wn = kind == 0 ? wq : wk;
    if (L.norm) {
      ss = warp_sum(ss);
      rstd = rsqrtf(ss / d + L.eps);
    }
    __syncwarp();
    for (int i = lane * 2; i < d; i += 64) {
      float o[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int idx = i + e;
        float val = sm[warp][idx] * rstd;
        if (L.norm) val *= (L.zero_centered ? 1.f : 0.f) + __bfloat162float(wn[idx]);
        if (idx < L.rot) {
          int partner, fi;
          float sign;
          if (L.interleaved) {
            partner = idx ^ 1;
            fi = idx >> 1;
            sign = (idx & 1) ? 1.f : -1.f;
          } else {
            partner = idx < half ? idx + half : idx - half;
            fi = idx < half ? idx : idx - half;
            sign = idx < half ? -1.f : 1.f;
          }
          float pv = sm[warp][partner] * rstd;
          if (L.norm) pv *= (L.zero_centered ? 1.f : 0.f) + __bfloat162float(wn[partner]);
          const float c = cosb[t * half + fi], s = sinb[t * half + fi];
          val = val * c + sign * pv * s;
        }
        o[e] = val;
      }
      *reinterpret_cast<uint32_t*>(dst + i) = pack_bf16x2(o[0], o[1]);
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(WARPS * 32)
qkv_bwd_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
               const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cosb, const float* __restrict__ sinb,
               const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
               const __nv_bfloat16* __restrict__ dv, const __nv_bfloat16* __restrict__ dgate,
               __nv_bfloat16* __restrict__ dqkv, float* __restrict__ dwq, float* __restrict__ dwk,
               float* __restrict__ partials, long long T,
               QkvLayout L) {
  __shared__ float sx[WARPS][MAX_D];   // raw input head
  __shared__ float sg[WARPS][MAX_D];   // gradient after inverse rotation
  __shared__ float sdw[WARPS][2][MAX_D];   // one slot per warp: summed in warp order below, no atomics
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slots = L.ng * (L.qpg * (1 + L.gate) + 2);
  const int nq = L.ng * L.qpg, d = L.d, half = L.rot / 2;
  for (int i = threadIdx.x; i < WARPS * 2 * MAX_D; i += blockDim.x) (&sdw[0][0][0])[i] = 0.f;
  __syncthreads();
  // every lane always touches the same head positions, so the norm-weight gradients are summed in registers over all
  // the heads a warp visits and meet in shared memory once, after the loop
  float dw_acc[2][MAX_D / 32];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < MAX_D / 32; ++b) dw_acc[a][b] = 0.f;
  // a block walks tokens, its warps walk the heads of the token: no 64-bit division on the hot path
  for (long long t = blockIdx.x; t < T; t += gridDim.x)
  for (int slot = warp; slot < slots; slot += WARPS) {
    int kind, head;
    decode_slot(L, slot, kind, head);
    const __nv_bfloat16* src = qkv + t * L.ld + (long long)slot * d;
    __nv_bfloat16* dst = dqkv + t * L.ld + (long long)slot * d;
    const __nv_bfloat16* gsrc = kind == 0 ? dq + (t * nq + head) * d
                                : kind == 1 ? (dgate ? dgate + (t * nq + head) * d : nullptr)
                                : kind == 2 ? dk + (t * L.ng + head) * d
                                            : dv + (t * L.ng + head) * d;
    if (kind == 1 || kind == 3 || (!L.norm && L.rot == 0)) {
      for (int i = lane * 8; i < d; i += 256)
        *reinterpret_cast<uint4*>(dst + i) = gsrc ? *reinterpret_cast<const uint4*>(gsrc + i) : make_uint4(0, 0, 0, 0);
      continue;
    }
    float ss = 0.f;
    for (int i = lane * 2; i < d; i += 64) {
      float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(src + i));
      float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gsrc + i));
      sx[warp][i] = f.x;
      sx[warp][i + 1] = f.y;
      sg[warp][i] = g.x;
      sg[warp][i + 1] = g.y;
      ss += f.x * f.x + f.y * f.y;
    }
    float rstd = 1.f;
    if (L.norm) {
      ss = warp_sum(ss);
      rstd = rsqrtf(ss / d + L.eps);
    }
    __syncwarp();
    const __nv_bfloat16* wn = kind == 0 ? wq : wk;
    // pass 1: gradient w.r.t. the normalised (pre-rotation) head, dot product for the norm backward
    float gn[MAX_D / 32];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < MAX_D / 64; ++j) {
      const int i = lane * 2 + j * 64;
      if (i < d) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int idx = i + e;
          float g = sg[warp][idx];
          if (idx < L.rot) {
            int partner, fi;
            float sign;  // transpose of the forward rotation
            if (L.interleaved) {
              partner = idx ^ 1;
              fi = idx >> 1;
              sign = (idx & 1) ? -1.f : 1.f;
            } else {
              partner = idx < half ? idx + half : idx - half;
              fi = idx < half ? idx : idx - half;
              sign = idx < half ? 1.f : -1.f;
            }
            const float c = cosb[t * half + fi], s = sinb[t * half + fi];
            g = g * c + sign * sg[warp][partner] * s;
          }
          gn[2 * j + e] = g;
          if (L.norm) {
            const float wv = (L.zero_centered ? 1.f : 0.f) + __bfloat162float(wn[idx]);
            dot += g * wv * sx[warp][idx];
          }
        }
      }
    }
    float c3 = 0.f;
    if (L.norm) {
      dot = warp_sum(dot);
      c3 = dot * rstd * rstd * rstd / d;
    }
#pragma unroll
    for (int j = 0; j < MAX_D / 64; ++j) {
      const int i = lane * 2 + j * 64;
      if (i < d) {
        float o[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int idx = i + e;
          const float g = gn[2 * j + e];
          if (L.norm) {
            const float wv = (L.zero_centered ? 1.f : 0.f) + __bfloat162float(wn[idx]);
            o[e] = g * wv * rstd - sx[warp][idx] * c3;
            const float contrib = g * sx[warp][idx] * rstd;
            if (kind == 0) dw_acc[0][2 * j + e] += contrib; else dw_acc[1][2 * j + e] += contrib;
          } else {
            o[e] = g;
          }
        }
        *reinterpret_cast<uint32_t*>(dst + i) = pack_bf16x2(o[0], o[1]);
      }
    }
    __syncwarp();
  }
  if (L.norm) {
#pragma unroll
    for (int j = 0; j < MAX_D / 64; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int idx = lane * 2 + j * 64 + e;
        if (idx < d) {
          sdw[warp][0][idx] = dw_acc[0][2 * j + e];
          sdw[warp][1][idx] = dw_acc[1][2 * j + e];
        }
      }
  }
  __syncthreads();
  if (L.norm) {
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
      float a = 0.f, b = 0.f;
      for (int w = 0; w < WARPS; ++w) {
        a += sdw[w][0][i];
        b += sdw[w][1][i];
      }
      if (partials) {                       // fixed-order sum over CTAs in qkv_dw_reduce_kernel
        partials[((long long)blockIdx.x * 2) * d + i] = a;
        partials[((long long)blockIdx.x * 2 + 1) * d + i] = b;
      } else {
        if (dwq) atomicAdd(dwq + i, a);
        if (dwk) atomicAdd(dwk + i, b);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Fast path for head size 128 with rotate-half RoPE over the whole head (the Qwen3 / Llama layout): 16 lanes to a head, a lane holds
// elements 4l .. 4l + 3 and their rotation partners 64 + 4l .. , so the head never leaves registers.  A warp has one pair of heads
// and walks the tokens: what the heads are is found out once, and the next token's are loaded while it works on one.
// us, forward and backward, before (a warp to a head, 4 bytes a lane, heads of a token in turn) / now: 8192 tokens, 32 + 8 + 8 heads
// with norms 72, 114 / 51, 93, without 63, 75 / 51, 60; 16384, 40 + 8 + 8 131, 160 / 102, 126.  With one CTA an SM more (spills)
// 63, 134, with one less 57, 99; two pairs in flight (spills) 78, 179.
// WIDE: all tensors start on 8-byte boundaries.
template <bool WIDE>
__device__ __forceinline__ uint2 ld_bf4(const __nv_bfloat16* p) {
  if (WIDE) return *reinterpret_cast<const uint2*>(p);
  return make_uint2(reinterpret_cast<const uint32_t*>(p)[0], reinterpret_cast<const uint32_t*>(p)[1]);
}
template <bool WIDE>
__device__ __forceinline__ void st_bf4(__nv_bfloat16* p, uint2 v) {
  if (WIDE) {
    *reinterpret_cast<uint2*>(p) = v;
  } else {
    reinterpret_cast<uint32_t*>(p)[0] = v.x;
    reinterpret_cast<uint32_t*>(p)[1] = v.y;
  }
}
__device__ __forceinline__ void unpack4(uint2 v, float (&f)[4]) {
  const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
  const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  f[0] = x.x;
  f[1] = x.y;
  f[2] = y.x;
  f[3] = y.y;
}
__device__ __forceinline__ uint2 pack4(const float (&f)[4]) { return make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3])); }
// the sum over a head's 16 lanes of x + y
__device__ __forceinline__ float head_sum(float x, float y) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
  }
  return x + y;
}
// The head of a half of a warp, and the warp's walk over the tokens: first one and step.
struct HeadWalk {
  int at, slot, kind, head;                       // slot -1: no head
  long long t, step;
  __device__ __forceinline__ HeadWalk(const QkvLayout& L) {
    const int slots = L.ng * (L.qpg * (1 + L.gate) + 2), pairs = (slots + 1) / 2;
    const int id = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warps = (gridDim.x * blockDim.x) >> 5;   // the host sees that
    at = (threadIdx.x & 15) * 4;                                                                          // warps >= pairs
    slot = 2 * (id % pairs) + ((threadIdx.x >> 4) & 1);
    t = id / pairs;
    step = warps / pairs;
    if (t >= step) t = 1ll << 62;                 // the remainder of the warps
    kind = head = 0;
    if (slot < slots) decode_slot(L, slot, kind, head);
    else slot = -1;
  }
};
__device__ __forceinline__ void head_weights(const QkvLayout& L, const __nv_bfloat16* w, int at, float (&a)[4], float (&b)[4]) {
  unpack4(ld_bf4<false>(w + at), a);
  unpack4(ld_bf4<false>(w + at + 64), b);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    a[e] += L.zero_centered ? 1.f : 0.f;
    b[e] += L.zero_centered ? 1.f : 0.f;
  }
}
__device__ __forceinline__ void ld_angles(const float* __restrict__ tab, float (&f)[4]) {
  const float2 x = reinterpret_cast<const float2*>(tab)[0], y = reinterpret_cast<const float2*>(tab)[1];
  f[0] = x.x;
  f[1] = x.y;
  f[2] = y.x;
  f[3] = y.y;
}

template <bool WIDE>
__global__ void __launch_bounds__(WARPS * 32, FWD_CTAS)
qkv_fwd_fast_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                    const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cosb,
                    const float* __restrict__ sinb, __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k,
                    __nv_bfloat16* __restrict__ v, __nv_bfloat16* __restrict__ gate, long long T, QkvLayout L) {
  constexpr int D = 128;
  const HeadWalk h(L);
  const int nq = L.ng * L.qpg, heads = h.kind < 2 ? nq : L.ng;
  const bool rot = h.kind == 0 || h.kind == 2, live = h.slot >= 0;
  float wa[4] = {}, wb[4] = {};
  const __nv_bfloat16* src = qkv + (live ? h.slot : 0) * D + h.at;
  __nv_bfloat16* dst = (h.kind == 0 ? q : h.kind == 1 ? gate : h.kind == 2 ? k : v) + (long long)h.head * D + h.at;
  uint2 ra, rb;
  float c[4], sn[4];
  auto fetch = [&](long long t) {
    ra = rb = make_uint2(0, 0);
    if (t >= T) return;
    ra = ld_bf4<WIDE>(src + t * L.ld);
    rb = ld_bf4<WIDE>(src + t * L.ld + 64);
    ld_angles(cosb + t * 64 + h.at, c);
    ld_angles(sinb + t * 64 + h.at, sn);
  };
  fetch(h.t);
  if (L.norm) head_weights(L, h.kind == 0 ? wq : wk, h.at, wa, wb);
  for (long long t = h.t; t < T; t += h.step) {
    float a[4], b[4], x[4], y[4], cc[4], ss_[4];
    uint2 oa = ra, ob = rb;
    unpack4(ra, a);
    unpack4(rb, b);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      cc[e] = c[e];
      ss_[e] = sn[e];
    }
    fetch(t + h.step);
    if (L.norm) {
      const float ss = head_sum(a[0] * a[0] + a[1] * a[1] + b[0] * b[0] + b[1] * b[1],
                                a[2] * a[2] + a[3] * a[3] + b[2] * b[2] + b[3] * b[3]);
      const float rstd = rsqrtf(ss * (1.f / D) + L.eps);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e] *= rstd * wa[e];
        b[e] *= rstd * wb[e];
      }
    }
    if (rot) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = fmaf(a[e], cc[e], -__fmul_rn(b[e], ss_[e]));
        y[e] = fmaf(a[e], ss_[e], __fmul_rn(b[e], cc[e]));
      }
      oa = pack4(x);
      ob = pack4(y);
    }
    if (live) {
      st_bf4<WIDE>(dst + t * heads * D, oa);
      st_bf4<WIDE>(dst + t * heads * D + 64, ob);
    }
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(WARPS * 32, BWD_CTAS)
qkv_bwd_fast_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ wq,
                    const __nv_bfloat16* __restrict__ wk, const float* __restrict__ cosb,
                    const float* __restrict__ sinb, const __nv_bfloat16* __restrict__ dq,
                    const __nv_bfloat16* __restrict__ dk, const __nv_bfloat16* __restrict__ dv,
                    const __nv_bfloat16* __restrict__ dgate, __nv_bfloat16* __restrict__ dqkv,
                    float* __restrict__ dwq, float* __restrict__ dwk, float* __restrict__ partials, long long T,
                    QkvLayout L) {
  constexpr int D = 128;
  __shared__ float sdw[WARPS * 2][D];
  __shared__ int kinds[WARPS * 2];
  const HeadWalk h(L);
  const int nq = L.ng * L.qpg, heads = h.kind < 2 ? nq : L.ng;
  const bool rot = h.kind == 0 || h.kind == 2, live = h.slot >= 0;
  float wa[4] = {}, wb[4] = {}, acc[8] = {};
  const __nv_bfloat16* src = qkv + (live ? h.slot : 0) * D + h.at;
  const __nv_bfloat16* gsrc = h.kind == 0 ? dq : h.kind == 1 ? dgate : h.kind == 2 ? dk : dv;
  const bool given = gsrc != nullptr;
  gsrc += (long long)h.head * D + h.at;
  __nv_bfloat16* dst = dqkv + (live ? h.slot : 0) * D + h.at;
  uint2 ga, gb, xa, xb;
  float c[4], sn[4];
  auto fetch = [&](long long t) {
    ga = gb = xa = xb = make_uint2(0, 0);
    if (t >= T) return;
    if (given) {
      ga = ld_bf4<WIDE>(gsrc + t * heads * D);
      gb = ld_bf4<WIDE>(gsrc + t * heads * D + 64);
    }
    if (L.norm && rot) {
      xa = ld_bf4<WIDE>(src + t * L.ld);
      xb = ld_bf4<WIDE>(src + t * L.ld + 64);
    }
    ld_angles(cosb + t * 64 + h.at, c);
    ld_angles(sinb + t * 64 + h.at, sn);
  };
  fetch(h.t);
  if (L.norm) head_weights(L, h.kind == 0 ? wq : wk, h.at, wa, wb);
  for (long long t = h.t; t < T; t += h.step) {
    // transpose of the rotation
    float a[4], b[4], x[4], y[4], na[4], nb[4];
    uint2 oa = ga, ob = gb;
    unpack4(ga, a);
    unpack4(gb, b);
    unpack4(xa, x);
    unpack4(xb, y);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      na[e] = a[e] * c[e] + b[e] * sn[e];
      nb[e] = b[e] * c[e] - a[e] * sn[e];
    }
    fetch(t + h.step);
    if (L.norm) {
      const float ss = head_sum(x[0] * x[0] + x[1] * x[1] + y[0] * y[0] + y[1] * y[1],
                                x[2] * x[2] + x[3] * x[3] + y[2] * y[2] + y[3] * y[3]);
      const float dot = head_sum(na[0] * wa[0] * x[0] + na[1] * wa[1] * x[1] + nb[0] * wb[0] * y[0] + nb[1] * wb[1] * y[1],
                                 na[2] * wa[2] * x[2] + na[3] * wa[3] * x[3] + nb[2] * wb[2] * y[2] + nb[3] * wb[3] * y[3]);
      const float rstd = rsqrtf(ss * (1.f / D) + L.eps);
      const float c3 = dot * rstd * rstd * rstd * (1.f / D);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[e] += na[e] * x[e] * rstd;
        acc[4 + e] += nb[e] * y[e] * rstd;
        na[e] = na[e] * wa[e] * rstd - x[e] * c3;
        nb[e] = nb[e] * wb[e] * rstd - y[e] * c3;
      }
    }
    if (rot) {
      oa = pack4(na);
      ob = pack4(nb);
    }
    if (live) {
      st_bf4<WIDE>(dst + t * L.ld, oa);
      st_bf4<WIDE>(dst + t * L.ld + 64, ob);
    }
  }
  if (L.norm) {
    const int half = threadIdx.x >> 4;
#pragma unroll
    for (int e = 0; e < 8; ++e) sdw[half][h.at + (e & 3) + (e >> 2) * 64] = acc[e];
    if ((threadIdx.x & 15) == 0) kinds[half] = live ? h.kind : 3;
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
      float a = 0.f, b = 0.f;
      for (int w = 0; w < WARPS * 2; ++w) {
        if (kinds[w] == 0) a += sdw[w][i];
        if (kinds[w] == 2) b += sdw[w][i];
      }
      if (partials) {
        partials[((long long)blockIdx.x * 2) * D + i] = a;
        partials[((long long)blockIdx.x * 2 + 1) * D + i] = b;
      } else {
        if (dwq) atomicAdd(dwq + i, a);
        if (dwk) atomicAdd(dwk + i, b);
      }
    }
  }
}

// CTAs of the fast kernels, 0 where a warp for every pair of heads is more than there are
int fast_grid(const QkvLayout& L, long long T, int ctas_per_sm) {
  const long long pairs = (L.ng * (L.qpg * (1LL + L.gate) + 2) + 1) / 2, cap = (long long)device_sm_count() * ctas_per_sm;
  if (pairs > cap * WARPS) return 0;
  const long long blocks = (T * pairs + WARPS - 1) / WARPS;
  return (int)(blocks < cap ? blocks : cap);
}
bool on_8_bytes(std::initializer_list<const void*> ps) {
  uintptr_t bits = 0;
  for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
  return bits % 8 == 0;
}

}  // namespace

extern "C" {

int mcb_qkv_split_norm_rope_fwd(const void* qkv, const void* wq, const void* wk, const float* cosb, const float* sinb,
                                void* q, void* k, void* v, void* gate, long long T, int ng, int qpg, int d,
                                int has_gate, int rot, int interleaved, int norm, int zero_centered, float eps,
                                long long ld, void* stream_) {
  if (T == 0) return 0;
  if (d > MAX_D || d % 8 || rot > d || (rot & 1) || ld % 8) return -1;
  QkvLayout L{ng, qpg, d, has_gate, rot, interleaved, norm, zero_centered, eps, ld};
  long long blocks = T;
  long long cap = (long long)device_sm_count() * 16;
  const int fast = d == 128 && rot == 128 && !interleaved ? fast_grid(L, T, FWD_CTAS) : 0;
  if (fast > 0) {
    auto* kernel = on_8_bytes({qkv, q, k, v, gate}) ? qkv_fwd_fast_kernel<true> : qkv_fwd_fast_kernel<false>;
    kernel<<<fast, WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cosb, sinb, (__nv_bfloat16*)q,
        (__nv_bfloat16*)k, (__nv_bfloat16*)v, (__nv_bfloat16*)gate, T, L);
    return (int)cudaGetLastError();
  }
  qkv_fwd_kernel<<<(int)(blocks < cap ? blocks : cap), WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(
      (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cosb, sinb, (__nv_bfloat16*)q,
      (__nv_bfloat16*)k, (__nv_bfloat16*)v, (__nv_bfloat16*)gate, T, L);
  return (int)cudaGetLastError();
}

// CTAs the backward kernels launch for T tokens at most = rows of `partials` ([rows, 2, d] fp32) the caller provides
int mcb_qkv_bwd_partial_rows(long long T) {
  return T > 0 ? device_sm_count() * 8 : 0;
}

// dwq / dwk: fp32 [d], accumulated into (caller zeroes or carries them across micro-batches), or, with `dw_bf16` (needs
// `partials`), bf16 [d] and overwritten.  With `partials` the norm-weight gradients are summed in a fixed order
// (bit-reproducible); without, with atomics.
int mcb_qkv_split_norm_rope_bwd(const void* qkv, const void* wq, const void* wk, const float* cosb, const float* sinb,
                                const void* dq, const void* dk, const void* dv, const void* dgate, void* dqkv,
                                void* dwq_any, void* dwk_any, int dw_bf16, float* partials, long long T, int ng, int qpg,
                                int d, int has_gate, int rot, int interleaved, int norm, int zero_centered, float eps,
                                long long ld, void* stream_) {
  if (T == 0) return 0;
  if (d > MAX_D || d % 8 || rot > d || (rot & 1) || ld % 8) return -1;
  QkvLayout L{ng, qpg, d, has_gate, rot, interleaved, norm, zero_centered, eps, ld};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_);
  int grid = (int)min(T, (long long)mcb_qkv_bwd_partial_rows(T));
  if (!norm) partials = nullptr;
  if (norm && dw_bf16 && !partials) return -3;
  float* dwq = dw_bf16 ? nullptr : reinterpret_cast<float*>(dwq_any);
  float* dwk = dw_bf16 ? nullptr : reinterpret_cast<float*>(dwk_any);
  const int fast = d == 128 && rot == 128 && !interleaved ? fast_grid(L, T, BWD_CTAS) : 0;
  if (fast > 0) {
    grid = fast;
    auto* kernel = on_8_bytes({qkv, dq, dk, dv, dgate, dqkv}) ? qkv_bwd_fast_kernel<true> : qkv_bwd_fast_kernel<false>;
    kernel<<<grid, WARPS * 32, 0, s>>>(
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cosb, sinb,
        (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)dgate,
        (__nv_bfloat16*)dqkv, dwq, dwk, partials, T, L);
  } else {
    qkv_bwd_kernel<<<grid, WARPS * 32, 0, s>>>(
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)wq, (const __nv_bfloat16*)wk, cosb, sinb,
        (const __nv_bfloat16*)dq, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, (const __nv_bfloat16*)dgate,
        (__nv_bfloat16*)dqkv, dwq, dwk, partials, T, L);
  }
  if (partials && dw_bf16)                                                       // rows are [dwq | dwk]
    launch_reduce_partials<__nv_bfloat16>(partials, grid, 2 * d, reinterpret_cast<__nv_bfloat16*>(dwq_any),
                                          reinterpret_cast<__nv_bfloat16*>(dwk_any), d, s);
  else if (partials)
    launch_reduce_partials<float>(partials, grid, 2 * d, dwq, dwk, d, s);
  return (int)cudaGetLastError();
}

}  // extern "C"
