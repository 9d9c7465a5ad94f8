// What surrounds the router's kernels, one launch each: the load-balancing loss with its gradient, and the two bf16 terms in which the
// logits' gradient enters the gate's products.  As tensor operations they were nine launches before the experts' first product,
// with the host as the bound (4096 tokens, 128 experts: 75 us of it), and fourteen behind the last one, 2 us and a gap each.
//
// Compiled with full-precision math: the divisions of the tensor operations.
#include "../common/host_utils.cuh"
#include "../common/ptx.cuh"

using namespace mcb;

namespace {

// out = {c sum_e frac_e score_sum_e / tokens, that / coeff},  frac_e = counts_e / (tokens k); the sum in another order than a tensor
// operation's, the gradient with its bits
__global__ void __launch_bounds__(256)
router_aux_kernel(const int* __restrict__ counts, const float* __restrict__ score_sum, float* __restrict__ frac, float* __restrict__ out,
                  int E, float tokens, float copies, float c, float coeff) {
  __shared__ float red[8];
  float s = 0.f;
  for (int e = threadIdx.x; e < E; e += 256) {
    const float f = (float)counts[e] / copies;
    frac[e] = f;
    s += f * (score_sum[e] / tokens);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += red[i];
    out[0] = c * t;
    out[1] = out[0] / coeff;
  }
}

__global__ void router_aux_bwd_kernel(const float* __restrict__ g, const float* __restrict__ frac, float* __restrict__ out, int E,
                                      float tokens, float c) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < E) out[e] = (g[0] * c * frac[e]) / tokens;
}

// x [rows, E] -> [rows, 2 E]: its rounding to bf16 and that of the rounding error
__global__ void split_terms_kernel(const float4* __restrict__ x, uint2* __restrict__ out, long long n, int quads) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / quads;
    const float4 v = x[i];
    const uint2 hi = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi.y));
    uint2* at = out + row * 2 * quads + (i - row * quads);
    at[0] = hi;
    at[quads] = make_uint2(pack_bf16x2(v.x - a.x, v.y - a.y), pack_bf16x2(v.z - b.x, v.w - b.y));
  }
}

// x [2, n] -> bf16(x[0] + x[1])
__global__ void add_halves_kernel(const float4* __restrict__ x, uint2* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float4 a = x[i], b = x[n + i];
    out[i] = make_uint2(pack_bf16x2(a.x + b.x, a.y + b.y), pack_bf16x2(a.z + b.z, a.w + b.w));
  }
}

int blocks_for(long long n) {
  const long long want = (n + 255) / 256, cap = (long long)device_sm_count() * 8;
  return (int)(want < cap ? want : cap);
}

}  // namespace

extern "C" {

// counts [E] int32, score_sum [E] fp32, out [2] = {loss, loss / coeff}, frac [E] for the backward pass; c = coeff times the
// number of experts
int mcb_router_aux(const int* counts, const float* score_sum, float* frac, float* out, int E, float tokens, int k, float c, float coeff,
                   void* stream) {
  if (E <= 0) return -1;
  router_aux_kernel<<<1, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(counts, score_sum, frac, out, E, tokens, tokens * (float)k, c,
                                                                          coeff);
  return (int)cudaGetLastError();
}

// g [1]: gradient of the loss -> out [E]: of score_sum
int mcb_router_aux_bwd(const float* g, const float* frac, float* out, int E, float tokens, float c, void* stream) {
  if (E <= 0) return -1;
  router_aux_bwd_kernel<<<(E + 127) / 128, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(g, frac, out, E, tokens, c);
  return (int)cudaGetLastError();
}

// x [rows, E] fp32 -> out [rows, 2 E] bf16; E a multiple of 4, x on a 16-byte boundary, out on an 8-byte one
int mcb_split_terms(const float* x, void* out, long long rows, int E, void* stream) {
  if (E <= 0 || E % 4 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 7)) return -1;
  if (rows == 0) return 0;
  const long long n = rows * (E / 4);
  split_terms_kernel<<<blocks_for(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<const float4*>(x),
                                                                                      reinterpret_cast<uint2*>(out), n, E / 4);
  return (int)cudaGetLastError();
}

// x [2, n] fp32 -> out [n] bf16 = x[0] + x[1]; n a multiple of 4, x on a 16-byte boundary, out on an 8-byte one
int mcb_add_halves(const float* x, void* out, long long n, void* stream) {
  if (n % 4 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 7)) return -1;
  if (n == 0) return 0;
  add_halves_kernel<<<blocks_for(n / 4), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<const float4*>(x),
                                                                                         reinterpret_cast<uint2*>(out), n / 4);
  return (int)cudaGetLastError();
}

}  // extern "C"
