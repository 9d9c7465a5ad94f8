// Gradient of the per-head sink logits: one more softmax column with a zero value vector, so
//   d sink_h = -sum_i exp(sink_h - lse(h, i)) delta(h, i).
// One CTA per head, sums in a fixed order.  Bound: the latency of its loads, so four rows of a thread are in flight.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace {

constexpr int SINK_THREADS = 512;

__global__ void __launch_bounds__(SINK_THREADS)
attn_sink_grad_kernel(const float* __restrict__ sinks, const float* __restrict__ lse, const float* __restrict__ delta, int T,
                      void* __restrict__ out, int out_bf16) {
  __shared__ float red[SINK_THREADS / 32];
  const int h = blockIdx.x;
  const float sink = sinks[h];
  float acc = 0.f;
#pragma unroll 4
  for (int i = threadIdx.x; i < T; i += SINK_THREADS) {
    const long long at = (long long)h * T + i;
    acc += expf(sink - lse[at]) * delta[at];
  }
#pragma unroll
  for (int s = 16; s; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    for (int w = 0; w < SINK_THREADS / 32; ++w) sum += red[w];
    if (out_bf16) reinterpret_cast<__nv_bfloat16*>(out)[h] = __float2bfloat16(-sum);
    else reinterpret_cast<float*>(out)[h] = -sum;
  }
}

}  // namespace

extern "C" {

// d sinks [nq] (fp32, or bf16 with out_bf16) of the forward's sinks [nq] fp32, from lse and delta [nq, T].
int mcb_attn_sink_grad(const float* sinks, const float* lse, const float* delta, void* out, int out_bf16, int T, int nq,
                       void* stream_) {
  if (nq <= 0) return 0;
  attn_sink_grad_kernel<<<(unsigned)nq, SINK_THREADS, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(sinks, lse, delta, T, out,
                                                                                                  out_bf16);
  return (int)cudaGetLastError();
}

}  // extern "C"
