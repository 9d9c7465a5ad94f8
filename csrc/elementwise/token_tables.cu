// What a model's forward pass derives from its packing before the first layer, one launch each: the first token of every token's
// sequence, and the rotary tables.  As tensor operations (searchsorted, clamp, gather, conversions; product, cosine, sine)
// they were twelve launches and 65 us on the host; on the device they are a few microseconds either way.
//
// Compiled with full-precision math: the tables have the bits of torch's cos and sin.
#include "../common/host_utils.cuh"

namespace {

// cu ascends; tokens behind the last boundary count to the last sequence
template <class I>
__global__ void seq_starts_kernel(const I* __restrict__ cu, int n, int* __restrict__ out, long long T) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < T; t += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = n - 1;                       // boundaries 1 .. n - 1 at or below t
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if ((long long)cu[mid + 1] <= t) lo = mid + 1;
      else hi = mid;
    }
    out[t] = (int)cu[min(lo, n - 2)];
  }
}

template <class I>
__global__ void rope_tables_kernel(const I* __restrict__ pos, const float* __restrict__ inv, float scale, float* __restrict__ cos_out,
                                   float* __restrict__ sin_out, long long T, int R) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < T * R; i += (long long)gridDim.x * blockDim.x) {
    const float f = (float)pos[i / R] * inv[i % R];
    const float c = cosf(f), s = sinf(f);
    cos_out[i] = scale == 1.f ? c : c * scale;
    sin_out[i] = scale == 1.f ? s : s * scale;
  }
}

int blocks(long long n) {
  const long long want = (n + 255) / 256, most = 8ll * mcb::device_sm_count();
  return (int)(want < most ? want : most);
}

}  // namespace

extern "C" {

// cu [n] int32 (wide: int64), n >= 2 -> out [T] int32
int mcb_seq_starts(const void* cu, int wide, int n, int* out, long long T, void* stream) {
  if (T <= 0) return 0;
  if (n < 2) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (wide) seq_starts_kernel<<<blocks(T), 256, 0, s>>>((const long long*)cu, n, out, T);
  else seq_starts_kernel<<<blocks(T), 256, 0, s>>>((const int*)cu, n, out, T);
  return (int)cudaGetLastError();
}

// cos, sin [T, R] of pos [T] int32 (wide: int64) times inv [R], times `scale`
int mcb_rope_tables(const void* pos, int wide, const float* inv, float scale, float* cos_out, float* sin_out, long long T, int R,
                    void* stream) {
  if (T <= 0 || R <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (wide) rope_tables_kernel<<<blocks(T * R), 256, 0, s>>>((const long long*)pos, inv, scale, cos_out, sin_out, T, R);
  else rope_tables_kernel<<<blocks(T * R), 256, 0, s>>>((const int*)pos, inv, scale, cos_out, sin_out, T, R);
  return (int)cudaGetLastError();
}

}  // extern "C"
