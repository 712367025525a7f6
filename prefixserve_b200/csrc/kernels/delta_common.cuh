// What the kernels of the delta rules share.
#pragma once
#include "common.cuh"

namespace delta {

constexpr int MAX_TAPS = 16;
// Per token and head the recurrences are handed five numbers, [T, BD, H]: beta, decay, and three dot products that do
// not depend on the state: q.k of the token, and k.k' and q.k' with the key k' of the token before it in the portion.
constexpr int BD = 5;

__device__ __forceinline__ float softplusf_(float x) { return log1pf(expf(-fabsf(x))) + fmaxf(x, 0.f); }
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float siluf_(float x) { return x / (1.f + expf(-x)); }
// The same of several numbers, each by its own size: up to QUICK_UP_TO without a division, which takes twice as many instructions (2,000 tokens of 16 heads:
// delta_prepare_wide_kernel 28 us -> 21); whether one lies beyond is asked for once.  From float64 0.485 units of the last place (root of the mean square, evenly over
// [-80, 80]), as with the division.
template <int M, int N>
__device__ __forceinline__ void silu_all(float (&x)[M][N]) {
  float top = 0.f;
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) top = fmaxf(top, fabsf(x[i][j]));
  if (top <= QUICK_UP_TO) {
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) x[i][j] = divided(x[i][j], 1.f + expf(-x[i][j]));
  } else {
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float d = 1.f + expf(-x[i][j]);
        x[i][j] = fabsf(x[i][j]) <= QUICK_UP_TO ? divided(x[i][j], d) : x[i][j] / d;
      }
  }
}
// what makes a vector with this sum of squares a unit vector, over sqrt(dim) for queries (keys: 1).  (rsqrtf(dim) is off by up to two units of the last place,
// in every query alike.)
__device__ __forceinline__ float unit_factor(float squares, int dim) { return 1.f / sqrtf((float)dim) / sqrtf(squares + 1e-6f); }

__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
// zeros where there is nothing to copy (``src`` is then not read, but must be an address)
__device__ __forceinline__ void copy_async16_or_zero(float* dst, const float* src, bool there) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// One block per request, at the end of its portion: the slot's convolution inputs, which are the K-1 positions before the
// next token (the portion's last rows, or what was there before, moved up, when the portion is shorter).
template <typename T>
__device__ __forceinline__ void keep_conv_inputs(const T* __restrict__ proj, long long P, float* __restrict__ base, int t0, int t1,
                                                 int C, int K) {
  if (K <= 1 || t1 <= t0) return;
  const int n = t1 - t0;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float keep[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K - 1) break;
      const int back = K - 1 - k;  // this row is the input ``back`` positions before the next token
      keep[k] = back <= n ? to_float<T>(proj[(size_t)(t1 - back) * P + c]) : base[(size_t)(k + n) * C + c];
    }
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
      if (k >= K - 1) break;
      base[(size_t)k * C + c] = keep[k];
    }
  }
}

}  // namespace delta
