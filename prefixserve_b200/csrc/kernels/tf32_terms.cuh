// Products of float32 numbers on the tensor cores.
//
// mma.sync m16n8k8 multiplies numbers of 11 bits.  A float32 number enters as hi (rounded to nearest) + lo, what is left: the instruction
// takes 11 bits of that (22 in all), and what it does not look at, the rest, enters as a third term where sums have to come out as
// float32's own would.  The sums of the hi hi products leave the tensor cores after every eight terms and are added up in float32 with
// rounding to nearest, since the instruction cuts its sums off instead of rounding them.
#pragma once
#include "common.cuh"

namespace terms {

struct Split {
  uint32_t hi, lo;
};
__device__ __forceinline__ Split split(float x) {
  const uint32_t hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  return {hi, __float_as_uint(x - __uint_as_float(hi))};  // (the instruction does not look at lo's last 13 bits)
}
__device__ __forceinline__ uint32_t rest(uint32_t lo) { return __float_as_uint(__uint_as_float(lo) - __uint_as_float(lo & 0xffffe000u)); }
__device__ __forceinline__ Split split_product(float x, float factor) {  // of a product, without rounding it first
  const uint32_t hi = (__float_as_uint(x * factor) + 0x1000u) & 0xffffe000u;
  return {hi, __float_as_uint(fmaf(x, factor, -__uint_as_float(hi)))};
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// One step of eight terms: sum += hi hi (rounded to nearest), small += hi lo + lo hi; with PRODUCTS 4 also lo lo, with 6 also hi rest +
// rest hi: operands to their last bit.  Long sums go in several chains, which lose less.
template <int CHAINS>
struct Sums {
  float sum[CHAINS][4] = {}, small[2][4] = {};
  template <int PRODUCTS>
  __device__ __forceinline__ void step(const uint32_t (&ah)[4], const uint32_t (&al)[4], Split b0, Split b1, int chain = 0) {
    static_assert(PRODUCTS == 4 || PRODUCTS == 6, "lo lo, or all");
    const float zero[4] = {};
    float d[4];
    if constexpr (PRODUCTS == 6) {
      const uint32_t ar[4] = {rest(al[0]), rest(al[1]), rest(al[2]), rest(al[3])};
      mma_tf32(small[0], ah, rest(b0.lo), rest(b1.lo), small[0]);
      mma_tf32(small[1], ar, b0.hi, b1.hi, small[1]);
    }
    mma_tf32(small[1], al, b0.lo, b1.lo, small[1]);
    mma_tf32(d, ah, b0.hi, b1.hi, zero);
    mma_tf32(small[0], ah, b0.lo, b1.lo, small[0]);
    mma_tf32(small[1], al, b0.hi, b1.hi, small[1]);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[chain][e] += d[e];
  }
  // the right operand's numbers are of eleven bits or fewer themselves (bfloat16); WHOLE: the left one's to their last bit
  template <bool WHOLE>
  __device__ __forceinline__ void step(const uint32_t (&ah)[4], const uint32_t (&al)[4], float b0, float b1, int chain = 0) {
    const float zero[4] = {};
    float d[4];
    if constexpr (WHOLE) {
      const uint32_t ar[4] = {rest(al[0]), rest(al[1]), rest(al[2]), rest(al[3])};
      mma_tf32(small[0], ar, __float_as_uint(b0), __float_as_uint(b1), small[0]);
    }
    mma_tf32(d, ah, __float_as_uint(b0), __float_as_uint(b1), zero);
    mma_tf32(small[1], al, __float_as_uint(b0), __float_as_uint(b1), small[1]);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[chain][e] += d[e];
  }
  __device__ __forceinline__ float total(int e) const {
    float s[CHAINS];
#pragma unroll
    for (int c = 0; c < CHAINS; ++c) s[c] = sum[c][e];
#pragma unroll
    for (int n = CHAINS / 2; n > 0; n >>= 1)
#pragma unroll
      for (int c = 0; c < n; ++c) s[c] += s[c + n];
    return s[0] + (small[0][e] + small[1][e]);
  }
  __device__ __forceinline__ void totals(float (&out)[4]) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) out[e] = total(e);
  }
};
using Sum = Sums<1>;

__device__ __forceinline__ bool is_finite(float x) { return fabsf(x) <= 3.402823466e38f; }
__device__ __forceinline__ bool all_finite(const float (&x)[4]) { return is_finite(x[0]) && is_finite(x[1]) && is_finite(x[2]) && is_finite(x[3]); }
// entry e of an array that stays in registers
__device__ __forceinline__ float pick(const float (&x)[4], int e) { return e < 2 ? (e ? x[1] : x[0]) : (e == 3 ? x[3] : x[2]); }
__device__ __forceinline__ void place(float (&x)[4], int e, float v) {
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = k == e ? v : x[k];
}
// a fragment of the left operand: this lane's number, ``down`` for the row eight further, ``along`` for the place four further
__device__ __forceinline__ void load_rows(const float* a, int down, int along, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const Split v = split(a[(e & 1) * down + (e >> 1) * along]);
    hi[e] = v.hi;
    lo[e] = v.lo;
  }
}

// A running product of decays with what its roundings lose carried along, rounded once where it is read.
struct Product {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float a) {
    const float p = hi * a;
    lo = fmaf(lo, a, fmaf(hi, a, -p));
    hi = p;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
};

}  // namespace terms
