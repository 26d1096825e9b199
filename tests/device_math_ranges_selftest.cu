// The reciprocals of csrc/device_math.cuh over the ranges they are used in,
// against the compiler's own (built with -prec-div=true): rcp_rn between 2^-126
// and 2^126, which holds what inverse_direction and the dominant axis of a ray
// give it, and rcp_small from 2^-128 to 2^124.  Prints per range the results that
// differ and the largest difference in ulps, and whether a divisor without a
// finite reciprocal gives a finite one.  Then the FP64 quotients by a divisor
// known beforehand (quotient) on 2^26 pairs, and how often the product with the
// reciprocal alone differs.
#include <cstdio>

#include "device_math.cuh"

using namespace dvsgb;

__device__ int ulps(float x, float y) {
  const int a = __float_as_int(x), b = __float_as_int(y);
  return abs((a < 0 ? (int)0x80000000 - a : a) - (b < 0 ? (int)0x80000000 - b : b));
}
// bits in [lo, hi], both signs
template <bool kSmall>
__global__ void compare(unsigned lo, unsigned hi, unsigned long long *differ, int *worst) {
  for (unsigned long long i = lo + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i <= hi;
       i += (unsigned long long)gridDim.x * blockDim.x)
    for (unsigned sign = 0; sign < 2; ++sign) {
      const float b = __uint_as_float((unsigned)i | sign << 31);
      const int d = ulps(kSmall ? rcp_small(b) : rcp_rn(b), 1.0f / b);
      if (d) {
        atomicAdd(differ, 1ull);
        atomicMax(worst, d);
      }
    }
}
__global__ void beyond(int *finite) {
  for (unsigned i = 1; i <= 0x00200000u; i += i < 0x1ff000u ? 4093u : 1u)  // up to 2^-128, whose reciprocal is no float
    if (isfinite(rcp_small(__uint_as_float(i)))) *finite = 1;
}

__device__ unsigned long long mix(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
// All 52 mantissa bits random, an exponent within 60 of 0.
__device__ double operand(unsigned long long seed) {
  const unsigned long long m = mix(seed), e = 1023ull - 60ull + mix(seed ^ 0x5555555555555555ull) % 121ull;
  return __longlong_as_double((long long)((m & 0x8000000000000000ull) | e << 52 | (m >> 12 & 0xfffffffffffffull)));
}
__global__ void quotients(unsigned long long n, unsigned long long *differ) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const double a = operand(2 * i), b = operand(2 * i + 1), y = 1.0 / b, want = a / b;
    if (quotient(a, b, y) != want) atomicAdd(differ, 1ull);
    if (a * y != want) atomicAdd(differ + 1, 1ull);
  }
}

int main() {
  unsigned long long *differ;
  int *worst;
  if (cudaMallocManaged(&differ, 4 * sizeof(*differ)) || cudaMallocManaged(&worst, 3 * sizeof(*worst))) return 2;
  for (int f = 0; f < 4; ++f) differ[f] = 0;
  for (int f = 0; f < 3; ++f) worst[f] = 0;
  compare<false><<<1216, 256>>>(0x00800000u, ((127u + 125u) << 23) | 0x7fffffu, differ, worst);
  compare<true><<<1216, 256>>>(0x00200001u, ((127u + 123u) << 23) | 0x7fffffu, differ + 1, worst + 1);
  beyond<<<1, 1>>>(worst + 2);
  quotients<<<1216, 256>>>(1ull << 26, differ + 2);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  printf("rcp_rn %llu %d\nrcp_small %llu %d\nbeyond_finite %d\n", differ[0], worst[0], differ[1], worst[1], worst[2]);
  printf("quotient %llu\nproduct %llu\n", differ[2], differ[3]);
  return 0;
}
