// The reciprocals of csrc/device_math.cuh over the ranges they are used in,
// against the compiler's own (built with -prec-div=true): rcp_rn between 2^-126
// and 2^126, which holds what inverse_direction and the dominant axis of a ray
// give it, and rcp_small from 2^-128 to 2^124.  Prints per range the results that
// differ and the largest difference in ulps, and whether a divisor without a
// finite reciprocal gives a finite one.
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

int main() {
  unsigned long long *differ;
  int *worst;
  if (cudaMallocManaged(&differ, 2 * sizeof(*differ)) || cudaMallocManaged(&worst, 3 * sizeof(*worst))) return 2;
  for (int f = 0; f < 2; ++f) differ[f] = 0;
  for (int f = 0; f < 3; ++f) worst[f] = 0;
  compare<false><<<1216, 256>>>(0x00800000u, ((127u + 125u) << 23) | 0x7fffffu, differ, worst);
  compare<true><<<1216, 256>>>(0x00200001u, ((127u + 123u) << 23) | 0x7fffffu, differ + 1, worst + 1);
  beyond<<<1, 1>>>(worst + 2);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  printf("rcp_rn %llu %d\nrcp_small %llu %d\nbeyond_finite %d\n", differ[0], worst[0], differ[1], worst[1], worst[2]);
  return 0;
}
