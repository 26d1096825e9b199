// The quotients and roots of csrc/device_math.cuh against the compiler's own
// (built with -prec-div=true -prec-sqrt=true): for n operand pairs spread over
// the trace's ranges, prints per function the results that differ and the
// largest difference in units of the last place.
#include <cstdio>
#include <cstdlib>

#include "device_math.cuh"

using namespace dvsgb;

__device__ unsigned mix(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (unsigned)(z ^ (z >> 31));
}
// A float with all 23 mantissa bits random and an exponent in [lo, hi].
__device__ float operand(unsigned long long seed, int lo, int hi, bool sign) {
  const unsigned a = mix(seed), b = mix(seed ^ 0x5555555555555555ull);
  const unsigned e = 127u + (unsigned)(lo + (int)(b % (unsigned)(hi - lo + 1)));
  return __uint_as_float((sign && (b >> 31) ? 0x80000000u : 0u) | (e << 23) | (a >> 9));
}
__device__ int ulps(float x, float y) {
  const int a = __float_as_int(x), b = __float_as_int(y);
  return abs((a < 0 ? (int)0x80000000 - a : a) - (b < 0 ? (int)0x80000000 - b : b));
}
__global__ void compare(unsigned long long n, unsigned long long *differ, int *worst) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const float a = operand(2 * i, -40, 40, true), b = operand(2 * i + 1, -40, 40, true);
    const float x = operand(3 * i + 7, -60, 60, false);
    const float got[4] = {div_rn(a, b), div_by(a, b, 1.0f / b), rcp_rn(b), sqrt_rn(x)};
    const float want[4] = {a / b, a / b, 1.0f / b, sqrtf(x)};
    for (int f = 0; f < 4; ++f) {
      const int d = ulps(got[f], want[f]);
      if (d) {
        atomicAdd(differ + f, 1ull);
        atomicMax(worst + f, d);
      }
    }
  }
}
__global__ void corners(float *out) {
  out[0] = sqrt_rn(0.0f);
  out[1] = div_rn(0.0f, 3.0f);
  out[2] = div_rn(6.0f, 3.0f);
  out[3] = rcp_rn(1e-20f);
  out[4] = sqrt_rn(4.0f);
}

int main(int argc, char **argv) {
  const unsigned long long n = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1ull << 28;
  unsigned long long *differ;
  int *worst;
  float *c;
  if (cudaMallocManaged(&differ, 4 * sizeof(*differ)) || cudaMallocManaged(&worst, 4 * sizeof(*worst)) ||
      cudaMallocManaged(&c, 5 * sizeof(*c)))
    return 2;
  for (int f = 0; f < 4; ++f) differ[f] = 0, worst[f] = 0;
  compare<<<1216, 256>>>(n, differ, worst);
  corners<<<1, 1>>>(c);
  if (cudaDeviceSynchronize() != cudaSuccess) return 2;
  const char *name[4] = {"div_rn", "div_by", "rcp_rn", "sqrt_rn"};
  for (int f = 0; f < 4; ++f) printf("%s %llu %d\n", name[f], differ[f], worst[f]);
  printf("corners %d\n", c[0] == 0.0f && c[1] == 0.0f && c[2] == 2.0f && c[3] == 1e20f && c[4] == 2.0f);
  return 0;
}
