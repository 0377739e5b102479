// Compares the integer-pipe products, reciprocals, quotients and roots
// (int_f64.cuh) with FP64 arithmetic over every seed argument: all 2^23 leading
// significand bits, with the bits below zero, all ones and mixed, in an even and
// an odd exponent.  Prints the number of mismatches of each.  Built by a C++
// compiler (the host's seeds) or by nvcc (the hardware's).
#include <cmath>
#include <cstdio>

#include "int_f64.cuh"

using namespace wenofd::dev;

enum { kMul, kReciprocal, kQuotient, kSqrt, kKinds };

WENOFD_HD u64 mixed(u64 z) {  // splitmix64
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

WENOFD_HD double number(u64 significand, int exponent) {
  const u64 u = (u64(1023 + exponent) << 52) | (significand & 0xfffffffffffffull);
  return bits_f64(u32(u >> 32), u32(u));
}

// Mismatches of the operands with leading bits `top`, added to bad[kKinds].
template <class Add>
WENOFD_HD void check(u32 top, Add add) {
  const u64 low[4] = {0ull, 0x1fffffffull, 1ull, mixed(top) & 0x1fffffffull};
  const u64 other[4] = {0ull, 0xfffffffffffffull, mixed(top + 0x100000000ull), u64(top) << 29};
  for (int k = 0; k < 4; ++k) {
    const u64 m = (u64(top) << 29) | low[k];
    const double x = number(m, 3), a = number(other[k], -2), b = number(other[3 - k], 40);
    const IntDivisor by(x);
    if (int_mul(x, a) != x * a) add(kMul);
    if (by.reciprocal() != 1.0 / x) add(kReciprocal);
    if (by.quotient(a) != a / x || by.quotient(-b) != -b / x) add(kQuotient);
    if (int_sqrt(number(m, 6)) != sqrt(number(m, 6)) || int_sqrt(x) != sqrt(x)) add(kSqrt);
  }
}

#ifdef __CUDACC__
__global__ void k_check(unsigned long long *bad) {
  for (u32 top = blockIdx.x * blockDim.x + threadIdx.x; top < (1u << 23); top += gridDim.x * blockDim.x)
    check(top, [&](int kind) { atomicAdd(&bad[kind], 1ull); });
}
#endif

int main() {
  unsigned long long bad[kKinds] = {};
#ifdef __CUDACC__
  unsigned long long *dev = nullptr;
  if (cudaMalloc(&dev, sizeof(bad)) != cudaSuccess || cudaMemset(dev, 0, sizeof(bad)) != cudaSuccess) return 1;
  k_check<<<1024, 256>>>(dev);
  if (cudaMemcpy(bad, dev, sizeof(bad), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  cudaFree(dev);
#else
  for (u32 top = 0; top < (1u << 23); ++top) check(top, [&](int kind) { bad[kind] += 1; });
#endif
  for (int k = 0; k < kKinds; ++k) std::printf("%llu ", bad[k]);
  std::printf("\n");
  return 0;
}
