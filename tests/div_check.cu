// Counts the quotients and reciprocals of seeded operands for which mixed::div_rn differs from
// the IEEE division: full mantissas and mantissas of 24 bits (an FP32 state), exponents within
// 2^+-32, both signs.
#include <cstdio>

#include "../pip_b200/csrc/pip_mixed_cell.cuh"

using namespace pip;

__device__ unsigned long long mix(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ double operand(unsigned long long s, bool brief) {
  unsigned long long m = s & 0x800fffffffffffffull;
  if (brief) m &= ~0x1fffffffull;
  return __longlong_as_double(
      (long long)(m | ((unsigned long long)(1023 + (int)((s >> 52) & 63) - 32) << 52)));
}

__global__ void check(unsigned long long n, unsigned long long *bad) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * (unsigned long long)blockDim.x) {
    const double a = operand(mix(2 * i), i & 1), x = operand(mix(2 * i + 1), i & 2);
    if (mixed::div_rn(a, x, rcp_(x)) != a / x) atomicAdd(&bad[0], 1ull);
    if (mixed::div_rn(a, x, 1.0 / x) != a / x) atomicAdd(&bad[1], 1ull);
    if (mixed::div_rn(a, 0.1 * x, rcp_(0.1 * x)) != a / (0.1 * x)) atomicAdd(&bad[2], 1ull);
  }
}

int main() {
  unsigned long long *bad, h[3];
  if (cudaMalloc(&bad, sizeof h) != cudaSuccess) return 1;
  cudaMemset(bad, 0, sizeof h);
  check<<<148 * 8, 256>>>(1ull << 30, bad);
  if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  printf("differ %llu %llu %llu\n", h[0], h[1], h[2]);
  return 0;
}
