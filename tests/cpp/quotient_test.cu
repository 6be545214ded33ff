// quotient_by (csrc/common.cuh) against the division on the device: prints the number of quotients and
// how many of them differ. Significands are random, or near the ends of their range (where the
// reciprocal's relative error is the largest) for numerator, divisor or both; divisors 2^-27..1.
#include <cstdint>
#include <cstdio>

#include "common.cuh"

namespace ves3d {
void set_error(const char*, ...) {}
std::atomic<long long>& launch_counter() {
  static std::atomic<long long> c{0};
  return c;
}
}  // namespace ves3d

__device__ uint64_t mix(uint64_t x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__device__ uint64_t significand(uint64_t r, int kind) {
  const uint64_t all = (1ull << 52) - 1;
  r &= all;
  const int low = 8 + (int)(mix(r) % 24);  // random bits that remain
  if (kind == 1) return r & ((1ull << low) - 1);
  if (kind == 2) return r | (all & ~((1ull << low) - 1));
  return r;
}

__global__ void compare(uint64_t n, unsigned long long* differ) {
  unsigned long long bad = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += gridDim.x * (uint64_t)blockDim.x) {
    const uint64_t a = mix(2 * i), b = mix(2 * i + 1), k = mix(a ^ b);
    const int es = -(int)(k % 27) - 1, en = (int)((k >> 8) % 930) - 900;
    const double s = __longlong_as_double((long long)((uint64_t)(1023 + es) << 52 | significand(b, (k >> 20) % 3)));
    double num = __longlong_as_double((long long)((uint64_t)(1023 + en) << 52 | significand(a, (k >> 24) % 3)));
    if (k >> 63) num = -num;
    const double q = ves3d::quotient_by(num, s, 1.0 / s), ref = num / s;
    bad += __double_as_longlong(q) != __double_as_longlong(ref);
  }
  if (bad) atomicAdd(differ, bad);
}

int main() {
  unsigned long long* d = nullptr;
  unsigned long long differ = 0;
  const uint64_t n = 1ull << 28;
  if (cudaMalloc((void**)&d, sizeof(*d)) || cudaMemset(d, 0, sizeof(*d))) return 1;
  compare<<<148 * 8, 256>>>(n, d);
  if (cudaMemcpy(&differ, d, sizeof(differ), cudaMemcpyDeviceToHost)) return 1;
  printf("%llu %llu\n", (unsigned long long)n, differ);
  return 0;
}
