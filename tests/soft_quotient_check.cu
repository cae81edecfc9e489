// Device check of mge::soft::quot and mulquot against the FP64 hardware, bit for
// bit, 2^24 triples of each of eight distributions.
#include <cstdio>

#include "soft_quotient_check.h"

using namespace mge::soft;

__device__ bool same(double x, double y) { return (isnan(x) && isnan(y)) || bits(x) == bits(y); }

__global__ void k_check(int kind, uint64_t n, unsigned long long* bad) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    double a, b, d;
    triple(kind, i, a, b, d);
    const Recip R = recip(d);
    if (!same(quot(a, R, d), __ddiv_rn(a, d)) || !same(mulquot(a, b, R, d), __ddiv_rn(__dmul_rn(a, b), d)))
      atomicAdd(bad, 1ull);
  }
}

int main() {
  unsigned long long *bad, total = 0;
  if (cudaMalloc(&bad, 8) != cudaSuccess) return 2;
  for (int kind = 0; kind < 8; kind++) {
    unsigned long long h = 0;
    cudaMemset(bad, 0, 8);
    k_check<<<152 * 8, 256>>>(kind, 1ull << 24, bad);
    if (cudaMemcpy(&h, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    total += h;
  }
  printf("mismatches %llu \n", total);
  return total ? 1 : 0;
}
