// Checks div_known (the streamline pass's quotient from a correctly rounded reciprocal)
// against IEEE division __fdiv_rn, bit for bit: 2^31 random pairs with divisors of every
// exponent from 2^-24 to 2^24 (in and around its fast range) and numerators of any bits
// (zeros, denormals, infinities and NaN among them: equal bits, or both NaN).
// Prints "<mismatches> <cases>" and exits 0; every index is bounded by its loop.
#include <cstdint>
#include <cstdio>

#include "wt_lattice.cuh"

__device__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}

__global__ void sweep(uint32_t n, uint32_t seed, bool any_bits, unsigned long long* bad) {
  const uint32_t stride = gridDim.x * blockDim.x;
  unsigned long long local = 0;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride) {
    const uint32_t h1 = hash32(t * 2u + seed), h2 = hash32(t * 2u + 1u + seed * 7919u), h3 = hash32(h1 ^ h2 * 31u);
    const uint32_t ea = 127u - 64u + (h3 & 0xffffu) % 129u;  // 2^-64 .. 2^64
    const float a = any_bits ? (h3 % 64u == 0 ? __uint_as_float(h1 & 0x80000000u) : __uint_as_float(h1))
                             : __uint_as_float(((h1 & 1u) << 31) | (ea << 23) | (h1 >> 9));
    const float b = __uint_as_float(((127u - 24u + (h3 >> 16) % 49u) << 23) | (h2 & 0x7fffffu));
    const bool fast = wt::div_range(b);
    const float q = wt::div_known(a, b, __frcp_rn(fast ? b : 1.0f), fast), want = __fdiv_rn(a, b);
    local += __float_as_uint(q) != __float_as_uint(want) && !(q != q && want != want);
  }
  atomicAdd(bad, local);
}

int main() {
  unsigned long long* dbad = nullptr;
  if (cudaMalloc(&dbad, sizeof(unsigned long long)) != cudaSuccess) return 2;
  cudaMemset(dbad, 0, sizeof(unsigned long long));
  sweep<<<1216, 256>>>(1u << 30, 5u, false, dbad);
  sweep<<<1216, 256>>>(1u << 30, 91u, true, dbad);
  unsigned long long hbad = 0;
  if (cudaMemcpy(&hbad, dbad, sizeof(hbad), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  printf("%llu %llu\n", hbad, 2ull << 30);
  cudaFree(dbad);
  return 0;
}
