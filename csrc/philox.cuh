// Counter-based random numbers of the samplers (Philox-4x32-10).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dice {

struct Philox {
  uint32_t key[2];
  __device__ __forceinline__ Philox(unsigned long long seed) {
    key[0] = static_cast<uint32_t>(seed);
    key[1] = static_cast<uint32_t>(seed >> 32);
  }
  __device__ __forceinline__ uint4 operator()(unsigned long long counter, unsigned long long stream) const {
    uint32_t c0 = static_cast<uint32_t>(counter), c1 = static_cast<uint32_t>(counter >> 32);
    uint32_t c2 = static_cast<uint32_t>(stream), c3 = static_cast<uint32_t>(stream >> 32);
    uint32_t k0 = key[0], k1 = key[1];
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
      const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
      const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
      c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    return make_uint4(c0, c1, c2, c3);
  }
};

// Maps 64 random bits to [0, high) by the multiply-high reduction (bias below high / 2^64).
__device__ __forceinline__ long long bounded(uint32_t a, uint32_t b, long long high) {
  const unsigned long long x = (static_cast<unsigned long long>(a) << 32) | b;
  return static_cast<long long>(__umul64hi(x, static_cast<unsigned long long>(high)));
}

}  // namespace dice
