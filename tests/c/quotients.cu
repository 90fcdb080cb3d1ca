// recip_rn and quot_rn of csrc/sph_device.cuh against the IEEE operations, on the device.
//
// Prints the number of wrong results of
//   1. recip_rn over every significand but all ones, at several exponents;
//   2. quot_rn over every divisor significand with the numerators whose quotient lies nearest a
//      rounding midpoint. For significands A, B (24 bits) and s = 24 (A >= B) or 25, the quotient's distance from
//      the midpoint M / 2^s (M odd) is k / (B 2^s), k = A 2^s - B M. The first quotient RN(a y) is within
//      1 ulp of a / b where A >= B and within 1.5 where A < B, the residual's own rounding included the
//      step's error before its last rounding is at most 2 2^-48 (A < B, where a midpoint is at least |k| 2^-49
//      away) and 2^-47 (A >= B: |k| 2^-48), so that only |k| <= 4 can round wrongly: all |k| <= 7 are tried;
//   3. quot_rn over pairs at the ends of the ranges that pair_safe admits, and drawn ones.
#include <cstdint>
#include <cstdio>

#include "sph_device.cuh"

namespace {

__device__ float make(uint32_t significand, int exponent) {  // significand / 2^23 * 2^exponent
  return __uint_as_float((uint32_t)(exponent + 127) << 23 | (significand & 0x7fffffu));
}

__device__ void check(float a, float b, unsigned long long* tried, unsigned long long* wrong) {
  atomicAdd(tried, 1ull);
  if (__float_as_uint(vxl::quot_rn(a, b, vxl::recip_rn(b))) != __float_as_uint(__fdiv_rn(a, b))) atomicAdd(wrong, 1ull);
}

__global__ void reciprocals(unsigned long long* out) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= 0x7fffffu) return;  // all ones: pair_safe keeps it out
  for (int e : {-60, -41, -30, -27, -1, 0, 1, 10, 21, 41, 60}) {
    const float b = make(m, e);
    if (__float_as_uint(vxl::recip_rn(b)) != __float_as_uint(__fdiv_rn(1.0f, b))) atomicAdd(out, 1ull);
  }
}

__global__ void hard(unsigned long long* out) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= 0x7fffffu) return;
  const uint32_t B = m | 0x800000u;
  for (uint32_t t = 0; t < 3; ++t) {
    if (B & ((1u << t) - 1u)) break;  // 2^t divides k only if it divides B
    if (!(B >> t & 1u)) continue;     // A 2^s - B M = k, M odd: k holds as many factors 2 as B
    const uint32_t N = B >> t;
    for (int k = -7; k <= 7; k += 2) {  // k 2^t, k odd
      if ((k < 0 ? -k : k) << t > 7) continue;
      for (uint32_t s = 24; s <= 25; ++s) {
        // A = k / 2^(s - t) modulo N, by halving
        uint32_t x = (uint32_t)((k % (int)N + (int)N) % (int)N);
        for (uint32_t i = 0; i < s - t; ++i) x = (x & 1u) ? (x + N) / 2 : x / 2;
        for (uint32_t A = x; A < (1u << 24); A += N) {
          if (A < 0x800000u || (A >= B) != (s == 24)) continue;
          check(make(A, 0), make(B, 0), out + 1, out + 2);
          check(make(A, -39), make(B, -30), out + 1, out + 2);
          check(make(A, 39), make(B, 20), out + 1, out + 2);
        }
      }
    }
  }
}

__global__ void drawn(unsigned long long* out) {
  uint64_t z = (uint64_t)(blockIdx.x * blockDim.x + threadIdx.x) * 0x9e3779b97f4a7c15ull + 1;
  for (int i = 0; i < 64; ++i) {  // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    uint64_t r = (z ^ z >> 30) * 0xbf58476d1ce4e5b9ull;
    r = (r ^ r >> 27) * 0x94d049bb133111ebull;
    r ^= r >> 31;
    const uint32_t A = (uint32_t)r & 0x7fffffu, B = (uint32_t)(r >> 23) & 0x7fffffu;
    if (B == 0x7fffffu) continue;
    const int ea = i % 4 == 0 ? -40 : (i % 4 == 1 ? 39 : (int)(r >> 46 & 63) - 32);  // the numerators' ends: 2^-40, 2^40
    const int eb = i / 4 % 4 == 0 ? -30 : (i / 4 % 4 == 1 ? 21 : (int)(r >> 52 & 31) - 16);
    check(make(A, ea), make(B, eb), out + 1, out + 2);
  }
}

}  // namespace

int main() {
  unsigned long long* d = nullptr;
  unsigned long long h[3] = {1, 0, 1};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
  reciprocals<<<(1 << 23) / 256, 256>>>(d);
  hard<<<(1 << 23) / 256, 256>>>(d);
  drawn<<<4096, 256>>>(d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("%llu reciprocals wrong, %llu quotients, %llu wrong\n", h[0], h[1], h[2]);
  return h[0] || h[2] ? 1 : 0;
}
