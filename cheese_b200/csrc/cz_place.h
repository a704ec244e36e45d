// The places that a counting sort gives its pairs, checked by a sum (device, and host for its test).
#pragma once
#include <cstdint>
#ifdef __CUDACC__
#define CZ_PLACE_HD __host__ __device__ __forceinline__
#else
#define CZ_PLACE_HD inline
#endif

namespace cz {

// A 64-bit mark of a place. Over all pairs i of a sort with places p(i), the sum of mark(p(i)) - mark(i) is 0 (mod 2^64)
// when the places are a permutation, and for any other places only by a chance of 2^-64.
CZ_PLACE_HD uint64_t place_mark(uint32_t p) {          // the finaliser of splitmix64 (Steele, Lea, Flood 2014)
  uint64_t x = ((uint64_t)p + 1) * 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}

}  // namespace cz
