// Hash of a blob's position, for the host's and the device's table of the
// blobs by position (host and device code; compiles without CUDA too).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define T2D_HASH_HD __host__ __device__ __forceinline__
#else
#define T2D_HASH_HD inline
#endif

namespace t2d {

T2D_HASH_HD uint64_t mix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

// From the coordinates' bits.  x enters unmixed and y mixed: with both mixed
// alike, all positions of x = y would share one hash (and (x, y) that of (y,
// x)), and a sheet along the diagonal one probe chain through every blob.
T2D_HASH_HD uint64_t position_hash(uint64_t x, uint64_t y) { return mix64(x ^ mix64(y)); }

}  // namespace t2d
