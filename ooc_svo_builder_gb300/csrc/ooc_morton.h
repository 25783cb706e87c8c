// Morton codes, on the host and on the device.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ooc {

// Morton codes: x -> bit 3i, y -> bit 3i+1, z -> bit 3i+2
// (libmorton morton3D_64_encode, morton.h:59-61).
__host__ __device__ __forceinline__ uint32_t spread3_10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}
__host__ __device__ __forceinline__ uint32_t compact3_10(uint32_t v) {
  v &= 0x09249249u;
  v = (v ^ (v >> 2)) & 0x030c30c3u;
  v = (v ^ (v >> 4)) & 0x0300f00fu;
  v = (v ^ (v >> 8)) & 0x030000ffu;
  v = (v ^ (v >> 16)) & 0x3ffu;
  return v;
}
// Local Morton code inside a stripe (coordinates < 1024, code < 2^30).
__host__ __device__ __forceinline__ uint32_t morton_local(uint32_t x, uint32_t y, uint32_t z) {
  return spread3_10(x) | (spread3_10(y) << 1) | (spread3_10(z) << 2);
}
__host__ __device__ __forceinline__ void morton_local_decode(uint32_t m, uint32_t& x, uint32_t& y, uint32_t& z) {
  x = compact3_10(m);
  y = compact3_10(m >> 1);
  z = compact3_10(m >> 2);
}
__host__ __device__ __forceinline__ uint64_t spread3_21(uint64_t v) {
  v &= 0x1fffffull;
  v = (v | (v << 32)) & 0x1f00000000ffffull;
  v = (v | (v << 16)) & 0x1f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  v = (v | (v << 2)) & 0x1249249249249249ull;
  return v;
}
__host__ __device__ __forceinline__ uint32_t compact3_21(uint64_t v) {
  v &= 0x1249249249249249ull;
  v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
  v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
  v = (v ^ (v >> 8)) & 0x1f0000ff0000ffull;
  v = (v ^ (v >> 16)) & 0x1f00000000ffffull;
  v = (v ^ (v >> 32)) & 0x1fffffull;
  return (uint32_t)v;
}
__host__ __device__ __forceinline__ uint64_t morton_global(uint32_t x, uint32_t y, uint32_t z) {
  return spread3_21(x) | (spread3_21(y) << 1) | (spread3_21(z) << 2);
}
__host__ __device__ __forceinline__ void morton_global_decode(uint64_t m, uint32_t& x, uint32_t& y, uint32_t& z) {
  x = compact3_21(m);
  y = compact3_21(m >> 1);
  z = compact3_21(m >> 2);
}

}  // namespace ooc
