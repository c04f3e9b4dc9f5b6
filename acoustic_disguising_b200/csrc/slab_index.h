// slab_index.h -- places in the CPML memory of the slabs.
//
// An array of one axis and side of the update (p, v) is [side][row][pitch]:
//   x: row = k*ny + j, pitch npp or nvp, side 1 from cell xs1 on
//   y: row = k*layers + layer, pitch nxp
//   z: row = layer*ny + j, pitch nxp
// Pitches and side lengths are multiples of four floats, so a place is counted
// in quads, 32 bits of them, for sides below 2^33 floats (solve_alloc refuses
// more; two buffers of two such sides do not fit the GPU's memory).  Sums are
// taken modulo 2^32, and the whole is less.
#ifndef ADF_SLAB_INDEX_H
#define ADF_SLAB_INDEX_H

#include <stdint.h>

#ifdef __CUDACC__
#define ADF_HD __host__ __device__ __forceinline__
#else
#define ADF_HD inline
#endif

namespace adf {

constexpr uint32_t kNoSlab = 0xFFFFFFFFu;
constexpr long long kMaxSideFloats = 1ll << 33;  // (every quad of two sides lies below kNoSlab)

// Quad of cell x (of its side) of a row.
ADF_HD uint32_t slab_quad(long long side_floats, int side, uint32_t row, int pitch, int x) {
  return (side ? (uint32_t)(side_floats >> 2) : 0u) + row * ((uint32_t)pitch >> 2) +
         ((uint32_t)x >> 2);
}

}  // namespace adf

#endif
