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

// What one of a warp's 32 lanes fetches ahead of plane k of the tile (x tile X of `xt`
// cells, y tile T) of a grid g (SolveDev): `floats` of array `array` (p x, y, z, v x, y,
// z) from quad `quad` on.  lane = tile row + 8 x (p y, v y, p z, v z); the v arrays
// have no halo row, whose two lanes take the rows of the x slabs (with `x_slabs`), one
// contiguous piece each.  zp, zv: the plane's layers in the z slabs, or kNoSlab.
struct SlabPiece {
  int array;
  uint32_t quad;
  int floats;
};
template <typename Grid>
ADF_HD SlabPiece slab_piece(const Grid& g, int X, int T, int xt, int lane, int k, bool x_slabs,
                            uint32_t zp, uint32_t zv) {
  const int row = lane & 7, arr = lane >> 3, j = T * g.ty - 1 + row, xb = X * xt;
  const bool v = arr & 1;
  if (row > g.ty || j >= g.ny) return SlabPiece{0, 0, 0};
  if (v && row == 0) {
    const bool lo = X == 0, hi = xb + xt >= g.nxp, xv = arr == 3;
    if (!x_slabs || (!lo && !hi)) return SlabPiece{0, 0, 0};
    const int pitch = xv ? g.nvp : g.npp, j0 = j < 0 ? 0 : j;
    const int j1 = j + g.ty + 1 < g.ny ? j + g.ty + 1 : g.ny;
    return SlabPiece{xv ? 3 : 0,
                     slab_quad(xv ? g.psi_v_side[0] : g.psi_p_side[0], !lo,
                               (uint32_t)(k * g.ny + j0), pitch, 0),
                     (j1 - j0) * pitch};
  }
  if (j < 0) return SlabPiece{0, 0, 0};
  SlabPiece f{(arr < 2 ? 1 : 2) + (v ? 3 : 0), 0, g.nxp - xb < xt ? g.nxp - xb : xt};
  if (arr < 2) {
    const int m = g.npml + (v ? 1 : 0), right = j >= m;  // layers
    if (right && j < g.ny - m) return SlabPiece{0, 0, 0};
    f.quad = slab_quad(v ? g.psi_v_side[1] : g.psi_p_side[1], right,
                       (uint32_t)(k * m + (right ? j - (g.ny - m) : j)), g.nxp, xb);
  } else {
    const uint32_t layer = v ? zv : zp;
    if (layer == kNoSlab) return SlabPiece{0, 0, 0};
    f.quad = layer + slab_quad(0, 0, (uint32_t)j, g.nxp, xb);
  }
  return f;
}

}  // namespace adf

#endif
