"""Index arithmetic of the CPML memory (csrc/slab_index.h) on the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "acoustic_disguising_b200", "csrc")

# Every array of a solve as solve_alloc lays it out, in 64 bits, against the step
# kernel's sums: the place in plane 0 plus k strides (x, y), the layer's plus the row's
# (z), and the whole place at once.
PLACES = r"""
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include "slab_index.h"
using namespace adf;
typedef long long ll;
static int bad = 0;
static ll top = 0;
static void check(uint32_t got, ll want, ll side) {
  if ((ll)got * 4 != want || want < 0 || want + 4 > 2 * side || got == kNoSlab) ++bad;
  top = std::max(top, want);
}
int main(int argc, char** argv) {
  const ll nx = atoll(argv[1]), ny = atoll(argv[2]), nz = atoll(argv[3]), n0 = atoll(argv[4]);
  const ll nxp = (nx + 3) / 4 * 4;
  for (ll n = n0; n <= n0 + 1; ++n) {  // the p side's layers, the v side's
    const ll xs1 = std::max(0ll, nx - n) / 4 * 4;
    const ll pitch = std::max((n + 3) / 4 * 4, nxp - xs1);
    const ll side[3] = {nz * ny * pitch, nz * n * nxp, n * ny * nxp};
    for (int a = 0; a < 3; ++a)
      if (side[a] >= kMaxSideFloats) ++bad;
    const ll ks[] = {0, 1, 31, 32, nz / 2, nz - 2, nz - 1};
    const ll js[] = {0, 1, 7, ny / 2, ny - 2, ny - 1}, ls[] = {0, n / 2, n - 1};
    for (int s = 0; s < 2; ++s)
      for (ll k : ks) {
        if (k < 0 || k >= nz) continue;
        for (ll j : js) {
          if (j < 0 || j >= ny) continue;
          for (ll x = 0; x < pitch; x += 4) {
            const ll want = s * side[0] + (k * ny + j) * pitch + x;
            check(slab_quad(side[0], s, (uint32_t)(k * ny + j), (int)pitch, (int)x), want, side[0]);
            check(slab_quad(side[0], s, (uint32_t)j, (int)pitch, (int)x) +
                      (uint32_t)k * slab_quad(0, 0, (uint32_t)ny, (int)pitch, 0), want, side[0]);
          }
        }
        for (ll l : ls)
          for (ll x = 0; x < nxp; x += 4) {
            const ll want = s * side[1] + (k * n + l) * nxp + x;
            check(slab_quad(side[1], s, (uint32_t)l, (int)nxp, (int)x) +
                      (uint32_t)k * slab_quad(0, 0, (uint32_t)n, (int)nxp, 0), want, side[1]);
          }
      }
    for (int s = 0; s < 2; ++s)
      for (ll l : ls)
        for (ll j : js)
          if (j >= 0 && j < ny)
            for (ll x = 0; x < nxp; x += 4)
              check(slab_quad(side[2], s, (uint32_t)(l * ny), (int)nxp, 0) +
                        slab_quad(0, 0, (uint32_t)j, (int)nxp, (int)x),
                    s * side[2] + (l * ny + j) * nxp + x, side[2]);
  }
  std::printf("%d %lld\n", bad, top);
  return 0;
}
"""


# What the lanes of a warp fetch ahead of a plane of a tile, against the slab rows of
# the tile, worked out cell by cell in 64 bits from the layout of solve_alloc.
PIECES = r"""
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <set>
#include <utility>
#include "slab_index.h"
using namespace adf;
typedef long long ll;
struct Grid {
  int ny, ty, nxp, npml, npp, nvp;
  ll psi_p_side[3], psi_v_side[3];
};
int main(int argc, char** argv) {
  const int nx = atoi(argv[1]), ny = atoi(argv[2]), nz = atoi(argv[3]), n = atoi(argv[4]);
  const int ty = atoi(argv[5]), xt = 64, nxp = (nx + 3) / 4 * 4;
  auto pitch = [&](int m) { return std::max((m + 3) / 4 * 4, nxp - std::max(0, nx - m) / 4 * 4); };
  Grid g{ny, ty, nxp, n, pitch(n), pitch(n + 1), {}, {}};
  for (int v = 0; v < 2; ++v) {
    const ll m = n + v, s[3] = {(ll)nz * ny * (v ? g.nvp : g.npp), nz * m * nxp, m * ny * nxp};
    for (int a = 0; a < 3; ++a) (v ? g.psi_v_side : g.psi_p_side)[a] = s[a];
  }
  auto side = [&](int array) { return (array >= 3 ? g.psi_v_side : g.psi_p_side)[array % 3]; };
  ll wrong = 0, fetched = 0;
  for (int k = 0; k < nz; ++k) {
    // (-1, m: the layer and its side; slab memory of the v side starts at plane 1)
    auto layer = [&](int v) {
      const int m = n + v;
      if (k < v) return kNoSlab;
      if (k < m) return slab_quad(g.psi_p_side[2], 0, (uint32_t)(k * ny), nxp, 0);
      if (k >= nz - m)
        return slab_quad(side(v ? 5 : 2), 1, (uint32_t)((k - (nz - m)) * ny), nxp, 0);
      return kNoSlab;
    };
    for (int T = 0; T < (ny + ty - 1) / ty; ++T)
      for (int X = 0; X < (nxp + xt - 1) / xt; ++X) {
        const int xb = X * xt, xe = std::min(xb + xt, nxp);
        std::set<std::pair<int, ll>> want, got;  // (array, float / 4)
        for (int r = 0; r <= ty; ++r) {
          const int j = T * ty - 1 + r;
          if (j < 0 || j >= ny) continue;
          for (int v = 0; v < 2; ++v) {
            const ll m = n + v;
            if (X == 0 || xe == nxp) {
              const ll p = v ? g.nvp : g.npp, s = X == 0 ? 0 : 1;
              for (ll x = 0; x < p; x += 4)
                want.insert({3 * v, (s * side(3 * v) + ((ll)k * ny + j) * p + x) / 4});
            }
            if (v && r == 0) continue;  // the halo row has no velocity update
            for (ll x = xb; x < xe; x += 4) {
              if (j < m) want.insert({1 + 3 * v, ((k * m + j) * nxp + x) / 4});
              else if (j >= ny - m)
                want.insert({1 + 3 * v, (side(1 + 3 * v) + (k * m + j - (ny - m)) * nxp + x) / 4});
              if (k >= v && k < m) want.insert({2 + 3 * v, (((ll)k * ny + j) * nxp + x) / 4});
              else if (k >= nz - m)
                want.insert({2 + 3 * v, (side(2 + 3 * v) + ((k - (nz - m)) * ny + j) * nxp + x) / 4});
            }
          }
        }
        for (int lane = 0; lane < 32; ++lane) {
          const SlabPiece f = slab_piece(g, X, T, xt, lane, k, true, layer(0), layer(1));
          for (int i = 0; i < f.floats; i += 4) {
            const ll at = (ll)f.quad * 4 + i;
            if (at < 0 || at + 4 > 2 * side(f.array)) ++wrong;
            got.insert({f.array, at / 4});
          }
          const SlabPiece h = slab_piece(g, X, T, xt, lane, k, false, layer(0), layer(1));
          if (h.floats != (f.array % 3 == 0 ? 0 : f.floats)) ++wrong;
        }
        if (got != want) ++wrong;
        fetched += (ll)got.size();
      }
  }
  std::printf("%lld %lld\n", wrong, fetched);
  return 0;
}
"""


def run_cpp(tmp_path, text, *args):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ is not available")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(text)
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True)
    return subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True,
                          text=True).stdout


@pytest.mark.parametrize("nx,ny,nz,npml,past", [
    (128, 4100, 4100, 63, 2 ** 31),   # 2.2e9 floats of x-slab memory a buffer
    (4, 8192, 8190, 63, 2 ** 32),     # the narrowest grid: the x slabs past 2^32 floats
    (512, 512, 2000, 63, 2 ** 25),
    (37, 29, 23, 5, 0),
    (9, 8, 41, 1, 0),
])
def test_slab_places(tmp_path, nx, ny, nz, npml, past):
    """No place of an array wraps or leaves its buffer, past 2^31 floats too."""
    bad, top = map(int, run_cpp(tmp_path, PLACES, nx, ny, nz, npml).split())
    assert bad == 0
    assert top >= past


@pytest.mark.parametrize("nx,ny,nz,npml,ty", [
    (163, 30, 29, 7, 7),    # three x tiles, the last y tile of two rows
    (129, 29, 21, 1, 7),    # one layer: velocity memory of two; an x tile of one quad
    (70, 23, 25, 9, 5),     # the right x slab begins in the tile before the last
    (40, 16, 18, 3, 7),     # one x tile with both slabs: the left one is fetched
])
def test_slab_pieces(tmp_path, nx, ny, nz, npml, ty):
    """The memory fetched ahead of every plane of every tile is that of the tile's slab
    rows, all of it, and lies inside its buffer."""
    wrong, fetched = map(int, run_cpp(tmp_path, PIECES, nx, ny, nz, npml, ty).split())
    assert wrong == 0
    assert fetched > 0


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,npml", [
    (12, 30, 28, 5),     # a quad with cells of both x slabs
    (100, 92, 90, 40),   # the halo column of the second x tile in the right slab, deep layers
    (66, 15, 20, 2),     # ... which is all of that tile
])
def test_slabs_of_narrow_tiles(adf, oracle, ctx, nx, ny, nz, npml):
    from test_fdtd_parity import assert_parity, make_case, run_both

    case = make_case(adf, oracle, nx, ny, nz, steps=20, npml=npml, shape="none", seed=nx, n_rec=6)
    gpu, cpu = run_both(adf, oracle, case)
    assert_parity(gpu, cpu, 1e-6)
