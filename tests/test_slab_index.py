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
