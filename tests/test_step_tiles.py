"""Step kernel against the oracle where its tiling can go wrong."""
import numpy as np
import pytest

from test_fdtd_parity import assert_parity, make_case, run_both


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,npml", [
    (130, 23, 20, 5),   # three x tiles, four y tiles, the last of each partial
    (64, 14, 17, 4),    # one x tile, two whole y tiles, a one-plane last chunk
    (67, 15, 33, 0),    # three cells in the second x tile, no CPML
])
def test_closed_cells_on_tile_edges(adf, oracle, ctx, nx, ny, nz, npml):
    """The mask is read only on planes of a tile (halo row and column included)
    that hold a closed bit: single closed cells on both sides of the tile
    edges, with any of the four bits closed, and nowhere else."""
    d, o, g, cp, _, field = make_case(adf, oracle, nx, ny, nz, steps=30, npml=npml, shape="none",
                                      seed=nx)
    rng = np.random.default_rng(ny)
    mask = np.ones((nx, ny, nz, 4), bool, order="F")
    for x in (5, 62, 63, 64, 65, 127, 128):
        for y in (6, 7, 13, 14):
            for z in (3, 15, 16):
                if x < nx and y < ny and z < nz and rng.random() < 0.4:
                    mask[x, y, z, rng.integers(4)] = False
    assert not mask.all()
    gpu, cpu = run_both(adf, oracle, (d, o, g, cp, mask, field))
    assert_parity(gpu, cpu, 1e-6)
