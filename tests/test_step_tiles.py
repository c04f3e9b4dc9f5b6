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


@pytest.mark.gpu
@pytest.mark.parametrize("nz", [4, 5, 13, 34])
def test_shallow_items(adf, oracle, ctx, nz):
    """A small run takes the shallowest work items: two planes, the last item
    one (the rigid plane alone) when nz is odd."""
    case = make_case(adf, oracle, 40, 30, nz, steps=25, npml=min(4, (nz - 2) // 2), shape="none",
                     seed=nz, n_rec=6)
    gpu, cpu = run_both(adf, oracle, case)
    assert_parity(gpu, cpu, 1e-6)


@pytest.mark.gpu
def test_depth_of_a_batch_changes_nothing(adf, ctx):
    """Ten solves share deeper items than one alone: the traces stay bit for
    bit those of the plain path."""
    from test_fdtd_parity import C0, DT, DX, RHO

    def request(n, k):
        d = adf.Domain(tmax=29.5 * DT, xmax=(n - 1) * DX / 2, nx=n, c0=C0, r0=RHO, cf=0.5)
        tf, _ = adf.impulsive_wavelet(d, 9000.0)
        rp, rn = adf.fibonacci_sphere(30, 0.5 * d.xmax)
        return adf.GfRequest(d, [0.3 * d.xmax, 0.02 * k * d.xmax, 0.0], [1.0, 0, 0, 0], tf, rp, rn,
                             npml=6, pml_fc=2000.0, scatterer="sphere",
                             scatterer_kw=dict(radius=0.2 * d.xmax))
    sizes = [96, 90, 85, 96, 64, 71, 96, 96, 80, 96]
    batch = [request(n, k) for k, n in enumerate(sizes)]
    alone = [request(n, k) for k, n in enumerate(sizes)]
    adf.gf_solve_batch(batch, batched=True)
    adf.gf_solve_batch(alone, batched=False)
    for a, b in zip(batch, alone):
        assert np.abs(a.p).max() > 0
        assert np.array_equal(a.p, b.p) and np.array_equal(a.vn, b.vn)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [None, "7,1", "7,2", "5,9", "7,32"])
def test_chunks_of_a_mixed_batch_change_nothing(adf, ctx, tile, monkeypatch):
    """Solves of unequal sizes and layer widths (none, and layers that leave few
    planes between them) in one batch: the chunks shrink towards the end, come from
    both ends in turn and keep to a tile's depth where one is given.  Every plane is
    stepped once: the traces are bit for bit those of each solve alone, and those of
    solves cut into equal chunks."""
    from test_fdtd_parity import C0, DT, DX, RHO

    def request(n, npml, k):
        d = adf.Domain(tmax=19.5 * DT, xmax=(n - 1) * DX / 2, nx=n, c0=C0, r0=RHO, cf=0.5)
        tf, _ = adf.impulsive_wavelet(d, 9000.0)
        rp, rn = adf.fibonacci_sphere(30, 0.4 * d.xmax)
        return adf.GfRequest(d, [0.35 * d.xmax, 0.01 * k * d.xmax, 0.0], [1.0, 0, 0, 0], tf, rp,
                             rn, npml=npml, pml_fc=2000.0, scatterer="sphere",
                             scatterer_kw=dict(radius=0.25 * d.xmax))
    sizes = [(96, 10), (30, 13), (101, 0), (64, 5), (33, 1), (110, 12), (96, 10), (47, 8), (83, 20)]
    if tile:
        monkeypatch.setenv("ADF_TILE", tile)
    batch = [request(n, npml, k) for k, (n, npml) in enumerate(sizes)]
    adf.gf_solve_batch(batch, batched=True)
    monkeypatch.setenv("ADF_TILE", "7,4")
    alone = [request(n, npml, k) for k, (n, npml) in enumerate(sizes)]
    adf.gf_solve_batch(alone, batched=False)
    for a, b in zip(batch, alone):
        assert np.abs(a.p).max() > 0
        assert np.array_equal(a.p, b.p) and np.array_equal(a.vn, b.vn)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,npml", [
    (163, 162, 161, 7),   # just above the size from which slab memory is fetched ahead
    (257, 260, 255, 9),   # ... and the x slabs' too, the right one in the last two x tiles
    (270, 141, 442, 1),   # one layer: velocity memory of two
])
def test_fetched_slab_memory(adf, oracle, ctx, nx, ny, nz, npml):
    """Grids whose slab memory is fetched into L2 ahead, of odd sizes: the fetches
    change nothing and stay inside the memory."""
    case = make_case(adf, oracle, nx, ny, nz, steps=8, npml=npml, shape="none", seed=nx, n_rec=6)
    gpu, cpu = run_both(adf, oracle, case)
    assert_parity(gpu, cpu, 1e-6)
