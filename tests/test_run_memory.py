"""run_fdtd's device memory: what fits a budget, and arrays larger than the memory
their layout is converted in."""
import numpy as np
import pytest

from test_fdtd_parity import _Cp, assert_parity, make_case, run_both, to_adf_grid

pytestmark = pytest.mark.gpu


def solve_bytes(nx, ny, nz, npml, ntx, nt, mask):
    """What a run is held to: fields, mask bits, CPML memory, ten traces, entries."""
    nxp, ty, n = (nx + 3) // 4 * 4, min(7, ny), npml
    b = 2 * 4 * nz * ny * nxp * 4
    if mask:
        b += ((nx + 7) // 8 + 3) // 4 * 4 * ny * nz * 4
    for m in (n, n + 1):
        b += 2 * 2 * 4 * (nz * ny * m + nz * m * nxp + m * ny * nxp)
    b += 10 * nt * ntx * 4 + ntx * 4 * 8 * 4 * 3 + -(-ny // ty) * nz * 4 * 4
    return b + (1 << 20)


@pytest.mark.parametrize("nx,ny,nz,npml,shape,n_rec", [
    (48, 44, 40, 6, "sphere", 40),
    (48, 44, 40, 0, "none", 4000),   # a trace larger than the field
    (30, 28, 26, 4, "sphere", 10),   # a grid with a conversion buffer of its own
])
def test_a_run_that_just_fits_its_budget(adf, oracle, nx, ny, nz, npml, shape, n_rec):
    case = make_case(adf, oracle, nx, ny, nz, steps=90, npml=npml, shape=shape, seed=1, n_rec=n_rec)
    d, o, g, cp, mask, field = case
    need = solve_bytes(nx, ny, nz, npml, g.idx[0].shape[1], d.nt, mask is not None)

    def run(own):
        gg, pc, f = to_adf_grid(adf, g), _Cp(adf, cp), field.copy(order="F")
        adf.run_fdtd(d, f, gg, pc, mask, ctx=own)
        return f, gg, pc
    with pytest.raises(adf.AdfError) as ei:
        run(adf.Context(0, need - 1))
    assert ei.value.code == -3
    gpu = run(adf.Context(0, need))
    go, co, f_cpu = g.copy(), cp.copy(), field.copy(order="F")
    oracle.run_fdtd(o, f_cpu, go, co, mask)
    assert_parity(gpu, (f_cpu, go, co), 1e-6)


def test_a_gf_request_that_just_fits_its_budget(adf, oracle):
    n, npml, n_rec, steps = 60, 6, 30, 20
    from test_fdtd_parity import C0, DT, DX, RHO

    d = adf.Domain(tmax=(steps - 0.5) * DT, xmax=(n - 1) * DX / 2, nx=n, c0=C0, r0=RHO, cf=0.5)
    tf, _ = adf.impulsive_wavelet(d, 9000.0)
    rp, rn = adf.fibonacci_sphere(n_rec, 0.5 * d.xmax)

    def request():
        return adf.GfRequest(d, [0.3 * d.xmax, 0.0, 0.0], [1.0, 0, 0, 0], tf, rp, rn, npml=npml,
                             pml_fc=2000.0, scatterer="sphere",
                             scatterer_kw=dict(radius=0.2 * d.xmax))
    need = solve_bytes(n, n, n, npml, 1 + n_rec, steps, True)
    need += (2 - 10) * steps * (1 + n_rec) * 4 + 4 * steps * 4 + 2 * steps * n_rec * 4
    need += (1 + n_rec) * 4 * 8 * 4
    plain, fits = request(), request()
    adf.gf_solve_batch([plain])
    with pytest.raises(adf.AdfError) as ei:
        adf.gf_solve_batch([request()], ctx=adf.Context(0, need - 1))
    assert ei.value.code == -3
    adf.gf_solve_batch([fits], ctx=adf.Context(0, need))
    assert np.abs(plain.p).max() > 0
    assert np.array_equal(plain.p, fits.p) and np.array_equal(plain.vn, fits.vn)


@pytest.mark.parametrize("nx,ny,nz,npml,nt,n_rec", [
    (12, 30, 28, 5, 3000, 300),      # columns of a trace in pieces of 87
    (30, 28, 26, 4, 300001, 2),      # a column longer than the buffer
    (8, 100, 99, 26, 40, 6),         # x-slab memory larger than the field
])
def test_arrays_in_pieces(adf, oracle, nx, ny, nz, npml, nt, n_rec):
    """Traces and CPML memory that cross in several pieces: every element arrives, goes
    through a few steps and comes back in its place."""
    case = make_case(adf, oracle, nx, ny, nz, steps=nt, npml=npml, shape="none", seed=3, n_rec=n_rec)
    d, o, g, cp, mask, field = case
    rng = np.random.default_rng(nx)
    for a in g.rec + g.src + [g.vn_rec, g.vn_src]:
        a[...] = rng.standard_normal(a.shape).astype(np.float32) * 1e-3
    for a in cp.mv + cp.mp:
        a[...] = rng.standard_normal(a.shape).astype(np.float32) * 1e-3
    gpu, cpu = run_both(adf, oracle, case, start=5, stop=9)
    assert_parity(gpu, cpu, 1e-6)
    (_, gg, pc), (_, go, co) = gpu, cpu
    rest = np.r_[0:4, 10:nt]  # rows that no step touched
    for a, b in zip(gg.rec + gg.src + [gg.vn_rec, gg.vn_src], go.rec + go.src + [go.vn_rec, go.vn_src]):
        assert np.array_equal(a[rest], b[rest])
