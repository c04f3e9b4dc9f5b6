"""Performance cases of the FDTD / Green's-function / KH library: what a user's
program has it do, through the Python entry points of acoustic_disguising_b200.

Medium and geometry follow the repository's own workloads (benchmark and
tests): 5 mm cells, air, CFL 0.5, CPML on all faces, Fibonacci shells, Ricker
and band-limited impulsive wavelets.  Each family has one builder (`prepare`),
one pass (`run`), its minimal traffic (`work`) and the same result in Float64
from plain torch (`exact`).
"""
import math

import numpy as np
import torch

import acoustic_disguising_b200 as A

DX, C0, RHO = 0.005, 343.0, 1.2
PML_R, PML_FC, F3DB = 1e-4, 2000.0, 2000.0


# ---------------------------------------------------------------------------
# the listed cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a quick look or a unit test of a host program: one short solve on an
        # odd-sized little box in Float32 arithmetic, all latency and launches
        dict(name="fdtd_tiny", family="fdtd", nx=40, ny=36, nz=33, npml=5, steps=60, nrec=8,
             shape="sphere", arith="fp32"),
        # the plain single solve: 96^3, 10-cell CPML, Ricker point source, 64
        # receivers, 800 steps
        dict(name="fdtd_plain", family="fdtd", nx=96, ny=96, nz=96, npml=10, steps=800, nrec=64,
             shape="none", arith="promote"),
        # impulsive Green's functions round a rigid sphere, batched: 256^3 and
        # a 2048-point shell (two of the 512 sources)
        dict(name="gf_sphere", family="gf", nx=256, ny=256, nz=256, npml=10, steps=1000, nrec=2048,
             solves=2, shape="sphere", arith="promote"),
        # one solve on the largest grid the library takes, 12-cell CPML and an
        # ellipsoid, recorded on an 8192-point shell
        dict(name="gf_large", family="gf", nx=512, ny=512, nz=512, npml=12, steps=240, nrec=8192,
             solves=1, shape="ellipsoid", arith="promote"),
        # requests of mixed grids, lengths and scatterers through the serving loop
        dict(name="serve_mixed", family="serve", sizes="96,128,160,128,96,192",
             steps="950,610,720,880,530,500", nrec=256),
        # a handful of control points: KH pressure, latency bound
        dict(name="kh_small", family="kh", kind="pressure", ns=200, nr=48, nt=700, dt=5e-6,
             r_surf=0.25, r_tgt=0.9),
        # KH pressure of a recorded surface at a whole far-field sphere
        dict(name="kh_far_field", family="kh", kind="pressure", ns=4096, nr=16384, nt=2048,
             dt=5e-6, r_surf=0.25, r_tgt=2.0),
        # KH normal velocity on a second surface, ragged sizes, wider window
        dict(name="kh_velocity", family="kh", kind="velocity", ns=1500, nr=2001, nt=1201,
             dt=3.6e-6, r_surf=0.25, r_tgt=0.8),
        # hologram synthesis: C_f/C_q injection on one surface, recording
        # shell, KH of the shell to the far field, traces handed over in HBM
        dict(name="hologram", family="holo", nx=192, ny=192, nz=192, npml=12, steps=500, nin=2048,
             nout=2048, nr=4096),
        # a run with the scatterer's Green's functions in the loop (recorded
        # shell drives the injection surface every step)
        dict(name="gf_loop", family="map", nx=128, ny=128, nz=128, npml=10, steps=300,
             kind="PVFromPin", contraction="fp64", lags=256, nsrc=256, nrec=256),
        # the same with a larger map and its older lags on the tensor cores
        dict(name="gf_loop_tf32x3", family="map", nx=96, ny=96, nz=96, npml=10, steps=500,
             kind="PFromPin", contraction="tf32x3", lags=300, nsrc=512, nrec=448),
        # post-processing of one source's recorded traces (denoise, cubic
        # B-spline resampling, physical units): 2048 receivers, p and v_n
        dict(name="postprocess", family="post", ncol=4096, nt_in=2000, nt_out=700),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _crossing(rng, n, most):
    """Steps of a run long enough for its waves to reach every face."""
    return _log(rng, 2.6 * n, max(2.7 * n, most))


def draw(rng):
    family = rng.choice(["fdtd", "fdtd", "gf", "gf", "serve", "kh", "kh", "holo", "map", "map",
                         "post"])
    if family == "fdtd":
        n = _log(rng, 32, 224)
        dims = [max(28, int(n * rng.uniform(0.75, 1.25))) for _ in range(3)]
        return dict(family="fdtd", nx=dims[0], ny=dims[1], nz=dims[2],
                    npml=rng.choice([5, 8, 10, 12]), steps=_crossing(rng, max(dims), 800),
                    nrec=_log(rng, 1, 2048), shape=rng.choice(["none", "sphere", "ellipsoid"]),
                    arith=rng.choice(["promote", "promote", "fp32"]))
    if family == "gf":
        n = _log(rng, 48, 360)
        dims = [max(40, min(512, int(n * rng.uniform(0.8, 1.25)))) for _ in range(3)]
        solves = _log(rng, 1, max(1.0, min(12.0, 2 * (256 / n) ** 3)))
        room = 2 * 1000 * 256 ** 3 / (solves * dims[0] * dims[1] * dims[2])
        return dict(family="gf", nx=dims[0], ny=dims[1], nz=dims[2], npml=rng.choice([8, 10, 12]),
                    steps=max(64, _log(rng, 64, max(65, min(1500, room)))),
                    nrec=_log(rng, 64, 2048), solves=solves,
                    shape=rng.choice(["none", "sphere", "cube", "ellipsoid"]),
                    arith=rng.choice(["promote", "promote", "fp32"]))
    if family == "serve":
        k = rng.randint(3, 7)
        return dict(family="serve", nrec=_log(rng, 64, 512),
                    sizes=",".join(str(rng.choice([96, 128, 160, 192])) for _ in range(k)),
                    steps=",".join(str(rng.randint(500, 1000)) for _ in range(k)))
    if family == "kh":
        kind = rng.choice(["pressure", "pressure", "velocity"])
        ns, nr, nt = _log(rng, 100, 4096), _log(rng, 20, 16384), _log(rng, 400, 2048)
        if kind == "velocity":
            nr = min(nr, 4000)
        dt = rng.choice([5e-6, 5e-6, 3.6e-6, 2.9e-6])
        return dict(family="kh", kind=kind, ns=ns, nr=nr, nt=nt, dt=dt, r_surf=0.25,
                    r_tgt=min(2.0, 0.25 + rng.uniform(0.15, 0.6) * nt * dt * C0))
    if family == "holo":
        n = _log(rng, 96, 192)
        return dict(family="holo", nx=n, ny=n, nz=n, npml=rng.choice([8, 10, 12]),
                    steps=_log(rng, 200, 500), nin=_log(rng, 256, 2048), nout=_log(rng, 256, 2048),
                    nr=_log(rng, 500, 4096))
    if family == "map":
        n = _log(rng, 72, 128)
        kind = rng.choice(["PVFromPin", "PFromPin", "PVFromPV"])
        tc = kind != "PVFromPV" and rng.random() < 0.4
        io = 512 if kind != "PVFromPV" else 200
        return dict(family="map", nx=n, ny=n, nz=n, npml=10, steps=_crossing(rng, n, 500), kind=kind,
                    contraction="tf32x3" if tc else "fp64", lags=_log(rng, 24, 300),
                    nsrc=_log(rng, 48, io), nrec=_log(rng, 48, io))
    return dict(family="post", ncol=_log(rng, 64, 4096), nt_in=_log(rng, 200, 3000),
                nt_out=_log(rng, 100, 1500))


# ---------------------------------------------------------------------------
# building blocks of the inputs
# ---------------------------------------------------------------------------
def _dt(cf=0.5):
    return cf * DX / C0 / math.sqrt(3.0)


def _domain(c):
    return A.Domain(tmax=(c["steps"] - 0.5) * _dt(), xmax=(c["nx"] - 1) * DX / 2,
                    ymax=(c["ny"] - 1) * DX / 2, zmax=(c["nz"] - 1) * DX / 2, nx=c["nx"],
                    ny=c["ny"], nz=c["nz"], c0=C0, r0=RHO, cf=0.5)


def _half(c):
    return (min(c["nx"], c["ny"], c["nz"]) - 1) * DX / 2


def _scatterer(shape, size, rng):
    """A rigid scatterer of half width about `size`, slightly off the centre."""
    centre = tuple(rng.uniform(-1.0, 1.0, 3) * DX)
    if shape == "sphere":
        return dict(radius=size, center=centre)
    if shape == "cube":
        return dict(length=1.6 * size, center=centre)
    if shape == "ellipsoid":
        return dict(semi_axes=(size, 0.75 * size, 0.5 * size), center=centre)
    return {}


def _ricker_noise(rng, nt, ns, dt, fc):
    """Ricker-filtered Gaussian noise (nt, ns), unit RMS per column."""
    half = int(2.0 / fc / dt)
    w = math.pi * fc * (np.arange(-half, half + 1) * dt)
    r = (1 - 2 * w * w) * np.exp(-w * w)
    nfft = 1 << int(math.ceil(math.log2(nt + len(r))))
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    x = torch.randn((ns, nt), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.rfft(torch.from_numpy(r).cuda(), nfft)
    y = torch.fft.irfft(torch.fft.rfft(x, nfft) * f, nfft)[:, half:half + nt]
    y = y / y.square().mean(dim=1, keepdim=True).sqrt()
    return y.float().contiguous().cpu().numpy().T


def _unit(rng):
    u = rng.standard_normal(3)
    return u / np.linalg.norm(u)


# ---------------------------------------------------------------------------
# prepare: what the program has in hand before the call
# ---------------------------------------------------------------------------
def _requests(c):
    """(grid, steps) of the requests of a serving case."""
    return list(zip(map(int, c["sizes"].split(",")), map(int, c["steps"].split(","))))


_server = None  # a serving program keeps one loop


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    family = c["family"]
    if family == "fdtd":
        d = _domain(c)
        inner = _half(c) - (c["npml"] + 3) * DX
        tf = A.ricker_wavelet(d, 2000.0, injection=False)
        rp, rn = A.fibonacci_sphere(c["nrec"], 0.8 * inner)
        src = 0.55 * inner * _unit(rng)
        txs = [A.Transceiver(src, np.array([1.0, 0, 0, 0]), tf)]
        txs += [A.Transceiver(rp[k], np.r_[0.0, rn[k]], np.zeros(d.nt)) for k in range(c["nrec"])]
        kw = _scatterer(c["shape"], 0.3 * inner, rng)
        return dict(c=c, d=d, g=A.transceivers_to_grid(d, txs), kw=kw, src_point=src,
                    cpml=A.Cpml(d, c["npml"], PML_R, PML_FC),
                    mask=A.build_update_mask(d, c["shape"], **kw), arith=c["arith"],
                    field=np.zeros((c["nx"], c["ny"], c["nz"], 4), np.float32, order="F"))
    if family == "gf":
        d = _domain(c)
        inner = _half(c) - (c["npml"] + 3) * DX
        tf, _ = A.impulsive_wavelet(d, F3DB)
        rp, rn = A.fibonacci_sphere(c["nrec"], 0.45 * inner)
        kw = _scatterer(c["shape"], 0.22 * inner, rng)
        reqs = [A.GfRequest(d, 0.6 * inner * _unit(rng), [1.0, 0, 0, 0], tf, rp, rn,
                            npml=c["npml"], pml_rcoef=PML_R, pml_fc=PML_FC, scatterer=c["shape"],
                            scatterer_kw=kw, arith=c["arith"]) for _ in range(c["solves"])]
        return dict(c=c, reqs=reqs)
    if family == "serve":
        global _server
        if _server is None:
            _server = A.Server(hbm_budget=120 << 30, work_waves=2.0)
        reqs = []
        for n, steps in _requests(c):
            q = dict(nx=n, ny=n, nz=n, steps=steps)
            d = _domain(q)
            xmax = _half(q)
            tf, _ = A.impulsive_wavelet(d, F3DB)
            shape = str(rng.choice(["none", "sphere", "cube", "ellipsoid"]))
            kw = _scatterer(shape, rng.uniform(0.1, 0.3) * xmax, rng)
            rp, rn = A.fibonacci_sphere(c["nrec"], 0.6 * xmax)
            reqs.append(A.GfRequest(d, 0.7 * xmax * _unit(rng), [1.0, 0, 0, 0], tf, rp, rn,
                                    npml=10, pml_rcoef=PML_R, pml_fc=PML_FC, scatterer=shape,
                                    scatterer_kw=kw))
        return dict(c=c, reqs=reqs, server=_server)
    if family == "kh":
        sp, sn = A.fibonacci_sphere(c["ns"], c["r_surf"])
        rp, rn = A.fibonacci_sphere(c["nr"], c["r_tgt"])
        p = _ricker_noise(rng, c["nt"], c["ns"], c["dt"], 2000.0)
        vn = _ricker_noise(rng, c["nt"], c["ns"], c["dt"], 2000.0) / np.float32(RHO * C0)
        dS = 4 * math.pi * c["r_surf"] ** 2 / c["ns"]
        return dict(c=c, sp=sp, sn=sn, rp=rp, rn=rn, vn=np.asfortranarray(vn),
                    p=np.asfortranarray(p), sigma=6.6e-6, aq=-RHO * dS * c["dt"], af=-dS * c["dt"],
                    out=np.zeros((c["nt"], c["nr"]), np.float32, order="F"))
    if family == "holo":
        d = _domain(c)
        inner = _half(c) - (c["npml"] + 3) * DX
        r_out, r_in = 0.85 * inner, 0.6 * inner
        op, on = A.fibonacci_sphere(c["nout"], r_out)
        ip, inn = A.fibonacci_sphere(c["nin"], r_in)
        zero = np.zeros(d.nt)
        txs = [A.Transceiver(op[k], np.r_[0.0, on[k]], zero) for k in range(c["nout"])]
        txs += [A.Transceiver(ip[k], np.r_[0.0, inn[k]], zero) for k in range(c["nin"])]
        g = A.transceivers_to_grid(d, txs)
        cf, cq, _ = A.injection_coefficients(d, r_in, c["nin"])
        drive = slice(c["nout"], c["nout"] + c["nin"])
        g.vn_src[:, drive] = cf * _ricker_noise(rng, d.nt, c["nin"], d.dt, 2000.0)
        g.src[0][:, drive] = cq * _ricker_noise(rng, d.nt, c["nin"], d.dt, 2000.0) / (RHO * C0)
        kw = _scatterer("ellipsoid", 0.4 * inner, rng)
        rp, _ = A.fibonacci_sphere(c["nr"], r_out + 0.3 * d.nt * d.dt * C0)
        dS = 4 * math.pi * r_out ** 2 / c["nout"]
        return dict(c=c, d=d, g=g, kw=kw, cpml=A.Cpml(d, c["npml"], PML_R, PML_FC),
                    mask=A.build_update_mask(d, "ellipsoid", **kw), arith="promote",
                    field=np.zeros((c["nx"], c["ny"], c["nz"], 4), np.float32, order="F"),
                    cols=np.arange(1, c["nout"] + 1, dtype=np.int64), op=op, on=on, rp=rp,
                    sigma=math.sqrt(math.log(2.0)) / (2 * math.pi * 20e3), aq=-RHO * dS * d.dt,
                    af=-dS * d.dt, out=np.zeros((int(d.nt), c["nr"]), np.float32, order="F"))
    if family == "map":
        d = _domain(c)
        inner = _half(c) - (c["npml"] + 3) * DX
        tf = A.ricker_wavelet(d, 2000.0, injection=False)
        rp, rn = A.fibonacci_sphere(c["nrec"], 0.8 * inner)   # recording shell (iRec)
        ip, inn = A.fibonacci_sphere(c["nsrc"], 0.6 * inner)  # injection surface (iSrc)
        src = 0.2 * inner * _unit(rng)
        txs = [A.Transceiver(src, np.array([1.0, 0, 0, 0]), tf * 1e3)]
        txs += [A.Transceiver(rp[k], np.r_[0.0, rn[k]], np.zeros(d.nt)) for k in range(c["nrec"])]
        txs += [A.Transceiver(ip[k], np.r_[0.0, inn[k]], np.zeros(d.nt)) for k in range(c["nsrc"])]
        i_rec = np.arange(2, 2 + c["nrec"], dtype=np.int64)
        i_src = np.arange(2 + c["nrec"], 2 + c["nrec"] + c["nsrc"], dtype=np.int64)
        n1, n2 = (c["nsrc"], c["nrec"]) if c["kind"] == "PVFromPin" else (c["nrec"], c["nsrc"])
        # loop gain about 0.05; the maps that turn p into v_n carry 1 / z0
        gain = 0.05 / math.sqrt(c["lags"] * c["nrec"] * c["nsrc"])
        z0 = RHO * C0
        units = {"PVFromPV": (1, 1 / z0, z0, 1), "PVFromPin": (1 / z0, 1), "PFromPin": (1, 1)}
        tens = [np.asfortranarray((rng.standard_normal((n2, n1, c["lags"]), dtype=np.float32) *
                                   np.float32(gain * u)).T) for u in units[c["kind"]]]
        if c["kind"] == "PVFromPV":
            gm = A.PVFromPV(*tens, i_src, i_rec)
        else:
            make = A.PVFromPin if c["kind"] == "PVFromPin" else A.PFromPin
            gm = make(*tens, i_src, i_rec, contraction=c["contraction"])
        return dict(c=c, d=d, g=A.transceivers_to_grid(d, txs), kw={}, mask=None, arith="promote",
                    src_point=src, cpml=A.Cpml(d, c["npml"], PML_R, PML_FC), gm=gm,
                    field=np.zeros((c["nx"], c["ny"], c["nz"], 4), np.float32, order="F"))
    t0 = rng.uniform(0.2, 0.8, c["ncol"]) * c["nt_in"]
    wd = rng.uniform(4, 25, c["ncol"])
    a = np.exp(-0.5 * ((np.arange(c["nt_in"])[:, None] - t0) / wd) ** 2)
    a = a * rng.normal(size=c["ncol"]) + rng.standard_normal((c["nt_in"], c["ncol"]),
                                                             dtype=np.float32) * 1e-6
    return dict(c=c, a=np.asfortranarray(a, np.float32), t_in0=-78 * _dt(), dt_in=_dt(),
                dt_out=_dt() * (c["nt_in"] - 1) / c["nt_out"] * 0.97, unit=-3.7e-4)


# ---------------------------------------------------------------------------
# run: one pass
# ---------------------------------------------------------------------------
def _shot(s):
    """The arrays of a new shot: quiet field, CPML memory and traces."""
    s["field"].fill(0)
    s["cpml"].reset()
    return s["g"].copy()


def run(s):
    family = s["c"]["family"]
    if family in ("fdtd", "map"):
        g = _shot(s)
        A.run_fdtd(s["d"], s["field"], g, s["cpml"], s["mask"], arith=s["arith"],
                   gf_map=s.get("gm"))
        out = dict(field=s["field"], p=g.rec[0], vn=g.vn_rec, psi_p=s["cpml"].mv,
                   psi_v=s["cpml"].mp)
        if family == "map":
            drive = s["gm"].i_src - 1
            out.update(p_src=g.src[0][:, drive], vn_src=g.vn_src[:, drive])
        return out
    if family == "gf":
        A.gf_solve_batch(s["reqs"])
        return [[r.p, r.vn] for r in s["reqs"]]
    if family == "serve":
        for r in s["reqs"]:
            s["server"].submit(r)
        s["server"].drain()
        return [[r.p, r.vn] for r in s["reqs"]]
    if family == "kh":
        if s["c"]["kind"] == "velocity":
            return A.kh_velocity(s["sp"], s["sn"], s["rp"], s["rn"], s["vn"], s["p"], s["c"]["dt"],
                                 s["sigma"], C0, s["aq"], s["af"], rho=RHO, out=s["out"])
        return A.kh_pressure(s["sp"], s["sn"], s["rp"], s["vn"], s["p"], s["c"]["dt"], s["sigma"],
                             C0, s["aq"], s["af"], out=s["out"])
    if family == "holo":
        g = _shot(s)
        A.run_fdtd_kh(s["d"], s["field"], g, s["cpml"], s["mask"], s["cols"], s["op"], s["on"],
                      s["rp"], s["sigma"], s["aq"], s["af"], out=s["out"])
        return dict(far=s["out"], field=s["field"], p=g.rec[0], vn=g.vn_rec, psi_p=s["cpml"].mv,
                    psi_v=s["cpml"].mp)
    return A.gf_postprocess(s["a"], s["t_in0"], s["dt_in"], s["c"]["nt_out"], 0.0, s["dt_out"],
                            unit=s["unit"], denoise=True)


# ---------------------------------------------------------------------------
# work: what one pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(nx, ny, nz, npml, masked):
    """One time step: the four channels read and written, half a byte of mask
    per cell, the CPML memory of both sides of each axis read and written."""
    cells = nx * ny * nz
    faces = ny * nz + nx * nz + nx * ny
    byt = 32.0 * cells + (0.5 * cells if masked else 0.0) + 16.0 * (2 * npml + 1) * faces
    return byt, 22.0 * cells + 8.0 * (2 * npml + 1) * faces


def _kh_work(ns, nr, nt, dt, sigma, rows=2):
    taps = math.floor(12 * sigma / dt) + 1
    return 4.0 * nt * (2 * ns + nr) + 48.0 * (ns + nr), 2.0 * rows * taps * ns * nr * float(nt)


def work(case):
    c = case
    family = c["family"]
    if family == "serve":
        b = f = 0.0
        for n, steps in _requests(c):
            sb, sf = _step_work(n, n, n, 10, True)
            b += steps * (sb + 8.0 * c["nrec"])
            f += steps * sf
        return dict(bytes=b, flops=f)
    if family == "kh":
        b, f = _kh_work(c["ns"], c["nr"], c["nt"], c["dt"], 6.6e-6)
        return dict(bytes=b, flops=f)
    if family == "post":
        return dict(bytes=4.0 * c["ncol"] * (c["nt_in"] + c["nt_out"]),
                    flops=c["ncol"] * (6.0 * c["nt_in"] + 30.0 * c["nt_out"]))
    sb, sf = _step_work(c["nx"], c["ny"], c["nz"], c["npml"], c.get("shape", "none") != "none")
    n = c.get("solves", 1) * c["steps"]
    b, f = n * sb, n * sf
    if family == "map":
        m = 4 if c["kind"] == "PVFromPV" else 2
        lags = sum(min(it, c["lags"]) for it in range(1, c["steps"]))
        b += 4.0 * m * c["lags"] * c["nsrc"] * c["nrec"]
        f += 2.0 * m * c["nsrc"] * c["nrec"] * lags
    if family == "holo":
        kb, kf = _kh_work(c["nout"], c["nr"], c["steps"], _dt(),
                          math.sqrt(math.log(2.0)) / (2 * math.pi * 20e3))
        b, f = b + kb + 4.0 * c["steps"] * 2 * (c["nin"] + c["nout"]), f + kf
    else:
        b += 8.0 * n * c["nrec"]
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# exact: the same results in Float64 (plain torch)
# ---------------------------------------------------------------------------
_F64 = dict(dtype=torch.float64, device="cuda")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float64)).cuda()


def _profiles(npml, dt):
    """CPML damping profiles: (a, b) of the grid and half-grid points, left and
    right."""
    alpha_max, thick = math.pi * PML_FC, DX * npml
    d0 = -3.0 * C0 * math.log(PML_R) / (2.0 * thick)

    def ab(dist):
        nd = dist / npml
        dd = d0 * nd * nd
        alpha = alpha_max * (1.0 - nd)
        b = np.exp(-(dd + alpha) * dt)
        return _t(dd * (b - 1.0) / (dd + alpha)), _t(b)

    on = np.linspace(0.0, npml - 1.0, npml)
    half = np.linspace(-0.5, npml - 0.5, npml + 1)
    half[0] = 0.0
    return dict(p=[ab(on[::-1]), ab(on)], v=[ab(half[::-1]), ab(half)])


def _open_cells(c, shape, kw):
    """Update mask [z][y][x] of P, Vx, Vy, Vz for a rigid scatterer, or None."""
    if shape == "none":
        return None
    ax = [_t(np.linspace(-(c[k] - 1) * DX / 2, (c[k] - 1) * DX / 2, c[k])) for k in
          ("nx", "ny", "nz")]
    x, y, z = (ax[i] - kw["center"][i] for i in range(3))
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    if shape == "sphere":
        p = x * x + y * y + z * z > kw["radius"] ** 2
    elif shape == "cube":
        h = kw["length"] / 2
        p = (x.abs() > h) | (y.abs() > h) | (z.abs() > h)
    else:
        s = kw["semi_axes"]
        p = (x / s[0]) ** 2 + (y / s[1]) ** 2 + (z / s[2]) ** 2 > 1.0
    m = [p]
    for axis in (2, 1, 0):
        o = torch.zeros_like(p)
        n = p.shape[axis]
        o.narrow(axis, 1, n - 1).copy_(p.narrow(axis, 1, n - 1) & p.narrow(axis, 0, n - 1))
        m.append(o)
    return m


class _Stencils:
    """interp_trilinear of one channel: record with weights W, inject with W^T;
    a transceiver's record includes the injections of those before it."""

    def __init__(self, c, points, chan):
        dims = (c["nx"], c["ny"], c["nz"])
        idx, frac = [], []
        for a in range(3):
            u = points[:, a] / DX + (dims[a] - 1) / 2 + (0.5 if chan == a + 1 else 0.0)
            i = np.ceil(u).astype(np.int64) - 1
            idx.append(i)
            frac.append(u - i)
        rows, cells, w = [], [], []
        for q in range(8):
            o = [q & 1, (q >> 1) & 1, q >> 2]
            cells.append(((idx[2] + o[2]) * dims[1] + idx[1] + o[1]) * dims[0] + idx[0] + o[0])
            w.append(np.prod([frac[a] if o[a] else 1 - frac[a] for a in range(3)], axis=0))
            rows.append(np.arange(len(points)))
        n = len(points)
        self.cells = torch.as_tensor(np.stack(cells, 1)).cuda()          # (ntx, 8)
        self.w = _t(np.stack(w, 1))
        uc, inv = torch.unique(self.cells, return_inverse=True)
        W = torch.sparse_coo_tensor(torch.stack([torch.arange(n, device="cuda").repeat_interleave(8),
                                                 inv.reshape(-1)]), self.w.reshape(-1),
                                    (n, uc.numel())).coalesce()
        S = torch.sparse.mm(W, W.t()).coalesce()
        r, k = S.indices()
        keep = r > k
        self.low = torch.sparse_coo_tensor(S.indices()[:, keep], S.values()[keep],
                                           (n, n)).coalesce().to_sparse_csr()

    def apply(self, f, s):
        flat = f.view(-1)
        rec = (flat[self.cells] * self.w).sum(1)
        if s is not None:
            rec = rec + (self.low @ s.unsqueeze(1)).squeeze(1)
            flat.index_add_(0, self.cells.reshape(-1), (self.w * s.unsqueeze(1)).reshape(-1))
        return rec


def _fdtd(c, points, dirs, src, vn_src, shape, kw, after=None):
    """nt steps from a quiet grid.  src: four (nt, ntx), vn_src (nt, ntx) or
    None, `after(it, rec_p, vn)` may change row it of both.  Returns the
    field, the p and v_n records and the CPML memory."""
    nx, ny, nz, n, nt = c["nx"], c["ny"], c["nz"], c["npml"], c["steps"]
    dt = _dt()
    fq, fv, rd = dt * RHO * C0 * C0, dt / RHO, 1.0 / DX
    P, VX, VY, VZ = (torch.zeros((nz, ny, nx), **_F64) for _ in range(4))
    V = {2: VX, 1: VY, 0: VZ}  # by torch axis
    mask = _open_cells(c, shape, kw)
    prof = _profiles(n, dt)
    stencils = [_Stencils(c, points, k) for k in range(4)]
    size = [nz, ny, nx]
    mp, mv = {}, {}
    for a in range(3):
        for side in range(2):
            s = list(size)
            s[a] = n
            mp[a, side] = torch.zeros(s, **_F64)
            s[a] = n + 1
            mv[a, side] = torch.zeros(s, **_F64)

    def along(v, a):
        return v.view([-1 if k == a else 1 for k in range(3)])

    def cpml(d, a, mem, ab, start, first, last, cut):
        """Memory of the cells first..last (global) of axis a; d starts at cell
        `start`, the other axes of the memory are cut like d."""
        l0 = first - cut["origin"]
        m = mem.narrow(a, l0, last - first + 1)
        for k in range(3):
            if k != a:
                m = m.narrow(k, cut["at"][k], d.shape[k])
        aa, bb = (along(q.narrow(0, l0, last - first + 1), a) for q in ab)
        part = d.narrow(a, first - start, last - first + 1)
        m.mul_(bb).add_(aa * part)
        part.add_(m)

    silent = [not bool(s.any()) and vn_src is None for s in src]
    rec_p, vn = (torch.zeros((nt, len(points)), **_F64) for _ in range(2))
    for it in range(nt):
        # rigid planes from the old field
        new_y = P[:nz - 1, ny - 1, :nx - 1] - fq * rd * (
            (VX[:nz - 1, ny - 1, 1:] - VX[:nz - 1, ny - 1, :-1]) - 2 * VY[:nz - 1, ny - 1, :-1] +
            (VZ[1:, ny - 1, :-1] - VZ[:-1, ny - 1, :-1]))
        new_z = P[nz - 1, :ny - 1, :nx - 1] - fq * rd * (
            (VX[nz - 1, :ny - 1, 1:] - VX[nz - 1, :ny - 1, :-1]) +
            (VY[nz - 1, 1:, :-1] - VY[nz - 1, :-1, :-1]) - 2 * VZ[nz - 1, :ny - 1, :-1])
        total = None
        for a in (2, 1, 0):
            d = V[a].diff(dim=a)
            for k in range(3):
                if k != a:
                    d = d.narrow(k, 0, size[k] - 1)
            d = d * rd
            if n > 1 or mask is not None:
                at = dict(at=[0, 0, 0])
                cpml(d, a, mp[a, 0], prof["p"][0], 0, 0, n - 1, dict(at, origin=0))
                cpml(d, a, mp[a, 1], prof["p"][1], 0, size[a] - n, size[a] - 2,
                     dict(at, origin=size[a] - n))
            total = d if total is None else total.add_(d)
        inner = P[:-1, :-1, :-1]
        if mask is None:
            inner.sub_(total, alpha=fq)
        else:
            inner.sub_(total.mul_(mask[0][:-1, :-1, :-1]), alpha=fq)
        del total, d
        P[:nz - 1, ny - 1, :nx - 1] = new_y
        P[nz - 1, :ny - 1, :nx - 1] = new_z
        r = [stencils[0].apply(P, None if silent[0] else src[0][it])]
        for a in (2, 1, 0):
            d = P.diff(dim=a) * rd
            at = dict(at=[0, 0, 0])
            cpml(d, a, mv[a, 0], prof["v"][0], 1, 1, n, dict(at, origin=0))
            cpml(d, a, mv[a, 1], prof["v"][1], 1, size[a] - n - 1, size[a] - 1,
                 dict(at, origin=size[a] - n - 1))
            if mask is not None:
                d.mul_(mask[3 - a].narrow(a, 1, size[a] - 1))
            V[a].narrow(a, 1, size[a] - 1).sub_(d, alpha=fv)
        for k, f in ((1, VX), (2, VY), (3, VZ)):
            r.append(stencils[k].apply(f, None if silent[k] else src[k][it]))
        rec_p[it] = r[0]
        vn[it] = r[1] * dirs[:, 1] + r[2] * dirs[:, 2] + r[3] * dirs[:, 3]
        if it + 1 < nt:
            if after is not None:
                after(it + 1, rec_p, vn)
            if vn_src is not None:
                for k in (1, 2, 3):
                    src[k][it + 1] += vn_src[it + 1] * dirs[:, k]
        VY[:, 0, :] = -VY[:, 1, :]
        VZ[0] = -VZ[1]
    julia = lambda q: q.permute(2, 1, 0)  # noqa: E731  (x, y, z) axis order
    field = torch.stack([julia(q) for q in (P, VX, VY, VZ)], dim=3)
    psi = [[torch.stack([julia(m[a, 0]), julia(m[a, 1])], dim=3) for a in (2, 1, 0)]
           for m in (mp, mv)]
    return field, rec_p, vn, psi


def _normcdf(x):
    return 0.5 * torch.special.erfc(-x / math.sqrt(2.0))


def _kh(sp, sn, rp, rn, in_q, in_f, dt, sigma, aq, af, velocity):
    """Windowed Gaussian KH sum: per surface point one product of the input's
    Toeplitz matrix with the targets' taps."""
    nt, ns = in_q.shape
    nr = rp.shape[0]
    hw = 6.0 * sigma / dt
    C = 1.0 / (math.sqrt(2 * math.pi) * sigma)
    out = torch.zeros((nt, nr), **_F64)
    cum = in_f.cumsum(0)
    for s in range(ns):
        v = rp - sp[s]
        dist = v.norm(dim=1)
        cs = (v @ sn[s]) / dist
        u = dist / (C0 * dt)
        lo = (u - hw).ceil().clamp(min=0).long()
        hi = (u + hw).floor().long()
        first = int(lo.min())
        width = int((hi - lo).max()) + 1
        nlag = int(hi.max()) - first + 2
        if first >= nt:
            continue
        k = torch.arange(width, device="cuda").unsqueeze(1) + lo  # (width, nr)
        tau = (k - u) * dt
        e = C * torch.exp(-tau * tau / (2 * sigma * sigma)) * (k <= hi)
        de = -tau / (sigma * sigma) * e
        i1, i2 = 1 / (4 * math.pi * dist), 1 / (4 * math.pi * dist ** 2)
        if velocity:
            cr = (v * rn).sum(1) / dist
            i3 = 1 / (4 * math.pi * dist ** 3)
            tq = aq * cr / RHO * (e * i2 + de / C0 * i1)
            ped = af * cr * cs / RHO * 2 * i3
            tf = (af * cr * cs / RHO * (e * 2 * i2 / C0 + de / (C0 * C0) * i1) +
                  ped * _normcdf(tau / sigma) * (k <= hi))
        else:
            tq = aq * de * i1
            tf = af * cs * (e * i2 + de / C0 * i1)
        parts, rows = [], []
        # taps past a pair's window are zero: they may land on any lag row
        row = (nlag - 1 - (k - first)).clamp(min=0)
        streams = [(in_q, tq, row), (in_f, tf, row)]
        if velocity:
            streams.append((cum, ped.unsqueeze(0), (nlag - 1 - (hi + 1 - first)).unsqueeze(0)))
        for x, taps, at in streams:
            m = torch.zeros((nlag, nr), **_F64)
            m.scatter_add_(0, at, taps)
            pad = torch.zeros(nt + nlag - 1 + first, **_F64)
            pad[first + nlag - 1:] = x[:, s]
            parts.append(m)
            rows.append(pad.unfold(0, nlag, 1)[:nt])
        out.addmm_(torch.cat(rows, dim=1), torch.cat(parts, dim=0))
    return out


def exact(case, seed):
    c, s = case, prepare(case, seed)
    family = c["family"]
    if family == "kh":
        return _kh(_t(s["sp"]), _t(s["sn"]), _t(s["rp"]), _t(s["rn"]), _t(s["vn"]), _t(s["p"]),
                   c["dt"], s["sigma"], s["aq"], s["af"], c["kind"] == "velocity").cpu().numpy()
    if family == "post":
        return _post(s)
    if family in ("gf", "serve"):
        out = []
        for r in s["reqs"]:
            q = dict(nx=r.dom.nx, ny=r.dom.ny, nz=r.dom.nz, npml=r.npml, steps=int(r.dom.nt))
            pts = np.vstack([r.src_point, r.rec_points])
            dirs = np.zeros((len(pts), 4))
            dirs[0], dirs[1:, 1:] = r.src_direction, r.rec_normals
            src = [torch.zeros((q["steps"], len(pts)), **_F64) for _ in range(4)]
            for k in range(4):
                src[k][:, 0] = _t(r.src_tf) * dirs[0, k]
            _, p, vn, _ = _fdtd(q, pts, _t(dirs), src, None, r.scatterer, r.scatterer_kw)
            out.append([p[:, 1:].cpu().numpy(), vn[:, 1:].cpu().numpy()])
            del p, vn, src
        return out
    g = s["g"]
    pts, dirs = _points(c, s), _t(g.direction.T)
    src = [_t(a) for a in g.src]
    vn_src, after = None, None
    if family == "holo":
        vn_src = _t(g.vn_src)
    if family == "map":
        vn_src = torch.zeros((c["steps"], len(pts)), **_F64)
        after = _extrapolation(c, s, src, vn_src)
    shape = "ellipsoid" if family == "holo" else c.get("shape", "none")
    field, p, vn, psi = _fdtd(c, pts, dirs, src, vn_src, shape, s["kw"], after)
    host = lambda q: q.cpu().numpy()  # noqa: E731
    out = dict(field=host(field), p=host(p), vn=host(vn), psi_p=[host(q) for q in psi[0]],
               psi_v=[host(q) for q in psi[1]])
    if family == "map":
        drive = torch.as_tensor(s["gm"].i_src - 1).cuda()
        out.update(p_src=host(src[0][:, drive]), vn_src=host(vn_src[:, drive]))
    if family == "holo":
        n = c["nout"]
        out["far"] = host(_kh(_t(s["op"]), _t(s["on"]), _t(s["rp"]), None, vn[:, :n], p[:, :n],
                              _dt(), s["sigma"], s["aq"], s["af"], False))
    return out


def _points(c, s):
    """The transceivers' positions, as prepare placed them."""
    inner = _half(c) - (c["npml"] + 3) * DX
    fib = lambda n, r: A.fibonacci_sphere(n, r)[0]  # noqa: E731
    if c["family"] == "fdtd":
        return np.vstack([s["src_point"], fib(c["nrec"], 0.8 * inner)])
    if c["family"] == "holo":
        return np.vstack([s["op"], fib(c["nin"], 0.6 * inner)])
    return np.vstack([s["src_point"], fib(c["nrec"], 0.8 * inner), fib(c["nsrc"], 0.6 * inner)])


def _extrapolation(c, s, src, vn_src):
    """extrapolate!: row it of the driven columns from the records so far."""
    gm, z0 = s["gm"], RHO * C0
    i_src = torch.as_tensor(gm.i_src - 1).cuda()
    i_rec = torch.as_tensor(gm.i_rec - 1).cuda()
    order = (1, 0, 2) if c["kind"] == "PVFromPin" else (2, 0, 1)  # -> (source, lag, receiver)
    T = [torch.as_tensor(t).cuda().double().permute(order).contiguous().flatten(1)
         for t in gm.tensors]
    nin = c["nrec"]

    def after(it, rec_p, vn):
        lags = min(it, c["lags"])
        p = rec_p[it - lags:it, i_rec].flip(0).reshape(-1)
        v = vn[it - lags:it, i_rec].flip(0).reshape(-1)
        if c["kind"] == "PVFromPV":
            pp, pv, vp, vv = (t[:, :lags * nin] for t in T)
            vn_src[it, i_src] = pv @ p + pp @ v
            src[0][it, i_src] = vv @ p + vp @ v
            return
        pin = (p - z0 * v) / 2
        a, b = (t[:, :lags * nin] @ pin for t in T)
        if c["kind"] == "PFromPin":
            a, b = (a + b) / z0, a - b
        vn_src[it, i_src] = a
        src[0][it, i_src] = b

    return after


def _post(s):
    a, c = s["a"], s["c"]
    n = a.shape[0]
    y = a.astype(np.float64)
    y[np.abs(y) < 1e-4 * a.max(axis=0).astype(np.float64)] = 0.0
    cf = np.zeros((n + 2, a.shape[1]))
    cf[1], cf[n] = y[0], y[n - 1]
    piv = np.zeros(n + 1)
    for i in range(2, n):
        rhs = 6.0 * y[i - 1]
        if i == 2:
            rhs = rhs - cf[1]
        if i == n - 1:
            rhs = rhs - cf[n]
        piv[i] = 1.0 / (4.0 - (piv[i - 1] if i > 2 else 0.0))
        cf[i] = (rhs - (cf[i - 1] if i > 2 else 0.0)) * piv[i]
    for i in range(n - 2, 1, -1):
        cf[i] -= piv[i] * cf[i + 1]
    cf[0], cf[n + 1] = 2 * cf[1] - cf[2], 2 * cf[n] - cf[n - 1]
    x = (np.arange(c["nt_out"]) * s["dt_out"] - s["t_in0"]) / s["dt_in"] + 1.0
    x = np.clip(x, 1.0, n)
    i = np.minimum(np.floor(x).astype(int), n - 1)
    d = (x - i)[:, None]
    e = 1.0 - d
    v = (cf[i - 1] * e ** 3 + cf[i] * (3 * d ** 3 - 6 * d ** 2 + 4) +
         cf[i + 1] * (-3 * d ** 3 + 3 * d ** 2 + 3 * d + 1) + cf[i + 2] * d ** 3) / 6.0
    return v * (s["dt_out"] / s["dt_in"]) / s["unit"]
