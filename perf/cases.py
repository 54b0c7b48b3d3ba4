"""The work whose speed is measured: calls, jobs, stages and products of the visibility path.

Each case is one use of the package through its public entry points, at a size
of this repository's own workloads (``matvis_b200.workloads``) or between them:

* ``call``: ``simulate_vis`` with host arrays in and a host array out;
* ``job``: a prepared and uploaded ``VisEngine`` run once over its times and
  frequencies, its visibilities left on the device (what a served job does);
* ``stages``: the plugin classes called one after another in the reference's
  loop order, one frequency, per time and source chunk;
* ``product``: the Hermitian product plugin on a caller's complex Z matrix.

``prepare`` builds the seeded inputs and the plan a program keeps, ``run`` is
one pass, ``work`` what a pass cannot do without and ``exact`` the FP64 result
of the same inputs from plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import matvis_b200 as mv
from matvis_b200 import workloads as wl
from matvis_b200.beamfits import BeamFits
from matvis_b200.engine import job_from_arrays

C_LIGHT = 299792458.0
#: Schwarzschild radius of the Sun (au), the apparent-place step's constant
SUN_RADIUS = 1.97412574336e-8

DEFAULTS = dict(
    kind="job", nant=64, nsrc=10000, nfreq=4, ntime=2, pol=True, layout="disc", sky="points", beam="grid", nbeam=1,
    precision=1, mode="fp16x3", pairs=0, rotation="lst", buffer=1.0, chunks=1,
)


def _case(**kw) -> dict:
    return dict(DEFAULTS, **kw)


def listed() -> list[dict]:
    return [
        # a first call of a new user, or one task of a small array's calibration: 16
        # antennas, 2,000 sources, double-precision output (the smallest workload here)
        _case(name="call-small", kind="call", nant=16, nsrc=2000, nfreq=2, ntime=4, pol=False, layout="square",
              beam="gauss", precision=2),
        # a script that simulates the 350-antenna array on an nside-64 map: every host
        # step of the call, the uploads and 63 MB of visibilities back
        _case(name="call-hera350", kind="call", nant=350, nsrc=49152, nfreq=8, ntime=2, layout="hera", sky="map",
              nbeam=4),
        # the served stream's median job: log-uniform antennas and sources, unpolarised
        _case(name="job-served-unpol", nant=90, nsrc=22361, nfreq=16, ntime=8, pol=False, beam="gauss"),
        # a small polarised served job: odd counts, few sources, launches count
        _case(name="job-served-small", nant=37, nsrc=5003, nfreq=7, ntime=5),
        # one time step of eight frequencies of the headline workload (HERA-350-like,
        # nside 128): what its job repeats 128 times
        _case(name="job-hera350", nant=350, nsrc=196608, nfreq=8, ntime=1, layout="hera", sky="map", nbeam=4),
        # the large-catalogue workload: 500,000 sources, source_buffer as the reference's default
        _case(name="job-hera350-500k", nant=350, nsrc=500000, nfreq=4, ntime=2, layout="hera", nbeam=4, buffer=0.55),
        # the more exact split for deep, high dynamic range work
        _case(name="job-tf32", nant=350, nsrc=49152, nfreq=3, ntime=1, layout="hera", sky="map", nbeam=4,
              mode="tf32x3"),
        # a sparse list of baselines on a million sources, one snapshot
        _case(name="job-pairs", nant=350, nsrc=1000000, nfreq=1, ntime=1, layout="hera", nbeam=4, pairs=5000),
        # a polarised sky: coherency fluxes rotated to the alt-az frame each time
        _case(name="job-polsky", nant=350, nsrc=49152, nfreq=4, ntime=2, layout="hera", sky="polmap", nbeam=4),
        # a measured beam that changes with frequency, apparent place refreshed each time
        _case(name="job-fits-erfa", nant=128, nsrc=30011, nfreq=6, ntime=3, beam="fits", rotation="erfa"),
        # the reference's own loop through the plugin classes, double precision, two chunks
        _case(name="stages", kind="stages", nant=61, nsrc=40000, nfreq=1, ntime=2, nbeam=4, precision=2, chunks=2),
        # the product plugin alone on a program's own Z (700 rows, complex64)
        _case(name="product-z", kind="product", nant=350, nsrc=24576, nfreq=1, ntime=1),
    ]


def _log_uniform(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c: dict) -> float:
    """Complex multiply-adds of the product, and of the panel, of one pass."""
    feeds = 2 if c["pol"] else 1
    rows, cols = c["nant"] * feeds, c["nsrc"] / 2 * feeds
    slices = c["nfreq"] * c["ntime"]
    per = (rows * (rows + 1) / 2 if not c["pairs"] else c["pairs"] * feeds * feeds * 12) + 60.0 * rows
    return slices * per * cols


def _panel_bytes(c: dict) -> float:
    feeds = 2 if c["pol"] else 1
    rows = -(-c["nant"] * feeds // 128) * 128
    per = {"tf32x3": 16, "bf16x6": 12}.get(c["mode"], 8)
    return min(c["nfreq"], 8) * rows * c["nsrc"] * c["buffer"] / c["chunks"] * feeds * per


def draw(rng) -> dict:
    top = max(_cost(c) for c in listed())
    kind = rng.choice(["call", "job", "job", "job", "job", "stages", "product"])
    c = _case(kind=kind)
    c["nant"] = _log_uniform(rng, 16, 512)
    c["nsrc"] = _log_uniform(rng, 1000, 500000)
    c["pol"] = rng.random() < 0.6
    c["layout"] = rng.choice(["disc", "disc", "square"])
    c["nfreq"] = rng.randint(1, 32)
    c["ntime"] = rng.randint(1, 16)
    c["mode"] = rng.choice(["fp16x3"] * 4 + ["tf32x3", "bf16x6"])
    c["nbeam"] = rng.choice([1, 1, 4])
    if c["pol"]:
        c["beam"] = rng.choice(["grid", "grid", "grid", "fits"])
        if kind in ("call", "job") and c["beam"] == "grid" and rng.random() < 0.2:
            c["sky"] = "polpoints"
    else:
        c["beam"] = rng.choice(["gauss", "gauss", "grid"])
    if c["beam"] == "fits":
        c["nbeam"] = 1
    if kind in ("call", "job"):
        if rng.random() < 0.2:
            c["rotation"] = "erfa"
        if rng.random() < 0.2:
            c["chunks"] = rng.choice([2, 3])
        if rng.random() < 0.2:
            c["pairs"] = min(_log_uniform(rng, 50, 5000), c["nant"] * (c["nant"] - 1) // 2)
            c["sky"] = "points"
        if kind == "call":
            c["nsrc"] = min(c["nsrc"], 100000)
    else:
        c["nfreq"], c["ntime"] = 1, (1 if kind == "product" else rng.randint(1, 3))
        c["mode"] = "fp16x3"
        c["beam"] = "grid" if c["pol"] else rng.choice(["gauss", "grid"])
        c["nbeam"] = 1 if c["beam"] == "gauss" else rng.choice([1, 4])
        c["precision"] = rng.choice([1, 2])
        c["chunks"] = rng.choice([1, 2]) if kind == "stages" else 1
        c["nsrc"] = min(c["nsrc"], 100000)
    while _cost(c) > top or _panel_bytes(c) > 24e9 or c["nfreq"] * c["ntime"] * c["nant"] ** 2 > 4e7:
        if c["ntime"] > 1:
            c["ntime"] = (c["ntime"] + 1) // 2
        elif c["nfreq"] > 1:
            c["nfreq"] = (c["nfreq"] + 1) // 2
        else:
            c["nsrc"] = max(1000, int(c["nsrc"] * 0.6))
    return c


# ----------------------------------------------------------------- inputs
def _inputs(c: dict, seed: int) -> dict:
    """Host inputs of a simulation, from the seed alone."""
    rng = np.random.default_rng(97003 + seed)
    nant, nf = c["nant"], c["nfreq"]
    if c["layout"] == "hera":
        antpos = wl.hera350(rng)[:nant]
    elif c["layout"] == "square":
        antpos = np.column_stack([rng.uniform(-50, 50, nant), rng.uniform(-50, 50, nant), np.zeros(nant)])
    else:
        antpos = wl.uniform_disc(rng, nant, 300.0)
        antpos[:, 2] = rng.normal(0.0, 0.3, nant)
    if c["sky"] in ("map", "polmap"):
        ra, dec = wl.healpix_ring_centres(int(round(math.sqrt(c["nsrc"] / 12))))
        flux0 = rng.lognormal(0.0, 1.0, len(ra))
    else:
        ra, dec = wl.isotropic(rng, c["nsrc"])
        flux0 = wl.powerlaw_flux(rng, c["nsrc"])
    freqs = np.linspace(100e6, 200e6, nf + 2)[1:-1] if c["beam"] == "fits" else np.sort(rng.uniform(100e6, 200e6, nf))
    alpha = rng.normal(-0.8, 0.2, len(ra))
    fluxes = flux0[:, None] * (freqs[None, :] / 150e6) ** alpha[:, None]
    if c["sky"].startswith("pol"):
        fluxes = wl.polarised_sky(dict(fluxes=fluxes), seed=seed)
    lsts = rng.uniform(0, 2 * np.pi) + np.arange(c["ntime"]) * 2 * np.pi * 600 / wl.SIDEREAL_DAY_S
    if c["beam"] == "gauss":
        beams = [mv.GaussianBeam(sigma=float(s)) for s in rng.uniform(0.15, 0.3, c["nbeam"])]
    else:
        beams = wl.dipole_beams(rng, c["nbeam"])
    if c["beam"] == "fits":
        g = beams[0]
        data = np.stack([g.data, 0.9 * g.data], axis=2).astype(np.complex128)
        beams = [BeamFits("efield", data, g.az, g.za, np.array([100e6, 200e6]), ["x", "y"])]
    beam_idx = rng.integers(0, c["nbeam"], nant) if c["nbeam"] > 1 else None
    pairs = None
    if c["pairs"]:
        iu, ju = np.triu_indices(nant, k=1)
        pick = rng.choice(len(iu), size=c["pairs"], replace=False)
        pairs = np.column_stack([iu[pick], ju[pick]])
    astrom = wl.synthetic_astrom(lsts, wl.HERA_LAT, seed=seed) if c["rotation"] == "erfa" else None
    return dict(antpos=antpos, ra=ra, dec=dec, fluxes=fluxes, freqs=freqs, lsts=lsts, beams=beams, beam_idx=beam_idx,
                pairs=pairs, astrom=astrom)


def _product_z(c: dict, seed: int) -> torch.Tensor:
    """Z as a program has it: lognormal source amplitudes times a random phase per antenna row."""
    feeds = 2 if c["pol"] else 1
    g = torch.Generator(device="cuda").manual_seed(4201 + seed)
    m, k = c["nant"] * feeds, c["nsrc"] * feeds
    amp = torch.exp(0.5 * torch.randn(k, generator=g, device="cuda", dtype=torch.float64))
    ph = 2 * math.pi * torch.rand((m, k), generator=g, device="cuda", dtype=torch.float32)
    z = torch.polar(torch.ones_like(ph), ph).mul_(amp.to(torch.float32))
    return z if c["precision"] == 1 else z.to(torch.complex128)


def prepare(case: dict, seed: int):
    c = dict(DEFAULTS, **case)
    kind = c["kind"]
    if kind == "product":
        feeds = 2 if c["pol"] else 1
        mp = mv.B200MatMul(1, feeds, c["nant"], None, precision=c["precision"], gemm_mode=c["mode"])
        mp.setup()
        return dict(kind=kind, mp=mp, z=_product_z(c, seed))
    i = _inputs(c, seed)
    if kind == "call":
        kw = dict(polarized=c["pol"], precision=c["precision"], beam_idx=i["beam_idx"], antpairs=i["pairs"],
                  gemm_mode=c["mode"], min_chunks=c["chunks"], source_buffer=c["buffer"],
                  matprod_method="VectorDot" if c["pairs"] else "MatMul")
        if i["astrom"] is not None:
            kw.update(coord_method="CoordinateRotationERFA", coord_method_params={"astrom": i["astrom"]})
        ants = {k: tuple(p) for k, p in enumerate(i["antpos"])}
        return dict(kind=kind, args=(ants, i["fluxes"], i["ra"], i["dec"], i["freqs"], i["lsts"], i["beams"],
                                     wl.HERA_LAT), kw=kw)
    if kind == "job":
        spec = job_from_arrays(ants=i["antpos"], fluxes=i["fluxes"], ra=i["ra"], dec=i["dec"], freqs=i["freqs"],
                               lsts=i["lsts"], latitude=wl.HERA_LAT, beams=i["beams"], beam_idx=i["beam_idx"],
                               polarized=c["pol"], precision=c["precision"], antpairs=i["pairs"],
                               gemm_mode=c["mode"], matprod="VectorDot" if c["pairs"] else "MatMul",
                               source_buffer=c["buffer"], nchunks=c["chunks"], astrom=i["astrom"])
        eng = mv.VisEngine(spec)
        eng.upload()
        return dict(kind=kind, eng=eng)
    nant, feeds = c["nant"], 2 if c["pol"] else 1
    coords = mv.CoordinateRotationLST(flux=np.sqrt(0.5 * i["fluxes"][:, 0]), times=i["lsts"],
                                      telescope_loc=wl.HERA_LAT, skycoords=(i["ra"], i["dec"]),
                                      chunk_size=-(-len(i["ra"]) // c["chunks"]), source_buffer=1.0,
                                      precision=c["precision"])
    beam = mv.B200BeamInterpolator(beam_list=i["beams"], beam_idx=i["beam_idx"], polarized=c["pol"], nant=nant,
                                   freq=float(i["freqs"][0]), nsrc=coords.nsrc_alloc, precision=c["precision"])
    tau = mv.TauCalculator(antpos=i["antpos"], freq=float(i["freqs"][0]), nsrc=coords.nsrc_alloc,
                           precision=c["precision"])
    zc = mv.ZMatrixCalc(nant=nant, nfeed=feeds, nax=feeds, nsrc=coords.nsrc_alloc)
    mp = mv.B200MatMul(nchunks=c["chunks"], nfeed=feeds, nant=nant, antpairs=None, precision=c["precision"])
    for o in (coords, beam, tau, zc, mp):
        o.setup()
    return dict(kind=kind, coords=coords, beam=beam, tau=tau, zc=zc, mp=mp, nt=len(i["lsts"]), chunks=c["chunks"],
                feeds=feeds)


def run(state):
    kind = state["kind"]
    if kind == "call":
        return mv.simulate_vis(*state["args"], **state["kw"])
    if kind == "job":
        return state["eng"].run()
    mp = state["mp"]
    if kind == "product":
        return mp(state["z"], 0)
    coords, beam = state["coords"], state["beam"]
    vis = np.zeros((state["nt"], mp.npairs, state["feeds"], state["feeds"]),
                   dtype=np.complex64 if mp.precision == 1 else np.complex128)
    counts = []
    for t in range(state["nt"]):
        coords.rotate(t)
        for c in range(state["chunks"]):
            crd, flux, n = coords.select_chunk(c, t)
            a = beam(crd[0], crd[1], check=t == 0 and c == 0)
            ext = state["tau"](crd)
            mp(state["zc"](flux, a, ext, beam.beam_idx), c)
            counts.append(n)
        mp.sum_chunks(vis[t])
    return dict(vis=vis, counts=np.array(counts), topo=coords.all_coords_topo, flux=flux)


def work(case: dict) -> dict:
    """One pass: sky, beams (or Z) read once, visibilities written once; the upper
    triangle (or the listed pairs) of V = conj(Z) Z^T once in complex arithmetic."""
    c = dict(DEFAULTS, **case)
    feeds = 2 if c["pol"] else 1
    rows, nfreq, ntime = c["nant"] * feeds, c["nfreq"], c["ntime"]
    npairs = c["pairs"] or c["nant"] ** 2
    out = nfreq * ntime * npairs * feeds * feeds * 8 * c["precision"]
    if c["kind"] == "product":
        k = c["nsrc"] * feeds
        return {"bytes": 8.0 * c["precision"] * rows * k + out, "flops": 4.0 * rows * (rows + 1) * k}
    k = c["nsrc"] / 2 * feeds  # half the sky is up
    per = 8.0 * c["pairs"] * feeds * feeds if c["pairs"] else 4.0 * rows * (rows + 1)
    grid = 0 if c["beam"] == "gauss" else c["nbeam"] * feeds * feeds * 91 * 361 * 8 * (2 if c["beam"] == "fits" else 1)
    sky = c["nsrc"] * (24 + nfreq * (16 if c["sky"].startswith("pol") else 4))
    return {"bytes": float(sky + grid + out), "flops": nfreq * ntime * per * k}


# ------------------------------------------------------------ FP64 restatement
def _rotation(lst: float, lat: float) -> np.ndarray:
    return np.array([[-np.sin(lst), np.cos(lst), 0.0],
                     [-np.sin(lat) * np.cos(lst), -np.sin(lat) * np.sin(lst), np.cos(lat)],
                     [np.cos(lat) * np.cos(lst), np.cos(lat) * np.sin(lst), np.sin(lat)]])


def _apparent(p: torch.Tensor, a: dict) -> torch.Tensor:
    """Light deflection, aberration, bias-precession-nutation of (3, N) directions."""
    dev = p.device
    e = torch.tensor(np.asarray(a["eh"]), dtype=torch.float64, device=dev)[:, None].expand_as(p)
    v = torch.tensor(np.asarray(a["v"]), dtype=torch.float64, device=dev)[:, None]
    q = (p * (p + e)).sum(0).clamp(min=1e-6)
    p = p + SUN_RADIUS / a["em"] / q * torch.linalg.cross(p, torch.linalg.cross(e, p, dim=0), dim=0)
    pdv = (v * p).sum(0)
    w1, w2 = 1.0 + pdv / (1.0 + a["bm1"]), SUN_RADIUS / a["em"]
    p = p * a["bm1"]
    p = p + v * w1 + w2 * (v - pdv * p)
    p = p / p.norm(dim=0)
    return torch.tensor(np.asarray(a["bpn"]).reshape(3, 3), dtype=torch.float64, device=dev) @ p


def _earth(a: dict) -> np.ndarray:
    ce, se = math.cos(a["eral"]), math.sin(a["eral"])
    sx, cx, sy, cy = math.sin(a["xpl"]), math.cos(a["xpl"]), math.sin(a["ypl"]), math.cos(a["ypl"])
    pole = np.array([[cx, 0, sx], [sx * sy, cy, -cx * sy], [-sx * cy, sy, cx * cy]])
    site = np.array([[0, 1, 0], [-a["sphi"], 0, a["cphi"]], [a["cphi"], 0, a["sphi"]]])
    return site.dot(pole.dot(np.array([[ce, se, 0], [-se, ce, 0], [0, 0, 1]])))


def _turn(r, p: torch.Tensor) -> torch.Tensor:
    """r @ p, each row as (r0 x + r1 y) + r2 z, so that the horizon cut is the framework's."""
    r = np.asarray(r, dtype=np.float64)
    return torch.stack([(float(r[k, 0]) * p[0] + float(r[k, 1]) * p[1]) + float(r[k, 2]) * p[2] for k in range(3)])


def _zenith(e, n):
    lsq = n * n + e * e
    zeta = torch.where(lsq < 1, (1 - lsq).clamp(min=0).sqrt(), torch.zeros_like(lsq))
    return 0.5 * math.pi - torch.asin(zeta)


def _beam_values(c, i, freq, crd) -> torch.Tensor:
    """(nbeam, feed, axis, n) complex128."""
    e, n = crd[0], crd[1]
    za = _zenith(e, n)
    az = torch.remainder(0.5 * math.pi - torch.atan2(e, n), 2 * math.pi)
    out = []
    for b in i["beams"]:
        if c["beam"] == "gauss":
            out.append(torch.exp(-za * za / (2 * b.sigma**2)).to(torch.complex128)[None, None])
            continue
        g = torch.as_tensor(np.asarray(b.data), device=crd.device)
        if c["beam"] == "fits":
            w = (freq - 100e6) / 100e6
            g = (1 - w) * g[:, :, 0] + w * g[:, :, 1]
        g = g.to(torch.complex128)
        if not c["pol"]:
            g = (g[:, :1].abs() ** 2).sum(0, keepdim=True).to(torch.complex128)
        row, col = za / float(b.za[1] - b.za[0]), (az - float(np.min(b.az))) / float(b.az[1] - b.az[0])
        nza, naz = g.shape[-2:]
        inside = (row >= 0) & (row <= nza - 1) & (col >= 0) & (col <= naz - 1)
        r0, c0 = row.floor().clamp(0, nza - 1).long(), col.floor().clamp(0, naz - 1).long()
        r1, c1 = (r0 + 1).clamp(max=nza - 1), (c0 + 1).clamp(max=naz - 1)
        fr, fc = row - r0, col - c0
        v = (1 - fr) * ((1 - fc) * g[..., r0, c0] + fc * g[..., r0, c1])
        v = v + fr * ((1 - fc) * g[..., r1, c0] + fc * g[..., r1, c1])
        v = torch.where(inside, v, torch.zeros_like(v))
        if not c["pol"]:
            v = v.real.sqrt().to(torch.complex128)
        out.append(v.transpose(0, 1))
    return torch.stack(out)


def _frame_turn(ra, dec, crd, rigid) -> tuple[torch.Tensor, torch.Tensor]:
    """cos X, sin X of the coherency's turn from the (ra, dec) to the (alt, az) basis."""
    dev = crd.device
    r = torch.tensor(np.array([[0.0, 1, 0], [1, 0, 0], [0, 0, 1]]) @ np.asarray(rigid), dtype=torch.float64, device=dev)
    alt = 0.5 * math.pi - _zenith(crd[0], crd[1])
    az = torch.remainder(torch.atan2(crd[0], crd[1]), 2 * math.pi)

    def unit(lon, lat):
        return torch.stack([lat.cos() * lon.cos(), lat.cos() * lon.sin(), lat.sin()])

    def theta_hat(theta, phi):
        return torch.stack([phi.cos() * theta.cos(), phi.sin() * theta.cos(), -theta.sin()])

    r1, to = r @ unit(ra, dec), unit(az, alt)
    axis = torch.linalg.cross(r1, to, dim=0)
    sp, cp = axis.norm(dim=0), (r1 * to).sum(0)
    psi = torch.atan2(sp, cp)
    u = torch.where(sp > 0, axis / torch.where(sp > 0, sp, torch.ones_like(sp)), torch.zeros_like(axis))
    back = theta_hat(math.pi / 2 - alt, az)
    # the transpose of the turn by psi about u, applied to the alt-az basis vector
    back = back - psi.sin() * torch.linalg.cross(u, back, dim=0) \
        + (1 - psi.cos()) * torch.linalg.cross(u, torch.linalg.cross(u, back, dim=0), dim=0)
    back = r.T @ back
    phi_hat = torch.stack([-ra.sin(), ra.cos(), torch.zeros_like(ra)])
    return (back * theta_hat(math.pi / 2 - dec, ra)).sum(0), (back * phi_hat).sum(0)


def _exact_vis(c: dict, i: dict):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    ra, dec = i["ra"], i["dec"]
    eci = torch.tensor(np.asarray([np.cos(ra) * np.cos(dec), np.cos(dec) * np.sin(ra), np.sin(dec)]), **f64)
    ant = torch.tensor(i["antpos"], **f64)
    flux = torch.tensor(i["fluxes"], device=dev)
    nant, feeds = c["nant"], 2 if c["pol"] else 1
    idx = torch.zeros(nant, dtype=torch.long, device=dev) if i["beam_idx"] is None else torch.tensor(i["beam_idx"], device=dev)
    npairs = c["pairs"] or nant * nant
    vis = torch.zeros((len(i["freqs"]), len(i["lsts"]), npairs, feeds, feeds), dtype=torch.complex128, device=dev)
    ups, topo = [], None
    for t, lst in enumerate(i["lsts"]):
        if i["astrom"] is not None:
            a = i["astrom"][t]
            rigid, topo = _earth(a) @ np.asarray(a["bpn"]).reshape(3, 3), _turn(_earth(a), _apparent(eci, a))
        else:
            rigid = _rotation(lst, wl.HERA_LAT)
            topo = _turn(rigid, eci)
        up = torch.nonzero(topo[2] > 0)[:, 0]
        ups.append(up)
        for s0 in range(0, len(up), 1 << 16):
            sel = up[s0:s0 + (1 << 16)]
            crd = topo[:, sel]
            beam = None
            if c["sky"].startswith("pol"):
                cx, sx = _frame_turn(torch.tensor(ra, **f64)[sel], torch.tensor(dec, **f64)[sel], crd, rigid)
                turn = torch.stack([torch.stack([cx, sx]), torch.stack([-sx, cx])]).to(torch.complex128)
            for f, freq in enumerate(i["freqs"]):
                if beam is None or c["beam"] == "fits":
                    beam = _beam_values(c, i, freq, crd)
                path = (ant @ crd) * (freq / C_LIGHT)
                ext = torch.polar(torch.ones_like(path), 2 * math.pi * (path - path.round()))
                y = ext[:, None, None, :] * beam[idx]  # (A, F, X, n)
                if c["sky"].startswith("pol"):
                    coh = torch.einsum("ban,nbc,cdn->nad", turn, flux[sel, f], turn)
                    w = torch.einsum("apxn,nxy->apyn", y, coh)
                else:
                    w = y * (0.5 * flux[sel, f])
                w, y = w.reshape(nant * feeds, -1), y.reshape(nant * feeds, -1)
                g = (y.conj() @ w.T).reshape(nant, feeds, nant, feeds)  # [i, q, j, p]
                g = g.permute(0, 2, 3, 1)
                if i["pairs"] is None:
                    vis[f, t] += g.reshape(nant * nant, feeds, feeds)
                else:
                    pr = torch.as_tensor(i["pairs"], device=dev)
                    vis[f, t] += g[pr[:, 0], pr[:, 1]]
    return vis, topo, ups


def exact(case: dict, seed: int):
    c = dict(DEFAULTS, **case)
    feeds = 2 if c["pol"] else 1
    if c["kind"] == "product":
        z = _product_z(c, seed).to(torch.complex128)
        g = torch.zeros((z.shape[0],) * 2, dtype=torch.complex128, device=z.device)
        for k in range(0, z.shape[1], 1 << 16):
            g += z[:, k:k + (1 << 16)].conj() @ z[:, k:k + (1 << 16)].T
        return g.reshape(c["nant"], feeds, c["nant"], feeds).permute(0, 2, 3, 1).reshape(-1, feeds, feeds).contiguous()
    i = _inputs(c, seed)
    vis, topo, ups = _exact_vis(c, i)
    if c["kind"] == "stages":
        size = -(-len(i["ra"]) // c["chunks"])
        last = ups[-1][ups[-1] >= (c["chunks"] - 1) * size]
        flux = torch.zeros(size, dtype=torch.float64, device=vis.device)
        flux[:len(last)] = torch.tensor(np.sqrt(0.5 * i["fluxes"][:, 0]), device=vis.device)[last]
        return dict(vis=vis[0].cpu().numpy(), counts=None, topo=topo, flux=flux)
    if c["pol"] or c["kind"] == "job":
        return vis.cpu().numpy() if c["kind"] == "call" else vis
    return vis[..., 0, 0].cpu().numpy()
