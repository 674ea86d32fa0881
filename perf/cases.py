"""Timed cases of the framework's work, through its public entry points.

A simulation step is a particle half (coordinate push, current and charge
deposit, gather, momentum push) and a field half (Fourier-Bessel transforms,
coupling operators, Poisson correction, PSATD update), in two precisions:

  * the FP64 drop-in of the reference's kernel module (``fimera``, called by
    ``ChimeraRun``), and
  * the split-precision form (``SplitRun``; its layers through the C ABI of
    include/chimera_gb300.h).

The cases are those halves over the range of grids and particle counts of the
repository's workloads (256 x 32 to 4096 x 512, 1 to 3 stored modes, up to 50
million electrons), for the plain and the envelope solver, and three whole
steps.  A pass is one step (or one half of it) on state that stays on the GPU;
fields and particles go on from where the pass before left them, as in a run.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from chimera_gb300 import ChimeraRun, Solver, Specie, _lib, fimera
from chimera_gb300.messages import msg
from chimera_gb300.solvers import spectral_operators
from chimera_gb300.split import SplitRun

msg.quiet = True

DX, DR = 0.04, 0.4       # cells of the laser-wakefield set-ups (wavelengths)
KX0_FEL = 2 * math.pi * 2.0e4  # carrier wavenumber of the FEL set-ups (per undulator period)
DX_FEL = 200e-4 / 2.8    # FEL box length (undulator periods), over nx cells
DR_FEL = 1000e-4 / 2.8   # FEL grid radius, over nkr cells
GAMMA_FEL = 200.0
VB_FEL = math.sqrt(1 - 1.5 / GAMMA_FEL ** 2)  # the beam's velocity in an undulator of strength 1


def listed():
    return [
        # the smallest call: a free-electron-laser step on a small envelope
        # grid, its kernels replayed from a CUDA graph (long undulator runs
        # take thousands of these; launches and gaps count)
        dict(name="fel_step_256x32", kind="fel_step", nx=256, nkr=32, modes=3, parts=130000),
        # the laser-wakefield demo's step in the split form: moving window with
        # absorption and injected plasma, small grid
        dict(name="lwfa_step_512x64", kind="lwfa_step", split=True, nx=512, nkr=64, modes=2,
             ppc_x=2, ppc_r=2, ppc_t=4),
        # the same demo step in the FP64 drop-in, on a grid without powers of two
        dict(name="lwfa_step64_600x50", kind="lwfa_step", split=False, nx=600, nkr=50, modes=2,
             ppc_x=2, ppc_r=2, ppc_t=4),
        # the field half of the split step at the largest laser-wakefield grid
        dict(name="fields_4096x512x3", kind="fields", nx=4096, nkr=512, modes=3),
        # and on an ordinary one, ragged in both directions
        dict(name="fields_1500x100x2", kind="fields", nx=1500, nkr=100, modes=2),
        # the particle half of the split step: 50 million electrons, 3 modes
        dict(name="parts_4096x512x3_50M", kind="parts", nx=4096, nkr=512, modes=3, ppc_x=2, ppc_r=2,
             ppc_t=12),
        # and an ordinary run's 4 million in 2 modes
        dict(name="parts_1024x128x2_4M", kind="parts", nx=1024, nkr=128, modes=2, ppc_x=2, ppc_r=4,
             ppc_t=8),
        # the field half of the FP64 drop-in: the small demo grid ...
        dict(name="fields64_512x64x2", kind="fields64", env=False, nx=512, nkr=64, modes=2),
        # ... and the 2048 x 256 set-up
        dict(name="fields64_2048x256x2", kind="fields64", env=False, nx=2048, nkr=256, modes=2),
        # the envelope solver's field half in FP64 at the FEL grid
        dict(name="fields64_env_2048x128", kind="fields64", env=True, nx=2048, nkr=128, modes=3),
        # the particle half of the FP64 drop-in, 4 million electrons
        dict(name="parts64_2048x128x2_4M", kind="parts64", env=False, nx=2048, nkr=128, modes=2,
             ppc_x=2, ppc_r=2, ppc_t=4),
        # an FEL beam's particle half in FP64: envelope deposit and gather, undulator
        dict(name="parts64_env_1M", kind="parts64", env=True, nx=2048, nkr=128, modes=3,
             parts=1000003),
    ]


def _smooth(n):
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    """One more case: the kinds above, grids spread over their logarithm."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid_x(lo, hi):  # an even cell count with small prime factors
        n = 2 * log_int(lo // 2, hi // 2)
        while not _smooth(n):
            n += 2
        return min(n, hi)

    kind = rng.choice(["fel_step", "lwfa_step", "fields", "fields", "parts", "parts", "fields64",
                       "fields64", "fields64", "parts64", "parts64"])
    if kind == "fel_step":
        return dict(kind=kind, nx=grid_x(256, 512), nkr=log_int(24, 64), modes=3,
                    parts=log_int(50000, 1000000))
    if kind == "lwfa_step":
        return dict(kind=kind, split=rng.random() < 0.5, nx=grid_x(256, 640), nkr=log_int(32, 80),
                    modes=rng.choice([1, 2, 3]), ppc_x=2, ppc_r=2, ppc_t=rng.choice([2, 4, 6]))
    if kind == "fields":
        return dict(kind=kind, nx=grid_x(256, 4096), nkr=log_int(32, 512),
                    modes=rng.choice([1, 2, 3]))
    if kind == "parts":
        return dict(kind=kind, nx=grid_x(256, 4096), nkr=log_int(32, 256),
                    modes=rng.choice([1, 2, 3]), ppc_x=2, ppc_r=2, ppc_t=rng.choice([2, 3, 4, 6, 8]))
    if kind == "fields64":
        env = rng.random() < 0.3
        return dict(kind=kind, env=env, nx=grid_x(256, 2048), nkr=log_int(32, 256),
                    modes=3 if env else rng.choice([1, 2, 3]))
    if rng.random() < 0.3:
        return dict(kind=kind, env=True, nx=grid_x(256, 2048), nkr=log_int(32, 128), modes=3,
                    parts=log_int(50000, 2000000))
    return dict(kind=kind, env=False, nx=grid_x(256, 2048), nkr=log_int(32, 128),
                modes=rng.choice([1, 2, 3]), ppc_x=2, ppc_r=2, ppc_t=rng.choice([2, 3, 4]))


# ---------------------------------------------------------------------------
# operators and helpers
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _operators(nkr, modes, env):
    """The DHT and coupling matrices a Solver builds for an r grid, as FP64
    numpy (K, N, modes), and the radial wavenumbers (nkr, modes).  They do not
    depend on the inputs, so a program builds them once per grid."""
    dr = DR_FEL / nkr if env else DR
    nko = (modes - 1) // 2 if env else modes - 1
    nr = nkr + 1
    rgrid = dr * (np.arange(nr) - 0.5)
    A = dict(Nx=2, Nkr=nkr, Nko=nko, lengthR=rgrid[-1] + dr, kx=np.array([0.0, 1.0]), RgridFull=rgrid)
    if env:
        A["KxShift"] = 1.0
    _, _, Dp, Dm, _, _, _, _, _ = spectral_operators(A, 1)
    In, Out, _, _, _, _, kr_g, _, _ = spectral_operators(A, 0)
    dx = DX
    vgrid = (rgrid > 0.0) / (2 * np.pi * dx * dr * rgrid)
    cur = In * vgrid[None, 1:, None]
    f = lambda a: np.asfortranarray(np.swapaxes(a, 0, 1))  # noqa: E731
    return dict(In=f(cur), Out=f(Out), Dp=f(Dp), Dm=f(Dm), kr=np.ascontiguousarray(kr_g[0]), dr=dr,
                rgrid=rgrid)


def _dims(case):
    return case["nx"], case["nkr"] + 1, case["nkr"], case["modes"]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _noise(shape, gen, scale, dtype=torch.complex128):
    """Complex Gaussian noise on a Fortran-ordered grid."""
    t = fimera.fortran_empty(shape, dtype)
    flat = torch.view_as_real(t.permute(*reversed(range(t.dim()))))
    flat.normal_(0.0, scale, generator=gen)
    return t


def _col(a, dtype=torch.float64):
    """numpy -> Fortran-ordered CUDA tensor."""
    a = np.asfortranarray(a)
    return torch.from_numpy(a).cuda().to(dtype)


def _fortran(t, dtype=None):
    out = fimera.fortran_empty(tuple(t.shape), dtype or t.dtype, t.device)
    out.copy_(t)
    return out


def _clone(t):
    return _fortran(t)


def _spectrum(case):
    """kx, kr, w and the solver's real spectral factors on the GPU (FP64)."""
    nx, nr, nkr, nm = _dims(case)
    env = bool(case.get("env"))
    o = _operators(nkr, nm, env)
    dx = DX_FEL / nx if env else DX
    kenv = torch.from_numpy(2 * np.pi * np.fft.fftfreq(nx, dx)).cuda()
    kx = kenv + KX0_FEL if env else kenv
    kr = torch.from_numpy(o["kr"]).cuda()
    w = torch.sqrt(kx[:, None, None] ** 2 + kr[None] ** 2)
    filt = torch.cos(0.5 * dx * kenv)[:, None, None] ** 2 * torch.cos(0.5 * o["dr"] * kr)[None] ** 2
    return o, dx, kenv, kx, w, (2 * np.pi) ** 2 / nx * filt


def _psatd(w, dt, kx=None):
    """The update's coefficients: five real ones with space charge, or (kx
    given) the envelope solver's three complex ones."""
    c, s = torch.cos(dt * w), torch.sin(dt * w)
    if kx is None:
        CE = [c, s / w, -s / w, (dt * w * c - s) / w ** 3 / dt, (s - dt * w) / w ** 3 / dt]
        CG = [-w * s, c, 1 - c, (1 - c - dt * w * s) / w ** 2 / dt, (c - 1) / w ** 2 / dt]
    else:
        k = 0.9999 * kx[:, None, None]
        den = w ** 2 - k ** 2
        ph, e = torch.exp(-0.5j * k * dt), torch.exp(1j * k * dt)
        CE = [c, s / w, ph * 1j * k / den * (1.0 - e * (w / (1j * k) * s + c))]
        CG = [-w * s, c, ph * w ** 2 / den * (1.0 + e * (1j * k / w * s - c))]
        CE, CG = ([a.to(torch.complex128) for a in v] for v in (CE, CG))
    return _fortran(torch.stack(CE, -1)), _fortran(torch.stack(CG, -1))


class _Ops(C.Structure):
    """chm_sp_ops of include/chimera_gb300.h"""
    _fields_ = [("K", C.c_int32), ("N", C.c_int32), ("nmodes", C.c_int32), ("pad", C.c_int32),
                ("f32", C.c_void_p), ("bf16", C.c_void_p * 3)]


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _prepared(mats):
    K, N, nm = mats.shape
    d = _col(mats)
    buf = torch.empty(_lib.query("chm_sp_ops_bytes", K, N, nm), dtype=torch.uint8, device="cuda")
    ops = _Ops()
    _lib.call("chm_sp_prepare_ops", C.addressof(ops), d.data_ptr(), K, N, nm, buf.data_ptr(),
              buf.numel(), _stream())
    return ops, buf


# ---------------------------------------------------------------------------
# particles
# ---------------------------------------------------------------------------
def _plasma(case, seed):
    """A thermal plasma with a wake-like momentum pattern in the right half of
    the box, cell by cell (r rows of x cells) with random in-cell positions, as
    a plasma is some hundred steps into a run; FP64 coords and momenta (3, n),
    weights (n)."""
    nx, nr, nkr, nm = _dims(case)
    g = _gen(seed)
    ppc = case["ppc_x"] * case["ppc_r"] * case["ppc_t"]
    cx0 = nx // 2
    ncx, ncr = nx - 1 - cx0, nkr - 1
    n = ncx * ncr * ppc
    i = torch.arange(n, device="cuda") // ppc
    u = torch.rand((3, n), device="cuda", dtype=torch.float64, generator=g)
    x = (cx0 + i % ncx + u[0]) * DX
    r = (i // ncx + u[1]) * DR
    th = 2 * math.pi * u[2]
    del i
    coords = torch.stack([x, r * torch.cos(th), r * torch.sin(th)])
    mom = torch.empty_like(coords).normal_(0.0, 1e-3, generator=g)
    mom[0] += 0.05 * torch.sin(2 * math.pi * x / 20.0) * torch.exp(-(r / 15.0) ** 2)
    w = -0.002 * DR * DX * 2 * math.pi / ppc * r
    return coords, mom, w


def _beam(case, seed):
    """An FEL beam: a uniform cylinder in the middle of the box, relativistic
    along x; FP64 coords and momenta (3, n), weights (n)."""
    g = _gen(seed)
    n = case["parts"]
    u = torch.rand((3, n), device="cuda", dtype=torch.float64, generator=g)
    lb = 80e-4 / 2.8
    r, th = lb * torch.sqrt(u[1]), 2 * math.pi * u[2]
    coords = torch.stack([lb * (u[0] - 0.5), r * torch.cos(th), r * torch.sin(th)])
    mom = torch.empty_like(coords).normal_(0.0, 0.004, generator=g)
    mom[0] = GAMMA_FEL + 5.0 * mom[0]
    w = torch.full((n,), -1e-4 / n, dtype=torch.float64, device="cuda")
    return coords, mom, w


# ---------------------------------------------------------------------------
# whole steps
# ---------------------------------------------------------------------------
def _prepare_lwfa(case, seed):
    np.random.seed(seed % (1 << 31))
    nx, nkr = case["nx"], case["nkr"]
    grid = (-nx * DX + 4.0, 4.0, nkr * DR, DX, DR)
    prof = lambda x: (np.asarray(x) >= grid[0]).astype(float)  # noqa: E731
    solver = Solver({"Grid": grid, "TimeStep": DX, "MaxAzimuthMode": case["modes"] - 1,
                     "Features": ("SpaceCharge", "StillAsBackground")})
    solver.add_gauss_beam({"a0": 1.0, "k0": 1.0, "x0": -4.0, "x_foc": 0.0, "Lx": 4.0, "LR": 6.0})
    el = {"Grid": grid, "TimeStep": DX, "Density": 0.002,
          "FixedCell": (case["ppc_x"], case["ppc_r"], case["ppc_t"]), "Features": ("NoSorting",)}
    io = dict(el, Charge=1.0, Mass=1836.0, Features=("Still", "NoSorting"))
    electrons, ions = Specie(el), Specie(io)
    parts = electrons.gen_parts(Domain=(grid[0] + 1.5 * DX, grid[1], 0.0, grid[2]), ProfileFunc=prof)
    electrons.add_particles(*parts)
    parts[-1] = parts[-1] * -1
    ions.add_particles(*parts)
    comps = {"Solvers": (solver,), "Particles": (electrons, ions),
             "MovingFrames": ({"TimeStep": DX, "Steps": 1, "Velocity": 1.0, "AbsorbLayer": 64,
                               "AddPlasma": prof, "Features": ("IonsOnTop",)},)}
    return dict(run=SplitRun(comps) if case["split"] else ChimeraRun(comps), istep=0,
                split=case["split"])


def _prepare_fel(case, seed):
    nx, nkr = case["nx"], case["nkr"]
    vb, kres, dt = VB_FEL, 2 * GAMMA_FEL ** 2 / 1.5, 1.0 / 30
    grid = (-0.5 * DX_FEL, 0.5 * DX_FEL, DR_FEL, DX_FEL / nx, DR_FEL / nkr)
    solver = Solver({"Grid": grid, "TimeStep": dt, "MaxAzimuthMode": (case["modes"] - 1) // 2,
                     "KxShift": kres, "Rcut": 0.7 * DR_FEL, "CoPropagative": vb,
                     "Features": {"NoPoissonCorrection": True, "NoAntiEcho": True}})
    solver.add_gauss_beam({"a0": 0.15, "k0": kres, "x0": -30e-4 / 2.8, "x_foc": 25.0,
                           "Lx": 15e-4 / 2.8, "LR": 180e-4 / 2.8})
    beam = Specie({"Grid": grid, "TimeStep": dt, "Charge": -1.0, "Mass": 1.0,
                   "MomentaMeans": (GAMMA_FEL, 0.0, 0.0),
                   "Devices": ([fimera.undul_analytic, np.array([1.0, 1.0, 1.0, 1.0e6])],)})
    beam.add_particles(*_beam(case, seed))
    run = SplitRun({"Solvers": (solver,), "Particles": (beam,),
                    "MovingFrames": ({"TimeStep": dt, "Steps": 1, "Velocity": vb,
                                      "Features": ("Staged", "NoSorting")},)})
    return dict(run=run, istep=0)


def _split_outputs(run):
    """Fields and the moving particles of a split run (x in cells)."""
    b = run.parts[0].buf
    return [run.EG, run.EB, run.Jfb, b["ix"] + b["fx"], b["y"], b["z"], b["px"], b["py"], b["pz"]]


def _run_lwfa(s):
    s["istep"] += 1
    run = s["run"]
    run.make_step(s["istep"])
    if s["split"]:
        return _split_outputs(run)
    D, P = run.Solvers[0].Data, run.Particles[0].Data
    return [D["EG_fb"], D["EB"], D["J_fb"], D["Rho_fb"], P["coords"], P["momenta"], P["weights"]]


def _run_fel(s):
    s["istep"] += 1
    s["run"].graph_step(s["istep"])
    return _split_outputs(s["run"])


# ---------------------------------------------------------------------------
# the field half
# ---------------------------------------------------------------------------
def _field_inputs(case, seed):
    """Deposited grids with the amplitude profile of a plasma (a noise floor,
    stronger on the axis) and a spectral field falling off with kr: FP64."""
    nx, nr, nkr, nm = _dims(case)
    g = _gen(seed)
    o, dx, kenv, kx, w, fact = _spectrum(case)
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None, None]
    r = torch.from_numpy(o["rgrid"]).cuda()[None, :, None]
    amp = torch.abs(r) * (0.2 + torch.exp(-(r / (0.1 * nr * o["dr"])) ** 2
                                          - ((x - 0.7 * nx) / (0.1 * nx)) ** 2))
    J = _noise((nx, nr, nm, 3), g, 1e-3)
    J *= amp[..., None]
    rho = _noise((nx, nr, nm), g, 1e-3)
    rho *= amp
    J[:, 0] = 0
    rho[:, 0] = 0
    EG = _noise((nx, nkr, nm, 6), g, 1e-2)
    fall = torch.exp(-torch.from_numpy(o["kr"]).cuda() * o["dr"])
    EG[..., :3] *= fall[None, :, :, None]
    EG[..., 3:] *= (fall[None] * w)[..., None]
    gprv = _noise((nx, nkr, nm, 3), g, 1e-4)
    return dict(o=o, kenv=kenv, kx=kx, w=w, fact=fact, J=J, rho=rho, EG=EG, gprv=gprv, leftX=3.3)


SCALE = 2.0 ** 52  # fixed-point scale of the deposit accumulators made here


def _prepare_fields(case, seed):
    nx, nr, nkr, nm = _dims(case)
    f = _field_inputs(case, seed)
    o = f["o"]

    def acc(t):  # the deposit's int64 {re, im} accumulator (no ghost content)
        flat = torch.view_as_real(t.permute(*reversed(range(t.dim())))).reshape(-1)
        return torch.round(flat * SCALE).to(torch.int64)

    CE, CG = _psatd(f["w"], DX)
    s = dict(case=case, accJ=acc(f["J"]), accR=acc(f["rho"]),
             scale=torch.tensor([SCALE, 1.0], dtype=torch.float64, device="cuda"),
             kx64=f["kx"], kx32=f["kx"].to(torch.float32), fact=_fortran(f["fact"], torch.float32),
             pf=_fortran(1.0 / f["w"] ** 2, torch.float32), c1=_fortran(CE, torch.float32),
             c2=_fortran(CG, torch.float32), EG=_fortran(f["EG"], torch.complex64),
             gprv=_fortran(f["gprv"], torch.complex64), leftX=f["leftX"])
    s["ops"] = {k: _prepared(o[k]) for k in ("In", "Out", "Dp", "Dm")}
    z = lambda *shape: fimera.fortran_zeros(shape, torch.complex64)  # noqa: E731
    s.update(J=z(nx, nkr, nm, 3), R=z(nx, nkr, nm), gnxt=z(nx, nkr, nm, 3), B=z(nx, nkr, nm, 3),
             EB=z(nx, nr, nm, 6),
             ws=torch.empty(_lib.query("chm_sp_fb_ws_bytes", nx, nr, nkr, nm), dtype=torch.uint8,
                            device="cuda"))
    return s


def _run_fields(s):
    nx, nr, nkr, nm = _dims(s["case"])
    st, ws, wsb = _stream(), s["ws"].data_ptr(), s["ws"].numel()
    In, Out, Dp, Dm = (C.addressof(s["ops"][k][0]) for k in ("In", "Out", "Dp", "Dm"))
    p = lambda k: s[k].data_ptr()  # noqa: E731
    for out, acc, nc in (("J", "accJ", 3), ("R", "accR", 1)):
        _lib.call("chm_sp_fb_in_acc", p(out), p(acc), p("scale"), None, None, s["leftX"], p("kx64"),
                  In, p("fact"), nx, nr, nkr, nm, nc, ws, wsb, st, None)
    _lib.call("chm_sp_fb_grad", p("gnxt"), p("R"), Dp, Dm, p("kx32"), nx, nkr, nm, ws, wsb, st)
    _lib.call("chm_sp_poisson_psatd", p("J"), p("gprv"), p("gnxt"), p("pf"), 1.0 / DX, Dp, Dm,
              p("kx32"), nx, nkr, nm, 3, 1, p("EG"), p("c1"), p("c2"), 5, ws, wsb, st)
    _lib.call("chm_sp_rot_b", p("B"), s["EG"][..., 3:].data_ptr(), p("pf"), Dp, Dm, p("kx32"), nx,
              nkr, nm, ws, wsb, st)
    _lib.call("chm_sp_fb_eb_out", p("EB"), p("EG"), p("B"), s["leftX"], p("kx64"), Out, nx, nr, nkr,
              nm, ws, wsb, st, None)
    return [s["J"], s["R"], s["gnxt"], s["EG"], s["B"], s["EB"]]


def _prepare_fields64(case, seed):
    nx, nr, nkr, nm = _dims(case)
    f = _field_inputs(case, seed)
    o = f["o"]
    env = case["env"]
    dt = 1.0 / 30 if env else DX
    z = lambda *shape: fimera.fortran_zeros(shape)  # noqa: E731
    s = {k: f[k] for k in ("J", "rho", "EG", "gprv", "kenv", "kx", "leftX")}
    s.update(env=env, pf=_fortran(1.0 / f["w"] ** 2), fact=_fortran(f["fact"]),
             Jfb=z(nx, nkr, nm, 3), B=z(nx, nkr, nm, 3), EB=z(nx, nr, nm, 6),
             **{k: _col(o[k]) for k in ("In", "Out", "Dp", "Dm")})
    s["c1"], s["c2"] = _psatd(f["w"], dt, f["kx"] if env else None)
    if not env:
        s.update(R=z(nx, nkr, nm), gnxt=z(nx, nkr, nm, 3), vec=z(nx, nkr, nm, 3))
    return s


def _run_fields64(s):
    D = (s["Dp"], s["Dm"], s["kx"])
    s["Jfb"] = fimera.fb_vec_in(s["Jfb"], s["J"], s["leftX"], s["kenv"], s["In"])
    s["Jfb"] = fimera.omp_mult_vec(s["Jfb"], s["fact"])
    if s["env"]:
        s["EG"] = fimera.maxwell_push_wo_spchrg(s["EG"], s["Jfb"], s["c1"], s["c2"])
        s["B"] = fimera.fb_rot_env(s["B"], s["EG"][..., 3:], *D)
    else:
        s["R"] = fimera.fb_scl_in(s["R"], s["rho"], s["leftX"], s["kenv"], s["In"])
        s["R"] = fimera.omp_mult_scl(s["R"], s["fact"])
        s["gnxt"] = fimera.fb_grad(s["gnxt"], s["R"], *D)
        for _ in range(3):
            s["vec"].copy_(s["Jfb"])
            s["vec"] = fimera.fb_graddiv(s["vec"], *D)
            s["Jfb"] = fimera.poiss_corr(s["Jfb"], s["vec"], s["gprv"], s["gnxt"], 1.0 / DX, s["pf"])
        s["EG"] = fimera.maxwell_push_with_spchrg(s["EG"], s["Jfb"], s["gprv"], s["gnxt"], s["c1"],
                                                  s["c2"])
        s["B"] = fimera.fb_rot(s["B"], s["EG"][..., 3:], *D)
    s["B"] = fimera.omp_mult_vec(s["B"], s["pf"])
    s["EB"] = fimera.fb_eb_out(s["EB"], s["EG"], s["B"], s["leftX"], s["kenv"], s["Out"],
                               eb_mode=2 if s["env"] else 1)
    return [s["Jfb"], s["EG"], s["B"], s["EB"]] + ([] if s["env"] else [s["R"], s["gnxt"]])


# ---------------------------------------------------------------------------
# the particle half
# ---------------------------------------------------------------------------
def _eb(case, seed, scale, dtype):
    """Node fields as fb_eb_out leaves them: noise in r rows 1.., the ghost
    row the (signed) image of row 1."""
    nx, nr, nkr, nm = _dims(case)
    EB = _noise((nx, nr, nm, 6), _gen(seed + 77), scale, dtype)
    sign = torch.full((nm,), -1.0, device="cuda")
    if not case.get("env"):
        sign[0] = 1.0
    EB[:, 0] = EB[:, 1] * sign[None, :, None].to(EB.dtype)
    return EB


def _prepare_parts(case, seed):
    nx, nr, nkr, nm = _dims(case)
    coords, mom, w = _plasma(case, seed)
    assert coords.dtype == mom.dtype == w.dtype == torch.float64  # (the C ABI takes pointers)
    n = int(w.shape[0])
    cap = _lib.query("chm_sp_capacity", n)
    alloc = lambda: [torch.zeros(cap, dtype=torch.int32 if k == 0 else torch.float32,  # noqa: E731
                                 device="cuda") for k in range(8)]
    bufs = alloc()
    _lib.call("chm_sp_from_f64", *[b.data_ptr() for b in bufs], None, 0, coords.data_ptr(),
              coords.stride(0), coords.stride(1), mom.data_ptr(), mom.stride(0), mom.stride(1),
              w.data_ptr(), w.stride(0), 0.0, DX, n, _stream())
    del coords, mom, w
    scale = torch.zeros(2, dtype=torch.float64, device="cuda")
    sws = torch.empty(_lib.query("chm_sp_scale_ws_bytes"), dtype=torch.uint8, device="cuda")
    _lib.call("chm_sp_weight_scale", scale.data_ptr(), bufs[7].data_ptr(), n, sws.data_ptr(),
              sws.numel(), _stream())
    sp = _spectrum(case)
    grid = nx * nr * nm * 2
    s = dict(case=case, n=n, bufs=bufs, spare=alloc(), steps=0,
             dead=torch.zeros(cap, dtype=torch.uint8, device="cuda"),
             count=torch.zeros(1, dtype=torch.int64, device="cuda"),
             sort_ws=torch.empty(_lib.query("chm_sp_sort_ws_bytes", n), dtype=torch.uint8,
                                 device="cuda"))
    _resort(s)
    return dict(s, scale=scale, EB=_eb(case, seed, 2e-4, torch.complex64),
                accJ=torch.zeros(3 * grid, dtype=torch.int64, device="cuda"),
                accR=torch.zeros(grid, dtype=torch.int64, device="cuda"),
                J=fimera.fortran_zeros((nx, nkr, nm, 3), torch.complex64),
                R=fimera.fortran_zeros((nx, nkr, nm), torch.complex64), kx64=sp[3],
                fact=_fortran(sp[5], torch.float32), In=_prepared(sp[0]["In"]),
                ws=torch.empty(_lib.query("chm_sp_fb_ws_bytes", nx, nr, nkr, nm), dtype=torch.uint8,
                               device="cuda"))


def _resort(s):
    """The re-sort by deposit cell that a run makes every 64 steps
    (SplitRun.sort_every)."""
    nx, nr, nkr, nm = _dims(s["case"])
    _lib.call("chm_sp_sort_cells", *[b.data_ptr() for b in s["bufs"]], s["dead"].data_ptr(), s["n"],
              0, 0.0, nx, nr, 1.0 / DR, *[b.data_ptr() for b in s["spare"]], s["count"].data_ptr(),
              s["sort_ws"].data_ptr(), s["sort_ws"].numel(), _stream())
    s["bufs"], s["spare"] = s["spare"], s["bufs"]
    s["n"] = int(s["count"].item())


def _run_parts(s):
    """Push and deposit, the deposits' transforms (what the step reads of
    them), gather and momentum push; the re-sort at its cadence."""
    nx, nr, nkr, nm = _dims(s["case"])
    st = _stream()
    if s["steps"] and s["steps"] % 64 == 0:
        _resort(s)
    s["steps"] += 1
    ptrs = [b.data_ptr() for b in s["bufs"]]
    p = lambda k: s[k].data_ptr()  # noqa: E731
    s["accJ"].zero_()
    s["accR"].zero_()
    _lib.call("chm_sp_push_deposit", *ptrs, s["n"], 0, 0.0, 1.0 / DX, 1.0 / DR, DX, nx, nr, nm, 1,
              p("accJ"), p("scale"), p("accR"), p("scale"), st, None)
    for out, acc, nc in (("J", "accJ", 3), ("R", "accR", 1)):
        _lib.call("chm_sp_fb_in_acc", p(out), p(acc), p("scale"), None, None, 0.0, p("kx64"),
                  C.addressof(s["In"][0]), p("fact"), nx, nr, nkr, nm, nc, p("ws"), s["ws"].numel(),
                  st, None)
    _lib.call("chm_sp_gather_push", *ptrs, s["n"], 0, 0.0, 1.0 / DR, p("EB"), nx, nr, nm,
              -2 * math.pi * DX, st, None)
    b = s["bufs"]
    return [s["J"], s["R"], b[0] + b[1]] + b[2:7]


def _prepare_parts64(case, seed):
    nx, nr, nkr, nm = _dims(case)
    env = case["env"]
    coords, mom, w = _beam(case, seed) if env else _plasma(case, seed)
    if env:
        dx, dr, left = DX_FEL / nx, DR_FEL / nkr, -0.5 * DX_FEL
    else:
        # (the cell order of the generator; deposits take any order)
        dx, dr, left = DX, DR, 0.0
    z = lambda *shape: fimera.fortran_zeros(shape)  # noqa: E731
    s = dict(case=case, env=env, x=coords, p=mom, w=w, h=torch.zeros_like(coords),
             EBp=torch.zeros((6, coords.shape[1]), dtype=torch.float64, device="cuda"),
             EB=_eb(case, seed, 2e-4, torch.complex128), J=z(nx, nr, nm, 3),
             rgrid=torch.from_numpy(dr * (np.arange(nr) - 0.5)).cuda(), dx=dx, dr=dr, left=left,
             dt=1.0 / 30 if env else DX, und=np.array([1.0, 1.0, -10.0, 1.0e6]))
    if not env:
        s["rho"] = z(nx, nr, nm)
    return s


def _run_parts64(s):
    # (an FEL window moves with the beam in two halves: chimera_main.py:286-304)
    half = 0.5 * VB_FEL * s["dt"] if s["env"] else 0.0
    s["left"] += half
    g = (s["left"], s["rgrid"], 1.0 / s["dx"], 1.0 / s["dr"])
    fimera.push_coords(s["x"], s["p"], s["h"], s["dt"])
    s["J"].zero_()
    s["EBp"].zero_()
    if s["env"]:
        fimera.dep_curr_env(s["h"], s["p"], s["w"], s["J"], *g, KX0_FEL)
        s["left"] += half
        g = (s["left"],) + g[1:]
        fimera.proj_fld_env(s["x"], s["w"], s["EB"], s["EBp"], *g, KX0_FEL)
        fimera.undul_analytic(s["x"], s["EBp"], 0.0, s["und"])
    else:
        fimera.dep_curr(s["h"], s["p"], s["w"], s["J"], *g)
        s["rho"].zero_()
        fimera.dep_dens(s["x"], s["w"], s["rho"], *g)
        fimera.proj_fld(s["x"], s["w"], s["EB"], s["EBp"], *g)
    fimera.push_velocs(s["p"], s["EBp"], -2 * math.pi * s["dt"])
    return [s["x"], s["h"], s["p"], s["EBp"], s["J"]] + ([] if s["env"] else [s["rho"]])


# ---------------------------------------------------------------------------
_PREPARE = dict(lwfa_step=_prepare_lwfa, fel_step=_prepare_fel, fields=_prepare_fields,
                parts=_prepare_parts, fields64=_prepare_fields64, parts64=_prepare_parts64)
_RUN = dict(lwfa_step=_run_lwfa, fel_step=_run_fel, fields=_run_fields, parts=_run_parts,
            fields64=_run_fields64, parts64=_run_parts64)


def prepare(case, seed):
    return dict(kind=case["kind"], state=_PREPARE[case["kind"]](case, seed))


def run(state):
    return _RUN[state["kind"]](state["state"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _num_parts(case):
    if "parts" in case:
        return case["parts"]
    ppc = case["ppc_x"] * case["ppc_r"] * case["ppc_t"]
    ncx = case["nx"] - 1 - (case["nx"] // 2 if case["kind"] != "lwfa_step" else 0)
    return ncx * (case["nkr"] - 1) * ppc


def _field_work(case, c, acc, env):
    """Field half with c-byte complex values and acc-byte deposit nodes: the
    deposits in, EG in and out, the coefficients, the gradients and the node
    fields out; the products' operations."""
    nx, nr, nkr, nm = _dims(case)
    P, S = nx * nkr * nm, nx * nr * nm
    dep, ncoef, grads = (3, 3, 0) if env else (4, 5, 6)
    b = dep * S * acc + 12 * P * c + 2 * ncoef * P * (c if env else c // 2) + P * c
    b += (3 + 3 + grads) * P * c + 6 * S * c
    if env:
        products = (3 + 6) * nm + 6 * (nm - 1)
    else:
        # fb_in 4 and fb_out 6 a mode; the gradient 2 nm - 1; the curl 3 (2 nm - 1);
        # three corrections of a divergence (2 (2 nm + 1) - 2) and a gradient (2 nm)
        products = 10 * nm + (2 * nm - 1) + 3 * (2 * nm - 1) + 3 * (2 * (2 * nm - 1) + 2 * nm)
    return b, 4.0 * nx * nkr * nkr * products


def work(case):
    nx, nr, nkr, nm = _dims(case)
    kind, n = case["kind"], None
    S = nx * nr * nm
    if kind in ("fields", "fields64"):
        env = bool(case.get("env"))
        b, f = _field_work(case, 8 if kind == "fields" else 16, 16, env)
        return dict(bytes=b, flops=f)
    n = _num_parts(case)
    comp = 1 if (kind == "fel_step" or case.get("env")) else 3
    per = nm * (8 * comp + (8 if comp == 3 else 0) + 48) + 120  # node values and pushes
    if kind == "parts":
        # 32 bytes read and 16 + 12 written per particle; node fields, transforms
        return dict(bytes=n * 60 + 6 * S * 8 + 4 * nx * nkr * nm * 8,
                    flops=n * per + 4.0 * nx * nkr * nkr * nm * 4)
    if kind == "parts64":
        # coords, momenta, weights in; coords, half-step coords, fields and momenta out
        return dict(bytes=n * (56 + 24 + 24 + 48 + 24) + 6 * S * 16 + (3 if comp == 1 else 4) * S * 16,
                    flops=n * per)
    split = kind == "fel_step" or case["split"]
    b, f = _field_work(dict(case), 8 if split else 16, 16, kind == "fel_step")
    return dict(bytes=b + n * (60 if split else 176), flops=f + n * per)


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
def _mm(a, m):
    """Complex (nx, K) times real (K, N), as a real product."""
    return torch.complex(a.real.contiguous() @ m, a.imag.contiguous() @ m)


def _ex_in(v, In, kx, leftX, fact):
    f = torch.fft.fft(v[:, 1:], dim=0)
    sh = torch.exp(-1j * kx * leftX)[:, None]
    out = torch.empty((v.shape[0], In.shape[1]) + tuple(v.shape[2:]), dtype=torch.complex128, device="cuda")
    for m in range(v.shape[2]):
        for c in range(v.shape[3]):
            out[:, :, m, c] = _mm(f[:, :, m, c], In[:, :, m]) * sh * fact[:, :, m]
    return out


def _ex_out(v, Out, kx, leftX, env):
    nx, nkr, nm, nc = v.shape
    sh = torch.exp(1j * kx * leftX)[:, None]
    eb = torch.zeros((nx, Out.shape[1] + 1, nm, nc), dtype=torch.complex128, device="cuda")
    for m in range(nm):
        lone = m == 0 and not env
        for c in range(nc):
            t = torch.fft.ifft(_mm(v[:, :, m, c], Out[:, :, m]) * sh, dim=0) * nx
            t = t * ((0.5 if lone else 1.0) / math.pi)
            eb[:, 1:, m, c] = t
            eb[:, 0, m, c] = t[:, 0] if (lone or nm == 1) else -t[:, 0]
    return eb


def _refl(p):
    """The m = -1 plane: -conj of the m = 1 plane at -kx."""
    q = -torch.conj(p)
    return torch.cat([q[:1], torch.flip(q[1:], (0,))])


def _nb(planes, D, m, step, nm):
    """Neighbour product of mode m: planes[m + step] times D[m], with the
    reflected mode below the axis (plain solver with nm > 1 stored modes);
    None where there is none."""
    k = m + step
    if k < 0:
        src = _refl(planes[1]) if nm > 1 else None
    else:
        src = planes[k] if k < len(planes) else None
    return None if src is None else _mm(src, D[:, :, m])


def _ex_grad(scl, Dp, Dm, kx, nm):
    """Gradient of the scalar modes scl (list) into nm modes (plain solver)."""
    out = torch.zeros(tuple(scl[0].shape) + (nm, 3), dtype=torch.complex128, device="cuda")
    for m in range(nm):
        out[:, :, m, 0] = 1j * kx[:, None] * scl[m]
        lo, hi = _nb(scl, Dm, m, -1, nm), _nb(scl, Dp, m, 1, nm)
        if lo is not None:
            out[:, :, m, 1] -= lo
            out[:, :, m, 2] += 1j * lo
        if hi is not None:
            out[:, :, m, 1] += hi
            out[:, :, m, 2] += 1j * hi
    return out


def _ex_graddiv(v, Dp, Dm, kx):
    """grad(div(v)) of the plain solver, the divergence carried to one mode
    more than v has."""
    nm = v.shape[2]
    v2, v3 = ([v[:, :, m, c] for m in range(nm)] for c in (1, 2))
    scl = []
    for m in range(nm + 1):
        r = 1j * kx[:, None] * v[:, :, m, 0] if m < nm else torch.zeros_like(v2[0])
        lo2, lo3 = _nb(v2, Dm, m, -1, nm), _nb(v3, Dm, m, -1, nm)
        if lo2 is not None:
            r = r + 1j * lo3 - lo2
        if m < nm - 1:
            r = r + 1j * _nb(v3, Dp, m, 1, nm) + _nb(v2, Dp, m, 1, nm)
        scl.append(r)
    return _ex_grad(scl, Dp, Dm, kx, nm)


def _ex_rot(v, Dp, Dm, kx, env):
    nm = v.shape[2]
    P = [[v[:, :, m, c] for m in range(nm)] for c in range(3)]
    out = torch.zeros_like(v)
    ikx = 1j * kx[:, None]
    for m in range(nm):
        out[:, :, m, 1] = -ikx * P[2][m]
        out[:, :, m, 2] = ikx * P[1][m]
        md = m + 1 if env else m
        for step, D in ((1, Dp), (-1, Dm)):
            k = m + step
            if k < 0 and not env and nm > 1:
                src = [_refl(P[c][1]) for c in range(3)]
            elif 0 <= k < nm:
                src = [P[c][k] for c in range(3)]
            else:
                continue
            q = [_mm(a, D[:, :, md]) for a in src]
            out[:, :, m, 1] += 1j * q[0]
            if step == 1:
                out[:, :, m, 0] -= 1j * q[1] - q[2]
                out[:, :, m, 2] -= q[0]
            else:
                if not env:
                    out[:, :, m, 0] -= 1j * q[1] + q[2]
                out[:, :, m, 2] += q[0]
    return out


def _ex_fields(case, seed):
    f = _field_inputs(case, seed)
    o, env = f["o"], bool(case.get("env"))
    single = case["kind"] == "fields"
    q = (lambda t: t.to(torch.complex64).to(torch.complex128)) if single else (lambda t: t)
    qr = (lambda t: t.to(torch.float32).to(torch.float64)) if single else (lambda t: t)
    fix = (lambda t: torch.complex(torch.round(t.real * SCALE) / SCALE,
                                   torch.round(t.imag * SCALE) / SCALE)) if single else (lambda t: t)
    In, Out, Dp, Dm = (torch.from_numpy(np.ascontiguousarray(o[k])).cuda()
                       for k in ("In", "Out", "Dp", "Dm"))
    kx, kenv, leftX = f["kx"], f["kenv"], f["leftX"]
    fact, pf = qr(f["fact"]), qr(1.0 / f["w"] ** 2)[..., None]
    EG = q(f["EG"])
    E, G = EG[..., :3], EG[..., 3:]
    J = _ex_in(fix(f["J"]), In, kenv, leftX, fact)
    c1, c2 = _psatd(f["w"], 1.0 / 30 if env else DX, f["kx"] if env else None)
    if single:
        c1, c2 = qr(c1), qr(c2)
    a = [c1[..., i, None] for i in range(c1.shape[-1])]
    b = [c2[..., i, None] for i in range(c2.shape[-1])]
    extra = []
    if env:
        En = a[0] * E + a[1] * G + a[2] * J
        Gn = b[0] * E + b[1] * G + b[2] * J
    else:
        R = _ex_in(fix(f["rho"])[..., None], In, kenv, leftX, fact)[..., 0]
        nm = R.shape[2]
        gn = _ex_grad([R[:, :, m] for m in range(nm)], Dp, Dm, kx, nm)
        gp = q(f["gprv"])
        for _ in range(3):
            J = J + pf * (_ex_graddiv(J, Dp, Dm, kx) + (gn - gp) / DX)
        En = a[0] * E + a[1] * G + a[2] * J + a[3] * gp + a[4] * gn
        Gn = b[0] * E + b[1] * G + b[2] * J + b[3] * gp + b[4] * gn
        extra = [R, gn]
    B = _ex_rot(Gn, Dp, Dm, kx, env) * pf
    EGn = torch.cat([En, Gn], -1)
    EB = _ex_out(torch.cat([En, B], -1), Out, kenv, leftX, env)
    fo = lambda t: _laid_out(t)  # noqa: E731
    if single:
        return [fo(t) for t in (J, extra[0], extra[1], EGn, B, EB)]
    return [fo(t) for t in [J, EGn, B, EB] + extra]


def _laid_out(t):
    return _fortran(t.contiguous())


def _ex_cells(x, y, z, left, dx, dr, nr):
    """Cell indices, linear weights and the unit phase of positions (FP64)."""
    r = torch.sqrt(y * y + z * z)
    fx = (x - left) * (1.0 / dx)
    ix = torch.floor(fx)
    fr = (r + 0.5 * dr) * (1.0 / dr)
    ir = torch.floor(fr)
    ok = (r < dr * (nr - 1.5)) & (ir >= 0) & (ir <= nr - 2)
    return ix.long(), fx - ix, ir.long(), fr - ir, torch.complex(y / r, z / r), ok


def _ex_deposit(vals, cells, nx, nr, modes, env_phase=None):
    """Linear deposit of per-particle values (list, one per component) into
    (nx, nr, nm, ncomp), with the ghost row folded."""
    ix, sx, ir, sr, ph, ok = cells
    nm = len(modes)
    out = torch.zeros((nx, nr, nm, len(vals)), dtype=torch.complex128, device="cuda")
    flat = torch.view_as_real(out)
    for mi, m in enumerate(modes):
        pm = torch.conj(ph) ** m if m >= 0 else ph ** (-m)
        for c, v in enumerate(vals):
            if v is None:
                continue
            val = v * pm if env_phase is None else v * pm * env_phase
            for j in (0, 1):
                for k in (0, 1):
                    wgt = (sr if j else 1 - sr) * (sx if k else 1 - sx)
                    gx = ix + k
                    good = ok & (gx >= 0) & (gx < nx)
                    idx = torch.where(good, gx * nr + ir + j, 0)
                    t = torch.zeros(nx * nr, 2, dtype=torch.float64, device="cuda")
                    a = torch.view_as_real(val * torch.where(good, wgt, 0.0))
                    t[:, 0].index_add_(0, idx, a[:, 0])
                    t[:, 1].index_add_(0, idx, a[:, 1])
                    flat[:, :, mi, c] += t.view(nx, nr, 2)
    out[:, 1] -= out[:, 0]
    out[:, 0] = 0
    return out


def _ex_gather(EB, cells, modes, env_phase=None):
    ix, sx, ir, sr, ph, ok = cells
    nx = EB.shape[0]
    F = torch.zeros((6, ix.shape[0]), dtype=torch.float64, device="cuda")
    for mi, m in enumerate(modes):
        pm = ph ** m if m >= 0 else torch.conj(ph) ** (-m)
        if env_phase is not None:
            pm = pm * env_phase
        for j in (0, 1):
            for k in (0, 1):
                wgt = (sr if j else 1 - sr) * (sx if k else 1 - sx)
                gx = ix + k
                good = ok & (gx >= 0) & (gx < nx)
                pw = pm * torch.where(good, wgt, 0.0)
                gx, jr = gx.clamp(0, nx - 1), (ir + j).clamp(0, EB.shape[1] - 1)
                for c in range(6):
                    f = EB[gx, jr, mi, c]
                    F[c] += pw.real * f.real - pw.imag * f.imag
    return F


def _ex_boris(p, F, dt):
    h = 0.5 * dt
    um = p + h * F[:3]
    t = h * F[3:] / torch.sqrt(1.0 + (um * um).sum(0))
    s = 2 * t / (1 + (t * t).sum(0))
    cross = lambda a, b: torch.linalg.cross(a, b, dim=0)  # noqa: E731
    return um + cross(um + cross(um, t), s) + h * F[:3]


def _ex_push(x, p, dt):
    v = p / torch.sqrt(1.0 + (p * p).sum(0))
    xn = x + dt * v
    return xn, 0.5 * (x + xn), v


def _ex_parts64(case, seed):
    s = _prepare_parts64(case, seed)
    nx, nr, nkr, nm = _dims(case)
    env, dx, dr = s["env"], s["dx"], s["dr"]
    half = 0.5 * VB_FEL * s["dt"] if env else 0.0
    modes = list(range(-(nm // 2), nm // 2 + 1)) if env else list(range(nm))
    xn, h, v = _ex_push(s["x"], s["p"], s["dt"])
    lh = s["left"] + half
    ch, cn = _ex_cells(*h, lh, dx, dr, nr), _ex_cells(*xn, lh + half, dx, dr, nr)
    carry = lambda x, sg: torch.exp(sg * 1j * (x * KX0_FEL)) if env else None  # noqa: E731
    vals = [None, None, v[2] * s["w"]] if env else [v[c] * s["w"] for c in range(3)]
    J = _ex_deposit(vals, ch, nx, nr, modes, carry(h[0], -1))
    F = _ex_gather(s["EB"], cn, modes, carry(xn[0], 1))
    if env:
        a0, lam, X0, L = s["und"]
        ku = 2 * math.pi / lam
        amp = a0 * torch.where((xn[0] > X0) & (xn[0] < X0 + L), 1.0, 0.0)
        amp = amp * torch.where(xn[0] < X0 + lam, (xn[0] - X0) / lam, 1.0)
        F[4] += amp * torch.sin(ku * (xn[0] - X0)) * torch.cosh(ku * xn[1])
        F[3] += amp * torch.cos(ku * (xn[0] - X0)) * torch.sinh(ku * xn[1])
    p = _ex_boris(s["p"], F, -2 * math.pi * s["dt"])
    out = [xn, h, p, F, _laid_out(J)]
    if not env:
        out.append(_laid_out(_ex_deposit([s["w"]], cn, nx, nr, modes)[..., 0]))
    return out


def _ex_parts(case, seed):
    s = _prepare_parts(case, seed)
    nx, nr, nkr, nm = _dims(case)
    n = s["n"]
    slot = torch.arange(n, device="cuda")
    slot = (slot // 512) * 512 + 32 * (slot % 16) + (slot // 16) % 32
    b = [t[slot].to(torch.float64) for t in s["bufs"]]
    x = torch.stack([(b[0] + b[1]) * DX, b[2], b[3]])
    p, w = torch.stack(b[4:7]), b[7]
    del b
    xn, h, v = _ex_push(x, p, DX)
    modes = list(range(nm))
    J = _ex_deposit([v[c] * w for c in range(3)], _ex_cells(*h, 0.0, DX, DR, nr), nx, nr, modes)
    del h, v
    cn = _ex_cells(*xn, 0.0, DX, DR, nr)
    R = _ex_deposit([w], cn, nx, nr, modes)
    In = torch.from_numpy(np.ascontiguousarray(_operators(nkr, nm, False)["In"])).cuda()
    fact = s["fact"].to(torch.float64)
    Jf = _ex_in(J, In, s["kx64"], 0.0, fact)
    Rf = _ex_in(R, In, s["kx64"], 0.0, fact)[..., 0]
    p = _ex_boris(p, _ex_gather(s["EB"].to(torch.complex128), cn, modes), -2 * math.pi * DX)

    def tiles(t):  # particle order -> slots (unused slots as they were: zero)
        full = torch.zeros(s["bufs"][0].shape[0], dtype=torch.float64, device="cuda")
        full[slot] = t
        return full

    return [_laid_out(Jf), _laid_out(Rf), tiles(xn[0] / DX)] + [tiles(t) for t in (*xn[1:], *p)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fields", "fields64"):
        return _ex_fields(case, seed)
    if kind == "parts":
        return _ex_parts(case, seed)
    if kind == "parts64":
        return _ex_parts64(case, seed)
    # (a whole step chains every layer; the layers' own cases hold them)
    return None
