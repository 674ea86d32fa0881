"""The FP64 particle kernels against sums in longer precision: deposits (through
the shared box and straight to the grid, one dominating particle, particles on
the axis, outside and at rest, an r spacing that takes the weights out of
[0, 1]), gathers and the momentum push.

Bounds, u = 2^-53: a stencil weight is off by the rounding of (x - x0) / dx,
3 u nx, of r / dr, 4 u nr, and a few u; a phase by a few u and by that of the
carrier's argument; a deposited value by a quantum, 2^-60 of the sum of the
weights, besides; sums by u per term of the sum of absolute values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD, CLD = np.longdouble, np.clongdouble
NX, NR, LEFT, DX, DR = 300, 40, -1.3, 0.07, 0.11


def _particles(n, order, rng, nr=NR):
    x = LEFT + DX * rng.uniform(-1.6, NX + 0.6, n)
    r = DR * rng.uniform(0, nr + 0.4, n)
    th = rng.uniform(0, 2 * np.pi, n)
    c = np.asfortranarray([x, r * np.cos(th), r * np.sin(th)])
    p = np.asfortranarray(rng.standard_normal((3, n)) * 10.0 ** rng.integers(-3, 3, n))
    w = rng.uniform(-0.5, 1, n)
    if n > 9:
        c[1:, 0] = 0.0
        p[:, 1] = 0.0
        w[2] = 0.0
        c[0, 3] = LEFT + 5 * DX
        c[1:, 4] = (DR * 3, 0.0)
        c[0, 5] = np.nan
        c[2, 6] = np.inf
    if order == "cells":
        k = np.lexsort((np.floor(np.hypot(c[1], c[2]) / DR), np.floor((c[0] - LEFT) / DX)))
        c, p, w = (np.asfortranarray(a[..., k]) for a in (c, p, w))
    elif order == "one":
        c[0], c[1], c[2] = LEFT + 3.3 * DX, 2.4 * DR, 0.3 * DR
    return c, p, w


def _rgrid():
    return DR * (np.arange(NR) - 0.5)


def _stencil(c, ok, rg, dr_inv):
    """per particle: cell, x and r weights, phase y - i z over r"""
    x, y, z = (c[k].astype(LD) for k in range(3))
    r = np.sqrt(y * y + z * z)
    fx = (x - LD(LEFT)) * LD(1 / DX)
    fr = (r - LD(rg[0])) * LD(dr_inv)
    with np.errstate(invalid="ignore"):
        ok = ok & (r < rg[-1]) & np.isfinite(fx) & (fr >= 0) & (np.floor(fr) <= NR - 2)
    ix, ir = np.floor(fx[ok]).astype(int), np.floor(fr[ok]).astype(int)
    sx = fx[ok] - ix
    sr = (r[ok] - rg[ir].astype(LD)) * LD(dr_inv)
    rr = np.where(r[ok] > 0, r[ok], 1)
    return ok, ix, ir, (1 - sx, sx), (1 - sr, sr), (y[ok] / rr - 1j * (z[ok] / rr)).astype(CLD), r[ok]


def _modes(nm, env):
    return range(-((nm - 1) // 2), (nm - 1) // 2 + 1) if env else range(nm)


def _deposit(kind, c, p, w, nm, kx0, rg, dr_inv):
    env, curr = kind.endswith("env"), kind.startswith("dep_curr")
    ok = (w != 0) & ((np.abs(p).sum(0) != 0) if curr else True)
    ok, ix, ir, sx, sr, ph, _ = _stencil(c, ok, rg, dr_inv)
    wl, pl = w[ok].astype(LD), p[:, ok].astype(LD)
    v = pl / np.sqrt(1 + (pl ** 2).sum(0))
    wc = wl * np.exp(-1j * (c[0, ok].astype(LD) * LD(kx0)).astype(CLD)) if env else wl
    out = np.zeros((NX, NR, nm, 3 if curr else 1), CLD)
    mag = np.zeros((NX, NR), LD)   # sums of |w| over the particles that touch a node
    cnt = np.zeros((NX, NR), LD)
    mags = wl ** 2 if kind == "dep_dens_env" else np.abs(wl)
    for j in range(2):
        for k in range(2):
            inx = (ix + k >= 0) & (ix + k < NX)
            at = (ix[inx] + k, ir[inx] + j)
            S = (sx[k] * sr[j])[inx]
            np.add.at(mag, at, mags[inx])
            np.add.at(cnt, at, 1)
            for s, m in enumerate(_modes(nm, env)):
                q = ph ** abs(m)
                q = np.conj(q) if m < 0 else q
                for l in range(out.shape[3]):
                    if kind == "dep_curr_env" and l != 2:
                        continue
                    val = {"dep_curr": lambda: v[l] * wl, "dep_dens": lambda: wl,
                           "dep_curr_env": lambda: v[2] * wc, "dep_dens_env": lambda: wc * wc}[kind]()
                    np.add.at(out[:, :, s, l], at, (q * val)[inx] * S)
    top = max([1.0] + [float(np.abs(s).max()) for s in sr if s.size])
    with np.errstate(invalid="ignore"):
        arg = float(np.abs(kx0 * c[0, ok]).max()) if env and ok.any() else 0.0
    B = float((w[np.isfinite(w)] ** 2).sum() if kind == "dep_dens_env" else np.abs(w).sum())
    tol = mag * (U * ((3 * NX + 4 * NR + 20 + 4 * nm) + 3 * arg) * top) + cnt * (2.0 ** -60 * B)
    out[:, 1] -= out[:, 0]
    out[:, 0] = 0
    tol[:, 1] += tol[:, 0]
    return out, tol.astype(float)


@pytest.mark.parametrize("order", ["random", "cells", "one"])
@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 6001])
@pytest.mark.parametrize("kind,nm", [("dep_curr", 1), ("dep_curr", 2), ("dep_curr", 3), ("dep_dens", 2),
                                     ("dep_curr_env", 3), ("dep_dens_env", 1), ("dep_dens_env", 3)])
@pytest.mark.parametrize("stretch", [1.0, 1.15])
def test_deposit(cuda, kind, nm, n, order, stretch):
    import torch
    from chimera_gb300 import fimera as fm
    rng = np.random.default_rng(n + nm)
    c, p, w = _particles(n, order, rng)
    rg, dr_inv, kx0 = _rgrid(), stretch / DR, 40.0
    env, curr = kind.endswith("env"), kind.startswith("dep_curr")
    want, tol = _deposit(kind, c, p, w, nm, kx0, rg, dr_inv)
    grid = fm.fortran_zeros((NX, NR, nm, 3) if curr else (NX, NR, nm))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda().T if a.ndim == 2 else torch.from_numpy(a).cuda()  # noqa: E731
    args = (T(c), T(p), T(w)) if curr else (T(c), T(w))
    getattr(fm, kind)(*args, grid, LEFT, rg, 1 / DX, dr_inv, *((kx0,) if env else ()))
    got = grid.cpu().numpy().reshape(NX, NR, nm, -1)
    err = np.abs(got - want).astype(float)
    assert np.all(err <= tol[:, :, None, None] + U * np.abs(got))


@pytest.mark.parametrize("env,nm", [(False, 1), (False, 2), (False, 4), (True, 1), (True, 3)])
def test_gather(cuda, env, nm):
    import torch
    from chimera_gb300 import fimera as fm
    rng = np.random.default_rng(7 + nm)
    c, _, w = _particles(3001, "random", rng)
    rg, dr_inv, kx0 = _rgrid(), 1 / DR, 40.0
    fld = np.asfortranarray(rng.standard_normal((NX, NR, nm, 6)) + 1j * rng.standard_normal((NX, NR, nm, 6)))
    f0 = np.asfortranarray(rng.standard_normal((6, w.size)))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.transpose())).cuda().permute(*reversed(range(a.ndim)))  # noqa: E731
    got = T(f0)
    name = "proj_fld_env" if env else "proj_fld"
    getattr(fm, name)(T(c), T(w), T(fld), got, LEFT, rg, 1 / DX, dr_inv, *((kx0,) if env else ()))
    ok, ix, ir, sx, sr, ph, r = _stencil(c, w != 0, rg, dr_inv)
    ph = np.conj(ph)
    if env:
        ph = np.where(r > 0, ph, 1)
    want, mag = f0.astype(LD).copy(), np.zeros((6, int(ok.sum())))
    car = np.exp(1j * (c[0, ok].astype(LD) * LD(kx0)).astype(CLD)) if env else 1
    for s, m in enumerate(_modes(nm, env)):
        q = ph ** abs(m)
        q = car * (np.conj(q) if m < 0 else q)
        for j in range(2):
            for k in range(2):
                inx = (ix + k >= 0) & (ix + k < NX)
                F = np.where(inx[:, None], fld[np.clip(ix + k, 0, NX - 1), ir + j, s], 0)
                want[:, ok] += ((q * (sx[k] * sr[j]))[:, None] * F).real.T
                mag += np.abs(F).T
    with np.errstate(invalid="ignore"):
        arg = float(np.abs(kx0 * c[0, ok]).max()) if env else 0.0
    err = np.abs(got.cpu().numpy() - want).astype(float)
    assert np.all(err[:, ~ok] == 0)
    assert np.all(err[:, ok] <= U * ((3 * NX + 4 * NR + 30 + 12 * nm + 3 * arg) * mag + 2 * np.abs(f0[:, ok])))


@pytest.mark.parametrize("n", [1, 255, 2000])
def test_push_velocs(cuda, n):
    import torch
    from chimera_gb300 import fimera as fm
    rng = np.random.default_rng(n)
    p = np.asfortranarray(rng.standard_normal((3, n)) * 10.0 ** rng.integers(-4, 4, n))
    f = np.asfortranarray(rng.standard_normal((6, n)) * 10.0 ** rng.integers(-4, 3, n))
    dt = 0.37
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda().T  # noqa: E731
    got = fm.push_velocs(T(p), T(f), dt).cpu().numpy()
    h = LD(dt) / 2
    um = p.astype(LD) + h * f[:3].astype(LD)
    t = h * f[3:].astype(LD) / np.sqrt(1 + (um ** 2).sum(0))
    s = 2 * t / (1 + (t ** 2).sum(0))
    u0 = um + np.cross(um, t, axis=0)
    want = um + np.cross(u0, s, axis=0) + h * f[:3].astype(LD)
    size = np.abs(p).sum(0) + dt * np.abs(f[:3]).sum(0)
    tn = np.abs(t).sum(0)
    assert np.all(np.abs(got - want).astype(float) <= 40 * U * size * (1 + tn).astype(float) ** 2)
