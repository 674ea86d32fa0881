"""The envelope solver's particle kernels at the sizes where their split over
warps can go wrong (csrc/split_particles.cu).

Gather and push: a beam of few tiles gets fewer slots a warp than the same
particles with so many zero-weight ones behind them that warps take whole runs;
a particle's result is its own, so the bits are equal.

Push and deposit: the runs of few tiles are summed in four pieces; on both sides
of that line, against the FP64 deposit at the same FP32 positions.  Bound, u =
2^-24: 17 roundings of the sums and some 40 of a value (push, 1 / gamma, carrier,
phases, weights) times the sum of absolute values that a node gets; a half-step position is off by a few u
of a cell in x and 4 u nr in r, which moves weight between neighbouring nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NR, DX, DR, KX0, DT = 256, 33, 0.05, 0.2, 30.0, 0.045
MANY = 152 * 32 * 512 + 77


def _beam(torch, n, total, order):
    g = torch.Generator().manual_seed(n)
    u = lambda: torch.rand(n, generator=g)  # noqa: E731
    phys = np.arange(n)
    phys = (phys & ~511) | ((phys & 15) << 5) | ((phys >> 4) & 31)
    a = [torch.zeros(-(-total // 512) * 512, dtype=torch.int32 if k == 0 else torch.float32) for k in range(8)]
    ix = torch.randint(-1, NX + 2, (n,), generator=g, dtype=torch.int32)
    r, th = u() * (0.95 * NR * DR), u() * 6.28318
    vals = [ix, u(), r * th.cos(), r * th.sin(), 100 * u(), 0.1 * (u() - 0.5), 0.2 * u(), u()]
    if order:  # runs of one cell
        k = torch.from_numpy(np.lexsort(((vals[2] ** 2 + vals[3] ** 2).sqrt().numpy() // DR, ix.numpy())))
        vals = [v[k] for v in vals]
    if n > 5:
        vals[7][3] = 0.0
        vals[2][4] = vals[3][4] = 0.0
    for b, v in zip(a, vals):
        b[torch.from_numpy(phys)] = v
    return [b.cuda() for b in a], torch.from_numpy(phys).cuda()


@pytest.mark.parametrize("n", [1, 15, 512, 513, 30001])
@pytest.mark.parametrize("nm", [1, 3, 5])
def test_gather_of_few_tiles(cuda, nm, n):
    import torch
    from chimera_gb300 import _lib
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator().manual_seed(3)
    eb = torch.view_as_complex(torch.randn((6, nm, NR, NX, 2), generator=g)).contiguous().cuda()
    und = np.array([0.5, 20.0, -50.0, 1000.0, 0.0])
    out = []
    for total in (n, MANY):
        P, phys = _beam(torch, n, total, False)
        tab = torch.zeros(NX + 4, dtype=torch.complex64, device="cuda")
        _lib.call("chm_sp_carrier", tab.data_ptr(), tab.numel(), KX0, 0.0, DX, 1, st, None)
        _lib.call("chm_sp_gather_push_env", *[b.data_ptr() for b in P], total, 1, 0.25, 1 / DR, eb.data_ptr(),
                  NX, NR, nm, 0.1, tab.data_ptr(), tab.numel(), KX0 * DX, 1, und.ctypes.data, None, 0, 0.0,
                  DX, st, None)
        out.append([b[phys].clone() for b in P])
    for a, b in zip(*out):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("order", [False, True])
@pytest.mark.parametrize("n", [1, 15, 17, 512, 513, 30001, 152 * 8 * 512, 152 * 8 * 512 + 1])
@pytest.mark.parametrize("nm", [1, 3, 5])
def test_deposit_in_pieces(cuda, nm, n, order):
    import torch
    from chimera_gb300 import _lib
    from chimera_gb300 import fimera as fm
    st = torch.cuda.current_stream().cuda_stream
    P, _ = _beam(torch, n, n, order)
    ptr = [b.data_ptr() for b in P]
    x = fm.fortran_zeros((3, n), torch.float64)
    p = fm.fortran_zeros((3, n), torch.float64)
    w = torch.zeros(n, dtype=torch.float64, device="cuda")
    _lib.call("chm_sp_to_f64", *ptr, n, x.data_ptr(), x.stride(0), x.stride(1), p.data_ptr(), p.stride(0),
              p.stride(1), w.data_ptr(), w.stride(0), 0.0, DX, st)
    wsum = float(w.sum())
    e = 61.0 - np.ceil(np.log2(wsum))
    scale = torch.tensor([2.0 ** e, wsum], dtype=torch.float64, device="cuda")
    tab = torch.zeros(NX + 4, dtype=torch.complex64, device="cuda")
    _lib.call("chm_sp_carrier", tab.data_ptr(), tab.numel(), KX0, 0.0, DX, 1, st, None)
    acc = torch.zeros((3, nm, NR, NX, 2), dtype=torch.int64, device="cuda")
    _lib.call("chm_sp_push_deposit_env", *ptr, n, 1, 0.25, 1 / DX, 1 / DR, DT, DX, NX, NR, nm, acc.data_ptr(),
              scale.data_ptr(), tab.data_ptr(), tab.numel(), KX0 * DX, st, None)
    got = acc[2].double().cpu().numpy() / 2.0 ** e
    half = fm.fortran_zeros((3, n), torch.float64)
    fm.push_coords(x, p, half, DT)
    rg = DR * (np.arange(NR) - 0.5)
    J = fm.fortran_zeros((NX, NR, nm, 3))
    fm.dep_curr_env(half, p, w, J, 1.25 * DX, rg, 1 / DX, 1 / DR, KX0)
    D = fm.fortran_zeros((NX, NR, 1))
    fm.dep_dens(half, w, D, 1.25 * DX, rg, 1 / DX, 1 / DR)
    want = J[..., 2].cpu().numpy().transpose(2, 1, 0)
    mag = np.abs(D[..., 0].cpu().numpy().real.T)
    mag[0] = mag[1]  # (the ghost row is folded away)
    near = np.pad(mag, 1)
    near = sum(near[1 + a:1 + a + NR, 1 + b:1 + b + NX] for a in (-1, 0, 1) for b in (-1, 0, 1))
    J2 = got[..., 0] + 1j * got[..., 1]
    J2[:, 1] -= J2[:, 0]
    J2[:, 0] = 0
    tol = 2.0 ** -24 * ((17 + 40) + 4 * NR + 8) * 2 * near
    assert np.all(np.abs(J2 - want) <= tol[None])
    assert n < 512 or np.abs(want).max() > 0
