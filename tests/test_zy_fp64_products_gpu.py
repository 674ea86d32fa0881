"""The FP64 form's products on the tensor cores (exact integer slices,
csrc/tc_ozaki.cu) against sums in longer precision, at the edges of the row
and column tiles and of the 256-value accumulation chunks.

Bound of an output, c the number of 256-value chunks: a chunk's sum has a unit
of 2^-54 of 2^(ea+eb) <= 4 max|a| max|b| (the row's and the column's largest
elements), is off by at most a unit and a half (the dropped digits and one
rounding) and is rounded once to FP64, and the chunks are added in FP64:
|err| <= c (2^-51.4 max|a| max|b| + 2^-52 sum |a b|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods(cuda):
    import torch
    from chimera_gb300 import _lib, fimera
    return torch, _lib, fimera


def _dev(torch, a):
    return torch.from_numpy(np.asfortranarray(a)).cuda()


def _product(mods, s, D):
    """s (nx, K) complex times D (K, K), as the upper-neighbour product of
    fb_grad's mode 0 (component 2, with a zero lower operator)."""
    torch, _lib, fm = mods
    nx, K = s.shape
    S = np.zeros((nx, K, 2), complex, order="F")
    S[:, :, 1] = s
    Dp = np.zeros((K, K, 3), order="F")
    Dp[:, :, 0] = D
    out = fm.fortran_zeros((nx, K, 2, 3))
    kx = torch.zeros(nx, dtype=torch.float64, device="cuda")
    fm.fb_grad(out, _dev(torch, S), _dev(torch, Dp), _dev(torch, np.zeros((K, K, 3))), kx)
    return out[:, :, 0, 1].cpu().numpy()


def _bound(a, b, K):
    c = -(-K // 256)
    big = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None]
    return c * (2.0 ** -51.4 * big + 2.0 ** -52 * (np.abs(a) @ np.abs(b)))


def _data(kind, nx, K, rng):
    s = rng.standard_normal((nx, K)) + 1j * rng.standard_normal((nx, K))
    D = rng.standard_normal((K, K))
    if kind == "peaked":  # rows falling off over 60 orders of magnitude
        s *= np.exp(-np.linspace(0, 12, K) ** 2)
    elif kind == "digits":  # every digit at its extreme
        v = float.fromhex("0x1.fefefefefefefp-1")
        s[...], D[...] = v * (1 - 1j), v
    elif kind == "scales":  # rows and columns of very different sizes
        s *= 10.0 ** rng.integers(-120, 120, (nx, 1))
        D *= 10.0 ** rng.integers(-30, 30, (1, K))
    return s, D


@pytest.mark.parametrize("kind", ["random", "peaked", "digits", "scales"])
@pytest.mark.parametrize("nx,K", [(1, 1), (3, 5), (65, 17), (64, 64), (129, 50), (37, 130), (64, 256),
                                  (33, 257), (20, 520)])
def test_product_within_its_bound(mods, nx, K, kind):
    rng = np.random.default_rng(100 * nx + K)
    s, D = _data(kind, nx, K, rng)
    got = _product(mods, s, D)
    for g, a in ((got.real, s.real), (got.imag, s.imag)):
        ref = a.astype(np.longdouble) @ D.astype(np.longdouble)
        assert np.all(np.abs(g - ref) <= _bound(a, D, K))
    assert mods[1].load().chm_sp_umma_status() == 0


def test_integers_are_exact(mods):
    rng = np.random.default_rng(4)
    s = rng.integers(-2 ** 26, 2 ** 26, (40, 256)).astype(float)
    D = rng.integers(-2 ** 18, 2 ** 18, (256, 256)).astype(float)
    got = _product(mods, s + 1j * s[::-1], D)
    want = s.astype(np.int64) @ D.astype(np.int64)  # below 2^52
    assert np.array_equal(got.real, want.astype(float))
    assert np.array_equal(got.imag, want[::-1].astype(float))


def test_infinities_and_nans_stay_in_their_rows_and_columns(mods):
    rng = np.random.default_rng(5)
    s = rng.standard_normal((48, 40)) + 1j * rng.standard_normal((48, 40))
    D = rng.standard_normal((40, 40))
    good = _product(mods, s, D)
    bad = s.copy()
    bad.real[3, 5] = np.inf
    bad.imag[7, 9] = np.nan
    got = _product(mods, bad, D)
    # fb_grad also reads row -x of the mode as the lower neighbour, times zero
    for part, row, x in ((got.real, 3, 45), (got.imag, 7, 41)):
        assert not np.isfinite(part[row]).any() and np.isnan(part[x]).all()
    keep = np.setdiff1d(np.arange(48), [3, 45])
    assert np.array_equal(got.real[keep], good.real[keep])
    D2 = D.copy()
    D2[4, 6] = -np.inf
    got = _product(mods, s, D2)
    assert np.array_equal(got.real[:, 6], np.where(s.real[:, 4] > 0, -np.inf, np.inf))
    assert np.array_equal(np.delete(got, 6, 1), np.delete(good, 6, 1))


@pytest.mark.parametrize("K,N", [(16, 16), (40, 100), (200, 72), (300, 256)])
def test_rectangular_product_no_less_exact_than_the_fp64_pipe(mods, K, N):
    """chm_fb_in of a line that is a delta in x (its transform is constant):
    on the tensor cores with the queried workspace, on the FP64 pipe with only
    the transform's own planes; both against the longer sum."""
    torch, _lib, fm = mods
    nx = 64
    rng = np.random.default_rng(K + N)
    v = rng.standard_normal(K) + 1j * rng.standard_normal(K)
    In = rng.standard_normal((K, N))
    vec = np.zeros((nx, K + 1, 1), complex, order="F")
    vec[0, 1:, 0] = v
    dv, dI = _dev(torch, vec), _dev(torch, In.reshape(K, N, 1))
    kx = torch.zeros(nx, dtype=torch.float64, device="cuda")
    full = _lib.query("chm_fb_ws_bytes", nx, K + 1, N, 1, 1)
    r256 = lambda b: (b + 255) // 256 * 256  # noqa: E731
    base = 2 * r256(16 * nx) + r256(16 * nx * max(K, N)) + 256
    ref = v.real.astype(np.longdouble) @ In.astype(np.longdouble)
    errs = []
    for nbytes in (full, base):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        out = fm.fortran_zeros((nx, N, 1))
        _lib.call("chm_fb_in", out.data_ptr(), dv.data_ptr(), 0.0, kx.data_ptr(), dI.data_ptr(), None, nx,
                  K + 1, N, 1, 1, ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
        got = out[:, :, 0].cpu().numpy().real
        assert np.array_equal(got, np.broadcast_to(got[:1], got.shape))
        d = (got[0] - ref).astype(float)
        assert np.all(np.abs(d) <= _bound(v.real[None], In, K)[0] * (1 if nbytes == full else K))
        errs.append(np.linalg.norm(d))
    assert errs[0] <= errs[1]
    with pytest.raises(_lib.ChimeraError):  # less than the transform's planes stays refused
        _lib.call("chm_fb_in", out.data_ptr(), dv.data_ptr(), 0.0, kx.data_ptr(), dI.data_ptr(), None, nx,
                  K + 1, N, 1, 1, ws.data_ptr(), base - 1, torch.cuda.current_stream().cuda_stream)
