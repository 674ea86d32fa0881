"""The FP64 form's products on the tensor cores (csrc/tc_ozaki.cu) where the
elements of a row or a column spread over many powers of two: the spectra of
smooth fields times the solver's own mode-coupling operators, and operands made
so that the large elements of a row meet the small ones of a column.

Truth: sums in longer precision (numpy longdouble).  Next to each product on the
tensor cores stands the FP64 pipe's, from the same entry point with a workspace
that has no room for the operand slices.

Bound of an output, c the number of 256-value chunks: an output that the slices
give has sum |a b| >= 2^-12 of 2^(ea + eb); what the slices leave out is 2^-66 of
2^(ea + eb) rms over random digits, 2^-62 are 16 deviations; a chunk is rounded
once.  An output summed in FP64 has K roundings:
|err| <= max(c (2^-50 + 2^-52), K 2^-53) sum |a b|."""
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


def _grad(mods, S, Dp, Dm, slices):
    """chm_fb_grad of a scalar of two modes; the products on the tensor cores
    (slices) or on the FP64 pipe."""
    torch, _lib, fm = mods
    nx, K, nm = S.shape
    out = fm.fortran_zeros((nx, K, nm, 3))
    kx = torch.zeros(nx, dtype=torch.float64, device="cuda")
    n = _lib.query("chm_fbmath_ws_bytes" if slices else "chm_fbmath_planes_bytes", nx, K, nm)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    t = [_dev(torch, a) for a in (S, Dp, Dm)]
    _lib.call("chm_fb_grad", out.data_ptr(), *(a.data_ptr() for a in t), kx.data_ptr(), nx, K, nm, 0, ws.data_ptr(),
              n, torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    assert _lib.load().chm_sp_umma_status() == 0
    return got


def _upper(mods, s, D, slices):
    """s (nx, K) complex times D (K, K): mode 1 as mode 0's upper neighbour."""
    nx, K = s.shape
    S = np.zeros((nx, K, 2), complex, order="F")
    S[:, :, 1] = s
    Dp = np.zeros((K, K, 3), order="F")
    Dp[:, :, 0] = D
    return _grad(mods, S, Dp, np.zeros((K, K, 3)), slices)[:, :, 0, 1]


def _errors(got, a, b):
    """(norm of the error over the result's, median and largest of |err| / sum |a b|)"""
    ref = a.astype(np.longdouble) @ b.astype(np.longdouble)
    err = np.abs((got - ref).astype(float))
    G = np.abs(a) @ np.abs(b)
    r = err[G > 0] / G[G > 0]
    assert np.all(err[G == 0] == 0)
    return np.linalg.norm(err) / np.linalg.norm(ref.astype(float)), np.median(r), r.max()


def _limit(K):
    return max(-(-K // 256) * (2.0 ** -50 + 2.0 ** -52), K * 2.0 ** -53)


def _operators(nkr, dr):
    from chimera_gb300.solvers import spectral_operators
    R = dr * (np.arange(nkr + 1) - 0.5)
    return spectral_operators(dict(Nx=4, Nkr=nkr, Nko=1, lengthR=dr * nkr, kx=np.arange(4.0), RgridFull=R), ext=1)


@pytest.mark.parametrize("nkr,dr", [(64, 0.4), (256, 0.4), (300, 0.2)])
@pytest.mark.parametrize("kind", ["gauss", "narrow", "steep", "pulse", "noise"])
def test_couplings_of_smooth_spectra_no_less_exact_than_the_fp64_pipe(mods, nkr, dr, kind):
    In, _, Dp, Dm = _operators(nkr, dr)[:4]
    r = dr * (np.arange(nkr) + 0.5)
    rng = np.random.default_rng(nkr)
    nx = 48
    white = rng.standard_normal((nx, nkr)) + 1j * rng.standard_normal((nx, nkr))
    if kind == "noise":
        s = white
    elif kind == "steep":
        s = white * np.exp(-np.linspace(0, 25, nkr))
    else:
        w = nkr * dr * (0.06 if kind == "narrow" else 0.2)
        f = (white[:, :1] if kind != "pulse" else np.exp(-np.linspace(-2, 2, nx)[:, None] ** 2 + 0j)) * np.exp(
            -(r / w) ** 2)
        if kind == "pulse":  # with the noise floor of a run's deposits
            f = f + 1e-8 * white
        s = f @ In[:, :, 0]
    for D in (Dp[:, :, 0], Dm[:, :, 1]):
        got, pipe = (_upper(mods, s, D, k) for k in (True, False))
        e = np.array([_errors(g, a, D) for g, a in ((got.real, s.real), (got.imag, s.imag)) if a.any()])
        p = np.array([_errors(g, a, D) for g, a in ((pipe.real, s.real), (pipe.imag, s.imag)) if a.any()])
        assert np.all(e[:, 2] <= _limit(nkr))
        assert np.all(e[:, :2] <= p[:, :2]), (e, p)


def _apart(K, rng):
    """a falling row meets columns that rise as powers of k"""
    k = np.arange(1, K + 1)
    a = rng.standard_normal((40, K)) * np.exp(-(k / 2.0) ** 2 / 4)
    return a, k[:, None] ** rng.integers(0, 9, K)[None] * rng.uniform(1, 2, (K, K))


def _blocks(K, rng):
    """a matrix of two blocks of very different size"""
    D = rng.standard_normal((K, K))
    h = K // 2
    D[h:, :h] = D[:h, h:] = 0
    D[h:, h:] *= 1e-30
    return rng.standard_normal((40, K)), D


def _digits(K, rng, vary=0):
    """every digit below the first at its extreme (or next to it), the largest
    elements apart; a scale of one for every K value"""
    def low(shape):
        return -sum(rng.integers(128 - vary, 129, shape) * 256.0 ** -i for i in range(1, 7)) / 64
    a, D = low((40, K)), low((K, K))
    a[:, 0] = 1 - 2.0 ** -53
    D[:, K - 1] = 1 - 2.0 ** -53
    D[1 % K, :] = 1 - 2.0 ** -53
    D[0, : K - 1] = 0.0
    return a, D


def _odd_digits(K, rng):
    """sums of S_5 and S_6 that pass 2^24 in odd steps"""
    return _digits(K, rng, 1)


def _tiny(K, rng):
    """products below and at the end of the normal range, and sums of zeros"""
    a, D = rng.standard_normal((40, K)), rng.standard_normal((K, K))
    a[:20] *= 1e-290
    a[30] = 0
    D *= 10.0 ** rng.integers(-40, 1, (1, K))
    D[:, K // 2] = 0
    D[K // 3] = 0
    return a, D


@pytest.mark.parametrize("K", [1, 17, 64, 256, 257])
@pytest.mark.parametrize("make", [_apart, _blocks, _digits, _odd_digits])
def test_large_elements_that_meet_small_ones(mods, make, K):
    a, D = make(K, np.random.default_rng(K))
    got = _upper(mods, a + 1j * a[::-1], D, True)
    for g, x in ((got.real, a), (got.imag, a[::-1])):
        assert _errors(g, x, D)[2] <= _limit(K)


@pytest.mark.parametrize("K", [5, 40, 260])
def test_small_sums_and_reflected_rows(mods, K):
    """The block of 1e-30 is below the slices' resolution: its outputs are FP64 sums,
    also as the reflected lower neighbour (whole rows of the warps in the FP64
    pipe's order, bit for bit; the 6 rows of the last tile one by one)."""
    rng = np.random.default_rng(K)
    nx, h = 67, K // 2
    s = rng.standard_normal((nx, K, 2)) + 1j * rng.standard_normal((nx, K, 2))
    D = np.zeros((K, K, 3))
    D[:, :, 0] = _blocks(K, rng)[1]
    refl = -s[(-np.arange(nx)) % nx, :, 1].conj()
    for Dp, Dm, a, sign in ((D, 0 * D, s[:, :, 1], 1), (0 * D, D, refl, -1)):
        got, pipe = (_grad(mods, s, Dp, Dm, k)[:, :, 0, 1] * sign for k in (True, False))
        assert np.array_equal(got[:64, h:], pipe[:64, h:]) and 0 < np.abs(got[:, h:]).max() < 1e-25
        for g, x in ((got.real, a.real), (got.imag, a.imag)):
            assert _errors(g, np.ascontiguousarray(x), D[:, :, 0])[2] <= _limit(K)


@pytest.mark.parametrize("K", [5, 40, 260])
def test_products_at_the_end_of_the_range(mods, K):
    """(within the bound, plus a unit of the smallest number a term)"""
    a, T = _tiny(K, np.random.default_rng(K))
    g = _upper(mods, a + 0j, T, True).real
    ref = a.astype(np.longdouble) @ T.astype(np.longdouble)
    assert np.all(np.abs(g - ref) <= _limit(K) * (np.abs(a) @ np.abs(T)) + K * 2.0 ** -1074)


@pytest.mark.parametrize("K,N", [(40, 100), (300, 256), (9001, 16)])
def test_transform_of_a_steep_profile(mods, K, N):
    """chm_fb_in (the phase and factor epilogue) of a line that is a delta in x,
    of two components that share the matrix, over a steep profile."""
    torch, _lib, fm = mods
    nx = 64
    rng = np.random.default_rng(K + N)
    v = rng.standard_normal((K, 2)) * np.exp(-np.linspace(0, 6, K) ** 2)[:, None]
    In = rng.standard_normal((K, N)) * np.linspace(1, 100, K)[:, None] ** 3
    fact = rng.uniform(1, 2, (nx, N))
    vec = np.zeros((nx, K + 1, 1, 2), complex, order="F")
    vec[0, 1:, 0, :] = v
    dv, dI, df = _dev(torch, vec), _dev(torch, In.reshape(K, N, 1)), _dev(torch, fact.reshape(nx, N, 1))
    kx = torch.zeros(nx, dtype=torch.float64, device="cuda")
    n = _lib.query("chm_fb_ws_bytes", nx, K + 1, N, 1, 2)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    out = fm.fortran_zeros((nx, N, 1, 2))
    _lib.call("chm_fb_in", out.data_ptr(), dv.data_ptr(), 0.0, kx.data_ptr(), dI.data_ptr(), df.data_ptr(), nx,
              K + 1, N, 1, 2, ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    assert not got.imag.any()
    for c in range(2):
        ref = (v[:, c].astype(np.longdouble) @ In.astype(np.longdouble))[None] * fact.astype(np.longdouble)
        G = (np.abs(v[:, c]) @ np.abs(In))[None] * fact
        # (two roundings more: the phase's and the factor's product)
        assert np.all(np.abs(got[:, :, 0, c].real - ref) <= (_limit(K) + 2.0 ** -52) * G)


def test_long_sums_in_fp64_do_not_run_into_the_wait_limit(mods):
    """Every output of the 32 rows below the slices' resolution, over 65536 terms:
    the FP64 pipe's bits, and no wait gives up meanwhile."""
    torch, _lib, fm = mods
    nx, K, N = 16, 65536, 16
    rng = np.random.default_rng(8)
    vec = np.zeros((nx, K + 1, 1), complex, order="F")
    vec[:, 1:, 0] = rng.standard_normal((nx, K)) + 1j * rng.standard_normal((nx, K))
    In = np.zeros((K, N), order="F")  # column 0 sets the scales; the others live where it is small
    In[: K // 2, 0] = 1.0
    In[K // 2:] = 1e-30 * rng.standard_normal((K - K // 2, N))
    dv, dI = _dev(torch, vec), _dev(torch, In.reshape(K, N, 1))
    kx = torch.zeros(nx, dtype=torch.float64, device="cuda")
    got = []
    for name in ("chm_fb_ws_bytes", "chm_fb_planes_bytes"):
        n = _lib.query(name, nx, K + 1, N, 1, 1)
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        out = fm.fortran_zeros((nx, N, 1))
        _lib.call("chm_fb_in", out.data_ptr(), dv.data_ptr(), 0.0, kx.data_ptr(), dI.data_ptr(), None, nx, K + 1, N, 1,
                  1, ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
        got.append(out.cpu().numpy())
    assert _lib.load().chm_sp_umma_status() == 0
    assert np.array_equal(got[0][:, 1:], got[1][:, 1:]) and 0 < np.abs(got[0][:, 1:]).max() < 1e-20
