"""The transforms along x over lengths: every radix of the register passes
(csrc/fft_mixed.cuh) as first, middle and last pass, lengths that fill a block
unevenly, the power-of-two passes, and lengths with a prime factor above 13
that take the general passes; few lines and many (other radices); both
precisions, through the absorbing layer's filter (backward, profile at the
edges, forward).

Bound: Gentleman and Sande (1966) for a transform with prime factors p,
||err|| <= 1.06 u ||x|| sum (2 p)^(3/2), u the unit roundoff, for both
transforms and for numpy's own (the doubled factor), and 20 u for the phases
and the profile, whose values are at most 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 22, 26, 30, 33, 34, 35, 49, 51,
           64, 77, 81, 91, 100, 120, 121, 143, 169, 210, 243, 256, 323, 360, 384, 480, 500, 512, 600, 625,
           686, 858, 1000, 1001, 1024, 1100, 1331, 1500, 1536, 1800, 2000, 2041, 2048, 2197, 2310, 2401,
           3000, 3003, 3072, 3125, 3600, 4004, 4050, 4094, 4095, 4096]


def _factors(n):
    out, p = [], 2
    while n > 1:
        while n % p == 0:
            out.append(p)
            n //= p
        p += 1
    return out


def _case(n, rows, mode):
    rng = np.random.default_rng(n)
    shape = (n, rows, 1, 2)
    v = np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    kx = 2 * np.pi * np.fft.fftfreq(n, 0.1)
    nf = (n + 3) // 4
    prof = np.linspace(0.0, 1.0, nf + 1)[1:]
    left = -1.7
    sh = np.exp(1j * kx * left)[:, None, None, None]
    a = n * np.fft.ifft(v * sh, axis=0)
    if mode in (0, 2):
        a[:nf] *= prof[:, None, None, None]
    if mode in (1, 2):
        a[n - nf:] *= prof[::-1, None, None, None]
    return v, kx, prof, left, np.fft.fft(a, axis=0) / (n * sh)


def _check(got, want, v, n, u):
    c = 2 * 2 * 1.06 * sum((2.0 * p) ** 1.5 for p in _factors(n)) + 20
    err = np.linalg.norm(got - want, axis=0)
    assert np.all(err <= c * u * np.linalg.norm(v, axis=0))


@pytest.mark.parametrize("rows", [3, 311])
@pytest.mark.parametrize("n", LENGTHS)
def test_fp64(cuda, n, rows):
    import torch
    from chimera_gb300 import fimera
    v, kx, prof, left, want = _case(n, rows, n % 3)
    t = torch.from_numpy(v).cuda()
    got = fimera.fb_filtr(t, left, kx, prof, n % 3).cpu().numpy()
    _check(got, want, v, n, 2.0 ** -53)


@pytest.mark.parametrize("rows", [3, 311])
@pytest.mark.parametrize("n", LENGTHS)
def test_fp32(cuda, n, rows):
    import torch
    from chimera_gb300 import _lib
    v, kx, prof, left, _ = _case(n, rows, n % 3)
    v = v.astype(np.complex64)
    prof32 = prof.astype(np.float32)
    sh = np.exp(1j * kx * left)[:, None, None, None]
    a = n * np.fft.ifft(v.astype(complex) * sh, axis=0)
    nf = prof.size
    if n % 3 in (0, 2):
        a[:nf] *= prof32[:, None, None, None]
    if n % 3 in (1, 2):
        a[n - nf:] *= prof32[::-1, None, None, None]
    want = np.fft.fft(a, axis=0) / (n * sh)
    t = torch.from_numpy(np.ascontiguousarray(v.transpose(3, 2, 1, 0))).cuda()
    f = torch.from_numpy(prof32).cuda()
    k = torch.from_numpy(kx).cuda()
    ws = torch.empty(2 * (8 * n + 256), dtype=torch.uint8, device="cuda")
    _lib.call("chm_sp_fb_filtr", t.data_ptr(), left, k.data_ptr(), f.data_ptr(), nf, n % 3, n, rows, 1, 2,
              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream, None)
    got = t.cpu().numpy().transpose(3, 2, 1, 0)
    _check(got, want, v, n, 2.0 ** -24)
