"""The transforms along x with few lines and with many: the register passes choose
their radices by the number of lines (csrc/fft_mixed.cuh, at 2048 values an SM), and
short lengths reach the plan for many lines with tens of thousands of lines only.
Every length has launches on both sides of the line, with blocks of one warp and
more and lengths of a single pass.  Input, reference and bound as in
test_zy_fft_gpu.py."""
import numpy as np
import pytest
from test_zy_fft_gpu import _case, _check

pytestmark = pytest.mark.gpu

LENGTHS = [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 22, 30, 49, 64, 77, 90, 117, 120, 128, 143, 154,
           169, 182, 210, 225, 243, 256, 260, 300, 343, 360, 392, 450, 462, 500]


def _rows(n, many):
    import torch
    line = 2048 * torch.cuda.get_device_properties(0).multi_processor_count
    rows = line // (2 * n) + (1 if many else 0)  # of two components
    assert (2 * rows * n > line) == many
    return rows


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("n", LENGTHS)
def test_fp64(cuda, n, many):
    import torch
    from chimera_gb300 import fimera
    v, kx, prof, left, want = _case(n, _rows(n, many), n % 3)
    got = fimera.fb_filtr(torch.from_numpy(v).cuda(), left, kx, prof, n % 3).cpu().numpy()
    _check(got, want, v, n, 2.0 ** -53)


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("n", [n for n in LENGTHS if n & (n - 1)])
def test_fp32(cuda, n, many):
    import torch
    from chimera_gb300 import _lib
    rows = _rows(n, many)
    v, kx, prof, left, _ = _case(n, rows, n % 3)
    v = v.astype(np.complex64)
    prof32 = prof.astype(np.float32)
    nf = prof.size
    sh = np.exp(1j * kx * left)[:, None, None, None]
    a = n * np.fft.ifft(v.astype(complex) * sh, axis=0)
    if n % 3 in (0, 2):
        a[:nf] *= prof32[:, None, None, None]
    if n % 3 in (1, 2):
        a[n - nf:] *= prof32[::-1, None, None, None]
    want = np.fft.fft(a, axis=0) / (n * sh)
    t = torch.from_numpy(np.ascontiguousarray(v.transpose(3, 2, 1, 0))).cuda()
    f, k = torch.from_numpy(prof32).cuda(), torch.from_numpy(kx).cuda()
    ws = torch.empty(2 * (8 * n + 256), dtype=torch.uint8, device="cuda")
    _lib.call("chm_sp_fb_filtr", t.data_ptr(), left, k.data_ptr(), f.data_ptr(), nf, n % 3, n, rows, 1, 2,
              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream, None)
    _check(t.cpu().numpy().transpose(3, 2, 1, 0), want, v, n, 2.0 ** -24)
