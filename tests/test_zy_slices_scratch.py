"""Scratch of the FP64 products' operand slices: a batch holds at most 48 products,
so more planes take no more; and such a transform is right (GPU)."""
import numpy as np
import pytest


def test_slices_of_at_most_one_batch():
    from chimera_gb300 import _lib
    q = lambda nm, ncomp: _lib.query("chm_fb_slices_bytes", 256, 129, 128, nm, ncomp)  # noqa: E731
    plane = q(1, 2) - q(1, 1)
    matrix = q(2, 1) - q(1, 2)
    rest = q(1, 1) - plane - matrix
    assert plane > 0 and matrix > 0 and rest >= 0
    for nm, ncomp in ((16, 3), (20, 3), (48, 1), (60, 1), (60, 3)):
        assert q(nm, ncomp) == min(nm * ncomp, 48) * plane + min(nm, 48) * matrix + rest


@pytest.mark.gpu
@pytest.mark.parametrize("nm,ncomp", [(16, 3), (17, 3), (33, 3)])
def test_transform_of_more_planes_than_a_batch(cuda, nm, ncomp):
    """Against the FP64 pipe (a workspace without room for the slices): K + 2
    roundings of sum |a b| each, and the transform's own."""
    import torch
    from chimera_gb300 import _lib, fimera as fm
    nx, nr, nkr = 36, 23, 20
    rng = np.random.default_rng(nm)
    dev = lambda a: torch.from_numpy(np.asfortranarray(a)).cuda()  # noqa: E731
    v = rng.standard_normal((nx, nr, nm, ncomp)) + 1j * rng.standard_normal((nx, nr, nm, ncomp))
    In = rng.standard_normal((nr - 1, nkr, nm))
    dv, dI, kx = dev(v), dev(In), torch.zeros(nx, dtype=torch.float64, device="cuda")
    got = []
    for name in ("chm_fb_ws_bytes", "chm_fb_planes_bytes"):
        n = _lib.query(name, nx, nr, nkr, nm, ncomp)
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        out = fm.fortran_zeros((nx, nkr, nm, ncomp))
        _lib.call("chm_fb_in", out.data_ptr(), dv.data_ptr(), 0.0, kx.data_ptr(), dI.data_ptr(), None, nx, nr, nkr,
                  nm, ncomp, ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
        got.append(out.cpu().numpy())
    f = np.fft.fft(v[:, 1:], axis=0)
    want = np.einsum("xrmc,rkm->xkmc", f, In)
    bound = np.einsum("xrmc,rkm->xkmc", np.abs(f.real) + np.abs(f.imag), np.abs(In))
    assert np.all(np.abs(got[0] - got[1]) <= 2 * (nr + 1) * 2.0 ** -53 * bound)
    assert np.linalg.norm(got[0] - want) <= 1e-13 * np.linalg.norm(want)
