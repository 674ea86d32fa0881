"""The wait limit of the FP64 form's products on the tensor cores (csrc/tc_ozaki.cu):
with a limit of 0 every pipeline wait gives up at once.  The kernel then reports it,
its outputs hold NaN, it frees its tensor memory, and the next launch at the default
limit is right.  (No wait depends on anything but the launch itself.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,K,nm", [(40, 24, 2), (1024, 256, 2), (300, 300, 3)])
def test_wait_limit_reports_fills_with_nan_and_recovers(cuda, nx, K, nm):
    import torch
    from chimera_gb300 import _lib, fimera as fm
    lib = _lib.load()
    rng = np.random.default_rng(nx)
    dev = lambda a: torch.from_numpy(np.asfortranarray(a)).cuda()  # noqa: E731
    vec = dev(rng.standard_normal((nx, K, nm, 3)) + 1j * rng.standard_normal((nx, K, nm, 3)))
    Dp, Dm = (dev(rng.standard_normal((K, K, nm + 1))) for _ in range(2))
    kx = dev(rng.standard_normal(nx))
    run = lambda: fm.fb_rot(fm.fortran_zeros((nx, K, nm, 3)), vec, Dp, Dm, kx).cpu().numpy()  # noqa: E731
    good = run()
    assert np.isfinite(good).all() and lib.chm_sp_umma_status() == 0
    prev = lib.chm_sp_set_umma_spin_limit(0)
    try:
        got = run()
    finally:
        lib.chm_sp_set_umma_spin_limit(prev)
    assert np.isnan(got).all()  # every output takes part of a product
    assert 11 <= lib.chm_sp_umma_status() <= 15
    assert lib.chm_sp_umma_status() == 0  # read and reset
    assert np.array_equal(run(), good)
    assert lib.chm_sp_umma_status() == 0
