"""An FP64 transform whose device has no memory for the operand slices still runs:
its products go to the FP64 pipe, with the FP64 pipe's bits."""
import types

import numpy as np
import pytest
import torch

from chimera_gb300 import _lib, fimera


@pytest.fixture
def refuse(monkeypatch):
    """workspace() without memory for slices of `limit` bytes or more."""
    asked, real = [], fimera.workspace
    state = types.SimpleNamespace(limit=0, asked=asked, fake=False)

    def workspace(nbytes, device=None, kind=""):
        asked.append((kind, nbytes))
        if kind == "slices" and nbytes >= state.limit:
            raise torch.cuda.OutOfMemoryError("no memory")
        return torch.empty(nbytes, dtype=torch.uint8) if state.fake else real(nbytes, device, kind)

    monkeypatch.setattr(fimera, "workspace", workspace)
    monkeypatch.setattr(fimera, "_slices_refused", {})
    monkeypatch.setattr(fimera, "_ws_cache", {})  # (a larger one has room for the slices)
    return state


def test_scratch_without_memory(refuse, monkeypatch):
    refuse.fake, refuse.limit = True, 1000
    need = {"chm_fb_planes_bytes": 500, "chm_fb_slices_bytes": 1000}
    monkeypatch.setattr(_lib, "query", lambda name, *a: need[name])
    assert fimera._scratch("fb")[1:] == (500, None, 0)
    assert fimera._scratch("fb")[1:] == (500, None, 0)
    assert refuse.asked.count(("slices", 1000)) == 1  # refused once, not asked for again
    need["chm_fb_slices_bytes"] = 900  # a smaller call still gets its slices
    ws = fimera._scratch("fb")
    assert ws[1] == 500 and ws[2] and ws[3] == 900


@pytest.mark.gpu
def test_transform_without_memory_for_slices(cuda, refuse):
    nx, K, nm = 64, 40, 2
    rng = np.random.default_rng(3)
    dev = lambda a: torch.from_numpy(np.asfortranarray(a)).cuda()  # noqa: E731
    vec = dev(rng.standard_normal((nx, K, nm, 3)) + 1j * rng.standard_normal((nx, K, nm, 3)))
    Dp, Dm = (dev(rng.standard_normal((K, K, nm + 1))) for _ in range(2))
    kx = dev(rng.standard_normal(nx))
    run = lambda: fimera.fb_rot(fimera.fortran_zeros((nx, K, nm, 3)), vec, Dp, Dm, kx)  # noqa: E731
    got = run().cpu().numpy()
    out = fimera.fortran_zeros((nx, K, nm, 3))
    n = _lib.query("chm_fbmath_planes_bytes", nx, K, nm)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _lib.call("chm_fb_rot", out.data_ptr(), vec.data_ptr(), Dp.data_ptr(), Dm.data_ptr(), kx.data_ptr(), nx, K, nm, 0,
              ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(got, out.cpu().numpy())
    refuse.limit = float("inf")
    fimera._slices_refused.clear()
    tc = run().cpu().numpy()
    assert not np.array_equal(tc, got) and np.linalg.norm(tc - got) <= 1e-14 * np.linalg.norm(got)
