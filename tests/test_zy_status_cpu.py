"""The step loop reads the products' device error flag every check_every steps and
before a snapshot, and raises on it (a fake of the library's status call)."""
import pytest

from chimera_gb300 import _lib, fimera
from chimera_gb300.chimera_main import ChimeraRun


class FakeLib:
    code = 0
    reads = 0

    def chm_sp_umma_status(self):
        self.reads += 1
        code, self.code = self.code, 0
        return code


@pytest.fixture
def lib(monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(_lib, "load", lambda: fake)
    return fake


def test_check_status(lib):
    fimera.check_status()
    lib.code = 13
    with pytest.raises(_lib.ChimeraError, match="13"):
        fimera.check_status()
    fimera.check_status()


def test_step_loop_and_snapshot(lib, tmp_path):
    run = ChimeraRun({"MovingFrames": ()})
    for i in range(63):
        run.make_step(i)
    assert lib.reads == 0
    lib.code = 14
    with pytest.raises(_lib.ChimeraError):
        run.make_step(63)
    lib.code = 14
    with pytest.raises(_lib.ChimeraError):
        run.drop_snap(str(tmp_path / "s_"))
    assert not list(tmp_path.iterdir())
    run.check_every = 0
    lib.code = 14
    for i in range(64):
        run.make_step(64 + i)
    assert lib.code == 14
