"""_lib.raw_stream where torch has, or lacks, its raw-stream function (fakes)."""
import types

import torch

from chimera_gb300 import _lib


def test_raw_stream(monkeypatch):
    stream = lambda i=None: types.SimpleNamespace(cuda_stream=100 + (2 if i is None else i))  # noqa: E731
    monkeypatch.setattr(torch.cuda, "current_stream", stream)
    want = [(None, 102), (torch.device("cuda", 1), 101), (torch.device("cuda"), 102)]
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 2, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 100 + i, raising=False)
    assert [_lib.raw_stream(d) for d, _ in want] == [s for _, s in want]
    monkeypatch.delattr(torch._C, "_cuda_getDevice")
    assert [_lib.raw_stream(d) for d, _ in want] == [s for _, s in want]
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    assert [_lib.raw_stream(d) for d, _ in want] == [s for _, s in want]
