"""Following torch's current stream with and without torch's raw stream handle
(CPU: torch and the library are stand-ins)."""
from types import SimpleNamespace

import pytest

from memory_database_b200 import olapcore


@pytest.mark.parametrize("raw_handle", [True, False])
def test_follows_the_current_stream(monkeypatch, raw_handle):
    current, seen = {0: 0, 1: 4242}, []
    torch = SimpleNamespace(_C=SimpleNamespace(), cuda=SimpleNamespace())
    if raw_handle:
        torch._C._cuda_getCurrentRawStream = lambda device: current[device]
    else:
        torch.cuda.current_stream = lambda device: SimpleNamespace(cuda_stream=current[device])
    monkeypatch.setattr(olapcore, "_torch", lambda: torch)
    monkeypatch.setattr(olapcore, "lib", SimpleNamespace(
        olap_ctx_set_stream=lambda h, s: seen.append(None if s is None else s.value) or 0))
    c = object.__new__(olapcore.Context)
    c._h, c.device, c._fixed_stream, c._cur_stream = 1, 1, False, None
    try:
        c.follow_torch_stream()
        c.follow_torch_stream()  # unchanged: no second call
        current[1] = 0
        c.follow_torch_stream()
        assert seen == [4242, None]
    finally:
        c._h = None
