"""A recorded call on a device that is not the current one goes through PyTorch's device guard, which
leaves the current device without a context if it has none (no GPU needed)."""

from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from grg_spmv_b200.backends.b200 import B200Runtime  # noqa: E402
from grg_spmv_b200.backends.b200 import _native as nat  # noqa: E402


@pytest.mark.parametrize("current,expected", [(1, ["launch"]), (0, ["enter 1", "launch", "exit"])])
def test_recorded_launch_guards_the_device(monkeypatch, current, expected):
    log = []

    class Guard:
        def __init__(self, device) -> None:
            self.index = torch.device(device).index

        def __enter__(self) -> None:
            log.append(f"enter {self.index}")

        def __exit__(self, *exc) -> None:
            log.append("exit")

    class Recording:
        def launch(self, args, stream_ptr) -> int:
            assert (args, stream_ptr) == ("args", 77)
            log.append("launch")
            return nat.OK

    monkeypatch.setattr(torch.cuda, "current_device", lambda: current)
    monkeypatch.setattr(torch.cuda, "device", Guard)
    runtime = B200Runtime.__new__(B200Runtime)
    runtime.device, runtime.stream_ptr = torch.device("cuda", 1), 77
    runtime._launch("args", Recording())
    assert log == expected
