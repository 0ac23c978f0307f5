"""A batch whose buffers were exchanged makes its copies on the stream that runs it."""

import contextlib

import pytest
import torch

from pyftle_b200 import _lib, batch as B


class _Tensor:
    def __init__(self, address):
        self.address = address

    def data_ptr(self):
        return self.address

    def numel(self):
        return 0


@pytest.mark.parametrize("stream", [None, "side"])
def test_exchanged_buffers_are_bound_inside_the_runs_stream(monkeypatch, stream):
    active, seen = [None], []

    @contextlib.contextmanager
    def on(s):
        active.append(s)
        yield
        active.pop()

    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(B, "stream_ptr", lambda s=None: 0)
    monkeypatch.setattr(B._lib, "call", lambda name, *args: seen.append((name, active[-1])))
    b = B.WindowBatch.__new__(B.WindowBatch)
    b.spatial_order, b._copies, b.schedule, b.count = True, False, B.Schedule(), 1
    window = B.WindowSpecRun(_Tensor(64), 0.0, 0.1, 1, ftle=_Tensor(128))
    b.windows = [window]
    b.desc = (_lib.FtleWindow * 1)()
    b.desc[0].positions, b.desc[0].ftle = 64, 128
    monkeypatch.setattr(b, "_plan", lambda order: _Tensor(256))
    monkeypatch.setattr(b, "_gather", lambda: seen.append(("gather", active[-1])))
    monkeypatch.setattr(b, "_scatter", lambda: seen.append(("scatter", active[-1])))

    def bind(copies):
        b._copies = copies
        seen.append(("bind", active[-1]))

    monkeypatch.setattr(b, "_bind", bind)
    b.run(stream=stream)
    assert seen == [("ftle_windows_run_mixed", stream)]  # nothing exchanged: no copies
    seen.clear()
    window.ftle = _Tensor(512)
    b.run(stream=stream)
    assert seen == [(what, stream) for what in ("bind", "gather", "ftle_windows_run_mixed",
                                                "scatter")]
