"""The autotuner's clock starts once the call it times has settled."""
import pytest


class _Clock:
    now = 0.0


class _Event:
    def __init__(self, enable_timing=True):
        self.t = 0.0

    def record(self, stream):
        self.t = _Clock.now

    def elapsed_time(self, other):
        return other.t - self.t


@pytest.mark.parametrize("slow", [0, 1, 3, 7])
def test_slow_first_calls_are_not_timed(monkeypatch, slow):
    import torch
    from libfastlib_b200 import tune
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: None)
    calls = [0]

    def fn():
        calls[0] += 1
        _Clock.now += 10.0 * 1.5 ** (slow - calls[0]) if calls[0] <= slow else 1.0

    assert tune._time(fn, 5) == pytest.approx(1.0)
