"""A kernel that gave up a wait makes the next check raise, once, and generation and the trace runner check.  The flags are faked here."""
import pytest
import torch

from krasis_b200 import capi, scheduler, seqops


class _Flags:
    def __init__(self, up=0):
        self.up = up

    def exchange(self, device, put, up):
        up._obj.value, self.up = self.up, put
        return 0

    kb2_wait_timeouts = kb2_seq_wait_timeouts = exchange


def test_raised_flags_are_reported_once(monkeypatch):
    core, seq = _Flags(), _Flags()
    monkeypatch.setattr(capi, "_lib", core)
    monkeypatch.setattr(seqops, "_lib", seq)
    capi.check_waits()
    seqops.check_waits()
    core.up = 2
    with pytest.raises(capi.Kb2Error, match="gave up"):
        capi.check_waits()
    capi.check_waits()
    core.up = 1                                  # the serving path reports the core library's kernels too
    with pytest.raises(capi.Kb2Error, match="gave up"):
        seqops.check_waits()
    seq.up = 1
    with pytest.raises(seqops.SeqOpsError, match="gave up"):
        seqops.check_waits()
    seqops.check_waits()
    monkeypatch.setattr(capi, "_lib", None)      # a process without the core library
    seq.up = 1
    with pytest.raises(seqops.SeqOpsError):
        seqops.check_waits()


def test_generation_checks(monkeypatch):
    asked = []
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(seqops, "check_waits", lambda device=0: asked.append(device))
    s = scheduler.Scheduler.__new__(scheduler.Scheduler)
    s.model = type("M", (), {"device": torch.device("cuda:1")})()
    s.can_admit = lambda n: True
    s.admit = lambda rid: scheduler.Request(rid, None, 0)
    s.finish = lambda rid: None
    s.step = lambda entries: torch.zeros(len(entries), 4)
    monkeypatch.setattr(scheduler, "Sampler", lambda *a: lambda logits: logits.argmax(1))
    assert s.generate([[1, 2], [3]], 2) == [[0, 0], [0, 0]]
    assert asked == [1]
    assert s.generate([], 2) == [] and asked == [1]
