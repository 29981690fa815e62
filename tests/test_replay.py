"""What a recorded step does when something fails in the middle: host logic, with the CUDA objects replaced by recorders."""
import pytest
import torch

from jaxpp_b200.runtime import replay


class _Log:
    def __init__(self, log, name):
        self.log, self.name = log, name

    def __getattr__(self, what):
        return lambda *args: self.log.append(f"{self.name}.{what}")


@pytest.fixture
def recording(monkeypatch):
    log = []
    rec = replay._Recording.__new__(replay._Recording)
    rec.device, rec.launches, rec.written = torch.device("cpu"), 1, []
    rec.static, rec.results, rec.outputs = [torch.zeros(4)], [torch.ones(3)], [("out", 0, 0)]
    rec.graph, rec.done = _Log(log, "graph"), _Log(log, "done")
    rec._plan()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: _Log(log, "stream"))
    return rec, log


def test_a_call_waits_for_the_last_one_and_is_waited_for(recording):
    rec, log = recording
    x = torch.arange(4.0)
    (out,) = rec.run([x])
    assert torch.equal(out[0], torch.ones(3)) and torch.equal(rec.static[0], x)
    assert log == ["stream.wait_event", "graph.replay", "done.record"]


def test_without_memory_for_the_results_nothing_runs(recording, monkeypatch):
    rec, log = recording

    def no_memory(*args, **kwargs):
        raise torch.OutOfMemoryError("none left")

    with monkeypatch.context() as m:
        m.setattr(torch, "empty_like", no_memory)
        with pytest.raises(torch.OutOfMemoryError):
            rec.run([torch.arange(4.0)])
    assert "graph.replay" not in log and torch.equal(rec.static[0], torch.zeros(4))


def test_an_error_behind_the_replay_leaves_it_waited_for(recording, monkeypatch):
    """The buffers are given back, or written by the next call on another stream, only behind ``done``."""
    rec, log = recording
    copy = replay._copy

    def fails_behind_the_replay(dst, src):
        if "graph.replay" in log:
            raise RuntimeError("copy failed")
        copy(dst, src)

    monkeypatch.setattr(replay, "_copy", fails_behind_the_replay)
    with pytest.raises(RuntimeError, match="copy failed"):
        rec.run([torch.arange(4.0)])
    assert log == ["stream.wait_event", "graph.replay", "done.record"]


def test_what_a_recording_covers():
    rec = replay._Recording.__new__(replay._Recording)
    buf = torch.zeros(64)
    rec.static, rec.results, rec.written = [torch.zeros(16), None, torch.zeros(4, 4), torch.zeros(0)], [], []
    rec._plan()
    ok = [buf[:16], None, buf[16:32].view(4, 4), buf[:0]]
    assert rec.covers(ok)
    for k, other in ((0, buf[:1]), (0, buf[:16].double()), (0, None), (1, buf[:16]), (2, buf[16:32]), (3, buf[:1])):
        assert not rec.covers([other if i == k else x for i, x in enumerate(ok)])
    overlapping = [buf[:16], None, buf[15:31].view(4, 4), buf[:0]]
    assert rec.covers(overlapping)              # nothing is updated in place
    rec.written = [0]
    assert rec.covers(ok) and not rec.covers(overlapping)
