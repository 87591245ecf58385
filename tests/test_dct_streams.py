"""A transform plan shared by streams: its solves are ordered."""

import threading

import pytest
import torch

from gradient_domain_b200 import _lib, solvers


class _Stream:
    """Stands in for a CUDA stream; `log` is the order of what every stream was given."""

    def __init__(self, number, log):
        self.cuda_stream, self.log = number, log

    def wait_event(self, event):
        self.log.append(("wait", self.cuda_stream, event.recorded))

    def synchronize(self):
        self.log.append(("synchronize", self.cuda_stream))


class _Event:
    def __init__(self, log):
        self.log, self.recorded = log, None

    def record(self, stream):
        self.recorded = (stream.cuda_stream, sum(e[0] == "solve" for e in self.log))

    def synchronize(self):
        self.log.append(("synchronize event", self.recorded))


@pytest.fixture
def plan(monkeypatch):
    """A DctPlan over a library and streams that only log, and a way to choose the stream."""
    log, current = [], {}

    class Library:
        def gd_dct_plan_create(self, h, w, out):
            out._obj.value = 1
            return 0

        def gd_dct_workspace_bytes(self, handle):
            return 256

        def gd_dct_plan_bind(self, *args):
            return 0

        def gd_dct_solve_neumann(self, handle, b, u, pitch, stream):
            log.append(("solve", stream))
            return 0

        def gd_dct_plan_destroy(self, handle):
            log.append(("destroy",))

    streams = [_Stream(k, log) for k in (7, 8, 9)]
    library = Library()
    current.update(stream=streams[0], capturing=False)
    monkeypatch.setattr(_lib, "lib", lambda: library)
    monkeypatch.setattr(_lib, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: current["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: current["capturing"])
    monkeypatch.setattr(torch.cuda, "Event", lambda **kw: _Event(log))
    made = solvers.DctPlan(4, 4)

    def solve(k, capturing=False):
        current.update(stream=streams[k], capturing=capturing)
        made.solve(torch.zeros(4, 4, dtype=torch.float64), torch.zeros(4, 4, dtype=torch.float64))

    return made, solve, log


def test_another_stream_waits_for_the_last_solve(plan):
    made, solve, log = plan
    for k in (0, 0, 1, 1, 2, 0):
        solve(k)
    assert log == [("solve", 7), ("solve", 7), ("wait", 8, (7, 2)), ("solve", 8), ("solve", 8),
                   ("wait", 9, (8, 4)), ("solve", 9), ("wait", 7, (9, 5)), ("solve", 7)]


def test_a_plan_is_destroyed_after_its_last_solve(plan):
    made, solve, log = plan
    solve(0)
    solve(1)
    solve(2, capturing=True)  # current stream when the plan goes: not where its work is
    del log[:]
    made.__del__()
    assert log[-1] == ("destroy",) and ("synchronize event", (8, 2)) in log


def test_a_plan_whose_set_up_failed_is_destroyed(plan, monkeypatch):
    made, solve, log = plan
    monkeypatch.setattr(type(_lib.lib()), "gd_dct_plan_bind", lambda *args: -1)
    monkeypatch.setattr(type(_lib.lib()), "gd_last_error", lambda self: b"no", raising=False)
    del log[:]
    with pytest.raises(_lib.GDError):
        solvers.DctPlan(4, 4)
    assert log[-1] == ("destroy",)


def test_capture_neither_waits_nor_is_waited_for(plan):
    made, solve, log = plan
    solve(0)
    solve(1, capturing=True)  # an event recorded outside may not enter the capture
    solve(0)
    assert log == [("solve", 7), ("solve", 8), ("solve", 7)]


@pytest.mark.gpu
def test_streams_sharing_a_plan_get_their_own_solutions():
    """Two threads, a stream each, solve different right-hand sides on one plan at once."""
    h, w, n = 480, 640, 40
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = torch.randn((2, n, h, w), generator=g, dtype=torch.float64, device="cuda")
    plan = solvers.DctPlan(h, w)
    want = torch.empty_like(b)
    for t in range(2):
        for k in range(n):
            plan.solve(b[t, k], want[t, k])
    torch.cuda.synchronize()
    got = torch.empty_like(b)

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for k in range(n):
                plan.solve(b[t, k], got[t, k])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert torch.equal(got, want)
