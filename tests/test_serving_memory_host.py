"""Memory of finished solves (no GPU): the server's own loop, iteration and
group code over stand-in fields that count themselves while they live."""

import gc
import weakref
from types import SimpleNamespace

import pytest

from cutile.runtime import native
from cutile.runtime.serving import SolveKind, SolveRequest, StencilServer, _Active

KINDS = [SolveKind("heat2d", {}, 1), SolveKind("wave2d", {}, 2), SolveKind("lap7", {}, 1)]


class Field:
    def __init__(self, nbytes):
        self.nbytes = nbytes


class CountingServer(StencilServer):
    """Device work replaced; ``live()`` is what the fields still referenced hold."""

    def __init__(self, budget):
        super().__init__(KINDS, budget_bytes=budget, device="cpu")
        self.fields = weakref.WeakSet()
        self.peak = 0
        import torch

        self._pool = torch.zeros(1, dtype=torch.uint8)

    def live(self):
        return sum(f.nbytes for f in self.fields)

    def program(self, kind, dtype):
        return (None, SimpleNamespace(handle=None), 0)

    def _admit(self, req, res, now):
        res.admitted = now
        P = self.kinds[req.kind].nstate + 1
        f = Field(self.memory_of(req))
        self.fields.add(f)
        self.peak = max(self.peak, self.live())
        return _Active(req=req, res=res, flat=f, bufs=[f] * P, desc=None, items=1, nbytes=f.nbytes)

    def _lanes(self, stream, groups):
        return [stream]

    def _stream(self):
        return None

    def _reserve(self):
        pass

    def _record(self, stream):
        return 0.0

    def _wait(self, mark):
        pass

    def _done(self, mark):
        return True

    def _mark_time(self, mark, start, t_start):
        return t_start


@pytest.fixture
def launches(monkeypatch):
    """csd_launch_batch as a list of its calls; no pinned memory."""
    import torch

    calls = []

    def launch_batch(handle, pool, starts, count, items, opts, stream):
        calls.append((count, items))
        return 0

    empty = torch.empty
    monkeypatch.setattr(torch, "empty",
                        lambda *a, pin_memory=False, **kw: empty(*a, **kw))
    monkeypatch.setattr(native, "library", lambda: SimpleNamespace(csd_launch_batch=launch_batch))
    monkeypatch.setattr(native, "stream_handle", lambda stream: None)
    return calls


@pytest.mark.parametrize("order", ["one kind after another", "mixed"])
def test_finished_solves_release_their_fields(launches, order):
    shape = {"heat2d": (66, 66), "wave2d": (66, 66), "lap7": (18, 18, 18)}
    kinds = [k.name for k in KINDS]
    names = ([k for k in kinds for _ in range(4)] if order == "one kind after another" else
             [kinds[i % 3] for i in range(12)])
    reqs = [SolveRequest(k, "float64", shape[k], 2 + i % 3) for i, k in enumerate(names)]
    probe = CountingServer(1)
    budget = 2 * max(probe.memory_of(r) for r in reqs)
    server = CountingServer(budget)
    gc.disable()      # references alone keep or free a field
    try:
        results = server.run(reqs, realtime=False, keep_state=False)
        assert server.stats.peak_bytes <= budget
        assert server.peak <= budget
        assert server.live() == 0
    finally:
        gc.enable()
    assert all(r.error is None for r in results)
    assert sum(count for count, _ in launches) == sum(r.steps for r in reqs)


def test_kept_states_alone_stay(launches):
    reqs = [SolveRequest("heat2d", "float64", (66, 66), 3) for _ in range(4)]
    server = CountingServer(10 * CountingServer(1).memory_of(reqs[0]))
    results = server.run(reqs, realtime=False, keep_state={2})
    assert server.live() == server.memory_of(reqs[0])
    assert len(results[2].state) == 1 and results[1].state == ()
