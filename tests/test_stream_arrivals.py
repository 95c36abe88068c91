"""CPU: the timed stream of the request server.  No request is submitted before
its arrival, none waits longer than the tick for those that arrive behind it, and
latencies count from the arrival."""
import time

import numpy as np

from desi_b200.serve import PcfServer, Request


class Instant(PcfServer):
    """Scheduler without slots: a request completes as it is submitted."""

    def __init__(self):
        self.at = {}

    def submit(self, req):
        req.t_submit = req.t_start = req.t_end = time.perf_counter()
        self.at[req.rid] = req.t_submit
        req.future.set_result({})
        return req.future


def _run(arrivals, monkeypatch, **kw):
    from desi_b200 import serve
    monkeypatch.setattr(serve._lib, "alloc_counters", lambda: {})
    srv = Instant()
    reqs = [Request("2iso", "d", "r", 10, 20.0, arrival=a, rid=i) for i, a in enumerate(arrivals)]
    t0 = time.perf_counter()
    rep = srv.run_stream(reqs, **kw)
    return np.array([srv.at[i] - t0 for i in range(len(reqs))]), rep


def test_never_before_arrival(monkeypatch):
    arrivals = [0.0, 0.002, 0.004, 0.0045, 0.02, 0.0235, 0.03, 0.0301]
    at, rep = _run(arrivals, monkeypatch)
    # (the stream's clock starts after t0, so its times here are later than its own)
    assert np.all(at >= np.array(arrivals)), at
    assert rep["requests"] == len(arrivals)


def test_latency_counts_from_arrival(monkeypatch):
    """With a tick of 30 ms, the first of three requests waits for it."""
    at, rep = _run([0.0, 0.01, 0.02], monkeypatch, tick_s=0.03)
    assert at.min() >= 0.02  # one group, behind its last arrival
    assert rep["latency_ms"]["max"] >= 29.0
    assert rep["latency_ms"]["p50"] >= 19.0


def test_without_a_tick_each_goes_at_its_arrival(monkeypatch):
    arrivals = np.array([0.0, 0.03, 0.06])
    at, _ = _run(list(arrivals), monkeypatch, tick_s=0.0)
    assert np.all(at >= arrivals)
    assert at[0] < 0.03 and at[1] < 0.06  # not held back for the ones behind
