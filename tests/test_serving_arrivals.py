"""Requests that reach an idle server within one poll interval of each other are served as one batch,
wherever between them the server happens to wake; later ones are not waited for.  Simulated time."""

import types

import pytest
import torch

import fvdb.serving as serving
from fvdb.serving import ContinuousBatcher, Executor, Request


class _Time:
    def __init__(self):
        self.now = 0.0

    def clock(self):
        self.now += 1e-7
        return self.now

    def sleep(self, seconds):
        self.now += seconds


class _Fake(Executor):
    def __init__(self, time):
        self.time, self.launched = time, []

    def footprint(self, req):
        return req.n_voxels

    def launch(self, batch, slot):
        self.launched.append([r.rid for r in batch])
        self.time.sleep(1e-4)
        return self.time.now + 1e-4

    def poll(self, handle):
        return self.time.clock() >= handle

    def finish(self, handle):
        pass


@pytest.mark.parametrize("gap,packed", [(0.0, True), (25e-6, True), (45e-6, True), (80e-6, False)])
@pytest.mark.parametrize("first", [0.0, 0.0100, 0.0105])
def test_arrivals_within_a_poll_interval(monkeypatch, gap, packed, first):
    t = _Time()
    monkeypatch.setattr(serving, "time", types.SimpleNamespace(sleep=t.sleep))
    ex = _Fake(t)
    srv = ContinuousBatcher(ex, hbm_budget=1 << 20, max_batch_voxels=1 << 10, slots=3, clock=t.clock)
    reqs = [Request(rid=i, ijk=torch.zeros((5, 3), dtype=torch.int32), features=torch.zeros(5, 1), arrival=a)
            for i, a in enumerate((first, first + gap))]
    out = srv.serve(reqs, poll_sleep=5e-5)
    assert all(r.done is not None and r.error is None for r in out)
    assert ex.launched == ([[0, 1]] if packed else [[0], [1]])
    assert out[0].done - out[0].arrival <= 5e-4
