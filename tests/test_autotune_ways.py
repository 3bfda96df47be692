"""The autotuner's choice between a queue and two launches (CPU, fake timings): the faster way is
applied, and again from memory and from a file; an entry written before there were two ways is
timed again."""
from __future__ import annotations

import json

import pytest
import torch

from psierra_b200 import autotune


class Pattern:
    two_pass = split = True
    queued_f = queued_k = False

    def tangent_in_two_passes(self, precision):
        return True


class Assembler:
    """What tune() uses of an assembler; ``way`` is the last thing that was set."""

    def __init__(self):
        self.device, self.npe, self.n_elements, self.n_nodes, self.precision = torch.device("cpu"), 4, 1000, 300, "fp64"
        self.pattern, self.way = Pattern(), None

    def set_queue(self, lag=None, blocks_per_sm=None, ring_slack=None, lag_f=None, split=None):
        self.way = ("queue", lag if lag is not None else lag_f, blocks_per_sm, ring_slack)

    def set_two_pass(self, f=True, k=True):
        # the two calls name one kind of sweep each: the one tuned, or the one left as it was
        if (f, k) == (not self.want_k, self.want_k):
            self.way = ("two-pass",)

    def new_f(self):
        return None

    def new_k(self, prec):
        return None


@pytest.fixture
def tune(monkeypatch):
    timed = []

    def run(two_pass_ms, want_k=True, **kw):
        asm = Assembler()
        asm.want_k = want_k

        def fake_time(a, *_):
            timed.append(a.way)
            return two_pass_ms if a.way == ("two-pass",) else abs(a.way[1] - 16) + 1.0

        monkeypatch.setattr(autotune, "_time", fake_time)
        timed.clear()
        return asm, autotune.tune(asm, None, want_k=want_k, lags=(8, 16), slacks=(12,), **kw), list(timed)

    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a, **k: "FakeGPU")
    monkeypatch.setattr(autotune, "_cache", {})
    return run


@pytest.mark.parametrize("want_k", [True, False])
@pytest.mark.parametrize("ms,way", [(0.5, ("two-pass",)), (1.5, ("queue", 16, 2, 12))])
def test_the_faster_way_is_kept_and_replayed(tune, tmp_path, ms, way, want_k):
    cache = str(tmp_path / "tune.json")
    asm, r, timed = tune(ms, want_k, cache_file=cache)
    assert asm.way == way and timed[-1] == ("two-pass",) and len(timed) == 3
    assert r["two_pass"] == (way == ("two-pass",)) and r["ms"] == min(ms, 1.0)  # what runs, and its time
    for forget in (False, True):  # from memory, from the file
        if forget:
            autotune._cache.clear()
        asm, r, timed = tune(99.0, want_k, cache_file=cache)
        assert asm.way == way and timed == [] and r["lag"] == 16
        assert r["two_pass"] == (way == ("two-pass",)) and r["ms"] is None


def test_entries_of_one_way_are_timed_again(tune, tmp_path):
    # a file of the time when every sweep was queued: same mesh, four values, no way
    cache = tmp_path / "tune.json"
    old = {"FakeGPU|npe4|E1000|N300|fp64|f1k1": [24, 2, 20, True]}
    cache.write_text(json.dumps(old))
    asm, r, timed = tune(0.5, cache_file=str(cache))
    assert len(timed) == 3 and asm.way == ("two-pass",)
    disk = json.loads(cache.read_text())
    assert len(disk) == 2 and {k: disk[k] for k in old} == old  # the other entries stay
