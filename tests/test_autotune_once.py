"""Candidates of the autotuner whose launches are equal are timed once, and each of them
gets that time (no GPU: the batch and the clock are fakes)."""
import itertools
import json
import types

import torch

from empm_b200 import autotune as A


class _Batch:
    """A batch that records the options each rollout ran with."""

    def __init__(self):
        for k, v in A.DEFAULTS.items():
            setattr(self, k, v)
        self.specs = [types.SimpleNamespace(n_grid=32, material="jelly")]
        self.n, self.cur, self.time, self.use_graph, self.solvers, self.runs = 1000, 0, 0.0, True, [], []
        for k in ("_x4", "_v4", "_C", "_F"):
            setattr(self, k, [torch.zeros(4), torch.zeros(4)])
        self.mu, self.lam, self.yield_stress = torch.zeros(4), torch.zeros(4), torch.zeros(4)

    def rollout(self, dt, n, block):
        self.runs.append(tuple(int(getattr(self, k)) for k in A.OPTION_NAMES))


def test_equal_launches_are_timed_once(monkeypatch):
    clock = itertools.count(1)

    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self):
            self.t = next(clock)

        def elapsed_time(self, other):
            return float(other.t)            # later candidates take longer

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(A, "_MEMORY", {})
    b = _Batch()
    res = A.tune_batch(b, 1e-4, substeps=4)
    seg = A.OPTION_NAMES.index("seg_cap")
    launches = [r[:seg] + r[seg + 1:] for r in b.runs]
    assert len(set(launches)) * 2 == len(b.runs) == 54          # a capture and a timed run each
    assert set(res["ms"]) == {json.dumps(c, sort_keys=True) for c in A.CANDIDATES}
    for c in A.CANDIDATES:
        assert res["ms"][json.dumps(c, sort_keys=True)] == res["ms"][json.dumps(dict(c, seg_cap=4), sort_keys=True)]
    assert res["options"] == A.CANDIDATES[0]
