"""EMPM_OPT_SEG_CAP is accepted and changes nothing: a rollout replays the graph that was
captured before it was set."""
import time

import pytest
import torch

from tests.test_gpu_cell_scatter import DT, _solver, _state

pytestmark = pytest.mark.gpu


def test_graphs_outlive_the_option():
    sv, md = _solver(2000, "jelly")
    a = _state("box", 2000)
    b = a.partial_clone()
    schedule = sv.build_schedule(0.0, DT, 400)

    def run():
        torch.cuda.synchronize()
        t = time.perf_counter()
        sv.rollout(md, a, b, DT, 400, schedule=schedule)
        return time.perf_counter() - t       # until it is on its way

    run()
    captures, replays = [], []
    for cap in (1, 2, 8, 16, 32, 4):
        sv.fuse = not sv.fuse                # an option that does change the launches
        captures.append(run())
        sv.seg_cap = cap
        replays.append(run())
    assert sorted(replays)[3] < 0.5 * min(captures), (replays, captures)
