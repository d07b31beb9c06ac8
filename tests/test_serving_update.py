"""A served request's blocks run the same update whatever the requests beside it (no
GPU: the library's rollout call is recorded)."""
import types

import pytest
import torch

from empm_b200 import _native as N
from empm_b200.serving import GpuExecutor


def _flags(kinds):
    calls = []
    tickets = [types.SimpleNamespace(id=i, n=4, progress=0, req=types.SimpleNamespace(grad=g, n_substeps=8))
               for i, g in enumerate(kinds)]
    plane = {k: [torch.zeros(64), torch.zeros(64)] for k in ("x4", "v4", "C", "F")}
    ex = types.SimpleNamespace(
        N=N, L=types.SimpleNamespace(empm_rollout_ex=lambda *a: calls.append(a) or N.EMPM_OK), ctx=None, cur=0, ai=0,
        arenas=[plane], Fe=torch.zeros(64), mat={k: [torch.zeros(16)] for k in ("vol", "mu", "lam", "ys")},
        fwd_stream=None, _sptr=lambda s: None, tables={t.id: ((N.EmpmStep * 8)(), False) for t in tickets})
    GpuExecutor.run_block(ex, tickets, 3)
    (call,) = calls
    return call[7]


@pytest.mark.parametrize("kinds", [(False,), (True,), (False, True), (False, False, True)])
def test_every_block_takes_the_tapes_update(kinds):
    assert _flags(kinds) == N.ROLLOUT_TAPE
