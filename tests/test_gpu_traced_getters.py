"""The state's matrices in functions that are traced: replayed, they are the state's, as
the tensor operations that make them record it."""
import pytest
import torch
from torch.fx.experimental.proxy_tensor import make_fx

from tests.test_gpu_cell_scatter import DEV, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tracer", ["jit", "fx", "compile"])
@pytest.mark.parametrize("name", ["particle_C", "particle_F_trial"])
def test_a_trace_reads_the_state(tracer, name):
    st = _state("box", 129)

    def f(x):
        return getattr(st, name).sum(0) * x

    x = torch.full((3, 3), 2.0, device=DEV)
    traced = {"jit": lambda: torch.jit.trace(f, x, check_trace=False), "fx": lambda: make_fx(f)(x),
              "compile": lambda: torch.compile(f, backend="eager")}[tracer]()
    junk = [torch.full((129, 3, 3), float("nan"), device=DEV) for _ in range(4)]   # what new memory may hold
    del junk
    assert torch.equal(traced(x), f(x))
    if tracer != "jit":                      # which folds what it takes for constant at its first run
        setattr(st, name, getattr(st, name) + 1.0)
        assert torch.equal(traced(x), f(x))
