"""Instances loaded by one launch, against assigning each array to its slice:
shared arrays, one row for all particles, other dtypes, arrays on both sides of the
size up to which they travel together, missing velocities, single instances
reloaded. Bit for bit."""
from dataclasses import replace

import numpy as np
import pytest
import torch

from empm_b200.batch import BatchedMPM, InstanceSpec
from empm_b200.mpm_data_structure import _f9_unpack

pytestmark = pytest.mark.gpu


def _spec(n, seed, **over):
    rng = np.random.default_rng(seed)
    f = lambda lo, hi, *s: rng.uniform(lo, hi, (n, *s)).astype(np.float32)  # noqa: E731
    s = InstanceSpec(x=f(0.3, 0.6, 3), v=f(-1, 1, 3), vol=f(1e-6, 2e-6), rho=f(900, 1100), E=f(1e4, 2e4), nu=f(0.2, 0.3),
                     yield_stress=f(1e3, 2e3), n_grid=32, material="plasticine")
    return replace(s, **over)


def _assigned(b, idx, before):
    """The state after assigning the arrays of the listed instances slice by slice."""
    out = {k: t.clone() for k, t in before.items()}
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float32).to(b.device)  # noqa: E731
    for i in idx:
        s, sl = b.specs[i], b._sl(i)
        out["x"][sl] = t(s.x)
        out["v"][sl] = t(s.v) if s.v is not None else 0.0
        for name, a in (("vol", s.vol), ("density", s.rho), ("E", s.E), ("nu", s.nu)):
            out[name][sl] = t(a)
        out["ys"][sl] = t(s.yield_stress) if s.yield_stress is not None else 0.0
        out["C"][sl], out["F"][sl] = 0.0, torch.eye(3, device=b.device)
    return out


def _state(b):
    c = b.cur
    return {"x": b._x4[c][:, :3].clone(), "v": b._v4[c][:, :3].clone(), "vol": b.vol.clone(), "density": b.density.clone(),
            "E": b.E.clone(), "nu": b.nu.clone(), "ys": b.yield_stress.clone(), "C": _f9_unpack(b._C[c], b.n).clone(),
            "F": _f9_unpack(b._F[c], b.n).clone()}


@pytest.mark.parametrize("sizes", [(1,), (1, 257, 3), (700, 700, 700), (64_000, 31, 70_001)])
@pytest.mark.parametrize("subset", [None, [0], [-1, 0]])
def test_loaded_instances_equal_assigned_slices(sizes, subset):
    specs = [_spec(n, k) for k, n in enumerate(sizes)]
    specs[0] = replace(specs[0], v=None, yield_stress=None, E=np.float64(3e4), rho=specs[0].rho.astype(np.float64),
                       nu=np.full(1, 0.25))
    if len(sizes) > 1 and sizes[1] == sizes[0]:
        specs[1] = replace(specs[0], v=np.array([0.5, -1.0, 2.0]), vol=specs[0].vol[None])
    b = BatchedMPM(specs)
    b.rollout(1e-4, 3)                                # state to overwrite, in the other buffers
    before = _state(b)
    b.load_state(subset)
    torch.cuda.synchronize()
    want = _assigned(b, range(len(sizes)) if subset is None else subset, before)
    got = _state(b)
    for k in want:
        assert torch.equal(got[k], want[k]), k
    mass = b.density * b.vol
    assert torch.equal(b._x4[b.cur][:, 3], mass)


def test_wrong_shapes_are_refused():
    for bad in (dict(E=np.zeros(5, np.float32)), dict(v=np.zeros((4, 3), np.float32))):
        with pytest.raises(RuntimeError):
            BatchedMPM([_spec(7, 0, **bad)])
