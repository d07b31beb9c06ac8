"""Single substeps take one constitutive update at every size and on every route: bodies
at rest, strained at random by 1e-5 to 1e-3, whose velocities after a substep are their
stress alone. The ordered P2G (from 65,536 particles on) and the direct one sum the
same terms in another order, so velocities agree within 8 sqrt(m) 2^-24 of the largest,
m particles on a node; the update without a decomposition differs from the one with it
by 1e-2 to 1e-4 of the stress."""
import numpy as np
import pytest
import torch

from tests.test_gpu_cell_scatter import DEV, DT, G, _solver, _state

pytestmark = pytest.mark.gpu


def _velocities(n, material, strain, path, inplace):
    sv, md = _solver(n, material)
    md.gravitational_accelaration = (0.0, 0.0, 0.0)
    sv.sort_every = 32 if path == "order" else 0
    a = _state("box", n)
    zero = torch.zeros(n, 3, device=DEV)
    a.particle_v, a.particle_C = zero, torch.zeros(n, 3, 3, device=DEV)
    rng = np.random.default_rng(7)
    a.particle_F_trial = torch.as_tensor((np.eye(3) + strain * rng.normal(size=(n, 3, 3))).astype(np.float32),
                                         device=DEV)
    if inplace:
        sv.p2g2p(md, a, 0, DT)
        return a.particle_v.double()
    b = a.partial_clone()
    sv.p2g2p_differentiable(md, a, b, DT)
    return b.particle_v.double()


@pytest.mark.parametrize("material", ["jelly", "plasticine"])
@pytest.mark.parametrize("strain", [1e-5, 1e-3])
@pytest.mark.parametrize("inplace", [False, True])
def test_ordered_substep_takes_the_direct_ones_update(material, strain, inplace):
    n = 70_001
    a, b = (_velocities(n, material, strain, p, inplace) for p in ("order", "direct"))
    tol = 8 * (27 * (8 + n / 900)) ** 0.5 * 2.0 ** -24 * float(b.abs().max())
    assert float(b.abs().max()) > 0
    assert float((a - b).abs().max()) <= tol, (float((a - b).abs().max()), tol)
