"""A checkpointed forward pass (EMPM_ROLLOUT_TAPE) reaches the states that the stored one
and the adjoint's re-run reach: bodies at rest with random strains of 1e-4, whose
velocities are their stress alone.

Both passes run the update with the decomposition, whose error is 2e-3 of such a stress;
sums in another order change the trial F of a particle in a hundred or so by its last
bit, and with it that error: 2e-3 / sqrt(100) of the largest velocity. Without the flag
every particle's stress differs by 2e-3."""
import numpy as np
import pytest
import torch

from empm_b200.adjoint import CheckpointedRollout
from tests.test_gpu_cell_scatter import DEV, DT, _solver, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("material", ["jelly", "plasticine"])
@pytest.mark.parametrize("n,steps", [(4001, 1), (4001, 3), (66_001, 1), (66_001, 3)])
def test_checkpointed_and_stored_passes_agree(n, steps, material):
    res = []
    for store in (True, False):
        sv, md = _solver(n, material)
        md.gravitational_accelaration = (0.0, 0.0, 0.0)
        a = _state("box", n)
        a.particle_v, a.particle_C = torch.zeros(n, 3, device=DEV), torch.zeros(n, 3, 3, device=DEV)
        rng = np.random.default_rng(9)
        a.particle_F_trial = torch.as_tensor((np.eye(3) + 1e-4 * rng.normal(size=(n, 3, 3))).astype(np.float32),
                                             device=DEV)
        tape = CheckpointedRollout(sv, md, a, DT, steps, checkpoint_every=3, store=store)
        tape.forward()
        assert tape.stored == store
        res.append(tape.final.particle_v.double().clone())
        tape.release()
    top = float(res[0].abs().max())
    assert top > 0
    assert float((res[0] - res[1]).abs().max()) <= 2e-4 * top, float((res[0] - res[1]).abs().max()) / top
