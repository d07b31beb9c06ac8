"""Every touched block is updated, whatever the share of a warp: grids from one
block per axis to more blocks than a launch's warps look at 32 at a time, and a
batch of uneven ones. A body that falls freely keeps F = I, so after k substeps
every velocity is v0 + k dt g (a block left out would hold its particles still);
the sums of a node's mass and momentum carry a few 2^-24, held to 1e-5 of |v|."""
import numpy as np
import pytest
import torch

from empm_b200.batch import BatchedMPM, InstanceSpec

pytestmark = pytest.mark.gpu


def _spec(G, n, seed):
    rng = np.random.default_rng(seed)
    full = lambda a: np.full(n, np.float32(a), np.float32)  # noqa: E731
    v = np.tile(np.float32([0.3, 0.5, -0.2]), (n, 1))
    return InstanceSpec(x=rng.uniform(0.55 if G < 8 else 0.3, 0.6 if G < 8 else 0.7, (n, 3)).astype(np.float32), v=v,
                        vol=full(0.06 / n), rho=full(1e3), E=full(1.0), nu=full(0.3), n_grid=G, material="jelly")


@pytest.mark.parametrize("grids", [[5], [16], [31], [86], [128], [300], [8, 130, 33, 5, 64]])
@pytest.mark.parametrize("sort_every", [0, 32])
def test_free_fall_reaches_every_block(grids, sort_every):
    b = BatchedMPM([_spec(G, 1500 + 97 * i, i) for i, G in enumerate(grids)])
    b.sort_every = sort_every
    b.rollout(1e-4, 5)
    torch.cuda.synchronize()
    want = torch.tensor([0.3, 0.5 - 9.8 * 5e-4, -0.2], dtype=torch.float64)
    assert b.read_status() == 0
    assert float((b.velocities().double().cpu() - want).abs().max()) <= 1e-5
