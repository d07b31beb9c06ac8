"""Fixed-corotated stress of small strains against 64 bits, where an error of the modulus'
rounding is an error of the stress: both updates (of rollouts, without a decomposition;
of single substeps and tapes, with it), F near the identity and under large rotations.

Tolerance: F - R is known to a few 2^-24 (the entries of R are rounded), which enters
the stress times 2 mu + 3 lam; 8 roundings without the decomposition, 40 with it (its
singular values carry those of U, V and the Jacobi sweeps), and 16 2^-24 of the stress
itself. A test of the tolerance: no stress at all must not pass."""
import ctypes

import numpy as np
import pytest
import torch

from tests.test_gpu_elastic_branch import LAM, MU, SOFT, YS, _reference, _rotations

pytestmark = pytest.mark.gpu


CASES = [("empm_debug_stress", 8, s) for s in (1e-6, 1e-5, 1e-3, 1e-2)] + [
    ("empm_debug_stress_tape", 40, s) for s in (2e-5, 1e-3, 1e-2)]


@pytest.mark.parametrize("rotated", [False, True])
@pytest.mark.parametrize("entry,roundings,strain,material", [
    (*c, m) for m in (0, 5) for c in CASES if m == 0 or c[2] <= 1e-3])   # plasticine inside its yield surface
def test_stress_of_small_strains(entry, roundings, strain, rotated, material):
    from empm_b200 import _native as N

    rng = np.random.default_rng(13)
    n = 4096
    F = np.eye(3) + strain * rng.normal(size=(n, 3, 3))
    if rotated:
        F = _rotations(rng, n) @ F
    F = F.astype(np.float32)
    _, tau, ys, _, _ = _reference(F.astype(np.float64), material == 5)
    assert (ys == YS).all()
    dev = "cuda:0"
    t = torch.as_tensor(F.reshape(n, 9), device=dev).contiguous()
    mu, lam, y = (torch.full((n,), v, device=dev) for v in (MU, LAM, YS))
    out_F, out_t = torch.empty_like(t), torch.empty_like(t)
    p = N.EmpmModelParams()
    p.n_grid, p.grid_lim, p.material, p.softening = 32, 1.0, material, SOFT
    N.check(getattr(N.lib(), entry)(ctypes.byref(p), t.data_ptr(), mu.data_ptr(), lam.data_ptr(), y.data_ptr(), 1e-4,
                                    out_F.data_ptr(), out_t.data_ptr(), n, None))
    torch.cuda.synchronize()
    size = np.abs(tau).max((1, 2))
    tol = roundings * 2.0 ** -24 * (2 * MU + 3 * LAM) + 16 * 2.0 ** -24 * size
    assert (size > tol).mean() > 0.5
    err = np.abs(out_t.double().cpu().numpy().reshape(n, 3, 3) - tau).max((1, 2))
    assert (err <= tol).all(), float((err / tol).max())
    eF = np.abs(out_F.double().cpu().numpy().reshape(n, 3, 3) - F).max()
    assert eF <= 40 * 2.0 ** -24             # inside the yield surface the trial F is the elastic one
