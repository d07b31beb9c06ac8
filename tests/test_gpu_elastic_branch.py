"""The fixed-corotated branch without a decomposition (jelly, plasticine inside
its yield surface) and its limits: strains from rounding level to half, large
rotations, F just inside and just outside the yield surface, and F that the
branch must hand to the general update (inverted, nearly singular, stretched
far), against the same map in 64 bits (numpy SVD).

Tolerance: single-precision singular values carry a few 1e-7 of the largest one
s, so stress entries carry a few 1e-7 of 2 mu s^2 + lam |J| (1 + |J|), and F_e
of s; both are held to 1e-5 of that."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MU, LAM, YS, SOFT = 8000.0, 12000.0, 500.0, 0.1


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def _cases(rng, kind, n=2048):
    if kind.startswith("strain"):
        S = np.eye(3) + float(kind[6:]) * rng.normal(size=(n, 3, 3))
        return _rotations(rng, n) @ S
    if kind == "yield":
        # deviatoric Hencky strain of norm (1 +- 1e-6 .. 1e-2) ys / (2 mu)
        d = rng.normal(size=(n, 3))
        d -= d.mean(1, keepdims=True)
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        off = 10.0 ** rng.uniform(-6, -2, n) * rng.choice([-1, 1], n)
        eps = d * (YS / (2 * MU) * (1 + off))[:, None] + 0.01 * rng.normal(size=(n, 1))
        A = _rotations(rng, n)
        return _rotations(rng, n) @ (A * np.exp(eps)[:, None, :]) @ A.transpose(0, 2, 1)
    s = {"stretched": rng.uniform(2.0, 6.0, (n, 3)), "flat": rng.uniform([0.8, 0.8, 0.01], [1.2, 1.2, 0.2], (n, 3)),
         "inverted": rng.uniform([1.1, 0.8, -0.6], [1.4, 1.0, -0.2], (n, 3))}[kind]
    A = _rotations(rng, n)
    return _rotations(rng, n) @ (A * s[:, None, :]) @ A.transpose(0, 2, 1)


def _reference(F, plastic):
    U, s, Vt = np.linalg.svd(F)
    for M, fix in ((U, lambda i: U[i, :, 2].__imul__(-1)), (Vt, lambda i: Vt[i, 2].__imul__(-1))):
        for i in np.nonzero(np.linalg.det(M) < 0)[0]:
            fix(i)
            s[i, 2] *= -1
    ys = np.full(len(F), YS)
    if plastic:
        eps = np.log(np.maximum(s, 0.01))
        hat = eps - eps.mean(1, keepdims=True)
        size = np.linalg.norm(hat, axis=1) + 1e-6
        over = 2 * MU * (size - 1e-6) > YS
        k = (size - YS / (2 * MU)) / size
        ys = np.where(over, YS - SOFT * np.abs(k) * (size - 1e-6), YS)
        s = np.where(over[:, None], np.exp(eps - k[:, None] * hat), s)
    Fe = (U * s[:, None, :]) @ Vt
    J = s.prod(1)
    tau = (U * (2 * MU * (s - 1) * s)[:, None, :]) @ U.transpose(0, 2, 1) + (LAM * J * (J - 1))[:, None, None] * np.eye(3)
    return Fe, tau, ys, np.abs(s).max(1), np.abs(J)


@pytest.mark.parametrize("material", [0, 5])
@pytest.mark.parametrize("kind", ["strain1e-6", "strain1e-3", "strain0.05", "strain0.2", "yield", "stretched", "flat",
                                  "inverted"])
def test_fixed_corotated_stress(material, kind):
    from empm_b200 import _native as N

    rng = np.random.default_rng(11)
    F = _cases(rng, kind).astype(np.float32)
    Fe, tau, ys, s, J = _reference(F.astype(np.float64), material == 5)
    n = len(F)
    dev = "cuda:0"
    t = torch.as_tensor(F.reshape(n, 9), device=dev).contiguous()
    mu, lam, y = (torch.full((n,), v, device=dev) for v in (MU, LAM, YS))
    out_F, out_t = torch.empty_like(t), torch.empty_like(t)
    p = N.EmpmModelParams()
    p.n_grid, p.grid_lim, p.material, p.softening = 32, 1.0, material, SOFT
    N.check(N.lib().empm_debug_stress(ctypes.byref(p), t.data_ptr(), mu.data_ptr(), lam.data_ptr(), y.data_ptr(),
                                      1e-4, out_F.data_ptr(), out_t.data_ptr(), n, None))
    torch.cuda.synchronize()
    eF = np.abs(out_F.double().cpu().numpy().reshape(n, 3, 3) - Fe).max((1, 2))
    et = np.abs(out_t.double().cpu().numpy().reshape(n, 3, 3) - tau).max((1, 2))
    assert (eF <= 1e-5 * s).all(), float((eF / s).max())
    scale = 2 * MU * s ** 2 + LAM * J * (1 + J)
    assert (et <= 1e-5 * scale).all(), float((et / scale).max())
    # softening: the strain past the surface is known to a few 1e-7
    assert (np.abs(y.double().cpu().numpy() - ys) <= 1e-5 * YS).all()
