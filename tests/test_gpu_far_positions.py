"""Particles so far from the grid that their cell does not fit an int: they contribute to
no node, the status names them, and the others' results are those without them, on
every route of a substep. (A base node of 2^31 - 1, to which the conversion saturates,
plus 2 is below the grid's size when it wraps: such a particle's nodes were taken for
nodes of the grid.) Tolerances of the per-cell scatter's tests."""
import pytest
import torch

from empm_b200 import _native as N
from tests.test_gpu_cell_scatter import DEV, DT, G, _solver, _state

pytestmark = pytest.mark.gpu
FAR = [(1e12, 0.5, 0.5), (0.5, -1e12, 0.5), (0.5, 0.5, 3e30), (7e7, 0.5, 0.5), (0.5, 0.5, -6.8e7), (60.0, 0.5, -40.0),
       (float("inf"), 0.5, 0.5), (0.5, float("-inf"), 0.5)]


@pytest.mark.parametrize("n,route", [
    (4001, "rollout"), (4001, "unsorted"), (4001, "tile"), (4001, "substep"), (4001, "inplace"), (66_001, "substep"),
    (66_001, "inplace"), (4001, "restart")])
def test_far_particles_touch_nothing(n, route):
    res = []
    for far in (True, False):
        m = n + len(FAR) if far else n
        sv, md = _solver(m, "jelly")
        a, full = _state("box", m), _state("box", n)
        put = lambda dst, src: dst[:n].copy_(src[:n])  # noqa: E731
        put(a._x4, full._x4), put(a._v4, full._v4), put(a.particle_vol, full.particle_vol)
        C, F = a.particle_C.clone(), a.particle_F_trial.clone()
        put(C, full.particle_C), put(F, full.particle_F_trial)
        a.particle_C, a.particle_F_trial = C, F
        if far:
            a._x4[n:, :3] = torch.tensor(FAR, device=DEV)
        b = a.partial_clone()
        if route in ("rollout", "unsorted", "tile"):
            sv.sort_every, sv.p2g_mode, sv.g2p_tile = {"rollout": (32, 2, False), "unsorted": (0, 2, False),
                                                       "tile": (32, 1, True)}[route]
            r = sv.rollout(md, a, b, DT, 1)
        elif route == "inplace":
            sv.p2g2p(md, a, 0, DT)
            r = a
        elif route == "restart":
            ctx = sv._context(md, m, a.device)
            target = a.particle_x + 0.01
            N.check(ctx.L.empm_restart_F(ctx.ptr, a._particles(), target.contiguous().data_ptr(), None, None, None),
                    ctx.ptr)
            r = a
        else:
            sv.p2g2p_differentiable(md, a, b, DT)
            r = b
        res.append([t[:n].double().clone() for t in (r.particle_x, r.particle_v, r.particle_C, r.particle_F_trial)])
        res[-1].append(sv.read_status())
    tol_v = (2e-5 + 8 * (27 * (8 + n / 900)) ** 0.5 * 2.0 ** -24) * float(res[1][1].abs().max())
    for got, want, tol in zip(res[0], res[1], (DT * tol_v + 1e-6, tol_v, 4 * G * tol_v, DT * G * tol_v + 2e-6)):
        assert torch.isfinite(got).all()
        assert float((got - want).abs().max()) <= tol
    assert res[0][4] & ~res[1][4]            # the bit of particles outside the grid
