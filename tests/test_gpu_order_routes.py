"""Single substeps in cell order on every route that can take it: the first one of a
context (whose buffers are part of its grid's allocation), particle modifiers, several
instances with different materials, positions outside the grid, a context made larger,
and grids with more blocks than particles, which keep the caller's order. Checked
against the direct kernel, which sums the same terms in another order, with the
tolerances of the per-cell scatter's tests (test_gpu_cell_scatter)."""
import ctypes

import numpy as np
import pytest
import torch

from empm_b200 import _native as N
from empm_b200.batch import BatchedMPM, InstanceSpec
from empm_b200.mpm_data_structure import _stream_ptr
from tests.test_gpu_cell_scatter import DEV, DT, G, _solver, _state

pytestmark = pytest.mark.gpu


def _fields(st):
    return [t.double().clone() for t in (st.particle_x, st.particle_v, st.particle_C, st.particle_F_trial)]


def _check(got, want, per_cell, grid=G):
    tol_v = (2e-5 + 8 * (27 * per_cell) ** 0.5 * 2.0 ** -24) * float(want[1].abs().max())
    for a, b, tol in zip(got, want, (DT * tol_v + 1e-6, tol_v, 4 * grid * tol_v, DT * grid * tol_v + 2e-6)):
        assert torch.isfinite(b).all()
        assert float((a - b).abs().max()) <= tol, (float((a - b).abs().max()), tol)


def test_the_first_substep_of_a_context_allocates_nothing():
    n = 200_000
    runs = []
    for _ in range(2):                       # the first run also loads the kernels
        sv, md = _solver(n, "jelly")
        sv.n_grid = md.n_grid = 128
        a = _state("box", n)
        b = a.partial_clone()
        ctx = sv._context(md, n, a.device)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        sv.p2g2p_differentiable(md, a, b, DT)
        torch.cuda.synchronize()
        runs.append(free - torch.cuda.mem_get_info()[0])
        assert sv._ctx is ctx
    assert runs[1] == 0, runs


@pytest.mark.parametrize("inplace", [False, True])
def test_particle_modifiers(inplace):
    n, res = 66_001, []
    for sort_every in (32, 0):
        sv, md = _solver(n, "plasticine")
        sv.sort_every = sort_every
        a = _state("box", n)
        sv.add_impulse_on_particles(a, (2e-4, 0.0, 1e-4), DT, [0.4, 0.4, 0.4], [0.08, 0.08, 0.08], num_dt=3)
        sv.enforce_particle_velocity_translation(a, [0.55, 0.5, 0.5], [0.04, 0.2, 0.2], [0.3, 0.0, -0.2], 0.0, 1.0)
        if inplace:
            sv.p2g2p(md, a, 0, DT)
            res.append(_fields(a))
        else:
            b = a.partial_clone()
            sv.p2g2p_differentiable(md, a, b, DT)
            res.append(_fields(b) + [a.particle_v.double().clone()])
    _check(*res, 8 + n / 900)
    if not inplace:                          # the velocity after the modifiers, in the input
        assert torch.equal(res[0][4], res[1][4])
        assert not torch.equal(res[0][4], _state("box", n).particle_v.double())


def test_positions_outside_the_grid():
    """Every fourth particle at the border or beyond; one velocity for all and no strain,
    so that no node's sum cancels."""
    n, res = 66_003, []
    for sort_every in (32, 0):
        sv, md = _solver(n, "jelly")
        md.gravitational_accelaration = (0.0, 0.0, 0.0)
        sv.sort_every = sort_every
        a = _state("outside", n)
        a.particle_v = torch.tensor([[0.5, -0.25, 1.0]], device=DEV).expand(n, 3).contiguous()
        a.particle_C = torch.zeros(n, 3, 3, device=DEV)
        a.particle_F_trial = torch.eye(3, device=DEV).expand(n, 3, 3).contiguous()
        b = a.partial_clone()
        sv.p2g2p_differentiable(md, a, b, DT)
        res.append(_fields(b))
        res[-1].append(sv.read_status())
    _check(*res, 8 + n / 900)
    assert res[0][4] == res[1][4] != 0       # the status bit of particles outside


def _specs():
    rng = np.random.default_rng(2)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    return [InstanceSpec(x=f(rng.uniform(0.3, 0.6, (n, 3))), vol=f(np.full(n, 0.027 / n)), rho=f(np.full(n, 1e3)),
                         E=f(np.full(n, 2e4)), nu=f(np.full(n, 0.3)), n_grid=g, v=f(rng.normal(0, 0.5, (n, 3))),
                         material=m, yield_stress=f(np.full(n, 1e3)))
            for n, g, m in ((30_001, 32, "jelly"), (40_007, 24, "sand"), (999, 16, "plasticine"))]


def test_several_instances():
    res = []
    for sort_every in (32, 0):
        b = BatchedMPM(_specs(), device=DEV)
        b.sort_every = sort_every
        b._apply_options()
        table, _ = b._schedule(DT, 1)
        mat = N.EmpmMaterial(b.vol.data_ptr(), b.mu.data_ptr(), b.lam.data_ptr(), b.yield_stress.data_ptr(), None,
                             b._Fe.data_ptr())
        for _ in range(2):                   # the second call finds the first one's buffers
            N.check(b.L.empm_substep(b.ptr, b._views(0), b._views(1), mat, table, _stream_ptr(b.device)), b.ptr)
        b.cur = 1
        F = b.F_trial().double().clone()
        b._F[1], keep = b._C[1], b._F[1]
        C = b.F_trial().double().clone()
        b._F[1] = keep
        res.append([b.positions().double().clone(), b.velocities().double().clone(), C, F])
    _check(*res, 8 + 40_007 / 250)


def test_a_context_made_larger():
    n, res = 70_003, []
    for sort_every in (32, 0):
        sv, md = _solver(n, "jelly")
        a = _state("box", n)
        b = a.partial_clone()
        L, p, ctx = N.lib(), md._params(), ctypes.c_void_p()
        small = N.EmpmModelParams.from_buffer_copy(bytes(p))
        small.n_grid = 16
        N.check(L.empm_ctx_create(small, 1000, 4, ctypes.byref(ctx)))
        N.check(L.empm_batch_reserve(ctx, n, (G // 4) ** 3, 2), ctx)
        N.check(L.empm_batch_reconfigure(ctx, (N.EmpmModelParams * 1)(p), (ctypes.c_int * 1)(n), 1,
                                         _stream_ptr(a.device)), ctx)
        N.check(L.empm_ctx_set_option(ctx, N.OPT_SORT_EVERY, sort_every), ctx)
        step = N.EmpmStep()
        sv._fill_step(step, 0.0, DT)
        for _ in range(2):
            N.check(L.empm_substep(ctx, a._particles(), b._particles(), sv._material(md, a), step,
                                   _stream_ptr(a.device)), ctx)
        torch.cuda.synchronize()
        res.append(_fields(b))
        N.check(L.empm_ctx_destroy(ctx))
    _check(*res, 8 + n / 900)


def test_more_blocks_than_particles():
    n, grid, res = 65_537, 180, []           # 45^3 blocks
    for sort_every in (32, 0):
        sv, md = _solver(n, "jelly")
        sv.n_grid = md.n_grid = grid
        sv.sort_every = sort_every
        a = _state("box", n)
        b = a.partial_clone()
        sv.p2g2p_differentiable(md, a, b, DT)
        res.append(_fields(b))
    _check(*res, 8, grid)
