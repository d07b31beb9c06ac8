"""Schedules filled by the library against the substep-by-substep Python fill
(no GPU): every byte of the tables, the moved points and the end time."""
import copy
import itertools
import random

import pytest

from empm_b200 import _native as N
from empm_b200.mpm_data_structure import Dirichlet_collider, GridCollider, Impulse_modifier, ParticleVelocityModifier
from empm_b200.mpm_solver_diff import MPMWARPDiff


def _solver(seed, n_colliders, n_modifiers):
    rng = random.Random(seed)
    vec = lambda: tuple(rng.uniform(-1, 1) for _ in range(3))  # noqa: E731
    sv = MPMWARPDiff()
    sv.initialize(4, n_grid=8, grid_lim=1.0, device="cpu")
    for _ in range(n_colliders):
        kind = rng.choice([N.COLL_SURFACE, N.COLL_GEOMETRY, N.COLL_GRID_VELOCITY, N.COLL_CUBOID_VELOCITY,
                           N.COLL_BOUNDING_BOX, N.COLL_GRID_MASK])
        p = GridCollider() if kind == N.COLL_GRID_MASK else Dirichlet_collider()
        p.point, p.start_time, p.end_time = vec(), rng.choice([0.0, 0, 1e-3, 2.5e-3]), rng.choice([999.0, 4e-3, 6e-3])
        if kind != N.COLL_GRID_MASK:
            p.velocity, p.size, p.radius, p.friction = vec(), vec(), rng.random(), rng.random()
            p.active, p.reset = rng.random() < 0.7, rng.choice([0, 1])
        moves = kind in (N.COLL_GRID_VELOCITY, N.COLL_CUBOID_VELOCITY)
        sv._register(p, kind, rng.randrange(4), modify=sv._move_point if moves else None)
    for _ in range(n_modifiers):
        p = rng.choice([Impulse_modifier, ParticleVelocityModifier])()
        p.start_time, p.end_time, p.velocity, p.force = rng.choice([0.0, 1e-3]), rng.choice([999.0, 5e-3]), vec(), vec()
        sv.particle_velocity_modifier_params.append(p)
    return sv


def _general(sv, t, dt, n):
    table = (N.EmpmStep * n)()
    for s in range(n):
        sv._fill_step(table[s], t, dt)
        sv._modify(t, dt)
        t = t + dt
    return table, t


@pytest.mark.parametrize("seed,n,t0,dt", [(s, n, t0, dt) for (n, t0, dt), s in itertools.product(
    [(1, 0.0, 1e-4), (2, 0.0, 1e-4), (120, 0.0, 1e-4), (77, 1.7e-3, 1.0 / 24 / 700), (64, 0.1, 1e-3)], range(6))])
def test_native_fill_equals_the_python_fill(seed, n, t0, dt):
    sv = _solver(seed, [0, 1, 3, 5, 9, N.EMPM_MAX_COLLIDERS][seed], [0, 1, 2, 0, 3, N.EMPM_MAX_MODIFIERS][seed])
    ref = copy.deepcopy(sv)
    want, t_want = _general(ref, t0, dt, n)
    got, t_got = sv.build_schedule(t0, dt, n)
    assert bytes(got) == bytes(want) and t_got == t_want
    for a, b in zip(sv.collider_params, ref.collider_params):
        assert a.point == b.point


def test_general_path_keeps_what_the_library_does_not_fill():
    sv = _solver(3, 3, 0)
    assert sv._windows(0.0, 1e-4) is not None
    assert sv._windows(0, 1e-4) is None and sv._windows(float("nan"), 1e-4) is None
    calls = []
    sv.modify_bc[1] = lambda t, dt, p: calls.append(t)
    assert sv._windows(0.0, 1e-4) is None
    sv.build_schedule(0.0, 1e-4, 4)
    assert len(calls) == 4


def test_bad_arguments_are_refused():
    L, end = N.lib(), N.ctypes.c_double()
    table = (N.EmpmStep * 2)()
    assert L.empm_schedule_fill(None, 1, 2, 0.0, 1e-4, None, None, end) == -1
    assert L.empm_schedule_fill(table, 0, 2, 0.0, 1e-4, None, None, end) == -1
    table[0].n_colliders = 1
    assert L.empm_schedule_fill(table, 1, 2, 0.0, 1e-4, None, None, end) == -1
