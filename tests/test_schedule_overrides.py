"""Solvers that resolve their substeps in their own way (a subclass or an instance that
replaces a step of it) get the schedule that their own methods make (no GPU)."""
import copy

import pytest

from empm_b200 import _native as N
from empm_b200.mpm_solver_diff import MPMWARPDiff
from tests.test_schedule_native import _general, _solver


class Slow(MPMWARPDiff):
    @staticmethod
    def _move_point(t, dt, param):
        MPMWARPDiff._move_point(t, 0.5 * dt, param)


class Late(MPMWARPDiff):
    def _gate(self, p, t32, dt):
        return MPMWARPDiff._gate(self, p, t32, dt) if t32 > 5e-4 else N.GATE_OFF


def _as(cls):
    sv = _solver(3, 9, 2)
    for i, p in enumerate(sv.collider_params):
        p._kind, p.active, p.end_time = N.COLL_CUBOID_VELOCITY, True, 999.0
        sv.modify_bc[i] = None
    sv.__class__ = cls
    sv.modify_bc = [sv._move_point] * len(sv.modify_bc)
    return sv


@pytest.mark.parametrize("how", ["slow", "late", "instance", "plain"])
def test_overridden_steps_are_run(how):
    sv = _as({"slow": Slow, "late": Late}.get(how, MPMWARPDiff))
    if how == "instance":
        sv._modify = lambda t, dt: None
    ref = copy.deepcopy(sv)
    if how == "instance":
        ref._modify = lambda t, dt: None
    want, t_want = _general(ref, 0.0, 1e-4, 12)
    got, t_got = sv.build_schedule(0.0, 1e-4, 12)
    assert bytes(got) == bytes(want) and t_got == t_want
    assert [p.point for p in sv.collider_params] == [p.point for p in ref.collider_params]
    assert (sv._windows(0.0, 1e-4) is None) == (how != "plain")
