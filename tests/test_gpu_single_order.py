"""Single substeps of many particles, whose P2G runs in cell order: sizes at the
line to the caller's order and past it, unsimulated particles, more particles per
cell than a group of the scatter holds, repeated calls.
Same oracle and tolerances as the per-cell scatter's tests (test_gpu_cell_scatter)."""
import pytest
import torch

from oracle import oracle as O
from tests.test_gpu_cell_scatter import DEV, DT, G, _solver, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,material", [
    ("box", 65_535, "jelly"), ("box", 65_536, "sand"), ("box", 65_537, "jelly"), ("selected", 70_001, "plasticine"),
    ("crowded", 80_001, "jelly")])
@pytest.mark.parametrize("inplace", [False, True])
def test_ordered_substep_matches_oracle(kind, n, material, inplace):
    res = {}
    for path in ("order", "direct"):
        sv, md = _solver(n, material)
        sv.sort_every = 32 if path == "order" else 0
        for _ in range(2):                        # the second call finds the first one's buffers
            a = _state(kind, n)
            if inplace:
                sv.p2g2p(md, a, 0, DT)
                r = a
            else:
                r = a.partial_clone()
                sv.p2g2p_differentiable(md, a, r, DT)
        res[path] = [t.double().clone() for t in (r.particle_x, r.particle_v, r.particle_C, r.particle_F_trial)]
        res[path].append(sv.read_status())
    f = lambda t: t.double().cpu().numpy()  # noqa: E731
    st = _state(kind, n)
    sim = O.OracleSim(f(st.particle_x), f(st.particle_v), f(st.particle_vol), f(st.particle_mass), 2e4, 0.3, n_grid=G,
                      material={"jelly": 0, "sand": 2, "plasticine": 5}[material], gravity=(0.0, -9.8, 0.0),
                      yield_stress=1e3, selection=st.particle_selection.cpu().numpy() if kind == "selected" else None)
    sim.C, sim.F_trial = f(st.particle_C).reshape(n, 9).copy(), f(st.particle_F_trial).reshape(n, 9).copy()
    sim.rollout(DT, 1)
    exact = [torch.as_tensor(t.reshape(n, *s), device=DEV) for t, s in
             ((sim.x, (3,)), (sim.v, (3,)), (sim.C, (3, 3)), (sim.F_trial, (3, 3)))]
    if kind == "selected":                        # an unsimulated particle's outputs are the call's, not the oracle's
        on = st.particle_selection == 0
        exact = [t[on] for t in exact]
        res = {k: [t[on] for t in v[:4]] + v[4:] for k, v in res.items()}
    per_cell = n / 8 if kind == "crowded" else 8 + n / 900
    tol_v = (2e-5 + 8 * (27 * per_cell) ** 0.5 * 2.0 ** -24) * float(exact[1].abs().max())
    for got, direct, want, tol in zip(res["order"], res["direct"], exact,
                                      (DT * tol_v + 1e-6, tol_v, 4 * G * tol_v, DT * G * tol_v + 2e-6)):
        assert torch.isfinite(got).all()
        err, own = float((got - want).abs().max()), float((direct - want).abs().max())
        assert err <= max(tol, 2 * own), (kind, n, err, own, tol)
    assert res["order"][4] == res["direct"][4]
