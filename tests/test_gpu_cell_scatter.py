"""The per-cell scatter and the fused kernels where group and tile sizes can go
wrong: one particle, warps and CTAs not filled, cells with more particles than a
group holds, every particle in its own cell, unsimulated particles among the
others, and particles whose stencil leaves the grid. Checked against the oracle in
64 bits, with the direct kernels (one reduction per particle and node) beside it.

Tolerance: sums of the m particles on a node (those of 27 cells) carry a few
sqrt(m) 2^-24 of their size, so velocities are held to 2e-5 + 8 sqrt(m) 2^-24 of the
largest, and C and F to that times 4 / dx and dt / dx. Where the sum on a node
nearly cancels (the border nodes of the bodies that leave the grid reach 100 m/s),
the error is that of its terms instead: there the scatter is held to twice the
error of the direct kernels, which sum the same terms."""
import numpy as np
import pytest
import torch

from empm_b200.mpm_data_structure import MPMModelStruct, MPMStateStruct
from empm_b200.mpm_solver_diff import MPMWARPDiff
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV, G, DT = "cuda:0", 32, 1e-4


def _state(kind, n, seed=5):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.3, 0.6, (n, 3))
    if kind == "crowded":      # all in a few cells
        x = 0.4 + rng.uniform(0, 1.5 / G, (n, 3))
    elif kind == "lattice":    # one particle per cell
        k = np.arange(n)
        x = (np.stack([k % 20, (k // 20) % 20, k // 400], 1) + 6.03 + 0.9 * rng.uniform(size=(n, 3))) / G
    elif kind == "outside":    # every fourth at the border or beyond
        x[::4] = rng.uniform(-0.02, 1.02, (len(x[::4]), 3))
    t = lambda a: torch.as_tensor(np.asarray(a, np.float32), device=DEV)  # noqa: E731
    st = MPMStateStruct()
    st.init(n, device=DEV)
    st.from_torch(t(x), t(np.full(n, 0.027 / n)), None, t(rng.normal(0, 0.5, (n, 3))), n_grid=G, device=DEV)
    st.reset_density(t(np.full(n, 1e3)), update_mass=True)
    st.particle_C = t(rng.normal(0, 1.0, (n, 3, 3)))
    st.particle_F_trial = t(np.eye(3) + 0.01 * rng.normal(size=(n, 3, 3)))
    if kind == "selected":
        st.set_selection(torch.as_tensor(rng.integers(0, 2, n), device=DEV))
    return st


def _solver(n, material):
    md = MPMModelStruct()
    md.init(n, device=DEV)
    md.init_other_params(n_grid=G)
    md.gravitational_accelaration = (0.0, -9.8, 0.0)
    sv = MPMWARPDiff()
    sv.initialize(n, n_grid=G, device=DEV)
    sv.set_parameters_dict(md, None, {"material": material})
    md.E.fill_(2e4)
    md.nu.fill_(0.3)
    md.yield_stress.fill_(1e3)
    md.finalize_mu_lam(n)
    return sv, md


@pytest.mark.parametrize("kind,n,material", [
    ("box", 1, "jelly"), ("box", 31, "plasticine"), ("box", 33, "jelly"), ("box", 65, "sand"), ("box", 127, "jelly"),
    ("crowded", 2500, "jelly"), ("crowded", 60_000, "plasticine"), ("lattice", 6000, "plasticine"),
    ("selected", 4001, "jelly"), ("outside", 4099, "jelly"), ("outside", 60_003, "neo-hookean"),
    ("box", 50_001, "plasticine")])
@pytest.mark.parametrize("steps", [1, 3])
def test_cell_scatter_matches_oracle(kind, n, material, steps):
    res = {}
    for path in ("sorted", "direct"):
        sv, md = _solver(n, material)
        sv.sort_every = 32 if path == "sorted" else 0
        a = _state(kind, n)
        b = a.partial_clone()
        r = sv.rollout(md, a, b, DT, steps)
        res[path] = [t.double().clone() for t in (r.particle_x, r.particle_v, r.particle_C, r.particle_F_trial)]
        res[path].append(sv.read_status())
    f = lambda t: t.double().cpu().numpy()  # noqa: E731
    st = _state(kind, n)
    sim = O.OracleSim(f(st.particle_x), f(st.particle_v), f(st.particle_vol), f(st.particle_mass), 2e4, 0.3, n_grid=G,
                      material={"jelly": 0, "sand": 2, "plasticine": 5, "neo-hookean": 6}[material],
                      gravity=(0.0, -9.8, 0.0), yield_stress=1e3,
                      selection=st.particle_selection.cpu().numpy() if kind == "selected" else None)
    sim.C, sim.F_trial = f(st.particle_C).reshape(n, 9).copy(), f(st.particle_F_trial).reshape(n, 9).copy()
    sim.rollout(DT, steps)
    exact = [torch.as_tensor(t.reshape(n, *s), device=DEV) for t, s in
             ((sim.x, (3,)), (sim.v, (3,)), (sim.C, (3, 3)), (sim.F_trial, (3, 3)))]
    per_cell = n / 8 if kind == "crowded" else 8 + n / 900
    tol_v = (2e-5 + 8 * (27 * per_cell) ** 0.5 * 2.0 ** -24) * float(exact[1].abs().max())
    for got, direct, want, tol in zip(res["sorted"], res["direct"], exact,
                                      (steps * DT * tol_v + 1e-6, tol_v, 4 * G * tol_v, steps * DT * G * tol_v + 2e-6)):
        assert torch.isfinite(got).all()
        err, own = float((got - want).abs().max()), float((direct - want).abs().max())
        assert err <= max(tol, 2 * own), (kind, n, err, own, tol)
    assert res["sorted"][4] == res["direct"][4]
