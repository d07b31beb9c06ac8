"""The work whose speed is looked after: what programs built on this library
have it do, with sizes from the library's own workloads and tests.

Kinds of case (see ``listed`` for what each listed one stands for):

  substep     one ``MPMWARPDiff.p2g2p_differentiable`` call
  frames      ``WarpMPMWrapper.advance_to`` from a given pose
  rollout     ``MPMWARPDiff.rollout`` of a plasticine scene with a moving tool
  population  ``BatchedMPM.load_state`` + ``rollout`` of an uneven batch
  generation  ``PopulationEvaluator.rollout`` + ``losses``: one CMA-ES generation
  gradient    ``MPMDifferentiableSimulation.apply`` + its backward
  segment     ``CheckpointedRollout.forward`` + ``backward`` (recomputed or stored)
  chamfer     ``chamfer_pairs`` and its gradient
  gaussians   one frame of ``MotionInterpolator``
  neighbours  ``knn_weights_sparse``

Inputs are synthetic, drawn from the seed. ``exact`` evaluates the same maps
with plain torch in 64 bits (matrix functions in place of an SVD).
"""
import math

import numpy as np
import torch

from empm_b200 import dynamic_utils as du
from empm_b200.adjoint import CheckpointedRollout
from empm_b200.batch import BatchedMPM, InstanceSpec
from empm_b200.cma_driver import PopulationEvaluator
from empm_b200.interface import MPMDifferentiableSimulation
from empm_b200.losses import chamfer_pairs
from empm_b200.mpm_data_structure import MPMModelStruct, MPMStateStruct
from empm_b200.mpm_solver_diff import MPMWARPDiff
from empm_b200.warp_mpm_wrapper import WarpMPMWrapper

DEV = "cuda:0"
GRAVITY = (0.0, -9.8, 0.0)
YIELD_FREE = ("jelly", "metal", "sand", "foam", "neo-hookean")   # materials whose scalars a substep leaves alone


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an interactive program stepping a small body itself: latency and launches
        {"name": "substep_4k", "kind": "substep", "material": "jelly", "n": 4000, "grid": 32},
        # the same on a large scene, as a step callback makes every substep a call of its own
        {"name": "substep_500k", "kind": "substep", "material": "sand", "n": 500_000, "grid": 128},
        # the interactive simulator: frames of 50 substeps of a 20k-particle body
        {"name": "frames_20k", "kind": "frames", "material": "jelly", "n": 20_000, "grid": 48, "frames": 4,
         "substeps": 50},
        # one large forward simulation, two bodies and a moving tool
        {"name": "rollout_500k", "kind": "rollout", "n": 500_000, "grid": 128, "steps": 100},
        # a CMA-ES population of uneven members over several grids
        {"name": "population_32", "kind": "population", "members": 32, "lo": 20_000, "hi": 300_000, "steps": 150},
        # one whole CMA-ES generation on a small body, with its losses
        {"name": "generation_12", "kind": "generation", "members": 12, "n": 2500, "grid": 32, "frames": 5,
         "substeps": 20},
        # one training iteration on a small body (odd size)
        {"name": "gradient_16k", "kind": "gradient", "material": "plasticine", "n": 16_001, "grid": 96, "steps": 60},
        # one training iteration at the full differentiable size
        {"name": "gradient_200k", "kind": "gradient", "material": "plasticine", "n": 200_000, "grid": 96,
         "steps": 100},
        # gradients of a rollout that is recomputed from checkpoints (tapes that do not fit)
        {"name": "segment_50k", "kind": "segment", "material": "neo-hookean", "n": 50_001, "grid": 64, "steps": 40,
         "store": False},
        # loss of a predicted cloud against an observed one, with its gradient
        {"name": "chamfer_100k", "kind": "chamfer", "pairs": 1, "n": 100_003, "m": 80_000},
        # one rendered frame: a million Gaussians follow 100k particles
        {"name": "gaussians_1m", "kind": "gaussians", "bones": 100_000, "n": 1_000_000, "k": 16, "quat": True},
        # a new scene: every Gaussian's nearest particles
        {"name": "neighbours_500k", "kind": "neighbours", "bones": 50_000, "n": 500_000, "k": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["substep", "frames", "rollout", "population", "generation", "gradient", "segment", "chamfer",
                       "gaussians", "neighbours"])
    if kind == "substep":
        return {"kind": kind, "material": rng.choice(YIELD_FREE), "n": _log(rng, 1000, 500_000),
                "grid": rng.randint(24, 128)}
    if kind == "frames":
        return {"kind": kind, "material": rng.choice(YIELD_FREE), "n": _log(rng, 2000, 100_000),
                "grid": rng.randint(32, 96), "frames": rng.randint(1, 4), "substeps": rng.randint(10, 50)}
    if kind == "rollout":
        return {"kind": kind, "n": _log(rng, 10_000, 500_000), "grid": rng.randint(48, 128),
                "steps": rng.randint(20, 100)}
    if kind == "population":
        return {"kind": kind, "members": rng.randint(2, 32), "lo": _log(rng, 2000, 20_000),
                "hi": _log(rng, 25_000, 300_000), "steps": rng.randint(20, 120)}
    if kind == "generation":
        return {"kind": kind, "members": rng.randint(4, 16), "n": rng.randint(800, 5000), "grid": rng.randint(24, 48),
                "frames": rng.randint(1, 5), "substeps": rng.randint(10, 25)}
    if kind == "gradient":
        return {"kind": kind, "material": rng.choice(["plasticine", "jelly"]), "n": _log(rng, 5000, 200_000),
                "grid": rng.randint(48, 96), "steps": rng.randint(10, 100)}
    if kind == "segment":
        return {"kind": kind, "material": rng.choice(["neo-hookean", "jelly"]), "n": _log(rng, 5000, 100_000),
                "grid": rng.randint(40, 96), "steps": rng.randint(10, 50), "store": rng.random() < 0.5}
    if kind == "chamfer":
        pairs = _log(rng, 1, 60)
        top = 100_000 / pairs
        return {"kind": kind, "pairs": pairs, "n": _log(rng, 600, max(1000, top)), "m": _log(rng, 600, max(1000, top))}
    if kind == "gaussians":
        return {"kind": kind, "bones": _log(rng, 5000, 100_000), "n": _log(rng, 30_000, 1_000_000),
                "k": rng.choice([5, 8, 16, 16]), "quat": rng.random() < 0.8}
    return {"kind": kind, "bones": _log(rng, 2000, 50_000), "n": _log(rng, 10_000, 500_000),
            "k": rng.choice([1, 5, 8, 16, 20])}


#: rough operations of one particle and substep: return map, scatter and gather of 27 nodes
FLOPS = 1300


def work(case):
    """Inputs read once and outputs written once, and the operations between
    them; what a path hands from one substep to the next is left out."""
    k = case["kind"]
    if k == "substep":
        return {"bytes": 208 * case["n"], "flops": FLOPS * case["n"]}
    if k == "frames":
        return {"bytes": (112 + 12 * (case["frames"] + 1)) * case["n"],
                "flops": FLOPS * case["n"] * case["frames"] * case["substeps"]}
    if k == "rollout":
        return {"bytes": 224 * case["n"], "flops": FLOPS * case["n"] * case["steps"]}
    if k == "population":
        n = sum(s["n"] for s in _members(case, 0))
        return {"bytes": 224 * n, "flops": FLOPS * n * case["steps"]}
    if k == "generation":
        n = case["members"] * case["n"]
        return {"bytes": (60 + 12 * (case["frames"] + 1)) * n,
                "flops": FLOPS * n * case["frames"] * case["substeps"] + 16 * n * case["frames"] * 200}
    if k in ("gradient", "segment"):
        return {"bytes": 300 * case["n"], "flops": 3.5 * FLOPS * case["n"] * case["steps"]}
    if k == "chamfer":
        p = case["pairs"] * (case["n"] + case["m"])
        return {"bytes": 24 * p, "flops": 8 * 200 * p}
    if k == "gaussians":
        return {"bytes": (56 + 4 * case["k"]) * case["n"] + (24 + 64) * case["bones"],
                "flops": case["n"] * case["k"] * 70 + case["bones"] * (16 * 30 + 600)}
    return {"bytes": 12 * (case["n"] + case["bones"]) + 12 * case["k"] * case["n"],
            "flops": 8 * 27 * 2 * case["k"] * case["n"]}


# ---------------------------------------------------------------------------
# inputs, from the seed alone (float32 on the device unless said otherwise)
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _full(n, v):
    return torch.full((n,), float(v), device=DEV)


def _side(n, grid, ppc=8.0):
    """Edge of a cube that holds n particles at about ppc per cell."""
    return min(max((n / (ppc * grid ** 3)) ** (1.0 / 3.0), 0.15), 0.6)


def _walls(grid):
    """Sticky floor between two node planes, slip walls."""
    return [dict(kind="surface", point=[0.0, 3.5 / grid, 0.0], normal=[0.0, 1.0, 0.0], surface="sticky"),
            dict(kind="bbox")]


def _body(case, seed, moving=True):
    """One body above the floor: positions, velocities and a strained state."""
    n, grid, g = case["n"], case["grid"], _gen(seed)
    side = _side(n, grid)
    lo = 0.15 + (0.7 - side) * _rand(g, 3)
    x = lo + side * _rand(g, n, 3)
    v = 0.2 * _randn(g, 3) + 0.05 * _randn(g, n, 3) if moving else torch.zeros(n, 3, device=DEV)
    eye = torch.eye(3, device=DEV)
    return {"x": x, "v": v, "F": eye + 0.01 * _randn(g, n, 3, 3), "C": 2.0 * _randn(g, n, 3, 3),
            "vol": _full(n, side ** 3 / n), "rho": _full(n, 1000.0), "E": _full(n, 2e4), "nu": _full(n, 0.3),
            "ys": _full(n, 2e3), "target": x + 0.01 * torch.sin(9.0 * x) + 0.005 * _randn(g, 3)}


def _scene(case, seed):
    """Two plasticine bodies of scattered stiffness; a tool comes down on one."""
    n, g = case["n"], _gen(seed)
    h = n // 2
    a = torch.tensor([0.15, 0.10, 0.15], device=DEV) + 0.3 * _rand(g, h, 3)
    b = torch.tensor([0.55, 0.10, 0.55], device=DEV) + 0.3 * _rand(g, n - h, 3)
    return {"x": torch.cat([a, b]), "v": 0.1 * _randn(g, n, 3) * 0.2 + torch.tensor([0.0, -0.5, 0.0], device=DEV),
            "vol": _full(n, 0.054 / n), "rho": _full(n, 1000.0),
            "E": torch.exp(math.log(1e3) + math.log(100.0) * _rand(g, n)), "nu": 0.2 + 0.25 * _rand(g, n),
            "ys": 500.0 + 4500.0 * _rand(g, n)}


TOOL = {"point": [0.3011, 0.4203, 0.3007], "size": [0.0517, 0.0513, 0.0519], "velocity": [0.0, -0.5, 0.0]}


def _members(case, seed):
    """The members of a population: sizes depend on the case alone (a caller's
    bodies are given), poses and materials on the seed."""
    fixed = np.random.default_rng(case["members"] * 7919 + case["lo"] + case["hi"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["members"]):
        n = int(np.exp(fixed.uniform(np.log(case["lo"]), np.log(case["hi"]))))
        grid = int(fixed.choice([48, 64, 96, 128]))
        side = _side(n, grid)
        out.append({"n": n, "grid": grid, "side": side, "lo": rng.uniform(0.1, 0.9 - side, 3),
                    "E": float(np.exp(rng.normal(np.log(2e4), 0.3))), "nu": float(np.clip(rng.normal(0.3, 0.05), 0.2, 0.45)),
                    "ys": float(np.exp(rng.normal(np.log(2e3), 0.3))), "seed": int(rng.integers(1 << 31))})
    return out


def _member_spec(m):
    rng = np.random.default_rng(m["seed"])
    n = m["n"]
    x = (m["lo"] + m["side"] * rng.random((n, 3), dtype=np.float32)).astype(np.float32)
    full = lambda v: np.full(n, np.float32(v), np.float32)  # noqa: E731
    v = np.zeros((n, 3), np.float32)
    v[:, 1] = -0.5
    return InstanceSpec(x=x, v=v, vol=full(m["side"] ** 3 / n), rho=full(1000.0), E=full(m["E"]), nu=full(m["nu"]),
                        yield_stress=full(m["ys"]), n_grid=m["grid"], material="plasticine", gravity=GRAVITY,
                        colliders=_walls(m["grid"]))


def _generation(case, seed):
    """The body, its observed frames and the candidates of one generation."""
    rng = np.random.default_rng(seed)
    n, grid = case["n"], case["grid"]
    x = (np.array([0.35, 0.15, 0.35]) + np.array([0.25, 0.2, 0.25]) * rng.random((n, 3))).astype(np.float32)
    v = np.zeros((n, 3), np.float32)
    v[:, 1] = -1.0
    full = lambda a: np.full(n, np.float32(a), np.float32)  # noqa: E731
    spec = InstanceSpec(x=x, v=v, vol=full(0.25 * 0.2 * 0.25 / n), rho=full(1000.0), E=full(2e4), nu=full(0.3),
                        n_grid=grid, material="jelly", gravity=GRAVITY, colliders=_walls(grid))
    fall = np.arange(case["frames"] + 1)[:, None, None] * case["substeps"] * 2e-4
    target = (x[None] + fall * np.array([0.1, -0.9, 0.05]) + rng.normal(0, 1e-3, (case["frames"] + 1, n, 3)))
    P = np.stack([rng.uniform(0.01, 0.06, case["members"]), rng.uniform(0.2, 0.4, case["members"])], 1)
    return spec, target.astype(np.float32), P


def _clouds(case, seed):
    """Predicted and observed points of the same moved bodies."""
    g, p = _gen(seed), case["pairs"]
    box = 0.3 + 0.2 * _rand(g, p, 1, 3)
    x = 0.2 + box * _rand(g, p, case["n"], 3)
    y = 0.2 + box * _rand(g, p, case["m"], 3)
    y = y + 0.01 * torch.sin(8.0 * y) + 0.005 * _randn(g, p, 1, 3)
    return x.reshape(-1, 3), y.reshape(-1, 3), 0.5 + _rand(g, p)


def _turn(a, degrees):
    axis = torch.tensor([0.3, 1.0, 0.2], dtype=torch.float64, device=DEV)
    axis, t = axis / axis.norm(), math.radians(degrees)
    K = torch.zeros(3, 3, dtype=torch.float64, device=DEV)
    K[0, 1], K[0, 2], K[1, 0], K[1, 2], K[2, 0], K[2, 1] = -axis[2], axis[1], axis[2], -axis[0], -axis[1], axis[0]
    R = torch.eye(3, dtype=torch.float64, device=DEV) + math.sin(t) * K + (1 - math.cos(t)) * (K @ K)
    c = a.double().mean(0)
    return ((a.double() - c) @ R.T + c).float()


def _gaussians(case, seed):
    g = _gen(seed)
    prev = 0.35 + 0.3 * _rand(g, case["bones"], 3)
    cur = _turn(prev, 2.0) + torch.tensor([0.002, -0.004, 0.001], device=DEV) + 2e-4 * _randn(g, case["bones"], 3)
    xyz = 0.33 + 0.34 * _rand(g, case["n"], 3)
    q = _randn(g, case["n"], 4)
    return prev, cur, xyz, q / q.norm(dim=1, keepdim=True)


def _near(queries, points, k, skip_self=False):
    """Exact k nearest points of every query by distance in 64 bits, [n, k]
    indices: candidates from the 27 cells around a query, and from all points
    where those do not hold the k nearest for certain."""
    p, q = points.double(), queries.double()
    want = k + (1 if skip_self else 0)
    lo, hi = p.min(0).values, p.max(0).values
    h = float(((hi - lo).prod() * max(2.0 * want, 8.0) / 4.2 / p.shape[0]) ** (1.0 / 3.0)) * 1.35
    dim = torch.clamp(((hi - lo) / h).long() + 1, min=1)
    cell = lambda a: torch.minimum(torch.clamp(((a - lo) / h).floor().long(), min=0), dim - 1)  # noqa: E731
    flat = lambda c: (c[:, 0] * dim[1] + c[:, 1]) * dim[2] + c[:, 2]  # noqa: E731
    key, order = torch.sort(flat(cell(p)), stable=True)
    total = int(dim.prod())
    start = torch.searchsorted(key, torch.arange(total + 1, device=DEV))
    most = int((start[1:] - start[:-1]).max())
    out = torch.empty(q.shape[0], k, dtype=torch.int64, device=DEV)
    step = max(1, int(2e8) // (27 * most))
    shift = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=DEV)] * 3, indexing="ij"), -1).reshape(27, 3)
    for s in range(0, q.shape[0], step):
        qs = q[s:s + step]
        c = cell(qs)[:, None] + shift
        ok = ((c >= 0) & (c < dim)).all(-1)
        f = torch.where(ok, (c[..., 0] * dim[1] + c[..., 1]) * dim[2] + c[..., 2], torch.zeros_like(c[..., 0]))
        pos = start[f][..., None] + torch.arange(most, device=DEV)
        good = ok[..., None] & (pos < start[f + 1][..., None])
        j = order[torch.clamp(pos, max=p.shape[0] - 1)].reshape(len(qs), -1)
        good = good.reshape(len(qs), -1)
        if skip_self:
            good &= j != torch.arange(s, s + len(qs), device=DEV)[:, None]
        d = torch.where(good, ((qs[:, None] - p[j]) ** 2).sum(-1), torch.full((), math.inf, dtype=torch.float64, device=DEV))
        best, at = torch.topk(d, min(k, d.shape[1]), dim=1, largest=False)
        found = torch.full((len(qs), k), -1, dtype=torch.int64, device=DEV)
        found[:, :best.shape[1]] = j.gather(1, at)
        # a point outside the 27 cells is further than the query's distance to their border
        edge = torch.minimum(qs - (lo + (cell(qs) - 1) * h), lo + (cell(qs) + 2) * h - qs)
        inner = cell(qs)
        edge = torch.where((inner - 1 <= 0) & (inner + 2 >= dim), torch.full_like(edge, math.inf), edge)
        sure = (best[:, -1] < edge.min(1).values.clamp(min=0) ** 2) & (best.shape[1] == k)
        rest = torch.nonzero(~sure).reshape(-1)
        for r in range(0, len(rest), 512):
            i = rest[r:r + 512]
            e = ((qs[i][:, None] - p[None]) ** 2).sum(-1)
            if skip_self:
                e[torch.arange(len(i), device=DEV), i + s] = math.inf
            found[i] = torch.topk(e, k, dim=1, largest=False).indices
        out[s:s + step] = found
    return out


# ---------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------
def _simulator(d, case, material, walls=True):
    n, grid = d["x"].shape[0], case["grid"]
    st = MPMStateStruct()
    st.init(n, device=DEV)
    st.from_torch(d["x"], d["vol"], None, d["v"], n_grid=grid, device=DEV)
    st.reset_density(d["rho"], update_mass=True)
    md = MPMModelStruct()
    md.init(n, device=DEV)
    md.init_other_params(n_grid=grid)
    md.gravitational_accelaration = GRAVITY
    solver = MPMWARPDiff()
    solver.initialize(n, n_grid=grid, device=DEV)
    solver.set_parameters_dict(md, st, {"material": material, "plastic_viscosity": 50.0, "friction_angle": 35.0})
    md.E.copy_(d["E"])
    md.nu.copy_(d["nu"])
    md.finalize_mu_lam(n)
    md.yield_stress.copy_(d["ys"])
    if walls:
        solver.add_surface_collider([0.0, 3.5 / grid, 0.0], [0.0, 1.0, 0.0], "sticky", 0.0)
        solver.add_bounding_box()
    return solver, md, st


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "substep":
        d = _body(case, seed)
        s["solver"], s["model"], s["state"] = _simulator(d, case, case["material"])
        s["state"].continue_from_torch(d["x"], d["v"], d["F"], d["C"])
        s["next"] = s["state"].partial_clone()
    elif k == "frames":
        d = _body(case, seed)
        mpm = WarpMPMWrapper(grid_size=case["grid"], frame_dt=2e-4 * (case["substeps"] + 0.5), sim_dt=2e-4, device=DEV)
        mpm.gravity = list(GRAVITY)
        mpm.material_params = {"material": case["material"], "plastic_viscosity": 50.0, "friction_angle": 35.0,
                               "yield_stress": 2000.0}
        mpm.add_particles(d["x"], d["v"], d["vol"], d["E"], d["nu"], d["rho"])
        mpm.surface_colliders.append([(0.0, 3.5 / case["grid"], 0.0), (0.0, 1.0, 0.0), "sticky", 0.0])
        mpm.initialize()
        mpm.mpm_solver.add_bounding_box()
        s["mpm"], s["x"], s["v"] = mpm, d["x"], d["v"]
    elif k == "rollout":
        d = _scene(case, seed)
        solver, md, st = _simulator(d, case, "plasticine", walls=False)
        solver.add_surface_collider([0.0, 3.5 / case["grid"], 0.0], [0.0, 1.0, 0.0], "sticky", 0.0)
        solver.set_velocity_on_cuboid(TOOL["point"], TOOL["size"], TOOL["velocity"])
        solver.add_bounding_box()
        s.update(solver=solver, model=md, state=st, other=st.partial_clone(), **d)
    elif k == "population":
        s["batch"] = BatchedMPM([_member_spec(m) for m in _members(case, seed)], device=DEV)
    elif k == "generation":
        spec, target, s["P"] = _generation(case, seed)
        s["evaluator"] = PopulationEvaluator(spec, torch.as_tensor(target, device=DEV), 2e-4, case["substeps"], device=DEV)
        s["evaluator"].rollout(s["P"])   # the batch is kept from one generation to the next
    elif k == "gradient":
        d = _body(case, seed)
        s["solver"], s["model"], s["state"] = _simulator(d, case, case["material"])
        s.update(x=d["x"], target=d["target"], ys=d["ys"])
        for name in ("v", "E", "nu", "rho"):
            s[name] = d[name].clone().requires_grad_(True)
    elif k == "segment":
        d = _body(case, seed)
        s["solver"], s["model"], s["state"] = _simulator(d, case, case["material"])
        s["state"].continue_from_torch(d["x"], d["v"], d["F"], d["C"])
        s["gx"], s["gv"] = d["x"] - d["target"], 0.01 * d["v"]
    elif k == "chamfer":
        s["x"], s["y"], s["w"] = _clouds(case, seed)
        s["x"].requires_grad_(True)
    elif k == "gaussians":
        s["prev"], s["cur"], s["xyz"], s["quat"] = _gaussians(case, seed)
        s["mover"] = du.MotionInterpolator(k_relations=case["k"], k_weights=case["k"])
        s["mover"].relations = _near(s["prev"], s["prev"], case["k"], True).to(torch.int32)
        s["mover"].weights_indices = _near(s["xyz"], s["prev"], case["k"]).to(torch.int32)
    else:
        s["prev"], _, s["xyz"], _ = _gaussians(case, seed)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "substep":
        s["solver"].p2g2p_differentiable(s["model"], s["state"], s["next"], 2e-4)
        r = s["next"]
        return {"x": r.particle_x, "v": r.particle_v, "C": r.particle_C, "F": r.particle_F_trial}
    if k == "frames":
        mpm = s["mpm"]
        mpm.mpm_solver.time = 0.0
        mpm.mpm_state.reset_state(s["x"], None, s["v"])
        frames = mpm.advance_to(case["frames"])
        return {"frames": frames, "v": mpm.mpm_state.particle_v}
    if k == "rollout":
        solver, md, st = s["solver"], s["model"], s["state"]
        solver.time = 0.0
        solver.collider_params[1].point = tuple(TOOL["point"])
        st.reset_state(s["x"], None, s["v"])
        md.finalize_mu_lam(st.n_particles)
        md.yield_stress.copy_(s["ys"])
        r = solver.rollout(md, st, s["other"], 1e-4, case["steps"])
        return {"x": r.particle_x, "v": r.particle_v, "F": r.particle_F_trial, "ys": md.yield_stress}
    if k == "population":
        b = s["batch"]
        b.cur, b.time = 0, 0.0
        b.load_state()
        b.rollout(2e-4, case["steps"])
        return {"x": b.positions(), "v": b.velocities(), "F": b.F_trial(), "ys": b.yield_stress}
    if k == "generation":
        ev = s["evaluator"]
        with torch.no_grad():
            frames = ev.rollout(s["P"])
            return {"frames": frames, "losses": ev.losses(frames)}
    if k == "gradient":
        solver, md = s["solver"], s["model"]
        solver.time = 0.0
        md.yield_stress.copy_(s["ys"])
        out = MPMDifferentiableSimulation.apply(solver, s["state"], md, case["steps"], 2e-4, case["steps"], s["x"],
                                                s["v"], s["E"], s["nu"], s["rho"])
        loss = (out - s["target"]).pow(2).mean()
        g = torch.autograd.grad(loss, (s["v"], s["E"], s["nu"], s["rho"]))
        return {"x": out.detach(), "loss": loss.detach(), "gv": g[0], "gE": g[1], "gnu": g[2], "grho": g[3]}
    if k == "segment":
        s["solver"].time = 0.0
        r = CheckpointedRollout(s["solver"], s["model"], s["state"], 2e-4, case["steps"], store=case["store"])
        end = r.forward()
        g = r.backward(g_x=s["gx"], g_v=s["gv"])
        r.release()
        return {"x": end.particle_x, "v": end.particle_v, "F": end.particle_F_trial,
                **{"g_" + n: g[n] for n in ("x", "v", "C", "F", "mu", "lam", "mass")}}
    if k == "chamfer":
        d = chamfer_pairs(s["x"], [case["n"]] * case["pairs"], s["y"], [case["m"]] * case["pairs"])
        return {"d": d.detach(), "g": torch.autograd.grad((d * s["w"]).sum(), s["x"])[0]}
    if k == "gaussians":
        x, q = s["mover"](s["prev"], s["cur"], s["xyz"], s["quat"] if case["quat"] else None)
        return {"xyz": x, "quat": q} if case["quat"] else {"xyz": x}
    w, idx = du.knn_weights_sparse(s["prev"], s["xyz"], case["k"])
    return {"w": w, "idx": idx}


# ---------------------------------------------------------------------------
# the same in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _mm(a, b):
    return (a.unsqueeze(-1) * b.unsqueeze(-3)).sum(-2)


def _t(a):
    return a.transpose(-1, -2)


def _eye_like(a):
    return torch.eye(3, dtype=a.dtype, device=a.device).expand_as(a)


def _tr(a):
    return a.diagonal(dim1=-2, dim2=-1).sum(-1)


def _cof(a):
    r0, r1, r2 = a[..., 0, :], a[..., 1, :], a[..., 2, :]
    return torch.stack([torch.cross(r1, r2, dim=-1), torch.cross(r2, r0, dim=-1), torch.cross(r0, r1, dim=-1)], -2)


def _det(a):
    return (a[..., 0, :] * torch.cross(a[..., 1, :], a[..., 2, :], dim=-1)).sum(-1)


def _polar(F):
    """R of F = R S by Newton's iteration X <- (X + X^-T) / 2."""
    X = F
    for _ in range(9):
        c = _cof(X)
        X = 0.5 * (X + c / (X[..., 0, :] * c[..., 0, :]).sum(-1)[..., None, None])
    return X


def _logm(C):
    """log of a symmetric positive matrix: 2 atanh((C - I)(C + I)^-1)."""
    I = _eye_like(C)  # noqa: E741
    A = C + I
    Y = _mm(C - I, _t(_cof(A)) / _det(A)[..., None, None])
    Z, acc = _mm(Y, Y), torch.zeros_like(Y)
    for m in range(14, -1, -1):
        acc = _mm(Z, acc) + I / (2 * m + 1)
    return 2.0 * _mm(Y, acc)


def _expm(A):
    I = _eye_like(A)  # noqa: E741
    acc = I
    for m in range(16, 0, -1):
        acc = I + _mm(A, acc) / m
    return acc


def _dev(A):
    return A - (_tr(A) / 3.0)[..., None, None] * _eye_like(A)


def _norm(A):
    return A.pow(2).sum((-1, -2)).sqrt()


def _where(mask, new, old):
    """old with new (the rows of mask) put in."""
    return old.index_put((torch.nonzero(mask).reshape(-1),), new)


def _material(name, F, mu, lam, ys, dt):
    """(elastic F, Kirchhoff stress, mu, lam, ys) of a trial F."""
    e3 = lambda a: a[..., None, None]  # noqa: E731
    C = _mm(_t(F), F)
    alpha = math.sqrt(2.0 / 3.0) * 2.0 * math.sin(35.0 / 180.0 * 3.14159265) / (3.0 - math.sin(35.0 / 180.0 * 3.14159265))
    if name in ("plasticine", "metal", "foam"):
        with torch.no_grad():
            over = 2.0 * mu * _norm(_dev(0.5 * _logm(C)))
            over = over - (ys if name != "foam" else math.sqrt(2.0 / 3.0) * ys) > 0
            over &= (ys > 0) if name == "plasticine" else torch.ones_like(over)
        if bool(over.any()):
            i = torch.nonzero(over).reshape(-1)
            Ci, mi, yi = C[i], mu[i], ys[i]
            eps = 0.5 * _logm(Ci)
            hat = _dev(eps)
            if name == "foam":
                s_norm = 2.0 * mi * _norm(hat)
                y = s_norm - math.sqrt(2.0 / 3.0) * yi
                mu_hat = mi * _tr(Ci) / 3.0
                new = s_norm - y / (1.0 + 50.0 / (2.0 * mu_hat * dt))
                k = 1.0 - new / s_norm
            else:
                size = _norm(hat) + 1e-6
                k = (size - yi / (2.0 * mi)) / size
                if name == "plasticine":
                    yi = yi - 0.1 * k * _norm(hat)
                    dead = yi <= 0
                    mu = _where(over, torch.where(dead, torch.zeros_like(mi), mi), mu)
                    lam = _where(over, torch.where(dead, torch.zeros_like(mi), lam[i]), lam)
                    ys = _where(over, yi, ys)
            F = _where(over, _mm(F[i], _expm(-e3(k) * hat)), F)
    elif name == "sand":
        eps = 0.5 * _logm(C)
        hat, tr = _dev(eps), _tr(eps)
        size = _norm(hat)
        dg = size + (3.0 * lam + 2.0 * mu) / (2.0 * mu) * tr * alpha
        flow = (dg > 0) & (tr <= 0)
        free = (dg > 0) & (tr > 0)
        scale = torch.where(flow, dg / size, torch.zeros_like(dg))
        U0 = _polar(F)
        F = torch.where(e3(free), U0, _mm(F, _expm(-e3(scale) * hat)))
    R = _polar(F)
    J = _det(F)
    root = _mm(F, _t(R))
    B = _mm(F, _t(F))
    I = _eye_like(F)  # noqa: E741
    if name in ("jelly", "plasticine"):
        tau = e3(2.0 * mu) * (B - root) + e3(lam * J * (J - 1.0)) * I
    elif name in ("metal", "foam"):
        L = _logm(B)
        tau = _mm(e3(mu) * L + e3(0.5 * lam * _tr(L)) * I, root)
    elif name == "sand":
        L = _logm(B)
        tau = e3(mu) * L + e3(0.5 * lam * _tr(L)) * I
    else:
        tau = _mm(e3(mu * J.pow(-2.0 / 3.0)) * _dev(B) + e3(0.5 * lam * (J * J - 1.0)) * I, root)
    return F, tau, mu, lam, ys


class _Domain:
    """Grids of one or more bodies, one after the other."""

    def __init__(self, counts, grids):
        self.off = np.concatenate([[0], np.cumsum([g ** 3 for g in grids])])
        long = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=DEV)  # noqa: E731
        rep = torch.as_tensor(np.asarray(counts, np.int64), device=DEV)
        self.G = torch.repeat_interleave(long(grids), rep)
        self.start = torch.repeat_interleave(long(self.off[:-1]), rep)
        self.nodes = int(self.off[-1])
        ijk, h, edge = [], [], []
        for g in grids:
            a = torch.arange(g, device=DEV)
            ijk.append(torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3))
            h.append(torch.full((g ** 3,), 1.0 / g, dtype=torch.float64, device=DEV))
            edge.append(torch.full((g ** 3,), g, dtype=torch.int64, device=DEV))
        self.ijk, h, edge = torch.cat(ijk), torch.cat(h), torch.cat(edge)
        self.pos = self.ijk.double() * h[:, None]
        self.floor = (self.pos[:, 1] - 3.5 * h < 0)[:, None]
        self.low, self.high = self.ijk < 3, self.ijk >= edge[:, None] - 3


_O = torch.stack(torch.meshgrid(*[torch.arange(3)] * 3, indexing="ij"), -1).reshape(27, 3)


def _substep(dom, material, x, v, C, F, mass, vol, mu, lam, ys, dt, tool=None):
    Fe, tau, mu, lam, ys = _material(material, F, mu, lam, ys, dt)
    o = _O.to(DEV)
    inv = dom.G.double()[:, None]
    with torch.no_grad():
        base = (x * inv - 0.5).floor().long()
        at = base[:, None] + o
        node = dom.start[:, None] + (at[..., 0] * dom.G[:, None] + at[..., 1]) * dom.G[:, None] + at[..., 2]
    fx = x * inv - base
    w3 = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2], 1)   # [N, offset, axis]
    d3 = torch.stack([fx - 1.5, -2.0 * (fx - 1.0), fx - 0.5], 1)
    wx, wy, wz = (w3[:, o[:, a], a] for a in range(3))
    dx, dy, dz = (d3[:, o[:, a], a] for a in range(3))
    w = wx * wy * wz
    dw = torch.stack([dx * wy * wz, wx * dy * wz, wx * wy * dz], -1) * inv[:, None]
    dpos = (o - fx[:, None]) / inv[:, None]
    wm = w * mass[:, None]
    S = -vol[:, None, None] * tau
    mom = wm[..., None] * (v[:, None] + torch.einsum("nab,nkb->nka", C, dpos)) + dt * torch.einsum("nab,nkb->nka", S, dw)
    grid = torch.zeros(dom.nodes, 4, dtype=x.dtype, device=DEV)
    grid = grid.index_add(0, node.reshape(-1), torch.cat([mom, wm[..., None]], -1).reshape(-1, 4))
    m = grid[:, 3:]
    has = m > 1e-15
    gv = torch.where(has, grid[:, :3] / torch.where(has, m, torch.ones_like(m)) +
                     dt * torch.tensor(GRAVITY, dtype=x.dtype, device=DEV), torch.zeros_like(grid[:, :3]))
    gv = torch.where(dom.floor, torch.zeros_like(gv), gv)
    if tool is not None:
        inside = ((dom.pos - tool[0]).abs() < tool[1]).all(1, keepdim=True)
        gv = torch.where(inside, tool[2].expand_as(gv), gv)
    gv = torch.where((dom.low & (gv < 0)) | (dom.high & (gv > 0)), torch.zeros_like(gv), gv)
    g = gv[node]
    nv = (w[..., None] * g).sum(1)
    nC = 4.0 * inv[..., None] ** 2 * torch.einsum("nk,nka,nkb->nab", w, g, dpos)
    grad = torch.einsum("nka,nkb->nab", g, dw)
    lo = 2.0 / inv
    nx = torch.minimum(torch.maximum(x + dt * nv, lo), 1.0 - lo)
    nF = _mm(_eye_like(F) + dt * grad, Fe)
    return nx, nv, nC, nF, mu, lam, ys


def _lame(E, nu):
    return E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))


def _start(d, names=("x", "v", "vol", "rho", "E", "nu", "ys")):
    d = {k: d[k].double() for k in names}
    n = d["x"].shape[0]
    eye = torch.eye(3, dtype=torch.float64, device=DEV).expand(n, 3, 3).clone()
    return d, eye, torch.zeros(n, 3, 3, dtype=torch.float64, device=DEV)


def _taped(dom, material, state, mass, vol, dt, steps):
    """steps substeps, each remembered by its inputs alone."""
    from torch.utils.checkpoint import checkpoint
    f = lambda *a: _substep(dom, material, *a[:4], mass, vol, *a[4:], dt)  # noqa: E731
    for _ in range(steps):
        state = checkpoint(lambda m, w, *a: _substep(dom, material, *a[:4], m, w, *a[4:], dt), mass, vol, *state,
                           use_reentrant=False)
    return state


def exact(case, seed):
    k = case["kind"]
    if k == "chamfer":
        return _exact_chamfer(case, seed)
    if k == "gaussians":
        return _exact_gaussians(case, seed)
    if k == "neighbours":
        prev, _, xyz, _ = _gaussians(case, seed)
        idx = _near(xyz, prev, case["k"])
        w = 1.0 / ((xyz.double()[:, None] - prev.double()[idx]).norm(dim=-1) + 1e-6)
        return {"w": w / w.sum(1, keepdim=True), "idx": None}
    if k == "generation":
        return _exact_generation(case, seed)
    if k in ("gradient", "segment"):
        return _exact_gradient(case, seed)
    with torch.no_grad():
        if k == "population":
            members = _members(case, seed)
            specs = [_member_spec(m) for m in members]
            cat = lambda name: torch.as_tensor(np.concatenate([getattr(s, name) for s in specs]), device=DEV)  # noqa: E731
            d = {"x": cat("x"), "v": cat("v"), "vol": cat("vol"), "rho": cat("rho"), "E": cat("E"), "nu": cat("nu"),
                 "ys": cat("yield_stress")}
            dom = _Domain([s.n for s in specs], [s.n_grid for s in specs])
            dt, steps, material = 2e-4, case["steps"], "plasticine"
        else:
            raw = _scene(case, seed) if k == "rollout" else _body(case, seed)
            d = raw
            dom = _Domain([case["n"]], [case["grid"]])
            material = "plasticine" if k == "rollout" else case["material"]
            dt = 1e-4 if k == "rollout" else 2e-4
            steps = {"substep": 1, "rollout": case.get("steps"), "frames": case.get("frames", 0) * case.get("substeps", 0)}[k]
        d, F, C = _start(d)
        if k == "substep":
            F, C = raw["F"].double(), raw["C"].double()
        mu, lam = _lame(d["E"], d["nu"])
        s = (d["x"], d["v"], C, F, mu, lam, d["ys"])
        point, size, vel = (torch.tensor(TOOL[a], dtype=torch.float64, device=DEV) for a in ("point", "size", "velocity"))
        frames = [d["x"]]
        for i in range(steps):
            tool = (point + i * dt * vel, size, vel) if k == "rollout" else None
            s = _substep(dom, material, *s[:4], d["rho"] * d["vol"], d["vol"], *s[4:], dt, tool)
            if k == "frames" and (i + 1) % case["substeps"] == 0:
                frames.append(s[0])
        if k == "substep":
            return {"x": s[0], "v": s[1], "C": s[2], "F": s[3]}
        if k == "frames":
            return {"frames": torch.stack(frames), "v": s[1]}
        return {"x": s[0], "v": s[1], "F": s[3], "ys": s[6]}


def _exact_generation(case, seed):
    spec, target, P = _generation(case, seed)
    lam_, n, F = case["members"], case["n"], case["frames"]
    with torch.no_grad():
        rep = lambda a: torch.as_tensor(a, device=DEV).repeat(lam_, *([1] * (a.ndim - 1)))  # noqa: E731
        each = lambda a: torch.repeat_interleave(torch.as_tensor(a, device=DEV), n).float()  # noqa: E731
        d = {"x": rep(spec.x), "v": rep(spec.v), "vol": rep(spec.vol), "rho": rep(spec.rho), "E": each(P[:, 0] * 1e6),
             "nu": each(P[:, 1]), "ys": torch.zeros(lam_ * n, device=DEV)}
        d, Fm, C = _start(d)
        dom = _Domain([n] * lam_, [case["grid"]] * lam_)
        mu, lam = _lame(d["E"], d["nu"])
        s = (d["x"], d["v"], C, Fm, mu, lam, d["ys"])
        frames = [s[0].reshape(lam_, n, 3)]
        for i in range(F * case["substeps"]):
            s = _substep(dom, "jelly", *s[:4], d["rho"] * d["vol"], d["vol"], *s[4:], 2e-4)
            if (i + 1) % case["substeps"] == 0:
                frames.append(s[0].reshape(lam_, n, 3))
        frames = torch.stack(frames)
        tgt = torch.as_tensor(target, device=DEV).double()
        loss = torch.zeros(lam_, dtype=torch.float64, device=DEV)
        for t in range(F):
            for i in range(lam_):
                e = ((frames[t, i][:, None] - tgt[t][None]) ** 2).sum(-1)
                loss[i] += e.min(1).values.mean() + e.min(0).values.mean()
            loss += (frames[t] - tgt[t]).pow(2).sum((1, 2)).sqrt() / n
        return {"frames": frames, "losses": 1e3 * loss}


def _exact_gradient(case, seed):
    raw = _body(case, seed)
    d, F, C = _start(raw)
    dom = _Domain([case["n"]], [case["grid"]])
    if case["kind"] == "gradient":
        v, E, nu, rho = (d[a].requires_grad_(True) for a in ("v", "E", "nu", "rho"))
        mu, lam = _lame(E, nu)
        s = _taped(dom, case["material"], (d["x"], v, C, F, mu, lam, d["ys"]), rho * d["vol"], d["vol"], 2e-4,
                   case["steps"])
        loss = (s[0] - raw["target"].double()).pow(2).mean()
        g = torch.autograd.grad(loss, (v, E, nu, rho))
        return {"x": s[0].detach(), "loss": loss.detach(), "gv": g[0], "gE": g[1], "gnu": g[2], "grho": g[3]}
    mu, lam = (a.requires_grad_(True) for a in _lame(d["E"], d["nu"]))
    mass = (d["rho"] * d["vol"]).requires_grad_(True)
    x, v = d["x"].requires_grad_(True), d["v"].requires_grad_(True)
    F, C = raw["F"].double().requires_grad_(True), raw["C"].double().requires_grad_(True)
    s = _taped(dom, case["material"], (x, v, C, F, mu, lam, d["ys"]), mass, d["vol"], 2e-4, case["steps"])
    gx, gv = (raw["x"] - raw["target"]).double(), (0.01 * raw["v"]).double()
    g = torch.autograd.grad((s[0] * gx).sum() + (s[1] * gv).sum(), (x, v, C, F, mu, lam, mass))
    return {"x": s[0].detach(), "v": s[1].detach(), "F": s[3].detach(),
            **{"g_" + a: b for a, b in zip(("x", "v", "C", "F", "mu", "lam", "mass"), g)}}


def _exact_chamfer(case, seed):
    x, y, w = _clouds(case, seed)
    p, n, m = case["pairs"], case["n"], case["m"]
    x, y, w = x.double().reshape(p, n, 3), y.double().reshape(p, m, 3), w.double()
    d = torch.zeros(p, dtype=torch.float64, device=DEV)
    g = torch.zeros_like(x)
    for i in range(p):
        for a, b, sign in ((x[i], y[i], 1), (y[i], x[i], -1)):
            near = torch.cat([((q[:, None] - b[None]) ** 2).sum(-1).argmin(1) for q in a.split(max(1, int(4e8) // len(b)))])
            diff = a - b[near]
            d[i] += diff.pow(2).sum(1).mean()
            if sign > 0:
                g[i] += 2.0 * w[i] / n * diff
            else:
                g[i].index_add_(0, near, -2.0 * w[i] / m * diff)
    return {"d": d, "g": g.reshape(-1, 3)}


def _exact_gaussians(case, seed):
    prev, cur, xyz, quat = _gaussians(case, seed)
    rel = _near(prev, prev, case["k"], True)
    idx = _near(xyz, prev, case["k"])
    b, x, q = prev.double(), xyz.double(), quat.double()
    motion = (cur - prev).double()
    c = b + motion
    Fm = torch.einsum("nka,nkb->nab", c[rel] - c[:, None], b[rel] - b[:, None])
    U, _, Vh = torch.linalg.svd(Fm)
    U = U * torch.where(torch.tensor([False, False, True], device=DEV), _det(U)[:, None], torch.ones(1, dtype=b.dtype, device=DEV))[:, None]
    Vh = Vh * torch.where(torch.tensor([False, False, True], device=DEV), _det(Vh)[:, None], torch.ones(1, dtype=b.dtype, device=DEV))[..., None]
    R = U @ Vh
    s = torch.sqrt(_tr(R) + 1.0 + 1e-8) * 2.0
    bq = torch.stack([0.25 * s, (R[:, 2, 1] - R[:, 1, 2]) / s, (R[:, 0, 2] - R[:, 2, 0]) / s,
                      (R[:, 1, 0] - R[:, 0, 1]) / s], 1)
    bq = bq / bq.norm(dim=1, keepdim=True)
    out, rot = [], []
    for i in torch.arange(case["n"], device=DEV).split(200_000):
        j = idx[i]
        w = 1.0 / ((x[i][:, None] - b[j]).norm(dim=-1) + 1e-6)
        w = w / w.sum(1, keepdim=True)
        out.append((w[..., None] * (torch.einsum("nkab,nkb->nka", R[j], x[i][:, None] - b[j]) + motion[j] + b[j])).sum(1))
        a = (w[..., None] * bq[j]).sum(1)
        a, o = a / a.norm(dim=1, keepdim=True), q[i]
        aw, ax, ay, az = a.unbind(1)
        ow, ox, oy, oz = o.unbind(1)
        rot.append(torch.stack([aw * ow - ax * ox - ay * oy - az * oz, aw * ox + ax * ow + ay * oz - az * oy,
                                aw * oy - ax * oz + ay * ow + az * ox, aw * oz + ax * oy - ay * ox + az * ow], 1))
    r = {"xyz": torch.cat(out)}
    if case["quat"]:
        r["quat"] = torch.cat(rot)
    return r
