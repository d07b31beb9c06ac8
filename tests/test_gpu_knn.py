"""The cell-grid neighbour search against the brute-force kernel, bit for bit
(indices, distances, ties in index order), where a grid can go wrong: flat and
degenerate clouds, clusters far apart, points on a lattice (ties everywhere),
queries far outside, coordinates far from the origin, and values that are not
finite. And chamfer distances of many pairs through the grid."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cloud(rng, kind, n):
    if kind == "box":
        return rng.uniform(0, 1, (n, 3))
    if kind == "plane":
        return rng.uniform(0, 1, (n, 3)) * [1, 1, 0]
    if kind == "line":
        return rng.uniform(0, 1, (n, 1)) * [[0.3, 0, 0]]
    if kind == "point":
        return np.full((n, 3), 0.25)
    if kind == "clusters":
        return rng.normal(0, 1e-3, (n, 3)) + rng.choice([0.0, 1.0, 50.0], (n, 1))
    if kind == "lattice":
        return rng.integers(0, 12, (n, 3)) / 8.0
    if kind == "far":
        return rng.uniform(0, 1, (n, 3)) + [1000.0, -500.0, 3e4]
    x = rng.uniform(0, 1, (n, 3))          # not finite
    x[::7, 0], x[3::11, 1], x[5::13, 2] = np.nan, np.inf, -np.inf
    return x


def _search(name, q, p, k, self_):
    from empm_b200 import _native as N
    L = N.lib()
    idx = torch.empty(len(q), k, dtype=torch.int64, device=DEV)
    dist = torch.empty(len(q), k, device=DEV)
    args = (q.data_ptr(), len(q), p.data_ptr(), len(p), k, int(self_), idx.data_ptr(), 8, dist.data_ptr())
    if name == "brute":
        N.check(L.empm_knn(*args, None))
    else:
        nb = ctypes.c_size_t()
        N.check(L.empm_knn_workspace(len(q), len(p), int(self_), ctypes.byref(nb)))
        assert nb.value > 0
        work = torch.empty(nb.value, dtype=torch.uint8, device=DEV)
        N.check(L.empm_knn_cells(*args, work.data_ptr(), nb.value, None))
    torch.cuda.synchronize()
    return idx, dist


@pytest.mark.parametrize("kind", ["box", "plane", "line", "point", "clusters", "lattice", "far", "nan"])
@pytest.mark.parametrize("k,n,nq", [(1, 2000, 1), (5, 2049, 700), (16, 6000, 3001), (32, 3000, 257)])
def test_cells_equal_brute_force(kind, k, n, nq):
    rng = np.random.default_rng(k)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float32), device=DEV).contiguous()  # noqa: E731
    p = t(_cloud(rng, kind, n))
    q = _cloud(rng, kind, nq)
    q[::5] = rng.uniform(-3, 4, q[::5].shape)      # some outside the points' box
    q[::17] = 1e6
    for queries, self_ in ((t(q), False), (p, True)):
        a, da = _search("brute", queries, p, k, self_)
        b, db = _search("cells", queries, p, k, self_)
        assert torch.equal(a, b)
        assert torch.equal(da.view(torch.int32), db.view(torch.int32))


@pytest.mark.parametrize("kind", ["box", "plane", "point", "clusters", "lattice", "nan"])
@pytest.mark.parametrize("sizes", [[(9001, 8000)], [(20_000, 9000), (1, 20_000), (17, 0), (0, 40), (5000, 4999)]])
def test_chamfer_cells_equal_brute_force(kind, sizes):
    """Neighbours bit for bit; the sums of n squared distances within n 2^-24."""
    from empm_b200 import _native as N
    L = N.lib()
    rng = np.random.default_rng(3)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float32), device=DEV).contiguous()  # noqa: E731
    xc, yc = [a for a, _ in sizes], [b for _, b in sizes]
    x = t(np.concatenate([_cloud(rng, kind, a) for a in xc]))
    y = t(np.concatenate([_cloud(rng, kind, b) for b in yc]))
    off = lambda c: torch.as_tensor(np.cumsum([0] + c).astype(np.int32), device=DEV)  # noqa: E731
    xo, yo = off(xc), off(yc)
    res = []
    for cells in (False, True):
        s = torch.empty(2, len(sizes), device=DEV)
        nx = torch.empty(len(x), dtype=torch.int32, device=DEV)
        ny = torch.empty(len(y), dtype=torch.int32, device=DEV)
        args = (x.data_ptr(), xo.data_ptr(), len(x), max(xc), y.data_ptr(), yo.data_ptr(), len(y), max(yc), len(sizes),
                s[0].data_ptr(), s[1].data_ptr(), nx.data_ptr(), ny.data_ptr())
        if cells:
            nb = ctypes.c_size_t()
            N.check(L.empm_chamfer_workspace(len(x), max(xc), len(y), max(yc), len(sizes), ctypes.byref(nb)))
            assert nb.value > 0
            work = torch.empty(nb.value, dtype=torch.uint8, device=DEV)
            N.check(L.empm_chamfer_cells(*args, work.data_ptr(), nb.value, None))
        else:
            N.check(L.empm_chamfer(*args, None))
        torch.cuda.synchronize()
        res.append((s.double().cpu(), nx, ny))
    assert torch.equal(res[0][1], res[1][1]) and torch.equal(res[0][2], res[1][2])
    n = torch.as_tensor([xc, yc], dtype=torch.float64)
    assert ((res[0][0] - res[1][0]).abs() <= 2 * n * 2.0 ** -24 * res[0][0] + 1e-30).all()


@pytest.mark.parametrize("n", [600, 1500])           # the brute-force search, the cell grid
def test_last_bit_of_the_distance_decides(n):
    """Pairs of points at equal true distance, (a, b, c) and (b, a, c) off their
    query: their order is that of dz^2 + (dx^2 + rounded dy^2), each sum rounded
    once. Offsets are multiples of 2^-16, so differences are exact in float32 and
    the sums before rounding in float64."""
    rng = np.random.default_rng(3)
    q = 8.0 * np.stack(np.unravel_index(np.arange(n), (12, 12, 12)), 1)
    o = rng.integers(1000, 60000, (n, 3)) / 65536.0
    pts = np.stack([q - o, q - o[:, [1, 0, 2]]], 1).reshape(-1, 3)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    dist = [f32(d[:, 2] ** 2 + f32(d[:, 0] ** 2 + f32(d[:, 1] ** 2))) for d in (o, o[:, [1, 0, 2]])]
    assert (dist[0] != dist[1]).sum() > n // 10
    want = np.where((dist[1] < dist[0])[:, None], [1, 0], [0, 1]) + 2 * np.arange(n)[:, None]
    t = lambda a: torch.as_tensor(a.astype(np.float32), device=DEV)  # noqa: E731
    idx, _ = _search("brute" if n < 1000 else "cells", t(q), t(pts), 2, False)
    assert np.array_equal(idx.cpu().numpy(), want)
