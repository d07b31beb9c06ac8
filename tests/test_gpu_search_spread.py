"""Nearest neighbours where the queries are not among the points, or the points are
spread unevenly: bodies side by side, a cloud over a flat sheet, points far away from
the others, most points in one cell. Results as brute force's, bit for bit, and no
arrangement may take much longer than it: twice its time and 0.2 ms for the sorting
(without the bounds of the search these take 3 to 30 times as long)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _clouds(kind, n, m, seed=1):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(0, 0.4, (n, 3)), rng.uniform(0, 0.4, (m, 3))
    if kind == "beside":
        x[:, 0] += 0.42
    elif kind == "far":
        x += [0.0, 4.0, -4.0]
    elif kind == "sheet":
        y[:, 2] = 0.0
        x[:, 2] = x[:, 2] * 0.01 + 0.3
    elif kind == "outlier":
        y[0], x[-1] = 40.0, -40.0
    elif kind == "outliers":
        y[:20], x[5:25] = rng.uniform(-40, 40, (20, 3)), rng.uniform(-40, 40, (20, 3))
    elif kind == "crowd":
        for a in (x, y):
            a[:len(a) * 9 // 10] = 0.2 + rng.normal(0, 0.002, (len(a) * 9 // 10, 3))
    elif kind == "corner":
        x, y = 0.4 * (x / 0.4) ** 5, 0.4 * (y / 0.4) ** 5
    elif kind == "one place":
        y[:] = 0.1
    t = lambda a: torch.as_tensor(a.astype(np.float32), device=DEV)  # noqa: E731
    return t(x), t(y)


KINDS = ["beside", "far", "sheet", "outlier", "outliers", "crowd", "corner", "one place"]


def _ms(f):
    f()
    best = float("inf")
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        f()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]))
    return best


def _knn_calls(x, y, k):
    from empm_b200 import _native as N
    L, res, calls = N.lib(), [], []
    stream = torch.cuda.current_stream().cuda_stream
    nb = ctypes.c_size_t()
    N.check(L.empm_knn_workspace(len(x), len(y), 0, ctypes.byref(nb)))
    assert nb.value > 0
    work = torch.empty(nb.value, dtype=torch.uint8, device=DEV)
    for cells in (False, True):
        idx = torch.full((len(x), k), -7, dtype=torch.int32, device=DEV)
        dist = torch.full((len(x), k), -7.0, device=DEV)
        a = (x.data_ptr(), len(x), y.data_ptr(), len(y), k, 0, idx.data_ptr(), 4, dist.data_ptr())
        res.append((idx, dist))
        calls.append((lambda a=a: N.check(L.empm_knn_cells(*a, work.data_ptr(), nb.value, stream))) if cells else
                     (lambda a=a: N.check(L.empm_knn(*a, stream))))
    return res, calls


def _chamfer_calls(x, xc, y, yc):
    from empm_b200 import _native as N
    L, res, calls = N.lib(), [], []
    stream = torch.cuda.current_stream().cuda_stream
    off = lambda c: torch.as_tensor(np.cumsum([0] + list(c)).astype(np.int32), device=DEV)  # noqa: E731
    xo, yo = off(xc), off(yc)
    nb = ctypes.c_size_t()
    N.check(L.empm_chamfer_workspace(len(x), max(xc), len(y), max(yc), len(xc), ctypes.byref(nb)))
    assert nb.value > 0
    work = torch.empty(nb.value, dtype=torch.uint8, device=DEV)
    for cells in (False, True):
        s = torch.empty(2, len(xc), device=DEV)
        nx, ny = (torch.full((len(a),), -7, dtype=torch.int32, device=DEV) for a in (x, y))
        a = (x.data_ptr(), xo.data_ptr(), len(x), max(xc), y.data_ptr(), yo.data_ptr(), len(y), max(yc), len(xc),
             s[0].data_ptr(), s[1].data_ptr(), nx.data_ptr(), ny.data_ptr())
        res.append((nx, ny, s))
        keep = (xo, yo, work)
        calls.append((lambda a=a, keep=keep: N.check(L.empm_chamfer_cells(*a, work.data_ptr(), nb.value, stream)))
                     if cells else (lambda a=a, keep=keep: N.check(L.empm_chamfer(*a, stream))))
    return res, calls


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,m,k", [(40_000, 30_011, 1), (6001, 6000, 5), (257, 2049, 16), (20_000, 20_001, 16),
                                   (5000, 7001, 32)])
def test_knn_of_uneven_clouds(kind, n, m, k):
    x, y = _clouds(kind, n, m)
    ((ia, da), (ib, db)), (brute, cells) = _knn_calls(x, y, k)
    tb, tc = _ms(brute), _ms(cells)
    assert torch.equal(ia, ib) and torch.equal(da.view(torch.int32), db.view(torch.int32))
    assert tc <= 2 * tb + 0.2, (kind, tb, tc)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("xc,yc", [([40_000], [30_011]), ([9000, 1, 6000], [8001, 300, 7999])])
def test_chamfer_of_uneven_clouds(kind, xc, yc):
    """The sums of n squared distances agree within 2 n 2^-24."""
    parts = [_clouds(kind, max(a, 40), max(b, 40), 3 + i) for i, (a, b) in enumerate(zip(xc, yc))]
    x = torch.cat([p[0][:a] for p, a in zip(parts, xc)]).contiguous()
    y = torch.cat([p[1][:b] for p, b in zip(parts, yc)]).contiguous()
    (a, b), (brute, cells) = _chamfer_calls(x, xc, y, yc)
    tb, tc = _ms(brute), _ms(cells)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    n = torch.as_tensor([xc, yc], dtype=torch.float64)
    sa, sb = a[2].double().cpu(), b[2].double().cpu()
    assert ((sa - sb).abs() <= 2 * n * 2.0 ** -24 * sa + 1e-30).all()
    assert tc <= 2 * tb + 0.2, (kind, tb, tc)
