"""Sums of squared distances of the chamfer search in cells against the same float32
distances added in 64 bits: one rounding to float32 at the end, 2^-24 of the sum (and
1e-9 for single distances whose own rounding falls the other way here). Pairs whose
clouds meet in a block and in a warp, one large pair, and queries left to brute force."""
import numpy as np
import pytest
import torch

from tests.test_gpu_search_spread import DEV, _chamfer_calls, _clouds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["box", "crowd", "beside"])
@pytest.mark.parametrize("xc,yc", [([100_003], [80_000]), ([2500] * 24, [2500] * 24),
                                   ([9000, 3, 1, 40, 5000], [8001, 2, 9, 33, 777])])
def test_sums_are_rounded_once(kind, xc, yc):
    parts = [_clouds(kind, max(a, 40), max(b, 40), 3 + i) for i, (a, b) in enumerate(zip(xc, yc))]
    x = torch.cat([p[0][:a] for p, a in zip(parts, xc)]).contiguous()
    y = torch.cat([p[1][:b] for p, b in zip(parts, yc)]).contiguous()
    res, calls = _chamfer_calls(x, xc, y, yc)
    calls[1]()
    torch.cuda.synchronize()
    nx, ny, s = (t.cpu().numpy() for t in res[1])
    x, y = x.cpu().numpy(), y.cpu().numpy()
    f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    for got, a, b, nn, counts in ((s[0], x, y, nx, xc), (s[1], y, x, ny, yc)):
        d = (a - b[nn]).astype(np.float64)           # differences rounded to float32
        d = f32(d[:, 2] ** 2 + f32(d[:, 0] ** 2 + f32(d[:, 1] ** 2)))
        want = np.add.reduceat(d, np.cumsum([0] + list(counts))[:-1])
        assert (np.abs(got - want) <= (2.0 ** -24 + 1e-9) * want).all(), np.abs(got / want - 1).max()
