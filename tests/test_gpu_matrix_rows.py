"""Matrix planes as rows, bit for bit against a concatenation of the planes, at the
edges of the kernel's blocks and 16-byte stores, NaN and infinities included; what the
kernel cannot take goes the concatenation's way."""
import pytest
import torch

from empm_b200 import _native as N
from empm_b200.mpm_data_structure import _f9_unpack

pytestmark = pytest.mark.gpu


def _cat(src, n):
    return torch.cat([src[:4 * n].view(n, 4), src[4 * n:8 * n].view(n, 4), src[8 * n:9 * n].view(n, 1)], 1).view(n, 3, 3)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 127, 128, 129, 130, 131, 255, 257, 50_001])
def test_rows_equal_concatenated_planes(n):
    src = torch.randn(9 * n + 5, device="cuda:0")
    src[::7], src[3::11] = float("nan"), float("inf")
    got, want = _f9_unpack(src, n), _cat(src, n)
    assert got.shape == want.shape and got.is_contiguous()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))


def test_other_sources_take_the_general_way():
    src = torch.randn(91, device="cuda:0")
    assert torch.equal(_f9_unpack(src[1:], 10), _cat(src[1:], 10))           # not aligned
    leaf = src[:90].clone().requires_grad_()
    _f9_unpack(leaf, 10).sum().backward()
    assert torch.equal(leaf.grad, torch.ones_like(leaf))
    assert N.lib().empm_matrix_rows(src.data_ptr() + 4, 10, src.data_ptr(), None) == -1
