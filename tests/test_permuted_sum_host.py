"""Axis-order changes below the size of the one-pass kernel: what torch is asked to copy."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from srf_b200.physics import permuted_sum

COPIES = {"aten::clone", "aten::copy_", "aten::_to_copy"}


class Copies(TorchDispatchMode):
    """Counts the elements that copying operators write."""

    def __init__(self):
        super().__init__()
        self.elements = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        out = func(*args, **(kwargs or {}))
        if func._schema.name in COPIES:
            self.elements += out.numel()
        return out


@pytest.mark.parametrize("shape,perm", [((5, 6, 7), (2, 1, 0)), ((5, 6, 7), (0, 2, 1)),
                                        ((3, 5, 6, 7), (0, 2, 3, 1)), ((5, 6, 7), (0, 1, 2))])
def test_one_view_is_copied_once(shape, perm):
    x = torch.arange(torch.Size(shape).numel(), dtype=torch.float32).reshape(shape)
    view = x.permute(*perm)
    with Copies() as c:
        out = permuted_sum([view])
    assert out.is_contiguous() and torch.equal(out, view)
    assert c.elements == (0 if view.is_contiguous() else x.numel())


def test_several_views_add_in_order():
    g = torch.Generator().manual_seed(1)
    a, b, c = (torch.randn(4, 5, 6, generator=g) for _ in range(3))
    views = [a, b.permute(0, 2, 1).contiguous().permute(0, 2, 1), c]
    out = permuted_sum(views)
    assert out.is_contiguous() and torch.equal(out, (a + b) + c)
    assert torch.equal(a, views[0])  # sources stay as they were
