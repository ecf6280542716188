"""Axis-order changes: what torch is asked to copy below the size of the one-pass kernel, and
what that kernel's entry point refuses on the host."""

import ctypes

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from srf_b200 import _lib, ops
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


class Cuda:
    """What ``ops.permutable`` looks at of a CUDA tensor."""

    is_cuda, dtype, requires_grad = True, torch.float32, False

    def __init__(self, *shape, neg=False):
        self.meta = torch.empty(shape, device="meta")
        self.shape, self.neg = self.meta.shape, neg

    def dim(self):
        return self.meta.dim()

    def numel(self):
        return self.meta.numel()

    def stride(self, k=None):
        return self.meta.stride() if k is None else self.meta.stride(k)

    def is_neg(self):
        return self.neg


def test_what_the_one_pass_kernel_takes():
    """Images and stacks that it cannot index, or that are negated on reading, stay with torch."""
    assert ops.permutable(Cuda(1290, 1290, 1290))
    assert not ops.permutable(Cuda(1291, 1291, 1291))        # 2^31 voxels and more
    assert ops.permutable(Cuda(4, 1290, 1290, 1290))
    assert ops.permutable(Cuda((1 << 31) - 1, 1, 2, 3))
    assert not ops.permutable(Cuda(1 << 31, 1, 2, 3))        # 2^31 tiles
    assert not ops.permutable(Cuda(64, 64, 64, neg=True))


def _call(dims, frames, strides, sources=(4096,), out=8192):
    n = len(sources)
    return _lib.load().srf_permute_sum(
        ctypes.c_void_p(out), (ctypes.c_int * 3)(*dims), frames, n,
        (ctypes.c_void_p * n)(*sources), (ctypes.c_int64 * len(strides))(*strides), None)


def test_entry_point_refuses_before_any_launch():
    """Strides that leave the frame, also where their sum passes 2^63, and counts of frames
    that no launch holds (status 1 invalid argument, 3 unsupported)."""
    assert _call((5, 4, 3), 1, (12, 3, 0)) == 1
    assert _call((5, 4, 3), 1, (13, 3, 1)) == 1
    assert _call((5, 4, 3), 1, (1 << 62, 3, 1)) == 1           # 4 * 2^62 = 0 mod 2^64
    assert _call((5, 4, 3), 1, (1, 1 << 61, 1 << 62)) == 1     # 3 * 2^61 + 2 * 2^62 < 0
    assert _call((5, 4, 3), 1, (12, 3, 1), (8192,)) == 1       # out among the sources
    assert _call((64, 16, 16), 1 << 62, (256, 16, 1)) == 3     # 4 tiles * 2^62 = 0 mod 2^64
    assert _call((16, 16, 16), 1 << 31, (256, 16, 1)) == 3
    assert _call((5, 0, 3), 1 << 62, (3, 3, 1)) == 0           # nothing to do
    assert _call((5, 4, 3), 0, (12, 3, 1)) == 0
