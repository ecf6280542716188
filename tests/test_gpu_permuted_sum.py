"""Transposes and sums of image stacks against torch's: bit-equal (the same additions in
the same order), at the edges of the kernel's 16 x 16 x 16 tiles."""

import itertools

import pytest
import torch

from srf_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (16, 16, 16), (17, 15, 33), (1, 40, 3), (64, 1, 5),
                                   (3, 2, 129)])
@pytest.mark.parametrize("frames", [0, 1, 3])
def test_permuted_sum(shape, frames):
    g = torch.Generator(device="cuda").manual_seed(5)
    views = []
    for perm in itertools.permutations(range(3)):
        size = [0, 0, 0]  # of the source whose view by `perm` has `shape`
        for k, p in enumerate(perm):
            size[p] = shape[k]
        if frames:
            src = torch.randn([frames] + size, generator=g, device="cuda")
            views.append(src.permute(0, *[p + 1 for p in perm]))
        else:
            views.append(torch.randn(size, generator=g, device="cuda").permute(*perm))
    for v in views:
        assert ops.permutable(v)
        assert torch.equal(ops.permuted_sum([v]), v.contiguous())
    for k in range(len(views)):
        a, b, c = (views[(k + i) % len(views)] for i in range(3))
        assert torch.equal(ops.permuted_sum([a, b]), a + b)
        assert torch.equal(ops.permuted_sum([a, b, c]), (a + b) + c)


def test_not_permutable():
    x = torch.zeros(8, 8, 8, device="cuda")
    assert not ops.permutable(x[:, ::2])
    assert not ops.permutable(x[:4, :4].permute(1, 0, 2))
    assert not ops.permutable(x.double())
    assert not ops.permutable(x.cpu())
    assert not ops.permutable(x.clone().requires_grad_(True))
    with pytest.raises(ValueError):
        ops.permuted_sum([x, x[:4]])
