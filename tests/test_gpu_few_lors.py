"""Which kernel family a TOR call takes by itself: the LOR-centric one (one launch) for few
LORs, the slabs (count, scan, fill and the op: four launches) else, on either side of the
line, where slices fill a warp and on flat grids, where they leave its lanes idle.

Tolerance 1e-5 relative L2 between the families (TOL of test_gpu_parity)."""

import numpy as np
import pytest
import torch

from srf_b200 import _lib, ops, tuning
from tests import _cases as K

pytestmark = pytest.mark.gpu
KW = 10.19


def _lors(n, size):
    g = np.random.default_rng(n)
    mid = (g.random((n, 3)) - 0.5) * np.array(size) * 0.9
    d = np.stack([g.uniform(-0.6, 0.6, n), g.uniform(-0.6, 0.6, n), np.ones(n)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rec = np.concatenate([mid - 150 * d, mid + 150 * d, mid, np.ones((n, 1))], 1)
    return torch.as_tensor(rec.astype(np.float32)).cuda()


@pytest.mark.parametrize("grid,voxel,n,few", [
    ((128, 128, 64), 3.2, 20_000, True),   # 20k * 36 * (64 - 32) = 2.3e7
    ((128, 128, 64), 3.2, 24_000, False),  # 2.8e7
    ((64, 64, 32), 6.4, 90_000, True),     # 90k * 16 * 16 = 2.3e7
    ((64, 64, 33), 6.4, 40_000, False),    # two rounds: 40k * 16 * 47.5 = 3.0e7
    ((64, 64, 8), 6.4, 50_000, True),      # 50k * 16 * 28 = 2.2e7
    ((64, 64, 8), 6.4, 60_000, False),     # 2.7e7
    ((128, 128, 1), 3.2, 21_000, True),    # 21k * 36 * 31.5 = 2.4e7
    ((128, 128, 1), 3.2, 100_000, False),
    ((256, 256, 128), 2.5, 18_000, True),  # more slabs than SMs: 18k * 49 * 64 = 5.6e7
    ((256, 256, 128), 2.5, 22_000, False),
])
def test_family_and_result(grid, voxel, n, few):
    g, size = list(grid), [k * voxel for k in grid]
    lors = _lors(n, size)
    img = torch.rand(g[::-1], device="cuda") + 0.1
    v = torch.rand(n, device="cuda") + 1.0
    a = (g, [0.0, 0.0, 0.0], size, KW, False, 6.0, 1139.77)
    m7 = lors[:, [0, 1, 2, 3, 4, 5, 9]].contiguous()
    calls = [lambda: ops.tor_projection(lors, img, *a, layout="nc"),
             lambda: ops.tor_backprojection(img, lors, v, *a, layout="nc"),
             lambda: ops.tor_backproject_adjoint(v, lors, *a, layout="nc"),
             lambda: ops.tor_maplors(img, *a[:3], m7, v, KW, False, layout="nc")]
    for call in calls:
        before = _lib.load().srf_launch_count()
        got = call()
        assert _lib.load().srf_launch_count() - before == (1 if few else 4)
        tuning.set_tuning(1 if few else 2, 0, 0)  # the other family
        try:
            other = call()
        finally:
            tuning.set_tuning()
        assert K.rel_l2(got.cpu().numpy(), other.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("frames,n,few", [(256, 100_000, True), (256, 150_000, False)])
def test_family_of_many_frames(frames, n, few):
    """256 slabs: 100k * 16 * 28 = 4.5e7, 150k 6.7e7."""
    g, size = [64, 64, 8], [409.6, 409.6, 51.2]
    lors = _lors(n, size)
    frame = (torch.arange(n, device="cuda") * frames // n).int()
    img = torch.rand([frames] + g[::-1], device="cuda") + 0.1
    before = _lib.load().srf_launch_count()
    ops.tor_projection_backprojection_batched(lors, frame, img, frames, g, [0.0, 0.0, 0.0], size,
                                              KW, False, 6.0, 1139.77, layout="nc")
    assert _lib.load().srf_launch_count() - before == (2 if few else 5)
