"""The slab kernels' walk where it can go wrong: every patch size, voxels that are not cubes
(boxes that the reference's window clips), LORs far from the slice axis, odd grids, row
bands, LOR counts around a warp, LORs that start and end inside the grid.

Tolerances: against the oracle's float mode 1e-5 relative L2 (TOL of test_gpu_parity: the
same float decisions, other roundings of the continuous terms only). A LOR at more than
~83 degrees from the slice axis goes through the general walk in both, same tolerance."""

import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from srf_b200 import ops, tuning
from tests import _cases as K

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _lors(n, size, seed, steep=0.0, inside=0.0):
    """[10, n] columns: LORs through the grid's inside around the slice axis; a share
    `steep` of them nearly in plane, a share `inside` with both ends in the grid."""
    g = np.random.default_rng(seed)
    mid = (g.random((n, 3)) - 0.5) * np.array(size) * 0.9
    d = np.stack([g.uniform(-1, 1, n), g.uniform(-1, 1, n), np.ones(n)], 1)
    flat = g.random(n) < steep
    d[flat, 2] = g.uniform(0.02, 0.2, flat.sum()) * g.choice([-1, 1], flat.sum())
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    half = np.where(g.random(n) < inside, 0.3 * min(size), 500.0)[:, None]
    f = g.uniform(0.4, 1.0, n)
    tof = mid + d * g.normal(0, 20.0, n)[:, None]
    return np.ascontiguousarray(np.concatenate(
        [mid - half * d, mid + half * d, tof, f[:, None]], 1).T.astype(np.float32))


@pytest.mark.parametrize("grid,voxel,kw,steep,inside,n", [
    ((40, 33, 21), (6.4, 6.4, 6.4), 4.0, 0.0, 0.3, 33),      # patch 2
    ((31, 47, 19), (3.7, 3.7, 3.7), 4.0, 0.1, 0.3, 500),     # patch 3
    ((64, 64, 32), (6.4, 6.4, 6.4), 10.19, 0.0, 0.0, 31),    # patch 4
    ((53, 29, 40), (4.0, 4.0, 4.0), 10.19, 0.1, 0.5, 700),   # patch 5
    ((37, 41, 24), (3.2, 3.2, 3.2), 10.19, 0.1, 0.2, 1000),  # patch 6
    ((37, 41, 24), (3.2, 4.5, 1.1), 10.19, 0.0, 0.2, 900),   # no cubes: the window clips
    ((41, 37, 24), (4.5, 3.2, 6.0), 10.19, 0.2, 0.2, 900),
    ((65, 66, 17), (2.5, 2.5, 2.5), 10.19, 0.1, 0.2, 600),   # patch 7
    ((70, 35, 9), (2.2, 2.2, 2.2), 10.19, 0.1, 0.2, 600),    # patch 8
    ((1, 1, 5), (3.2, 3.2, 3.2), 10.19, 0.0, 0.0, 64),
    ((300, 9, 130), (3.2, 3.2, 3.2), 10.19, 0.0, 0.5, 400),
])
@pytest.mark.parametrize("path", [(1, 0, 1), (1, 3, 2), (1, 9, 1)])  # slabs, few and many slices
def test_slab_walk(grid, voxel, kw, steep, inside, n, path):
    g, c = list(grid), [1.0, -2.0, 0.5]
    s = [a * b for a, b in zip(grid, voxel)]
    lors = _lors(n, s, 7 + n, steep, inside)
    img = np.random.default_rng(1).random((g[2], g[1], g[0])).astype(np.float32) + 0.1
    b, s2 = 6.0, 1139.77
    tuning.set_tuning(*path)
    try:
        L, I = torch.as_tensor(lors).cuda(), torch.as_tensor(img).cuda()
        pv = ops.tor_projection(L, I, g, c, s, kw, False, b, s2, layout="cn")
        ref = O.tor_projection(lors, img, g, c, s, kw, False, b, s2, mode="f32", contract=True)
        assert K.rel_l2(pv.cpu().numpy(), ref) <= TOL
        v = np.full(n, 3.0, np.float32)
        v[::5] = 0.0  # nothing
        V = torch.as_tensor(v).cuda()
        bp = ops.tor_backprojection(I, L, V, g, c, s, kw, False, b, s2, layout="cn")
        ref = O.tor_backprojection(lors, v, g, c, s, kw, False, b, s2, mode="f32", contract=True)
        assert K.rel_l2(bp.cpu().numpy(), ref) <= TOL
        m7 = np.ascontiguousarray(lors[[0, 1, 2, 3, 4, 5, 9]])
        mp = ops.tor_maplors(I, g, c, s, torch.as_tensor(m7).cuda(), V + 1.0, kw, False,
                             layout="cn")
        ref = O.tor_maplors(m7, v + 1.0, g, c, s, kw, False, mode="f32", contract=True)
        assert K.rel_l2(mp.cpu().numpy(), ref) <= TOL
    finally:
        tuning.set_tuning()
