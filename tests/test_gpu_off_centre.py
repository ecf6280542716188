"""Images far from the origin, where coordinates have few digits left for a voxel: the slab
kernels (whole slices, row bands, few slices) against the oracle's float mode, LOR by LOR. TOF
is off: its exponent, which the slab kernels take in double once per LOR and the reference per
slice from rounded crossings, differs out there without any decision being involved.

Tolerance 1e-5 per LOR (TOL of test_gpu_parity): both take the same float decisions; a voxel
at the cut-off that is left out is worth 1 % of one of the LOR's at most 26 x 9 voxels."""

import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from srf_b200 import ops, tuning
from tests import _cases as K

pytestmark = pytest.mark.gpu


def _lors(n, size, centre, slope=0.6):
    g = np.random.default_rng(5)
    mid = (g.random((n, 3)) - 0.5) * np.array(size) * 0.9 + np.array(centre)
    d = np.stack([g.uniform(-slope, slope, n), g.uniform(-slope, slope, n), np.ones(n)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rec = np.concatenate([mid - 300 * d, mid + 300 * d, mid, np.ones((n, 1))], 1)
    return torch.as_tensor(rec.astype(np.float32)).cuda()


@pytest.mark.parametrize("off", [0.0, 6e3, 2e4, 1e5, 8e5])
@pytest.mark.parametrize("grid,path", [((48, 44, 26), (1, 0, 0)), ((128, 128, 26), (1, 16, 0)),
                                       ((48, 44, 26), (1, 3, 0))])
def test_off_centre(grid, path, off):
    n, voxel, kw = 40_000, 3.2, 10.19
    g, size = list(grid), [k * voxel for k in grid]
    centre = [off, -off, 0.0]
    lors = _lors(n, size, centre)
    img = torch.rand(g[::-1], device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    img += 0.1
    a = (g, centre, size, kw, False, 6.0, 1.0e6)
    tuning.set_tuning(*path)
    try:
        pv = ops.tor_projection(lors, img, *a, layout="nc").cpu().numpy()
        bp = ops.tor_backprojection(img, lors, torch.ones(n, device="cuda"), *a, layout="nc")
    finally:
        tuning.set_tuning()
    soa = np.ascontiguousarray(lors.cpu().numpy().T)
    ref = O.tor_projection(soa, img.cpu().numpy(), *a, mode="f32", contract=True)
    assert np.count_nonzero(ref) > 0.9 * n
    assert np.max(np.abs(pv - ref) / np.maximum(np.abs(ref), 1e-3 * ref.max())) <= 1e-5
    ref = O.tor_backprojection(soa, np.ones(n, np.float32), *a, mode="f32", contract=True)
    assert K.rel_l2(bp.cpu().numpy(), ref) <= 1e-5


def test_off_centre_along_the_slices():
    """Planes that lie up to half a millimetre from where an even spacing would put them (floats
    are 1 mm apart there): every row of every band (128 x 128 slices, 16 per slab) that oblique
    LORs reach still has them."""
    grid, n, voxel, kw, off = [128, 128, 26], 40_000, 2.7, 10.19, 1.6e7
    size = [k * voxel for k in grid]
    centre = [0.0, 0.0, off]
    lors = _lors(n, size, centre, slope=1.5)
    img = torch.rand(grid[::-1], device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    img += 0.1
    a = (grid, centre, size, kw, False, 6.0, 1.0e6)
    tuning.set_tuning(1, 16, 0)
    try:
        pv = ops.tor_projection(lors, img, *a, layout="nc").cpu().numpy()
        bp = ops.tor_backprojection(img, lors, torch.ones(n, device="cuda"), *a, layout="nc")
    finally:
        tuning.set_tuning()
    soa = np.ascontiguousarray(lors.cpu().numpy().T)
    ref = O.tor_projection(soa, img.cpu().numpy(), *a, mode="f32", contract=True)
    assert np.count_nonzero(ref) > 0.9 * n
    assert np.max(np.abs(pv - ref) / np.maximum(np.abs(ref), 1e-3 * ref.max())) <= 1e-5
    ref = O.tor_backprojection(soa, np.ones(n, np.float32), *a, mode="f32", contract=True)
    assert K.rel_l2(bp.cpu().numpy(), ref) <= 1e-5
