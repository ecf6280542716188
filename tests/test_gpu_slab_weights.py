"""Weights of the slab kernels over the range that a float holds: factors above 1 (TOF sharper
than the tube), voxels that only the tails of the two Gaussians reach, TOF centres that are
not numbers or at infinity.

Tolerances. The slab kernels and the oracle take the same float decisions; their weights
differ by the exponent's error. A crossing point is off by up to 1.7e-5 mm here (the
quotient's half ulp along 280 mm, and its own rounding), which moves the exponent by
|C - X| 1.7e-5 / tse (TOF) and, against float64, d 1.7e-5 / sigma^2 (tube); sums of positive
weights are off by no more than their worst weight."""

import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from srf_b200 import ops, tuning
from tests import _cases as K

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def slabs():
    """The slab kernels, whatever the number of LORs."""
    tuning.set_tuning(1, 0, 0)
    yield
    tuning.set_tuning()


GRID = [48, 44, 26]
CENTER = [0.0, 0.0, 0.0]


def _lors(n, seed, spread=30.0, along=5.0):
    """[10, n] LORs around the slice axis, TOF centres `along` mm (sigma) from its middle."""
    g = np.random.default_rng(seed)
    mid = g.normal(0, 1, (n, 3)) * np.array([spread, spread, along])
    d = np.stack([g.uniform(-0.6, 0.6, n), g.uniform(-0.6, 0.6, n), np.ones(n)], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    f = g.uniform(0.5, 1.5, n)
    return np.ascontiguousarray(np.concatenate(
        [mid - 300 * d, mid + 300 * d, mid, f[:, None]], 1).T.astype(np.float32))


def _cu(a):
    return torch.as_tensor(a).cuda()


@pytest.mark.parametrize("voxel,kw", [(6.4, 8.0), (3.2, 8.0), (3.2, 10.19), (2.5, 10.19)])
@pytest.mark.parametrize("geo", [False, True])
@pytest.mark.parametrize("sharp", [0.8, 0.5, 0.2])
def test_tof_sharper_than_the_tube(voxel, kw, geo, sharp):
    """tse = sharp * tube variance: the weight grows towards the cut-off, to e^(4.5 (1/sharp - 1)).
    Tolerance 1e-4: three sigma of TOF, sqrt(tse) >= 0.55 mm: 3 * 1.7e-5 / 0.55."""
    n = 60_000
    size = [g * voxel for g in GRID]
    tse = sharp * kw * kw / 36 * (0.5 if geo else 1.0)
    tof = (0.5, tse - 0.25 / 12)
    lors = _lors(n, 3, spread=9.0 * voxel, along=7.0 * voxel)
    # LORs' scales from 2^-4 to 2^10 of the typical one, a few of them far
    g = np.random.default_rng(5)
    v = np.exp(g.normal(0, 0.4, n)).astype(np.float32)
    far = g.random(n) < 0.02
    v[far] *= (2.0 ** g.uniform(-10, 4, far.sum())).astype(np.float32)
    ref = O.tor_backprojection(lors, v, GRID, CENTER, size, kw, geo, *tof, mode="f32",
                               contract=True)
    if not np.isfinite(ref).all():  # the oracle's own 0 * exp(large) outside the cut-off
        ref = np.where(np.isfinite(ref), ref, O.tor_backprojection(
            lors, v, GRID, CENTER, size, kw, geo, *tof, mode="f64"))
    ok = np.isfinite(ref)
    assert ok.mean() > 0.9
    L = _cu(lors)
    bp = ops.tor_backprojection(torch.zeros(GRID[::-1], device="cuda"), L, _cu(v), GRID, CENTER,
                                size, kw, geo, *tof, layout="cn").cpu().numpy()
    assert np.isfinite(bp).all() and K.rel_l2(bp[ok], ref[ok]) <= 1e-4
    adj = ops.tor_backproject_adjoint(_cu(1.0 / v), L, GRID, CENTER, size, kw, geo, *tof,
                                      layout="cn").cpu().numpy()
    assert np.isfinite(adj).all() and K.rel_l2(adj[ok], ref[ok]) <= 1e-4


@pytest.mark.parametrize("op", ["back", "adjoint", "map"])
def test_every_voxel(op):
    """Relative error voxel by voxel, also where only tails reach: slices five sigma of TOF
    away, tube edges. Tolerance 1e-4: 5.1 * 1.7e-5 / 2.885 (three sigma of the tube) + 42 *
    2.1e-5 / 64 (the grid's end) = 4.4e-5, twice that for roundings of exponents near -18."""
    n, voxel, kw, tof = 60_000, 3.2, 10.19, (6.0, 61.0)
    size = [g * voxel for g in GRID]
    lors = _lors(n, 7, spread=20.0)
    v = np.random.default_rng(9).uniform(1.0, 30.0, n).astype(np.float32)
    L, V = _cu(lors), _cu(v)
    I = torch.zeros(GRID[::-1], device="cuda")
    if op == "map":
        m7 = np.ascontiguousarray(lors[[0, 1, 2, 3, 4, 5, 9]])
        ref = O.tor_maplors(m7, v, GRID, CENTER, size, kw, False, mode="f64")
        out = ops.tor_maplors(I, GRID, CENTER, size, _cu(m7), V, kw, False, layout="cn")
    else:
        ref = O.tor_backprojection(lors, v, GRID, CENTER, size, kw, False, *tof, mode="f64")
        out = (ops.tor_backprojection(I, L, V, GRID, CENTER, size, kw, False, *tof, layout="cn")
               if op == "back" else
               ops.tor_backproject_adjoint(_cu(1.0 / v), L, GRID, CENTER, size, kw, False, *tof,
                                           layout="cn"))
    out = out.cpu().numpy().astype(np.float64)
    some = ref > 0
    assert ref[some].min() < 1e-6 * ref.max() or op == "map"
    assert np.array_equal(out != 0, some)
    assert np.max(np.abs(out[some] - ref[some]) / ref[some]) <= 1e-4


@pytest.mark.parametrize("many", [0, 1, 200])  # 0: one LOR that meets one voxel, the corner
def test_centre_that_is_not_a_number(many):
    """Every voxel of such a LOR is not a number, as in the LOR-centric kernels; the others
    keep their sums (tolerance 1e-5, TOL of test_gpu_parity)."""
    n, voxel, kw, tof = 60_000, 3.2, 10.19, (6.0, 1139.77)
    size = [g * voxel for g in GRID]
    lors = _lors(n, 11)
    if many:
        lors[6 + np.arange(many) % 3, np.arange(many) * 290] = np.nan
    else:  # 3.5 mm from the corner column's axis along x and y: 4.95 of 5.1 mm
        x, y, z = (-s / 2 for s in size)
        lors[:, 0] = [x - 1.9, y - 1.9, z + 0.5, x - 1.9, y - 1.9, z + 2.5, np.nan, y, z, 1.0]
    L, V = _cu(lors), torch.full((n,), 2.0, device="cuda")
    img = torch.rand(GRID[::-1], device="cuda") + 0.1

    def run():
        a = (GRID, CENTER, size, kw, False, *tof)
        return [ops.tor_projection(L, img, *a, layout="cn"),
                ops.tor_backprojection(img, L, V, *a, layout="cn"),
                ops.tor_backproject_adjoint(V, L, *a, layout="cn")]

    slab = run()
    tuning.set_tuning(2, 0, 0)
    for got, ref in zip(slab, run()):
        nan = torch.isnan(ref)
        assert nan.any() and not nan.all()
        assert many or nan.sum() == 1
        assert torch.equal(torch.isnan(got), nan)
        assert K.rel_l2(got[~nan].cpu().numpy(), ref[~nan].cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("row", [6, 7, 8])
@pytest.mark.parametrize("value", [np.inf, -np.inf, 1e30])
def test_centre_at_infinity(row, value):
    """A LOR whose TOF centre is infinitely far away weighs nothing anywhere (tolerance for the
    rest as above)."""
    n, voxel, kw, tof = 60_000, 3.2, 10.19, (6.0, 1139.77)
    size = [g * voxel for g in GRID]
    lors = _lors(n, 13)
    away = np.arange(50) * 1100
    lors[row, away] = value
    rest = np.delete(lors, away, axis=1)
    L, V = _cu(lors), torch.full((n,), 2.0, device="cuda")
    img = torch.rand(GRID[::-1], device="cuda") + 0.1
    a = (GRID, CENTER, size, kw, False, *tof)
    pv = ops.tor_projection(L, img, *a, layout="cn").cpu().numpy()
    assert not pv[away].any()
    ref = O.tor_projection(rest, img.cpu().numpy(), *a, mode="f32", contract=True)
    assert K.rel_l2(np.delete(pv, away), ref) <= 1e-5
    ref = O.tor_backprojection(rest, np.full(rest.shape[1], 2.0, np.float32), *a, mode="f32",
                               contract=True)
    for got in (ops.tor_backprojection(img, L, V, *a, layout="cn"),
                ops.tor_backproject_adjoint(0.25 * V, L, *a, layout="cn")):
        assert K.rel_l2(got.cpu().numpy(), ref) <= 1e-5


def test_zero_values_and_weights_beyond_the_floats():
    """TOF so sharp that weights overflow towards the cut-off (e^220): a zero value leaves
    infinity times 0 there, not a number, as in the LOR-centric kernels, and 0 elsewhere."""
    n, voxel, kw, tof = 20, 6.4, 24.0, (0.5, 0.3)
    size = [g * voxel for g in GRID]
    lors = _lors(n, 17)
    at = np.arange(n)  # along z, centres in slice planes
    lors[0, at] = lors[3, at] = lors[6, at] = (at - 10) * 9.7
    lors[1, at] = lors[4, at] = lors[7, at] = (at % 5 - 2) * 11.3
    lors[2, at], lors[5, at], lors[8, at] = -300.0, 300.0, (at % 9 - 4 + 0.5) * voxel
    lors[9, at] = 1.0
    L, V = _cu(lors), torch.zeros(n, device="cuda")
    a = (GRID, CENTER, size, kw, False, *tof)
    got = ops.tor_backproject_adjoint(V, L, *a, layout="cn")
    tuning.set_tuning(2, 0, 0)
    ref = ops.tor_backproject_adjoint(V, L, *a, layout="cn")
    nan = torch.isnan(ref)
    assert nan.any() and not nan.all()
    assert torch.equal(torch.isnan(got), nan)
    assert not got[~nan].any() and not ref[~nan].any()
