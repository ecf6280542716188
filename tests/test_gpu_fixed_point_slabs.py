"""Scatter ops over slabs that accumulate in fixed point: sums that would wrap 32 bits, scales
far from the typical one, values of one and of both signs, few and many adds per voxel.

Reference: the oracle's float64 mode. Tolerance 1e-5 relative L2 (the bound of every TOR
back-projection here, FP64_TOL["default"] of test_gpu_parity)."""

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


TOL = 1e-5
GRID, VOXEL, KW = [48, 44, 26], 3.2, 10.19
SIZE = [g * VOXEL for g in GRID]
TOF = (6.0, 1139.77)


def _lors(n, seed, spread):
    """[10, n] LORs around the slice axis; `spread` mm is how far they pass from the axis."""
    g = np.random.default_rng(seed)
    mid = g.normal(0, 1, (n, 3)) * np.array([spread, spread, 5.0])
    d = np.stack([g.uniform(-0.6, 0.6, n), g.uniform(-0.6, 0.6, n), np.ones(n)], 1)
    d *= min(1.0, spread / 20.0 + 0.01) if spread < 20 else 1.0
    d[:, 2] = 1.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate(
        [mid - 300 * d, mid + 300 * d, mid, np.ones((n, 1))], 1).T.astype(np.float32))


def _back64(lors, v):
    return O.tor_backprojection(lors, v.astype(np.float32), GRID, [0, 0, 0], SIZE, KW, False,
                                *TOF, mode="f64")


def _values(kind, n, seed):
    g = np.random.default_rng(seed)
    v = np.exp(g.normal(0, 0.4, n))
    if kind == "outliers":  # 1 % from 2^-12 to 2^12 of the others
        far = g.random(n) < 0.01
        v[far] *= 2.0 ** g.uniform(-12, 12, far.sum())
    if kind == "decades":   # no typical value
        v = 10.0 ** g.uniform(-3, 3, n)
    if kind == "threshold":
        v[::3] = 1e-8
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["plain", "outliers", "decades", "threshold"])
@pytest.mark.parametrize("n,spread", [(300, 30.0), (40_000, 30.0), (100_000, 0.3)])
def test_backprojection(n, spread, kind):
    lors, v = _lors(n, n, spread), _values(kind, n, 3)
    L, V = torch.as_tensor(lors).cuda(), torch.as_tensor(v).cuda()
    I = torch.zeros(GRID[::-1], device="cuda")
    bp = ops.tor_backprojection(I, L, V, GRID, [0, 0, 0], SIZE, KW, False, *TOF, layout="cn")
    assert K.rel_l2(bp.cpu().numpy(), _back64(lors, v)) <= TOL


@pytest.mark.parametrize("sign", ["positive", "negative", "few", "both"])
@pytest.mark.parametrize("n,spread", [(40_000, 30.0), (60_000, 0.3)])
def test_adjoint(n, spread, sign):
    lors, v = _lors(n, n + 1, spread), _values("plain", n, 4)
    s = np.ones(n, np.float32)
    if sign == "negative":
        s[:] = -1
    elif sign == "few":
        s[::200] = -1
    elif sign == "both":
        s[::2] = -1
    L, V = torch.as_tensor(lors).cuda(), torch.as_tensor(s / v).cuda()
    out = ops.tor_backproject_adjoint(V, L, GRID, [0, 0, 0], SIZE, KW, False, *TOF, layout="cn")
    pos, neg = s > 0, s < 0
    ref = np.zeros(GRID[::-1])
    total = np.zeros(GRID[::-1])  # the size of what cancels
    for m, f in ((pos, 1.0), (neg, -1.0)):
        if m.any():
            b = _back64(np.ascontiguousarray(lors[:, m]), v[m])
            ref, total = ref + f * b, total + b
    diff = np.linalg.norm((out.cpu().numpy() - ref).ravel())
    assert diff <= TOL * np.linalg.norm(total.ravel())


@pytest.mark.parametrize("n,spread", [(40_000, 30.0), (60_000, 0.3)])
def test_map(n, spread):
    lors = _lors(n, n + 2, spread)
    m7 = np.ascontiguousarray(lors[[0, 1, 2, 3, 4, 5, 9]])
    v = np.ones(n, np.float32)
    v[5::1000] = -2.0
    out = ops.tor_maplors(torch.zeros(GRID[::-1], device="cuda"), GRID, [0, 0, 0], SIZE,
                          torch.as_tensor(m7).cuda(), torch.as_tensor(v).cuda(), KW, False,
                          layout="cn")
    ref = O.tor_maplors(m7, v, GRID, [0, 0, 0], SIZE, KW, False, mode="f64")
    assert K.rel_l2(out.cpu().numpy(), ref) <= TOL
