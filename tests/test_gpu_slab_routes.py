"""The slab kernels, forced, on calls that are small enough for the LOR-centric kernels to take
them by default: generated map LORs (whole slices and row bands, chunks), calls in chunks under
a scratch limit, and replay from a CUDA graph."""

import pytest
import torch

from srf_b200 import Image, SplitLoRsModel, _lib, ops, tuning
from srf_b200.batched import BatchedOSEM
from tests import _cases as K
from tests.test_generated_pairs import _fused_map_case

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def slabs():
    tuning.set_tuning(1, 0, 0)
    yield
    tuning.set_tuning()
    tuning.set_scratch_limit()


@pytest.mark.parametrize("case", ["random128", "random256band", "blockpairs"])
def test_generated_map(case):
    """random256band: the z group's 256 x 256 slices go in row bands of 49 rows."""
    _fused_map_case(case)


@pytest.mark.parametrize("axis", ["x", "z"])
def test_chunks_equal_one_pass(axis):
    """4096 LORs per chunk (one tile of the binning) against one pass; tolerance 1e-6, the
    order of float sums (test_gpu_large_fov)."""
    case = K.tor_case(n=30_000, seed=17, grid=(128, 128, 64), voxel=3.2, n_box=20_000)
    lors, img, g, c, s = K.tor_axis(case, axis)
    n = lors.shape[1]
    assert n > 4096
    b, s2 = K.tof_params(530.0)
    L, I = torch.as_tensor(lors).cuda(), torch.as_tensor(img).cuda()
    M = L[[0, 1, 2, 3, 4, 5, 9]].contiguous()

    def run():
        before = _lib.load().srf_launch_count()
        pv, bp = ops.tor_projection_backprojection(L, I, g, c, s, K.KW_CONFIG, False, b, s2,
                                                   layout="cn")
        m = ops.tor_maplors(I, g, c, s, M, pv + 1.0, K.KW_CONFIG, False, layout="cn")
        return (pv, bp, m), _lib.load().srf_launch_count() - before

    one, launches = run()
    assert launches == 5 + 4
    tuning.set_scratch_limit(4096)
    chunked, launches = run()
    assert launches == -(-n // 4096) * (5 + 4)
    for x, y in zip(chunked, one):
        assert torch.count_nonzero(y) > 0
        assert K.rel_l2(x.cpu().numpy(), y.cpu().numpy()) <= 1e-6


def test_graph_replay_equals_eager():
    """One iteration of four frames captured and replayed twice, images back to the start
    between; tolerance 1e-5 (test_gpu_recon's batched bound)."""
    grid, voxel = (48, 48, 24), 6.4
    size = [k * voxel for k in grid]
    b, s2 = K.tof_params(530.0)
    model = SplitLoRsModel(K.KW_CONFIG, False, tof_sigma2=s2, tof_bin=b)
    frames = [{a: torch.as_tensor(v.astype("float32")).cuda().contiguous()
               for a, v in K.tor_case(n=2000 + 500 * f, seed=50 + f, grid=grid)["groups"].items()}
              for f in range(4)]
    eff = Image(torch.full(grid, 0.9, device="cuda"), [0, 0, 0], size)
    x0 = torch.ones(grid, device="cuda")
    eager = BatchedOSEM(model, frames, eff, x0, n_subsets=2)
    graph = BatchedOSEM(model, frames, eff, x0, n_subsets=2, use_graph=True)
    ref = eager.step().clone()
    for _ in range(2):
        graph.x.copy_(x0.expand_as(graph.x))
        assert K.rel_l2(graph.step().cpu().numpy(), ref.cpu().numpy()) <= 1e-5
