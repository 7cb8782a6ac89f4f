"""The warp reconstruction against the brick kernel (an explicit brick selects
it): the same arithmetic in another decomposition, so every output is equal bit
for bit, and the brick kernel is held to step 0 and float64 elsewhere."""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api

pytestmark = pytest.mark.gpu


def _run(plan, vol):
    out = torch.full_like(vol, float("nan"))
    ranks = torch.empty(plan.n_patches, dtype=torch.int32, device="cuda")
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    plan.denoise(vol.data_ptr(), out.data_ptr(), ranks.data_ptr(), ws.data_ptr(), s)
    assert plan.status(ws.data_ptr(), s) == 0
    return out, ranks


# volume sides off the 2 x 2 x (4, 8) bricks, patches that end between a lane's two
# voxels, one-plane patches, gaps between patches, z-runs of more than 32 patches
# and of more rows than a buffer holds, ranks of zero and of more than a buffer's 40
# rows at T = 96 (rank 60)
@pytest.mark.parametrize("form", ["plain", "accurate"])
@pytest.mark.parametrize("T,size,patch,stride,rank", [
    (32, (9, 8, 13), (5, 5, 5), 1, 4), (32, (7, 9, 45), (3, 4, 3), 1, 0), (48, (12, 11, 11), (11, 11, 11), 3, 4),
    (48, (11, 13, 15), (5, 5, 5), 2, 9), (48, (12, 11, 17), (4, 4, 4), 7, 3), (48, (9, 9, 10), (7, 7, 1), 1, 30),
    (64, (10, 9, 12), (5, 5, 5), 2, 5), (64, (8, 9, 21), (6, 5, 3), 2, 20), (96, (11, 10, 9), (7, 7, 7), 2, 5),
    (96, (8, 7, 17), (7, 7, 7), 3, 60), (96, (7, 7, 23), (7, 7, 2), 1, 12),
])
def test_warp_equals_brick_kernel(cuda_ok, T, size, patch, stride, rank, form):
    rng = np.random.default_rng(T + rank)
    n = int(np.prod(size))
    vol = 0.05 * rng.standard_normal((n, T))
    if rank:
        vol += rng.standard_normal((n, rank)) @ rng.standard_normal((rank, T))
    vol = torch.from_numpy((vol + 7.0).reshape(*size, T).astype(np.float32)).cuda()
    shape = tuple(vol.shape)
    out, ranks = _run(api.get_plan(shape, patch, stride, form=form), vol)
    ref, rref = _run(api.get_plan(shape, patch, stride, form=form, brick=(3, 2, 3), split=4), vol)
    assert torch.equal(ranks, rref)
    assert (int(ranks.max()) > 40) == (rank == 60)
    assert torch.equal(out, ref)
