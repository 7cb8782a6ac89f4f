"""Small launches of the warp eigensolver (up to 48 frames) take a kernel of their
own: equal bit for bit to the same patches in one large launch."""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api

pytestmark = pytest.mark.gpu


# 4998 patches at once: the kernel of large launches. In batches, with remainders
@pytest.mark.parametrize("T", [2, 5, 16, 24, 31, 32, 33, 48])
@pytest.mark.parametrize("rank", [0, 3])
def test_batches_agree(cuda_ok, T, rank):
    rng = np.random.default_rng(T + rank)
    v = rng.standard_normal((24 * 20 * 17, T))
    if rank:
        v = 0.05 * v + rng.standard_normal((24 * 20 * 17, rank)) @ rng.standard_normal((rank, T))
    vol = torch.from_numpy(v.reshape(24, 20, 17, T).astype(np.float32)).cuda()
    want, ranks = api.denoise(vol, (4, 4, 4), 1, return_ranks=True)
    assert ranks.numel() == 4998
    for batch in (97, 2000, 4499):
        got, r = api.denoise(vol, (4, 4, 4), 1, batch=batch, return_ranks=True)
        assert torch.equal(got, want) and torch.equal(r, ranks)
