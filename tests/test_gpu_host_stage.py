"""Pageable input large enough to go through the plan's pinned slots, against the
same volume denoised on the device: equal bit for bit."""

import threading

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api

pytestmark = pytest.mark.gpu


# just above the size from which slots are used (32 MiB), slabs that end inside a
# chunk, few wide planes, and enough chunks for every slot to be used several times
@pytest.mark.parametrize("shape,patch,stride", [((61, 67, 43, 48), (7, 7, 7), 3), ((12, 128, 100, 64), (5, 5, 5), 4),
                                                ((96, 96, 48, 33), (7, 7, 5), 5)])
def test_pageable_input_equals_device(cuda_ok, shape, patch, stride):
    rng = np.random.default_rng(shape[0])
    vols = [rng.standard_normal(shape, dtype=np.float32) for _ in range(2)]
    assert vols[0].nbytes >= 32 << 20
    want = [api.denoise(torch.from_numpy(v).cuda(), patch, stride).cpu().numpy() for v in vols]
    for v, w in zip(vols, want):
        np.testing.assert_array_equal(api.denoise(v, patch, stride), w)
    # two threads, one plan
    got = [None, None]

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = api.denoise(vols[i], patch, stride)

    team = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    [t.start() for t in team]
    [t.join() for t in team]
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
