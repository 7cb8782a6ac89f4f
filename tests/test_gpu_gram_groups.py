"""The column Gram where many planes lie in the same windows (stride at or beyond
the patch side, a volume one patch deep): a lane's chain of additions is bounded.

Rows are a (+1, -1, +1, ...), whose temporal mean is exactly 0. A patch's first
plane has a^2 such that a lane's sum of it comes to just above 16, and every
later product is just below half of a unit in the last place of that: added one
after the other to it they are all lost, with an error of (later products of a
lane) u of the sum, u = 2^-24. A lane adds at most g planes before its sum goes
to the window (three; two where rows are padded or KS = 2), so the error is within
(n + 1) u, n = g ceil(px py / KS) products, log2(KS) exchanges, a window addition
per group of planes and the two-word windows' last one - far less than the loss
of an unbounded chain."""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api

pytestmark = pytest.mark.gpu


# frame count (a multiple of 4 or not, two CTAs per column), patch, stride, depth in
# patches, threads per block KS (by the frame count, or from the split asked for)
@pytest.mark.parametrize("T,patch,stride,nz,split,ks", [
    (48, (11, 11, 11), 11, 22, 0, 8), (64, (11, 11, 11), 13, 24, 0, 4), (96, (11, 11, 11), 3, 11, 0, 4),
    (65, (11, 11, 11), 11, 22, 0, 4), (31, (7, 7, 7), 7, 14, 0, 4), (20, (9, 9, 9), 9, 9, 0, 8),
    (96, (15, 15, 15), 15, 30, 0, 4), (31, (15, 15, 15), 2, 15, 0, 4), (126, (11, 11, 11), 11, 11, 0, 4),
    (64, (11, 11, 11), 11, 11, 1, 2), (32, (5, 5, 15), 15, 15, 0, 4),
])
def test_plane_groups_are_bounded(cuda_ok, T, patch, stride, nz, split, ks):
    px, py, pz = patch
    rows = px * py
    lane = rows // ks
    shape = (px, py, nz, T)
    first = np.float32(np.sqrt(16.01 / lane))
    later = np.float32(np.sqrt(0.98 * 2.0 ** -20))
    starts = sorted({*range(0, nz - pz + 1, stride), nz - pz})
    amp = np.full(nz, later, np.float32)
    amp[starts] = first
    sign = np.zeros(T, np.float32)
    sign[:T - T % 2] = np.tile([1, -1], T // 2)
    vol = np.broadcast_to(amp[:, None] * sign, (px, py, nz, T)).copy()
    plan = api.get_plan(shape, patch, stride, gram_split=split)
    P = plan.n_patches
    assert P == len(starts)
    d = torch.from_numpy(vol).cuda()
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    gram = torch.full((P, T, T), float("nan"), device="cuda")
    plan.stage_gram(d.data_ptr(), gram.data_ptr(), ws.data_ptr(), s)
    assert plan.status(ws.data_ptr(), s) == 0
    gram = gram.cpu().numpy().astype(np.float64)
    g = 2 if T % 4 or ks == 2 else 3
    n = g * -(-rows // ks) + (ks.bit_length() - 1) + -(-pz // g) + 1
    lost = lane * (pz - 1)  # products that an unbounded chain would lose
    assert n + 1 < 0.9 * lost
    u = 2.0 ** -24
    for k in range(P):
        x = vol[:, :, starts[k]:starts[k] + pz].reshape(-1, T).astype(np.float64)
        G = x.T @ x
        bound = (n + 1) * u * np.sqrt(np.outer(np.diag(G), np.diag(G)))
        assert np.all(np.abs(gram[k] - G) <= bound + 1e-30)
