"""The column Gram against float64 Grams of the same centred patches.

Tolerance (rigorous): a float32 sum of n products in any order is within
(n + 1) u sum |x_r x_c| of the exact one, u = 2^-24, and the sum of absolute
products is at most sqrt(G_rr G_cc). The kernel's longest chain is a plane's
rows, the lanes' exchange and the window's planes: n = px * py + pz + 4.
"""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api
from oracle import mppca as orc

pytestmark = pytest.mark.gpu


# quads of the 8 x 8 blocks even and odd in number (T % 8), one block (T = 4, 8),
# row counts off the split (odd patches, one-voxel planes), a stride beyond the
# patch (planes in no window), a border-shifted last corner, and window rings
# that do not fit shared memory (T = 96 and 128 at stride 1: columns cut); frame
# counts whose rows are padded (T % 4)
@pytest.mark.parametrize("shape,patch,stride,split", [
    ((7, 6, 9, 4), (3, 2, 3), 2, 0), ((9, 8, 7, 8), (3, 3, 3), 1, 4), ((8, 9, 13, 12), (5, 3, 4), 2, 1),
    ((9, 9, 12, 20), (1, 5, 5), 1, 0), ((9, 9, 12, 20), (5, 1, 5), 3, 2), ((12, 11, 17, 44), (5, 5, 5), 7, 0),
    ((12, 12, 14, 48), (5, 6, 5), 3, 4), ((12, 12, 16, 64), (5, 5, 5), 1, 0), ((13, 12, 15, 96), (11, 11, 11), 1, 0),
    ((8, 8, 12, 100), (5, 5, 5), 2, 0), ((8, 9, 14, 128), (7, 7, 7), 1, 4),
    ((7, 6, 9, 2), (3, 2, 3), 2, 0), ((7, 6, 9, 5), (3, 3, 3), 1, 0), ((8, 9, 13, 31), (5, 4, 4), 2, 2),
    ((9, 8, 11, 65), (5, 5, 5), 2, 0), ((13, 12, 15, 99), (11, 11, 11), 1, 0), ((8, 8, 9, 126), (6, 6, 5), 2, 1),
])
def test_column_gram_vs_float64(cuda_ok, shape, patch, stride, split):
    rng = np.random.default_rng(shape[3])
    T = shape[3]
    vol = (rng.standard_normal(shape) + 3 * rng.standard_normal(shape[:3] + (1,))).astype(np.float32)
    plan = api.get_plan(shape, patch, stride, gram_split=split)
    P = plan.n_patches
    d = torch.from_numpy(vol).cuda()
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    # a result block that is not 16-byte aligned takes scalar stores
    flat = torch.full((P * T * T + 1,), float("nan"), device="cuda")
    plan.stage_gram(d.data_ptr(), flat[1:].data_ptr(), ws.data_ptr(), s)
    gram = torch.full((P, T, T), float("nan"), device="cuda")
    plan.stage_gram(d.data_ptr(), gram.data_ptr(), ws.data_ptr(), s)
    assert plan.status(ws.data_ptr(), s) == 0
    assert torch.equal(flat[1:].view(P, T, T), gram)
    gram = gram.cpu().numpy().astype(np.float64)
    n = patch[0] * patch[1] + patch[2] + 4
    corners = orc.patch_corners(shape, patch, stride)
    for idx in range(0, P, max(1, P // 40)):
        i, j, k = corners[idx]
        x = vol[i:i + patch[0], j:j + patch[1], k:k + patch[2]].reshape(-1, T)
        xc = (x - x.mean(axis=1, keepdims=True)).astype(np.float64)
        G = xc.T @ xc
        bound = (n + 1) * 2.0 ** -24 * np.sqrt(np.outer(np.diag(G), np.diag(G)))
        assert np.all(np.abs(gram[idx] - G) <= bound + 1e-30)
        assert np.array_equal(gram[idx], gram[idx].T)
