"""The float64 near-tie pass against numpy's float64 results.

The eigensolve stage is handed Gram matrices whose eigenvalues sit on an MP tie,
so every patch is queued and recomputed in float64 from the centred volume: its
eigenvalues, rank and eigenvectors are then those of the float64 Gram matrix of
the patch's rows.

Tolerances: an eigenvalue is a float64 result (intervals of 1e-14 of the norm,
the reduction's own round-off below 1e-13 of it) rounded to float32, half an ulp
= 6e-8 relative; an eigenvector entry (magnitude <= 1) is rounded likewise, so
an entry of V V^T is within 2 * 6e-8 * sqrt(p) of the projector, p <= 8.
"""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api
from lowrank_gpu_fastest_b200.harness import make_phantom_lowrank
from oracle import mppca as orc

pytestmark = pytest.mark.gpu


def tied_gram(T, N):
    """Diagonal matrix (one null eigenvalue, noise eigenvalues b, one on the MP
    threshold to float32 rounding) that the float32 pass must queue."""
    t = T - 1
    b, s = 1.0, np.sqrt(t * N)
    top = b * (t * N + 4 * (t - 1) * s) / (t * N - 4 * s)
    return N * np.diag([0.0] + [b] * (t - 1) + [top]).astype(np.float32)


# edges of the 4 x 4 blocks (T % 4), of the threads per row (powers of two at
# T = 16, 32, 64, 128), of the single pass over the patch (T = 124 / 125), and
# patches of one staged chunk and of many
@pytest.mark.parametrize("T,patch", [(3, (5, 5, 5)), (8, (3, 3, 3)), (16, (4, 3, 2)), (17, (5, 5, 5)),
                                     (31, (5, 4, 3)), (32, (5, 5, 5)), (48, (7, 7, 7)), (65, (5, 5, 5)),
                                     (96, (11, 11, 11)), (124, (5, 5, 5)), (125, (5, 5, 6)), (128, (6, 5, 5))])
def test_near_tie_pass_vs_float64(cuda_ok, T, patch):
    shape, stride = (13, 12, 12, T), 3
    N = patch[0] * patch[1] * patch[2]
    vol = make_phantom_lowrank(shape, rank=3, seed=T)[0]
    plan = api.get_plan(shape, patch, stride)
    P = plan.n_patches
    d = torch.from_numpy(vol).cuda()
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    gram = torch.empty(P, T, T, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    plan.stage_gram(d.data_ptr(), gram.data_ptr(), ws.data_ptr(), s)  # leaves the centred volume in ws
    tied = torch.from_numpy(tied_gram(T, N)).cuda().expand(P, T, T).contiguous()
    lam = torch.empty(P, T, device="cuda")
    vecs = torch.zeros(P, T, T, device="cuda")
    ranks = torch.empty(P, dtype=torch.int32, device="cuda")
    plan.stage_eigh(tied.data_ptr(), lam.data_ptr(), vecs.data_ptr(), ranks.data_ptr(), ws.data_ptr(), s)
    torch.cuda.synchronize()
    lam, vecs, ranks = (t.cpu().numpy() for t in (lam, vecs, ranks))
    corners = orc.patch_corners(shape, patch, stride)
    for idx in range(0, P, max(1, P // 12)):
        i, j, k = corners[idx]
        x = vol[i:i + patch[0], j:j + patch[1], k:k + patch[2]].reshape(-1, T)
        xc = (x - x.mean(axis=1, keepdims=True)).astype(np.float64)  # float32 centred, as in ws
        ref, V64 = np.linalg.eigh(xc.T @ xc)
        assert np.all(np.abs(lam[idx] - ref) <= 6.1e-8 * np.abs(ref) + 1e-12 * ref[-1])
        p = orc.mp_rank_from_eigs(np.maximum(ref[::-1][:T - 1], 0) / N, N)
        assert int(ranks[idx]) == p
        V = vecs[idx].reshape(-1)[: T * p].reshape(p, T).T.astype(np.float64)
        top = V64[:, T - p:]
        if p and (p == T or ref[T - p] - ref[T - p - 1] > 1e-4 * ref[-1]):
            assert np.abs(V @ V.T - top @ top.T).max() <= 4e-7
