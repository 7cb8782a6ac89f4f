"""The float32 eigensolver on Gram matrices of its own choosing, through the
eigensolve stage, against numpy's float64 eigh of the same matrices.

Tolerances: a float32 Householder reduction and its back-transform are exact
for a matrix within c n u ||A|| of the given one (u = 2^-24; c = 8 here), so
eigenvalues are within that, a returned vector's residual within twice it, and
the vectors are orthonormal to c n u.
"""

import numpy as np
import pytest
import torch

from lowrank_gpu_fastest_b200 import api, rel_l2
from oracle import mppca as orc

pytestmark = pytest.mark.gpu


def _gram(rng, T, N, rank):
    """Gram matrix of a centred low-rank patch with noise, far from an MP tie."""
    while True:
        x = rng.standard_normal((N, T)) * 0.1
        for r in range(rank):
            x += (3.0 + r) * np.outer(rng.standard_normal(N), rng.standard_normal(T)) / np.sqrt(T)
        x -= x.mean(1, keepdims=True)
        g = (x.T @ x).astype(np.float32)
        g = np.maximum(g, g.T)
        eigs = np.maximum(np.linalg.eigvalsh(g.astype(np.float64))[::-1][:T - 1], 0) / N
        t = T - 1
        i = np.arange(t)
        lhs = (eigs - eigs[-1]) * (t - i) * (N - i)
        rhs = 4 * np.cumsum(eigs[::-1])[::-1] * np.sqrt(t * N)
        if np.abs(lhs / np.maximum(rhs, 1e-300) - 1)[: t - 1].min(initial=1.0) > 1e-3:
            return g


# the lanes' and rows' edges (16, 32, 48, 64 rows), frame counts whose rows are not
# float4-aligned, odd matrix counts (a warp solves two), more vectors than one
# chunk of eight, and the block solver's sizes
@pytest.mark.parametrize("T,rank", [(2, 1), (5, 1), (15, 2), (16, 3), (17, 3), (31, 4), (32, 10), (33, 4), (47, 5),
                                    (48, 19), (49, 3), (63, 6), (64, 17), (65, 3), (96, 9), (97, 2), (128, 5)])
def test_eigh_stage_vs_numpy(cuda_ok, T, rank):
    rng = np.random.default_rng(T)
    patch, stride = (6, 6, 6), 2
    shape = (12, 8, 6, T)  # 4 x 2 x 1 patches and one more in x
    N = 216
    plan = api.get_plan(shape, patch, stride)
    P = plan.n_patches
    g = np.stack([_gram(rng, T, N, rank if i % 2 else max(1, rank // 2)) for i in range(P)])
    flat = torch.empty(P * T * T + 1, device="cuda")
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    got = []
    for off in (0, 1):  # a caller's block that is not 16-byte aligned takes scalar loads
        block = flat[off:off + P * T * T]
        block.copy_(torch.from_numpy(g.reshape(-1)))
        lam = torch.empty(P, T, device="cuda")
        vecs = torch.zeros(P, T, T, device="cuda")
        ranks = torch.empty(P, dtype=torch.int32, device="cuda")
        plan.stage_eigh(block.data_ptr(), lam.data_ptr(), vecs.data_ptr(), ranks.data_ptr(), ws.data_ptr(), s)
        torch.cuda.synchronize()
        got.append([t.cpu().numpy() for t in (lam, vecs, ranks)])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    lam, vecs, ranks = got[0]
    tol = 8 * T * 2.0 ** -24
    for i in range(P):
        ref = np.linalg.eigvalsh(g[i].astype(np.float64))
        assert np.abs(lam[i] - ref).max() <= tol * ref[-1]
        p = orc.mp_rank_from_eigs(np.maximum(ref[::-1][:T - 1], 0) / N, N)
        assert int(ranks[i]) == p
        V = vecs[i].reshape(-1)[: T * p].reshape(p, T).T.astype(np.float64)
        assert np.abs(V.T @ V - np.eye(p)).max(initial=0) <= tol
        res = g[i].astype(np.float64) @ V - V * ref[::-1][:p]
        assert np.abs(res).max(initial=0) <= 2 * tol * ref[-1]


@pytest.mark.parametrize("T", [24, 48, 64])
def test_equal_signal_eigenvalues(cuda_ok, T):
    """Two components of equal strength: the kept eigenvalues agree to float32,
    where one eigenvector could come out twice. Against step 0 and float64."""
    shape, patch = (8, 8, 6, T), (8, 8, 4)
    rng = np.random.default_rng(1)
    x, y, z = np.meshgrid(*(np.arange(s) for s in shape[:3]), indexing="ij")
    k = 2 * np.pi * np.arange(T) / T
    # +-1 maps, orthogonal over every patch; zero-mean sinusoids, orthogonal over T
    vol = ((-1.0) ** x)[..., None] * np.sin(3 * k) + ((-1.0) ** y)[..., None] * np.cos(3 * k)
    vol = (vol + 1e-6 * rng.standard_normal(shape)).astype(np.float32)
    ref, ranks = orc.denoise(vol, patch, 2)
    ref64, _ = orc.denoise_fp64(vol, patch, 2)
    assert (ranks >= 2).all()
    d = torch.from_numpy(vol).cuda()
    out, got = api.denoise(d, patch, 2, form="accurate", return_ranks=True)
    # both components whole: dropping one would be an error of 0.7
    assert rel_l2(out.cpu().numpy(), ref64) <= 1e-6
    plain = api.denoise(d, patch, 2)
    assert rel_l2(plain.cpu().numpy(), ref) <= 1e-6


@pytest.mark.parametrize("T", [24, 32, 48, 64, 96, 127])
def test_round_off_vectors_are_orthonormal(cuda_ok, T):
    """Two equal components over round-off: the tridiagonal's tail vanishes, many kept
    eigenvalues are round-off, and their vectors coincide before they are made
    orthogonal. A projection leaves at least 0.03 of a vector, so T dot products of
    T terms, rounded by T 2^-24 each, put V^T V at most 2 T 2^-24 / 0.03 from 1; the
    two components' span moves by the reduction's T 2^-24 a few times over."""
    shape, patch = (8, 8, 6, T), (8, 8, 4)
    rng = np.random.default_rng(1)
    x, y, z = np.meshgrid(*(np.arange(s) for s in shape[:3]), indexing="ij")
    k = 2 * np.pi * np.arange(T) / T
    vol = ((-1.0) ** x)[..., None] * np.sin(3 * k) + ((-1.0) ** y)[..., None] * np.cos(3 * k)
    vol = (vol + 1e-6 * rng.standard_normal(shape)).astype(np.float32)
    plan = api.get_plan(shape, patch, 2)
    P = plan.n_patches
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    G = torch.empty(P, T, T, device="cuda")
    d = torch.from_numpy(vol).cuda()
    plan.stage_gram(d.data_ptr(), G.data_ptr(), ws.data_ptr(), s)
    lam, vecs = torch.empty(P, T, device="cuda"), torch.empty(P, T, T, device="cuda")
    ranks = torch.empty(P, dtype=torch.int32, device="cuda")
    plan.stage_eigh(G.data_ptr(), lam.data_ptr(), vecs.data_ptr(), ranks.data_ptr(), ws.data_ptr(), s)
    torch.cuda.synchronize()
    for i in range(P):
        p = int(ranks[i])
        assert p >= 2
        V = vecs[i].cpu().numpy().reshape(-1)[: T * p].reshape(p, T).T.astype(np.float64)
        assert np.abs(V.T @ V - np.eye(p)).max() <= 2 * T * 2.0 ** -24 / 0.03
        U = np.linalg.eigh(G[i].cpu().numpy().astype(np.float64))[1][:, -2:]
        assert np.linalg.norm(U - V[:, :2] @ (V[:, :2].T @ U)) <= 8 * T * 2.0 ** -24


@pytest.mark.parametrize("T", [33, 40, 48])
def test_small_launches_agree(cuda_ok, T):
    """A launch that fits the device at once takes another kernel: equal bit for bit to
    the same patches in one large launch (3179 of them), with and without a remainder."""
    rng = np.random.default_rng(T)
    vol = torch.from_numpy(rng.standard_normal((20, 20, 14, T)).astype(np.float32)).cuda()
    want, ranks = api.denoise(vol, (4, 4, 4), 1, return_ranks=True)
    for batch in (97, 2000):
        got, r = api.denoise(vol, (4, 4, 4), 1, batch=batch, return_ranks=True)
        assert torch.equal(got, want) and torch.equal(r, ranks)
