"""Workloads of the MP-PCA denoiser, as its users call it.

Each case is one call of a public entry point on one problem: a 4D volume
``(x, y, z, t)``, a patch shape, a stride and a form. The sizes are those of
the package's benchmark and serving mix (96x96x48x48 and 48x48x24x48 with 11^3
patches at stride 3; x, y in 64..128, z in 32..64, t in {32, 48, 64, 96},
patches 5^3 / 7^3 / 11^3, strides 1..3; the 128x128x64x96 request at stride 2)
and, around them, smaller, ragged and odd-frame volumes.

``listed()`` names the fixed cases, ``draw(rng)`` gives more of the same
ranges, ``prepare(case, seed)`` makes the inputs, ``run(state)`` is one pass,
``work(case)`` the bytes and operations a pass cannot do without and
``exact(case, seed)`` the same outputs from plain torch in float64.
"""

import math
import random
from concurrent.futures import ThreadPoolExecutor

import torch

import lowrank_gpu_fastest_b200 as lrd

# Entry points of a case ("entry"):
#   device  denoise() of a CUDA tensor: the volume of a GPU pipeline
#   host    denoise() of a NumPy array: the drop-in call of a script
#   pinned  denoise() of a pinned CPU tensor: a loader that stages its volumes
#   noise   denoise_with_noise(): the volume with its noise and rank maps
#   batch   denoise_batch() of ``volumes`` volumes of mixed shapes
PHANTOMS = ("unit", "baseline")  # signal in [0, 1]; signal on a ~1000 baseline


def _case(name, entry, shape, patch, stride, **kw):
    c = dict(entry=entry, nx=shape[0], ny=shape[1], nz=shape[2], nt=shape[3], px=patch[0], py=patch[1],
             pz=patch[2], stride=stride, form="plain", phantom="unit", rank=4, sigma=0.05, ranks=False)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    p5, p7, p11 = (5, 5, 5), (7, 7, 7), (11, 11, 11)
    return [
        # one patch: the smallest call there is (a region of interest); latency and launches only
        _case("one_patch", "device", (11, 11, 11, 48), p11, 3, ranks=True),
        # the small benchmark volume, resident on the GPU
        _case("small_volume", "device", (48, 48, 24, 48), p11, 3),
        # the headline volume, resident on the GPU, in the three arithmetic forms users pick between
        _case("headline_plain", "device", (96, 96, 48, 48), p11, 3),
        _case("headline_accurate", "device", (96, 96, 48, 48), p11, 3, form="accurate"),
        _case("headline_tensor", "device", (96, 96, 48, 48), p11, 3, form="tensor", ranks=True),
        # the drop-in call: NumPy in, NumPy out, intensities of a scanner (baseline ~1000)
        _case("headline_host", "host", (96, 96, 48, 48), p11, 3, phantom="baseline", rank=5),
        # dense small patches, few frames: many small eigenproblems
        _case("dense_5cubed_t32", "device", (96, 96, 48, 32), p5, 1, sigma=0.1),
        # ragged sizes, mid patch, 64 frames
        _case("ragged_7cubed_t64", "device", (101, 87, 43, 64), p7, 2, sigma=0.03, rank=8),
        # 64 directions and one reference frame: an odd frame count on odd sizes
        _case("odd_frames_t65", "device", (61, 53, 37, 65), p7, 2, ranks=True),
        # quality-control run: volume, ranks, noise estimates and noise map of a 96-frame series
        _case("noise_maps_t96", "noise", (64, 64, 48, 96), p11, 3, phantom="baseline", rank=5),
        # a batch of a mixed queue
        _case("mixed_batch", "batch", (128, 128, 64, 96), p11, 3, volumes=4, mix=9),
        # the largest request of the serving mix
        _case("largest_request", "device", (128, 128, 64, 96), p11, 2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Rough work of one volume: Gram and reconstruction plus the eigenproblem."""
    n = c["px"] * c["py"] * c["pz"]
    t = c["nt"]
    return _patches(c) * (0.1 * n * t * t + 20.0 * t ** 3)


def draw(rng):
    big = listed()[-1]
    while True:
        entry = rng.choice(["device"] * 6 + ["host", "pinned", "noise", "batch"])
        t = rng.choice([32, 48, 64, 96]) if rng.random() < 0.7 else rng.randint(16, 128)
        p = rng.choice([5, 7, 11])
        patch = (p, p, p) if rng.random() < 0.85 else tuple(rng.choice([5, 6, 7, 9, 11]) for _ in range(3))
        if patch[0] * patch[1] * patch[2] < t:
            continue
        shape = (_log_int(rng, 16, 128), _log_int(rng, 16, 128), _log_int(rng, 11, 64), t)
        phantom = rng.choice(["unit", "unit", "unit", "baseline"])
        c = _case(None, entry, shape, patch, rng.choice([1, 2, 3]),
                  form=rng.choice(["plain", "plain", "plain", "accurate", "tensor", "tensor_bf16"]),
                  phantom=phantom, rank=rng.choice([2, 4, 8]) if phantom == "unit" else 5,
                  sigma=round(math.exp(rng.uniform(math.log(0.01), math.log(0.2))), 4),
                  ranks=rng.random() < 0.3 and entry != "batch")
        if entry == "batch":
            c.update(volumes=rng.randint(2, 6), mix=rng.randint(0, 10 ** 6), form="plain")
        total = sum(_cost(v) for v in _volumes(c))
        memory = sum(_patches(v) * v["nt"] ** 2 * 4 for v in _volumes(c))
        if total <= _cost(big) and memory <= 6e9:
            return c


def _volumes(c):
    """The volumes of a case: itself, or the mixed shapes of a batch."""
    if c["entry"] != "batch":
        return [c]
    rng = random.Random(c["mix"])
    got = []
    while len(got) < c["volumes"]:
        p = rng.choice([5, 7, 11])
        v = dict(c, nx=rng.randint(48, c["nx"]) if c["nx"] > 48 else c["nx"],
                 ny=rng.randint(48, c["ny"]) if c["ny"] > 48 else c["ny"],
                 nz=rng.randint(24, c["nz"]) if c["nz"] > 24 else c["nz"],
                 nt=rng.choice([32, 48, 64, 96]), px=p, py=p, pz=p, stride=rng.choice([2, 3]),
                 sigma=rng.uniform(0.02, 0.1), entry="device")
        if p ** 3 >= v["nt"] and min(v["nx"], v["ny"], v["nz"]) >= p:
            got.append(v)
    return got


def _corners(size, patch, stride):
    return sorted({*range(0, size - patch + 1, stride), size - patch})


def _patches(c):
    return math.prod(len(_corners(c["n" + a], c["p" + a], c["stride"])) for a in "xyz")


def _phantom(c, seed):
    """A smooth rank-r signal plus white noise, on the GPU from the seed alone:
    spatial maps that are products of cosines times sinusoid time courses,
    either scaled into [0, 1] with noise ``sigma`` or 20 units strong on a
    baseline of 200..2200 with noise 4."""
    rng = random.Random(seed * 7919 + 13)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rng.randrange(1 << 40))
    sides = [c["nx"], c["ny"], c["nz"]]

    def field():
        axes = [torch.cos(2 * math.pi * rng.uniform(0.5, 3.0) * torch.linspace(0, 1, n, device="cuda")
                          + rng.uniform(0, 2 * math.pi)) for n in sides]
        return axes[0][:, None, None] * axes[1][None, :, None] * axes[2][None, None, :]

    time = torch.linspace(0, 1, c["nt"], device="cuda")
    vol = torch.zeros(*sides, c["nt"], device="cuda")
    for _ in range(c["rank"]):
        course = torch.sin(2 * math.pi * rng.uniform(1, 6) * time + rng.uniform(0, 6))
        vol += field()[..., None] * course
    if c["phantom"] == "unit":
        lo, hi = vol.min(), vol.max()
        vol = (vol - lo) / (hi - lo).clamp_min(1e-6)
        sigma = c["sigma"]
    else:
        vol = 20.0 * vol + 1000.0 * (1.2 + field())[..., None]
        sigma = 4.0
    vol += sigma * torch.randn(vol.shape, generator=gen, device="cuda")
    return vol


def prepare(case, seed):
    vols = [_phantom(v, seed * 16 + i) for i, v in enumerate(_volumes(case))]
    if case["entry"] == "host":
        vols = [v.cpu().numpy() for v in vols]
    elif case["entry"] == "pinned":
        vols = [v.cpu().pin_memory() for v in vols]
    return dict(case=case, vols=vols, patches=[(v["px"], v["py"], v["pz"]) for v in _volumes(case)],
                strides=[v["stride"] for v in _volumes(case)])


def run(state):
    c, vols = state["case"], state["vols"]
    patch, stride = state["patches"][0], state["strides"][0]
    if c["entry"] == "batch":
        return lrd.denoise_batch(vols, state["patches"], state["strides"], form=c["form"])
    if c["entry"] == "noise":
        return lrd.denoise_with_noise(vols[0], patch, stride, form=c["form"])
    res = lrd.denoise(vols[0], patch, stride, form=c["form"], return_ranks=c["ranks"])
    return list(res) if c["ranks"] else res


def work(case):
    """The volume in and the results out once; every voxel's outer product
    once (T (T + 1) operations: the Gram sums share them), the T^3-order
    tridiagonalisation per patch, and the projection and weighted sum of every
    voxel of every patch at the signal's rank."""
    nbytes = flops = 0.0
    for v in _volumes(case):
        t, p = v["nt"], _patches(v)
        vox = v["nx"] * v["ny"] * v["nz"]
        n = v["px"] * v["py"] * v["pz"]
        nbytes += 2.0 * 4 * vox * t
        if v["ranks"] or case["entry"] in ("noise", "batch"):
            nbytes += 4.0 * p
        if case["entry"] == "noise":
            nbytes += 4.0 * p + 4.0 * vox
        flops += vox * t * (t + 1.0) + p * (4.0 / 3.0 * t ** 3) + p * n * t * (4.0 * v["rank"] + 3.0)
    return {"bytes": nbytes, "flops": flops}


def _exact_volume(c, vol):
    """Step 0's denoiser in float64: per patch the centred Gram matrix, its
    eigenvectors, the Marchenko-Pastur count, the projection, and the average
    of the patches with weights 1 / (2 + rank)."""
    t, (px, py, pz) = c["nt"], (c["px"], c["py"], c["pz"])
    n = px * py * pz
    rows = vol.double().reshape(-1, t)
    mean = rows.mean(1, keepdim=True)
    centred = rows - mean

    def grid(a, b, d):
        a, b, d = (torch.as_tensor(list(s), device="cuda") for s in (a, b, d))
        return ((a[:, None, None] * c["ny"] + b[None, :, None]) * c["nz"] + d[None, None, :]).reshape(-1)

    base = grid(*(_corners(c["n" + a], c["p" + a], c["stride"]) for a in "xyz"))
    offs = grid(range(px), range(py), range(pz))
    out = torch.zeros_like(rows)
    wsum = torch.zeros(rows.shape[0], dtype=torch.float64, device="cuda")
    noise = torch.zeros_like(wsum)
    sigma2 = torch.zeros(base.numel(), dtype=torch.float64, device="cuda")
    i = torch.arange(t - 1, dtype=torch.float64)
    step = max(1, int(4e8 // (8 * n * t)))
    torch.set_num_threads(1)
    with ThreadPoolExecutor() as pool:
        for at in range(0, base.numel(), step):
            idx = base[at:at + step, None] + offs
            x = centred[idx.reshape(-1)].reshape(-1, n, t)
            gram = torch.bmm(x.mT, x).cpu()
            parts = list(pool.map(torch.linalg.eigh, gram.split(max(1, len(gram) // 64))))
            lam = torch.cat([p[0] for p in parts]).flip(1)[:, :t - 1].clamp_min(0) / n
            vec = torch.cat([p[1] for p in parts]).flip(2)
            tail = lam.flip(1).cumsum(1).flip(1)
            test = (lam - lam[:, -1:]) * (t - 1 - i) * (n - i) > 4 * tail * math.sqrt((t - 1) * n)
            rank = test.sum(1)
            left = (t - 1 - rank).clamp_min(1)
            s2 = torch.where(rank < t - 1, tail.gather(1, rank.clamp_max(t - 2)[:, None])[:, 0] / left, 0.0).cuda()
            keep = int(rank.max())
            vec = (vec[:, :, :keep] * (torch.arange(keep) < rank[:, None])[:, None, :]).cuda()
            w = (1.0 / (2.0 + rank.double())).cuda()
            xd = torch.bmm(torch.bmm(x, vec), vec.mT) + mean[idx.reshape(-1)].reshape(-1, n, 1)
            out.index_add_(0, idx.reshape(-1), (xd * w[:, None, None]).reshape(-1, t))
            wsum.index_add_(0, idx.reshape(-1), w[:, None].expand(-1, n).reshape(-1))
            noise.index_add_(0, idx.reshape(-1), (w * s2)[:, None].expand(-1, n).reshape(-1))
            sigma2[at:at + step] = s2
    wsum = wsum.clamp_min(1e-12)
    side = (c["nx"], c["ny"], c["nz"])
    return (out / wsum[:, None]).reshape(*side, t), sigma2, (noise / wsum).reshape(side)


def exact(case, seed):
    vols = _volumes(case)
    if sum(_patches(v) * v["nt"] ** 3 for v in vols) > 2.5e10:
        return None  # the float64 eigenproblems alone would take too long
    got = [_exact_volume(v, _phantom(v, seed * 16 + i)) for i, v in enumerate(vols)]
    if case["entry"] == "batch":
        return [g[0] for g in got]
    out, sigma2, noise = got[0]
    if case["entry"] == "noise":
        return dict(out=out, ranks=None, sigma2=sigma2, noise=noise)
    out = out.cpu() if case["entry"] in ("host", "pinned") else out
    return [out, None] if case["ranks"] else out
