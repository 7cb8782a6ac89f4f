"""The autotuner's file on disk: a choice that was timed on other kernels (an
entry of an older package, with another meaning of its Gram split) is passed
over, one of these kernels is used."""

import json

from lowrank_gpu_fastest_b200 import tune


def test_choices_of_other_kernels_are_passed_over(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("LRD_TUNE_CACHE", str(path))
    entry = {"brick": [3, 3, 3], "split": 2, "gram_split": 1, "eigh_block": 1, "recon_ms": 1.0}
    k = tune.key("sm_100:148", 32, (11, 11, 11), 3, "plain")
    path.write_text(json.dumps({k: entry}))  # as the package before these kernels wrote it
    assert tune._stored(k) is None
    monkeypatch.setattr(tune, "KERNELS", tune.KERNELS + 1)
    later = tune._slot(k)
    monkeypatch.undo()
    monkeypatch.setenv("LRD_TUNE_CACHE", str(path))
    path.write_text(json.dumps({k: entry, later: entry}))
    assert tune._stored(k) is None
    path.write_text(json.dumps({k: dict(entry, gram_split=4), tune._slot(k): entry}))
    assert tune._stored(k) == dict(brick=(3, 3, 3), split=2, gram_split=1, eigh_block=1)
