"""The autotuner's cache tells a class whose envs are divided among clusters of blocks from the
same class undivided, and tries the block sizes that its kernels have."""

import numpy as np
import pytest
import torch

from ffsrl import SimIntegratorDO, autotune, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu


def _plan(meshes):
    m, _ = sc.liver_model("cuda:0", len(meshes), meshes=meshes)
    return m, SimIntegratorDO("cuda:0").plan(m)


def test_divided_class_has_a_key_of_its_own(gpu):
    big, small = mg.ellipsoid_for_tets(12000, seed=1), mg.beam(2, 1, 1)
    keys = {}
    for others in (0, 1200):  # few envs: the big one is divided; many: it is not
        m, plan = _plan([big] + [small] * others)
        cls = next(c for c in autotune._classes(plan) if 0 in c["envs"])
        assert len(cls["envs"]) == 1
        assert (cls["split"] > 1) == (others == 0)
        keys[others] = autotune._key(plan, cls)
    assert keys[0] != keys[1200]


def test_divided_class_is_tuned_over_its_own_kernels(gpu, monkeypatch, tmp_path):
    monkeypatch.setenv("FFSRL_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    mesh = mg.ellipsoid_for_tets(3000, seed=2)
    m, plan = _plan([mesh] * 2)
    tried = []
    time = autotune._time
    monkeypatch.setattr(autotune, "_time", lambda plan, envs, reps: tried.append(plan.info()["block_threads"]) or time(plan, envs, reps))
    result = autotune.autotune(plan)
    assert [b for (b,) in tried] == [128, 256, 512, 768]  # each kernel once
    assert result[0]["block"] in (128, 256, 512, 768) and result[0]["prefetch"] == 0
    want = m.vertex.clone()
    plan.step(1)
    torch.cuda.synchronize()
    assert torch.isfinite(m.vertex).all() and not torch.equal(m.vertex, want)
    assert np.array_equal(autotune._classes(plan)[0]["envs"], [0, 1])
