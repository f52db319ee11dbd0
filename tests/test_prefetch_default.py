"""Records fetched into registers (kind 2) for a class with the plan's own block size: accepted
whatever that is for middle-sized envs, with the same bits; a block size that the caller has
set and that has no such kernel is still refused."""

import pytest
import torch

from ffsrl import SimIntegratorDO, _lib as L, autotune, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arithmetic", ["reference", "fast"])
def test_register_prefetch_of_default_classes(gpu, arithmetic):
    mesh = mg.ellipsoid_for_tets(6000, seed=3)  # 1,684 vertices; 1,100 envs are not divided
    out = []
    for kind in (0, 2):
        m, _ = sc.liver_model("cuda:0", 1100, meshes=[mesh] * 1100, substeps=2, iterations=3)
        plan = SimIntegratorDO("cuda:0", arithmetic=arithmetic).plan(m)
        cls = autotune._classes(plan)
        assert len(cls) == 1 and cls[0]["split"] == 1 and 1024 < cls[0]["max_nv"] <= 2560
        L.check(L.lib().ffsrl_batch_set_class_prefetch(plan.handle, 0, kind))
        plan.step(1)
        torch.cuda.synchronize()
        out.append(m.vertex.clone())
    assert torch.equal(*out)
    L.check(L.lib().ffsrl_batch_set_class_prefetch(plan.handle, 0, 0))
    L.check(L.lib().ffsrl_batch_set_class_block(plan.handle, 0, 768))
    assert L.lib().ffsrl_batch_set_class_prefetch(plan.handle, 0, 2) != L.OK
