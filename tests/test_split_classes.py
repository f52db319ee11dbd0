"""Envs too large for one block in a plan of many envs: each is split into two parts that just
fit, one env with the larger parts, the other with the longer exchange table.  A class of both
would need more shared memory than a block has, so that they get a class each; the plan is
made whatever their sizes, and its bits are those of the two envs in a plan of their own."""

import pytest
import torch

from ffsrl import SimIntegratorDO, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu


def _plan(meshes):
    m, _ = sc.liver_model("cuda:0", len(meshes), meshes=meshes, substeps=1, iterations=3)
    return m, SimIntegratorDO("cuda:0").plan(m)


def test_parts_and_exchange_tables_of_two_envs(gpu):
    small, wide = mg.beam(2, 1, 1), mg.ellipsoid_for_tets(53720)
    classes = set()
    # the long beam's parts grow by 13 vertices from each length to the next
    for length in range(552, 580):
        beam = mg.beam(length, 4, 4)
        m, plan = _plan([beam, wide] + [small] * 1078)
        classes.add(plan.info()["num_classes"])
        if length in (560, 566, 570):
            plan.step(1)
            few, alone = _plan([beam, wide])
            alone.step(1)
            torch.cuda.synchronize()
            for e in range(2):
                assert torch.equal(m.vertex[m.envSlice(e)], few.vertex[few.envSlice(e)])
            assert float((few.vertex - few.initialVertex).abs().max()) > 0.0
        del m, plan
    assert classes == {2, 3}  # below the joint limit one class for both, above it two
