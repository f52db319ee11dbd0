"""Constraints that are switched off in the reference-shaped step: an edge, a tet or a surface
triangle that is inactive (a hole) may hold ids that are no vertices' or envs' at all -- rows
that pad an array, or that a removal has overwritten -- and the step gives what it gives with
those of the intact mesh.  The first record of each array, whose row the threads past the
end load too, is among them."""

import numpy as np
import pytest
import torch

from ffsrl import SimIntegratorDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu

PBD = L.VOLUME | L.DISTANCE | L.DRAG | L.COLLIDE
XPBD = L.VOLUME_XPBD | L.DISTANCE_XPBD | L.DRAG | L.COLLIDE


@pytest.mark.parametrize("flags", [PBD, XPBD])
@pytest.mark.parametrize("tets,copies", [(300, 2), (1000, 1), (16000, 33)])  # 33: one lane a triangle
def test_ids_of_inactive_records_are_not_followed(gpu, flags, tets, copies):
    mesh = mg.ellipsoid_for_tets(tets, seed=7)
    out = []
    for garbage in (False, True):
        m, _ = sc.liver_model("cuda:0", copies, meshes=[mesh] * copies, substeps=2, iterations=3)
        m.constraintFlags = flags
        rng = np.random.Generator(np.random.PCG64(1))
        for ids, mask, off in ((m.tetrahedron, m.activeTetrahedron, 0.0), (m.edge, m.activeEdge, 0.0), (m.triangle, m.hole, 1)):
            n = mask.numel()
            pick = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, size=n // 5)]))
            pick = torch.as_tensor(pick, device="cuda:0")
            mask[pick] = off
            if garbage:
                rows = ids.view(n, -1)
                rows[pick[0::2]] = -(1 << 30)
                rows[pick[1::2]] = (1 << 30) + 7
                if ids is m.triangle:
                    m.triToEnv[pick] = -(1 << 28)
        m.graspNearest(torch.ones(copies, dtype=torch.int32, device="cuda:0"), radius=1.0)
        SimIntegratorDO("cuda:0", batched=False).stepModel(m, 1)
        torch.cuda.synchronize()
        out.append(m.vertex.cpu().numpy())
    assert np.isfinite(out[0]).all()
    # (float atomics: the sums' order differs from run to run)
    np.testing.assert_allclose(out[1], out[0], rtol=0, atol=1e-4 * np.abs(out[0]).max())
    assert np.abs(out[0] - m.initialVertex.cpu().numpy()).max() > 1e-4
