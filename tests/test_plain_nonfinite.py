"""Contact of the reference-shaped step with vertices that are no numbers any more: the triangles
of a vertex at infinity or NaN are not skipped as out of every capsule's reach; they spoil the
same vertices as in the CPU restatement, which tests every triangle."""

import numpy as np
import pytest
import torch

import oracle
from ffsrl import SimIntegratorDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("tets,copies", [(700, 2), (16000, 33)])  # four lanes a triangle, and one
def test_nonfinite_vertices_in_contact(gpu, oracle_lib, value, tets, copies):
    meshes = [mg.ellipsoid_for_tets(tets, seed=5)] * copies
    m, _ = sc.liver_model("cuda:0", copies, meshes=meshes, substeps=1, iterations=1)
    m.constraintFlags = L.COLLIDE
    x = m.vertex.cpu().numpy()
    tri = m.host["triangle"].reshape(-1, 3)
    far = tri[np.argmax(x[tri].mean(axis=1) @ np.array([1.0, -1.0, 0.0]))]  # a triangle away from the instrument
    m.vertex[int(far[0]), 0] = value
    o = oracle.OracleSim(m, {
        "vertex": m.vertex.cpu().numpy(), "velocity": m.velocity.cpu().numpy(),
        "laparoscope_base": m.laparoscopeBase.cpu().numpy(), "laparoscope_tip": m.laparoscopeTip.cpu().numpy(),
        "laparoscope_radius": m.laparoscopeRadius.cpu().numpy()})
    SimIntegratorDO("cuda:0", batched=False).stepModel(m, 1)
    torch.cuda.synchronize()
    o.step(1)
    got, want = np.isfinite(m.vertex.cpu().numpy()), np.isfinite(o.a["vertex"])
    assert not want[far].all(axis=1).all()
    assert np.array_equal(got, want)
