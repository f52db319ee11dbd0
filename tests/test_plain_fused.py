"""The reference-shaped step's joined launches (tets and edges in one grid, apply with drag,
bounds with the velocity update) against the CPU restatement: each subset of the constraints
that changes the grid's make-up, on tet counts below, at and above a block, ground contact
and a grasped vertex included."""

import numpy as np
import pytest
import torch

import oracle
from ffsrl import SimIntegratorDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu

POS_TOL = 1e-4  # of the parity tests


@pytest.mark.parametrize("flags", [L.VOLUME, L.DISTANCE, L.NEOHOOKEAN, L.VOLUME | L.DISTANCE, L.VOLUME | L.NEOHOOKEAN,
                                   L.NEOHOOKEAN | L.DISTANCE, L.VOLUME | L.NEOHOOKEAN | L.DISTANCE,
                                   L.VOLUME_XPBD | L.NEOHOOKEAN | L.DISTANCE, 0])
@pytest.mark.parametrize("tets,drag", [(100, True), (256, False), (700, True)])
def test_joined_launches(gpu, oracle_lib, flags, tets, drag):
    m, _ = sc.liver_model("cuda:0", 2, meshes=[mg.ellipsoid_for_tets(tets, seed=5)] * 2, substeps=3, iterations=4)
    m.constraintFlags = flags | (L.DRAG if drag else 0)
    m.groundLevel = float(m.vertex[:, 1].min()) + 0.05
    m.graspNearest(torch.ones(2, dtype=torch.int32, device="cuda:0"), radius=1.0)
    torch.cuda.synchronize()
    o = oracle.OracleSim(m, {
        "vertex": m.vertex.cpu().numpy(), "velocity": m.velocity.cpu().numpy(),
        "laparoscope_base": m.laparoscopeBase.cpu().numpy(), "laparoscope_tip": m.laparoscopeTip.cpu().numpy(),
        "laparoscope_radius": m.laparoscopeRadius.cpu().numpy(),
        "active_drag_constraint": m.activeDragConstraint.cpu().numpy()})
    SimIntegratorDO("cuda:0", batched=False).stepModel(m, 2)
    torch.cuda.synchronize()
    o.step(2)
    x, want = m.vertex.cpu().numpy(), o.a["vertex"]
    assert np.abs(x - want).max() < POS_TOL * np.abs(want).max()
    assert np.abs(want - m.initialVertex.cpu().numpy()).max() > 1e-4  # it moved


def test_contact_lanes(gpu):
    # a triangle's four lanes (small models) and its one (from 100,000 triangles on) give the
    # same responses: an env's contact on the positions as they are, alone and among its copies
    mesh = mg.ellipsoid_for_tets(16000, seed=6)
    out = []
    for copies in (1, 33):
        m, _ = sc.liver_model("cuda:0", copies, meshes=[mesh] * copies, substeps=1, iterations=1)
        m.constraintFlags = L.COLLIDE
        top = m.vertex[int(m.vertex[m.envSlice(0), 1].argmax())]  # the jaws' tips onto the surface
        m.moveTool((top - m.laparoscopeTip[0]).repeat(copies, 1))
        SimIntegratorDO("cuda:0", batched=False).stepModel(m, 1)
        torch.cuda.synchronize()
        for e in {0, copies - 1}:
            out.append((int(m.laparoscopeInCollision[e]), m.vertex[m.envSlice(e)].cpu().numpy()))
    assert len(mesh["triangle"]) < 100000 < 33 * len(mesh["triangle"])
    assert out[0][0] > 0
    for n, x in out[1:]:
        assert n == out[0][0]
        # sums of a few responses in any order: a few roundings of the position
        np.testing.assert_allclose(x, out[0][1], rtol=0, atol=8 * np.finfo(np.float32).eps * np.abs(x).max())
