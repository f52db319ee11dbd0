"""Envs stepped by a cluster of blocks: the same bits as one block gives them.

An env alone in a model is split over a cluster; among some hundred copies of itself it is
not (up to 7,000 vertices), or into fewer parts.  The fixed-point sums are exact, so the
split must not change a bit, whatever the constraint set, the arithmetic, the seams'
place, or the paths off the common one: terms too large for the 32-bit sums, tets without
a gradient, contacts on a seam."""

import numpy as np
import pytest
import torch

from ffsrl import SimIntegratorDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu

PBD = L.VOLUME | L.DISTANCE | L.DRAG | L.COLLIDE
XPBD = L.VOLUME_XPBD | L.DISTANCE_XPBD | L.DRAG | L.COLLIDE
NEO = L.VOLUME | L.DISTANCE | L.NEOHOOKEAN | L.DRAG | L.COLLIDE


def _step(mesh, copies, flags, arithmetic, steps, disturb):
    m, _ = sc.liver_model("cuda:0", copies, meshes=[mesh] * copies, substeps=3, iterations=5)
    m.constraintFlags = flags
    rng = np.random.Generator(np.random.PCG64(3))
    nv = len(mesh["vertex"])
    x = mesh["vertex"] + rng.normal(scale=0.02, size=(nv, 3)).astype(np.float32)
    free = np.nonzero(mesh["inverse_mass"] > 0)[0]
    m.graspNearest(torch.ones(copies, dtype=torch.int32, device="cuda:0"), radius=1.0)
    integ = SimIntegratorDO("cuda:0", arithmetic=arithmetic)
    integ.plan(m)
    if disturb:
        x[free[len(free) // 2]] += 60.0                        # terms beyond the 32-bit sums
        t = mesh["tetrahedron"][len(mesh["tetrahedron"]) // 3]
        x[t] = x[t[0]]                                          # a tet without a gradient
    m.vertex.copy_(torch.as_tensor(np.tile(x, (copies, 1))))
    integ.stepModel(m, steps)
    torch.cuda.synchronize()
    e = m.envSlice(copies - 1)
    return {"vertex": m.vertex[e].cpu().numpy(), "velocity": m.velocity[e].cpu().numpy(),
            "contacts": int(m.laparoscopeInCollision[copies - 1]), "status": integ.envStatus(m).tolist()}


# tet counts on both sides of two 100-tet parts, ragged middle sizes, one that fills 16
# parts, one too large for a block; the last two constraint sets leave more edges unfolded
@pytest.mark.parametrize("tets", [100, 205, 1000, 4321, 19000, 46640])
@pytest.mark.parametrize("flags,arithmetic", [(NEO, "reference"), (NEO, "fast"), (PBD, "reference"), (XPBD, "fast")])
@pytest.mark.parametrize("disturb", [False, True])
def test_split_env_gives_the_undivided_env_s_bits(gpu, tets, flags, arithmetic, disturb):
    mesh = mg.ellipsoid() if tets == 46640 else mg.ellipsoid_for_tets(tets, seed=1)
    steps = 1 if disturb else 2
    alone = _step(mesh, 1, flags, arithmetic, steps, disturb)
    many = _step(mesh, 40 if tets == 46640 else 320, flags, arithmetic, steps, disturb)
    assert np.isfinite(alone["vertex"]).all() and alone["status"] == [0]
    assert np.array_equal(alone["vertex"], many["vertex"])
    assert np.array_equal(alone["velocity"], many["velocity"])
    assert alone["contacts"] == many["contacts"]
    if not disturb:
        assert alone["contacts"] > 0  # the instrument is pressed into the surface


def test_autotuned_split_plan(gpu, tmp_path, monkeypatch):
    # the autotuner's block sizes on a split class: the same bits; its cache is read back
    monkeypatch.setenv("FFSRL_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    mesh = mg.ellipsoid_for_tets(3000, seed=2)
    out = []
    for tune in (False, True, True):
        m, _ = sc.liver_model("cuda:0", 2, meshes=[mesh] * 2)
        integ = SimIntegratorDO("cuda:0", autotune=tune)
        integ.stepModel(m)
        torch.cuda.synchronize()
        out.append(m.vertex.cpu().numpy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("arithmetic", ["reference", "fast"])
def test_classes_of_a_step_in_turn(gpu, arithmetic):
    # each class's kernel waits for the one ahead to have begun: a class left out breaks no
    # chain, a captured step keeps it, and the envs' bits do not depend on it
    sizes = (12000, 6000, 2500, 300)
    meshes = [mg.ellipsoid_for_tets(t, seed=4) for t in sizes]

    def fresh():
        m, _ = sc.liver_model("cuda:0", len(sizes), meshes=meshes)
        return m, SimIntegratorDO("cuda:0", arithmetic=arithmetic).plan(m)

    m, plan = fresh()
    rest = m.vertex.clone()
    assert plan.info()["num_classes"] > 2
    for _ in range(3):
        plan.step(1)
    torch.cuda.synchronize()
    want = m.vertex.clone()
    m, plan = fresh()
    for _ in range(3):
        plan.step_envs([0, 2])
    torch.cuda.synchronize()
    for e in range(len(sizes)):
        s = m.envSlice(e)
        assert torch.equal(m.vertex[s], (want if e in (0, 2) else rest)[s])
    m, plan = fresh()
    plan.step(1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.step(1)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(m.vertex, want)
