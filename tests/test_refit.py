"""The fused BVH refit (leaves of all envs, then one block per env climbing the tree in
shared memory) against the level-by-level refit, which follows the reference's launches:
the same boxes and traversal copies bit for bit, on trees of one leaf, trees that fill the
block's shared memory, trees that do not fit it or are numbered another way, for all envs
and for a list of them."""

import numpy as np
import pytest
import torch

from ffsrl import SimBVH, _lib as L, meshgen as mg, scenarios as sc
from ffsrl._lib import check, lib, ptr

pytestmark = pytest.mark.gpu


def _one_triangle():
    return mg.tiny_mesh([[0, 0, 0], [1, 0, 0], [0, 1, 0]], triangle=[[0, 1, 2]])


def _two_triangles():
    return mg.tiny_mesh([[0, 0, 0], [1, 0, 0], [0, 1, 0], [9, 0, 0], [10, 0, 0], [9, 1, 0]],
                        triangle=[[0, 1, 2], [3, 4, 5]])


def _boxes(bvh):
    torch.cuda.synchronize()
    return [t.cpu().numpy().copy() for t in (bvh.aabbMin, bvh.aabbMax, bvh.nodeBox, bvh.triPos)]


def _check(bvh, m):
    rng = torch.Generator(device="cuda:0").manual_seed(5)
    m.allVisPoint.add_(0.3 * torch.rand(m.allVisPoint.shape, generator=rng, device="cuda:0"))
    for t in (bvh.aabbMin, bvh.aabbMax, bvh.nodeBox, bvh.triPos):
        t.fill_(7.0)
    bvh.refitBVH(fused=False)
    want = _boxes(bvh)
    for t in (bvh.aabbMin, bvh.aabbMax, bvh.nodeBox, bvh.triPos):
        t.fill_(-7.0)
    bvh.refitBVH()
    for a, b in zip(_boxes(bvh), want):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))
    return want


@pytest.mark.parametrize("make,copies", [
    (_one_triangle, 1), (_two_triangles, 3), (mg.beam, 2),
    (lambda: mg.ellipsoid_for_tets(5000), 2), (mg.ellipsoid, 1),
    (lambda: mg.ellipsoid(h=0.4), 1),      # more nodes than a block's shared memory holds
    (lambda: mg.ellipsoid(), 153),         # more envs than SMs: half the shared memory each
    (mg.beam, 200)])
def test_fused_refit_equals_the_levels(gpu, make, copies):
    mesh = make()
    if len(mesh["tetrahedron"]):
        m, _ = sc.liver_model("cuda:0", copies, meshes=[mesh] * copies)
    else:
        from ffsrl import SimModelDO
        m = SimModelDO(mesh, copies, "cuda:0")
    bvh = SimBVH("cuda:0", m)
    want = _check(bvh, m)
    # a list of envs: only theirs are written
    ids = torch.tensor(sorted({0, copies - 1}), dtype=torch.int32, device="cuda:0")
    for t in (bvh.aabbMin, bvh.aabbMax, bvh.nodeBox, bvh.triPos):
        t.fill_(-7.0)
    import ctypes as C
    check(lib().ffsrl_bvh_refit_fused_envs(C.byref(bvh.desc), ptr(m.allVisPoint), ptr(m.allVisFace), ptr(ids),
                                           int(ids.numel()), None))
    got = _boxes(bvh)[0]
    n = bvh.numNodes
    for e in range(copies):
        a, b = got[e * n:(e + 1) * n], want[0][e * n:(e + 1) * n]
        assert np.array_equal(a, b) if e in (0, copies - 1) else np.all(a == -7.0)


def test_tree_numbered_another_way(gpu, tmp_path):
    # an empty leaf at node 1 moves every child pair to even numbers: refitted by levels
    m, _ = sc.liver_model("cuda:0", 2, meshes=[mg.beam()] * 2)
    t = dict(SimBVH("cuda:0", m).topologies[0])
    for k, v in (("left_node", -1), ("first_tri_id", 0), ("tri_count", 0), ("level", 1)):
        a = t[k].copy()
        if k == "left_node":
            a[a >= 0] += 1
        t[k] = np.insert(a, 1, v).astype(np.int32)
    for k in ("aabb_min", "aabb_max"):
        t[k] = np.insert(t[k], 1, 0.0, axis=0).astype(np.float32)
    path = str(tmp_path / "bvh.npz")
    np.savez(path, t["tri_id"], t["aabb_min"], t["aabb_max"], t["left_node"], t["first_tri_id"], t["tri_count"],
             t["level"])
    bvh = SimBVH("cuda:0", m, load=True, path=path)
    assert bvh.numNodes == len(t["level"])
    _check(bvh, m)
