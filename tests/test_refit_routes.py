"""Each route of the fused refit against the level-by-level refit, bit for bit: small trees (leaves
and climb in one launch), larger ones (a launch each), more envs than two an SM (leaves and
levels in one launch), trees too large for the shared memory they would share, trees of several
sizes in a model, and trees numbered another way on each route."""

import numpy as np
import pytest
import torch

from ffsrl import SimBVH, meshgen as mg, scenarios as sc
from test_refit import _check

pytestmark = pytest.mark.gpu


def _mesh(tets):
    return mg.beam() if tets == 0 else mg.ellipsoid() if tets == 46640 else mg.ellipsoid_for_tets(tets)


@pytest.mark.parametrize("tets,copies", [
    ([0], 1), ([0], 250), ([0], 310),              # small trees
    ([1500], 1), ([1500], 160), ([1500], 304), ([1500], 305), ([300, 5000, 1500], 9), ([300, 5000], 170),
    ([20000], 153), ([46640, 0], 3), ([46640, 0], 160)])
def test_each_route(gpu, tets, copies):
    pool = [_mesh(t) for t in tets]
    m, _ = sc.liver_model("cuda:0", copies, meshes=[pool[k % len(pool)] for k in range(copies)])
    _check(SimBVH("cuda:0", m), m)


@pytest.mark.parametrize("tets,copies", [(0, 2), (0, 310), (1500, 2)])
def test_tree_numbered_another_way(gpu, tmp_path, tets, copies):
    # an empty leaf at node 1 moves every child pair to even numbers
    m, _ = sc.liver_model("cuda:0", copies, meshes=[_mesh(tets)] * copies)
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
    _check(SimBVH("cuda:0", m, load=True, path=path), m)
