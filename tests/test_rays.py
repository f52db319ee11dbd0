"""The tiled ray-cast against the reference-shaped renderer, which traverses every ray in the
reference's order: the same depth bit for bit (no sum's order enters it) -- on ragged image
sizes, on both tile sizes, where a tile has more triangles than its list (quarters, and
rays traversed one by one), for cameras inside a mesh, along the axes, facing away and
with a quaternion that is no rotation, over axis-aligned planes, and for a list of envs."""

import ctypes as C

import numpy as np
import pytest
import torch

from ffsrl import SimBVH, WarpRaycastRendererDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu

_MESHES = {}


def _mesh(kind):
    if kind not in _MESHES:
        m = mg.ellipsoid() if kind == "dense" else mg.beam(jitter=0.0) if kind == "beam" else mg.ellipsoid_for_tets(1500)
        lo, hi = m["vertex"].min(axis=0) - 2.0, m["vertex"].max(axis=0) + 2.0
        box = mg.rigid_box([lo[0], lo[1] - 0.5, lo[2]], [hi[0], lo[1], hi[2]])
        _MESHES[kind] = mg.with_rigids(m, [box]) if kind != "dense" else m
    return _MESHES[kind]


def _camera(kind, meshes, seed):
    pos, rot = sc.env_cameras(meshes, seed=seed)
    c = np.stack([m["vertex"].mean(axis=0) for m in meshes])
    if kind == "inside":
        pos = c.astype(np.float32)
    elif kind == "away":
        pos = (2.0 * pos - c).astype(np.float32) + 40.0
    elif kind == "axis":  # straight along -z from a point level with the mesh's vertices
        pos = np.round(c).astype(np.float32) + np.float32([0.0, 0.0, 30.0])
        rot = np.tile(np.float32([0.0, 0.0, 0.0, 1.0]), (len(meshes), 1))
    elif kind == "scaled":
        rot = (rot * 1.1).astype(np.float32)
    elif kind == "near":
        pos = (c + 0.4 * (pos - c)).astype(np.float32)
    return pos, rot


@pytest.mark.parametrize("kind,envs,res,camera,mode", [
    ("plain", 1, 1, "out", 4), ("plain", 2, 7, "out", 3), ("plain", 1, 33, "out", 1), ("plain", 3, 50, "near", 0),
    ("plain", 1, 128, "out", 2), ("dense", 1, 8, "out", 4), ("dense", 2, 16, "out", 4), ("dense", 1, 128, "near", 3),
    ("beam", 2, 64, "axis", 3), ("plain", 2, 64, "axis", 4), ("plain", 2, 48, "inside", 4), ("plain", 2, 40, "away", 4),
    ("plain", 2, 40, "scaled", 4), ("plain", 70, 63, "out", 4), ("dense", 300, 17, "out", 4), ("beam", 18, 128, "axis", 4),
    # tiles of 8 whose patches have one warp each (more than 608, the cases above fewer)
    ("plain", 3, 128, "out", 4), ("dense", 10, 64, "near", 3), ("beam", 3, 125, "axis", 4)])
def test_tiles_give_the_traversal_s_depth(gpu, kind, envs, res, camera, mode):
    meshes = [_mesh(kind)] * envs
    m, _ = sc.liver_model("cuda:0", envs, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    ap = sc.fov_aperture(60.0)
    out = []
    for fused in (False, True):
        r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", verticalAperture=ap,
                                  horizontalAperture=ap, fused=fused, render_mode=mode)
        r.setCameras(*_camera(camera, meshes, seed=res))
        r.depth.fill_(-1.0)
        r.pixels.fill_(-1.0)
        r.renderNew(bvh, m)
        torch.cuda.synchronize()
        r.checkErrors()
        out.append(r)
    a, b = (r.depthImages().cpu().numpy() for r in out)
    np.testing.assert_array_equal(b, a)
    assert (a == 0.0).all() if camera == "away" else (a > 0.0).any()
    np.testing.assert_allclose(out[1].pixels.cpu().numpy(), out[0].pixels.cpu().numpy(), atol=2e-4)
    # a list of envs writes theirs alone
    r = out[1]
    want, ids = b.copy(), torch.tensor([envs - 1], dtype=torch.int32, device="cuda:0")
    r.depth.fill_(-1.0)
    L.check(L.lib().ffsrl_render_fused_envs(C.byref(r._desc(m)), C.byref(bvh.desc), L.ptr(ids), 1, None))
    got = r.depthImages().cpu().numpy()
    np.testing.assert_array_equal(got[envs - 1], want[envs - 1])
    assert envs == 1 or (got[:envs - 1] == -1.0).all()


@pytest.mark.parametrize("without", ["packed copies", "level lists"])
def test_optional_arrays_left_out(gpu, without):
    # the ray-cast needs neither the refit's packed copies (every ray is traversed) nor the
    # level lists (the walk starts at the root)
    meshes = [_mesh("plain")] * 2
    m, _ = sc.liver_model("cuda:0", 2, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    r = WarpRaycastRendererDO("cuda:0", m, resolution=40, mode="headless")
    r.setCameras(*_camera("out", meshes, seed=3))
    r.renderNew(bvh, m)
    want = r.depthImages().cpu().numpy().copy()
    if without == "packed copies":
        bvh.desc.node_box = bvh.desc.tri_pos = None
    else:
        bvh.desc.level_node = bvh.desc.level_start = bvh.desc.topo_level_offset = None
    r.depth.zero_()
    r.renderNew(bvh, m)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(r.depthImages().cpu().numpy(), want)
