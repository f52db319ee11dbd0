"""The ray-cast by tiles (images above 64 pixels, as their sizes and lenses decide)
against the reference-shaped renderer, which traverses every ray: the same depth bit for bit
from each of its three kernels -- tiles of 16 (many pixels), tiles of 8, and tiles of 8 with
two warps a patch (few pixels) -- for every kind of camera, where a tile has more triangles
than its list (quarters, rays traversed one by one), behind narrow lenses, where triangles
are hit at the same distance, where leaves box another face than the one they hold, on
triangles seen edge on, with vertices that are no numbers or overflow in products, without the arrays that the ray-cast can do without, and on a tree
deeper than the traversal's stack."""

import ctypes as C

import numpy as np
import pytest
import torch

import test_render_overflow
from ffsrl import SimBVH, SimModelDO, WarpRaycastRendererDO, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu

_MESHES = {}


def _kernel(bvh, envs, res, fov=21.73):
    """The kernel that images of this size take (the rule of the dispatch)."""
    lens = np.tan(np.radians(fov) / 2.0)
    pixels = (res / lens) ** 2  # of a unit angle's square
    work, dense = envs * pixels, bvh.desc.total_env_nodes / bvh.desc.num_envs / pixels
    tiles = envs * (-(-res // 16)) ** 2
    if work >= 2.4e6:
        t16 = dense < 0.64 and tiles >= 600
    elif work >= 1.2e6:
        t16 = dense < 0.32 and tiles >= 1024
    else:
        t16 = lens > 0.75 and (dense < 0.16 if work >= 8e5 else work >= 4e5 and dense < 0.02)
    if lens > 0.75:
        t8x2, t8 = work < 1e5 and dense < 0.08, False
    else:
        t8x2 = (work < 2e5 and dense < 0.16) or (work < 1e5 and dense < 0.32)
        t8 = dense < 0.16
    return "rays" if res <= 64 else "16" if t16 else "8x2" if t8x2 else "8" if t8 else "rays"


def _mesh(kind):
    if kind not in _MESHES:
        if kind == "dense":
            m = mg.ellipsoid()
        elif kind == "textured":
            m = mg.add_texture(mg.ellipsoid_for_tets(1500), size=64, seed=1)
        else:
            m = mg.beam(jitter=0.0) if kind == "beam" else mg.ellipsoid_for_tets(1500)
            lo, hi = m["vertex"].min(axis=0) - 2.0, m["vertex"].max(axis=0) + 2.0
            m = mg.with_rigids(m, [mg.rigid_box([lo[0], lo[1] - 0.5, lo[2]], [hi[0], lo[1], hi[2]])])
        _MESHES[kind] = m
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


def _compare(m, bvh, meshes, envs, res, camera, mode, seed):
    ap = sc.fov_aperture(60.0)
    out = []
    for fused in (False, True):
        r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", verticalAperture=ap,
                                  horizontalAperture=ap, fused=fused, render_mode=mode)
        r.setCameras(*_camera(camera, meshes, seed=seed))
        r.depth.fill_(-1.0)
        r.pixels.fill_(-1.0)
        r.renderNew(bvh, m)
        torch.cuda.synchronize()
        r.checkErrors()
        out.append(r)
    a, b = (r.depthImages().cpu().numpy() for r in out)
    assert np.array_equal(a, b), f"{(a != b).sum()} of {a.size} depths differ"
    assert camera == "away" or (a > 0.0).any()
    # (the two sum the vertex normals in different orders)
    np.testing.assert_allclose(out[1].pixels.cpu().numpy(), out[0].pixels.cpu().numpy(), atol=2e-4)
    # a list of envs writes theirs alone
    r = out[1]
    ids = torch.tensor([envs - 1], dtype=torch.int32, device="cuda:0")
    r.depth.fill_(-1.0)
    L.check(L.lib().ffsrl_render_fused_envs(C.byref(r._desc(m)), C.byref(bvh.desc), L.ptr(ids), 1, None))
    got = r.depthImages().cpu().numpy()
    np.testing.assert_array_equal(got[envs - 1], b[envs - 1])
    assert envs == 1 or (got[:envs - 1] == -1.0).all()


@pytest.mark.parametrize("kernel,kind,envs,res,camera,mode", [
    ("8x2", "plain", 1, 70, "out", 1), ("8x2", "plain", 2, 101, "axis", 4), ("8x2", "beam", 1, 128, "axis", 4),
    ("8x2", "dense", 1, 128, "out", 4), ("8x2", "plain", 2, 96, "inside", 4), ("8x2", "plain", 1, 80, "away", 4),
    ("8x2", "plain", 2, 88, "scaled", 2), ("8x2", "dense", 1, 150, "near", 3), ("8x2", "textured", 1, 128, "near", 1),
    ("8", "plain", 1, 300, "out", 3), ("8", "beam", 2, 220, "axis", 4), ("8", "dense", 3, 260, "out", 4),
    ("8", "plain", 2, 192, "inside", 4), ("8", "plain", 2, 205, "away", 4), ("8", "plain", 3, 161, "scaled", 4),
    ("8", "dense", 1, 300, "near", 0), ("8", "textured", 2, 200, "out", 1),
    ("16", "plain", 1, 700, "out", 1), ("16", "plain", 30, 128, "out", 3), ("16", "beam", 30, 125, "axis", 4),
    ("16", "dense", 2, 515, "near", 4), ("16", "dense", 100, 90, "out", 4), ("16", "plain", 2, 515, "inside", 4),
    ("16", "plain", 4, 320, "away", 4), ("16", "plain", 4, 325, "scaled", 4), ("16", "textured", 2, 512, "near", 1)])
def test_each_kernel(gpu, kernel, kind, envs, res, camera, mode):
    meshes = [_mesh(kind)] * envs
    m, _ = sc.liver_model("cuda:0", envs, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    assert _kernel(bvh, envs, res, 60.0) == kernel
    _compare(m, bvh, meshes, envs, res, camera, mode, res)


def _triangles(v, envs=1):
    """A model of separate triangles v [n, 3, 3] and its BVH."""
    mesh = mg.tiny_mesh(np.asarray(v, np.float32).reshape(-1, 3), triangle=np.arange(3 * len(v)).reshape(-1, 3))
    m = SimModelDO(mesh, envs, "cuda:0")
    return m, SimBVH("cuda:0", m)


def _differ(m, bvh, res, fov, pos, rot, mode):
    """Pixels whose depth or colour the two renderers give differently, and pixels with a hit
    (no two triangles share a point, so that no normal is a sum)."""
    images = []
    for fused in (False, True):
        r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", verticalAperture=sc.fov_aperture(fov),
                                  horizontalAperture=sc.fov_aperture(fov), fused=fused, render_mode=mode)
        r.setCameras(pos, rot)
        r.renderNew(bvh, m)
        torch.cuda.synchronize()
        r.checkErrors()
        images.append(torch.cat([r.pixels, r.depth[:, None]], dim=1).cpu().numpy())
    return int((images[0] != images[1]).any(axis=1).sum()), int((images[0][:, 3] > 0.0).sum())


@pytest.mark.parametrize("kernel,fov,res", [("8x2", 20.0, 70), ("8", 0.2, 128), ("8", 0.2, 256), ("16", 0.5, 480), ("16", 0.5, 1024),
                                            ("16", 1.0, 1024), ("16", 2.0, 1024), ("16", 5.0, 1024)])
@pytest.mark.parametrize("size", [1.0, 1.1])
def test_narrow_lenses(gpu, kernel, fov, res, size):
    # the sides of a tile are as little as some 1e-4 radians apart: triangles of a few rays'
    # width, so that many reach just across a side.  (Below 1e-2 a side a triangle's determinant
    # is under the test's limit, whatever the ray.)  size: of the camera's quaternion
    for seed in range(4):
        rng = np.random.Generator(np.random.PCG64(seed))
        n, t = max(300, int(4e-3 * res * res)), np.tan(np.radians(fov) / 2.0)
        width = np.exp(rng.uniform(np.log(2.0), np.log(12.0), n)) * t / res
        far = np.maximum(20.0, 0.03 / width) * rng.uniform(1.0, 3.0, n)
        d = np.stack([rng.uniform(-t, t, n), rng.uniform(-t, t, n), np.full(n, -1.0)], axis=1) * far[:, None]
        q = rng.normal(size=4)
        q *= size / np.linalg.norm(q)
        u, w = q[:3], q[3]
        c = d * (2.0 * w * w - 1.0) + 2.0 * (d @ u)[:, None] * u + 2.0 * w * np.cross(u, d)
        m, bvh = _triangles(c[:, None, :] + rng.normal(size=(n, 3, 3)) * (width * far)[:, None, None])
        assert _kernel(bvh, 1, res, fov) == kernel
        differ, hit = _differ(m, bvh, res, fov, np.zeros((1, 3)), q[None], 2)
        assert differ == 0 and hit > 300, f"seed {seed}: {differ} pixels differ, {hit} are hit"


@pytest.mark.parametrize("kernel,res", [("8x2", 128), ("8", 300), ("16", 700)])
def test_equally_near_triangles(gpu, kernel, res):
    # plates in coordinate planes, on a coarse grid: many rays hit two of them at the same
    # distance, which is that of their boxes, too; the normals tell which one was kept
    for seed in range(6):
        rng = np.random.Generator(np.random.PCG64(seed))
        v = []
        for _ in range(600):
            c = np.array([*(rng.integers(-12, 13, 2) / 2.0), rng.integers(-30, -9)])
            across = rng.permutation(3)[:2]
            b, d = c.copy(), c.copy()
            b[across[0]] += rng.choice([0.5, 1.0, 2.0]) * rng.choice([-1, 1])
            d[across[1]] += rng.choice([0.5, 1.0, 2.0]) * rng.choice([-1, 1])
            v.append([c, b, d])
        m, bvh = _triangles(v)
        assert _kernel(bvh, 1, res, 60.0) == kernel
        differ, hit = _differ(m, bvh, res, 60.0, np.zeros((1, 3)), np.array([[0.0, 0.0, 0.0, 1.0]]), 2)
        assert differ == 0 and hit > 1000, f"seed {seed}: {differ} pixels differ, {hit} are hit"


@pytest.mark.parametrize("kernel,envs,res", [("8x2", 2, 128), ("8", 3, 160), ("16", 40, 128)])
@pytest.mark.parametrize("foreign", [0.02, 0.5])
def test_leaves_that_box_another_face(gpu, kernel, envs, res, foreign):
    # refit_source: a leaf's box is another face's, nearer or farther than what it holds
    meshes = [_mesh("plain")] * envs
    m, _ = sc.liver_model("cuda:0", envs, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    assert _kernel(bvh, envs, res, 60.0) == kernel
    rng = np.random.Generator(np.random.PCG64(envs))
    n = m.numAllVisFaces
    src = np.arange(n, dtype=np.int32)
    pick = rng.random(n) < foreign
    src[pick] = rng.integers(0, n, size=int(pick.sum()))
    bvh.refitSource = torch.as_tensor(src, device="cuda:0")
    bvh.desc.refit_source = L.ptr(bvh.refitSource)
    bvh.refitBVH()
    for seed in range(4):
        _compare(m, bvh, meshes, envs, res, "out", 4, seed)


@pytest.mark.parametrize("kernel,res", [("8x2", 80), ("8", 256), ("16", 512)])
@pytest.mark.parametrize("depth", [1.0, 5.0])
def test_grazing_triangles(gpu, kernel, res, depth):
    # triangles that run along the rays: the test's determinant goes down to its limit, and the
    # distance it finds is off by up to some per cent, to both sides of the triangle's box
    for seed in range(6):
        rng = np.random.Generator(np.random.PCG64(seed))
        n = 1500
        a = np.concatenate([0.12 * rng.normal(size=(n, 2)), np.full((n, 1), -1.0)], axis=1) * rng.uniform(5.0, 40.0, (n, 1))
        u = a / np.linalg.norm(a, axis=1, keepdims=True)
        off = [u * rng.uniform(0.3, 1.0, (n, 1)) * depth * rng.choice([-1, 1], (n, 1)) +
               0.5 * rng.normal(size=(n, 3)) * np.exp(rng.uniform(-4.0, 0.0, (n, 1))) for _ in range(2)]
        m, bvh = _triangles(np.stack([a, a + off[0], a + off[1]], axis=1))
        assert _kernel(bvh, 1, res) == kernel
        differ, hit = _differ(m, bvh, res, 21.73, np.zeros((1, 3)), np.array([[0.0, 0.0, 0.0, 1.0]]), 2)
        assert differ == 0 and hit > 1000, f"seed {seed}: {differ} pixels differ, {hit} are hit"


@pytest.mark.parametrize("kernel,envs,res", [("8x2", 1, 100), ("8", 2, 205), ("16", 30, 128)])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf"), 1e15, -1e20, 1e25, 1e30, -1e35, -3e38])
def test_extreme_vertices(gpu, kernel, envs, res, value):
    mesh = mg.ellipsoid_for_tets(1500)
    for count in (1, 5, 200):
        m, _ = sc.liver_model("cuda:0", envs, meshes=[mesh] * envs)
        bvh = SimBVH("cuda:0", m)
        assert _kernel(bvh, envs, res, 60.0) == kernel
        rng = np.random.Generator(np.random.PCG64(count))
        m.allVisPoint.view(-1)[torch.as_tensor(rng.integers(0, m.allVisPoint.numel(), count), device="cuda:0")] = value
        bvh.refitBVH()
        images = []
        for fused in (False, True):
            r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", fused=fused, render_mode=4,
                                      verticalAperture=sc.fov_aperture(60.0), horizontalAperture=sc.fov_aperture(60.0))
            r.setCameras(*sc.env_cameras([mesh] * envs, seed=1))
            r.renderNew(bvh, m)
            torch.cuda.synchronize()
            images.append(r.depthImages().cpu().numpy().view(np.int32))
        assert np.array_equal(*images), f"{count}: {(images[0] != images[1]).sum()} depths differ"


@pytest.mark.parametrize("kernel,envs,res", [("8x2", 1, 80), ("8", 2, 100), ("16", 2, 400)])
@pytest.mark.parametrize("without", ["packed copies", "level lists"])
def test_optional_arrays_left_out(gpu, kernel, envs, res, without):
    meshes = [_mesh("plain")] * envs
    m, _ = sc.liver_model("cuda:0", envs, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    assert _kernel(bvh, envs, res) == kernel
    r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless")
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


@pytest.mark.parametrize("kernel,envs,res", [("8x2", 1, 80), ("8", 2, 180), ("16", 2, 400)])
def test_depth_equals_the_oracle_s(gpu, oracle_lib, kernel, envs, res):
    meshes = [_mesh("plain")] * envs
    m, _ = sc.liver_model("cuda:0", envs, meshes=meshes)
    bvh = SimBVH("cuda:0", m)
    assert _kernel(bvh, envs, res) == kernel
    r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", render_mode=3)
    r.setCameras(*_camera("out", meshes, seed=7))
    r.renderNew(bvh, m)
    torch.cuda.synchronize()
    color, depth, _ = oracle_lib.render(r, bvh, m.allVisPoint.cpu().numpy())
    np.testing.assert_array_equal(r.depthImages().cpu().numpy(), depth)
    np.testing.assert_allclose(r.pixels.view(color.shape).cpu().numpy(), color, atol=2e-4)


@pytest.mark.parametrize("kernel,res", [("8x2", 80), ("8", 200), ("16", 512)])
def test_overflow_is_reported(gpu, kernel, res):
    m = test_render_overflow._model("cuda:0")
    bvh = SimBVH("cuda:0", m)
    assert _kernel(bvh, 1, res) == kernel
    r = WarpRaycastRendererDO("cuda:0", m, resolution=res, mode="headless", render_mode=4)
    r.setCameras(*test_render_overflow._camera())
    r.renderNew(bvh, m)
    torch.cuda.synchronize()
    with pytest.raises(L.FFSRLError) as e:
        r.checkErrors()
    assert e.value.code == L.ERR_STACK_OVERFLOW
