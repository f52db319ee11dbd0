"""The work that programs have this framework do, as cases that can be timed and compared.

Three paths, each through the package's public classes:

* ``step``    -- ``SimIntegratorDO.stepModel``: one env-step of every environment from a
  saved state (a rollout that is branched or replayed from it), in the batched form with
  either arithmetic or in the reference-shaped form;
* ``observe`` -- ``SimBVH.refitBVH`` and ``WarpRaycastRendererDO.renderNew``: the images of
  the environments' current state;
* ``rl``      -- a whole RL step (effector action, env-step, refit, images) recorded once as
  a CUDA graph and replayed, as a training loop runs it.

Meshes are the seeded generators' (``ffsrl.meshgen``): the beam of 800 tets, the
12/8/6 cm ellipsoid of 46,640 tets, and ellipsoids of 500 to 20,000 tets spread evenly
over the logarithm.  A state is a mid-episode one: the mesh deformed by a few
millimetres and moving at a few centimetres per second, the instrument pressed into
the surface and holding a vertex.  The seed draws the deformation, the velocities, the
instrument's place, the cameras and which environment has which mesh.
"""

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ff-srl_gb300"))

from ffsrl import SimBVH, SimIntegratorDO, WarpRaycastRendererDO, _lib as L, meshgen as mg, scenarios as sc  # noqa: E402
from ffsrl.graphs import Graph  # noqa: E402

DEVICE = "cuda:0"
SHADINGS = {"grayscale": 0, "texture": 1, "normal": 2, "vertex_color": 3, "depth": 4}


def listed():
    return [
        # the smallest simulation there is: one beam, volume and distance constraints, the
        # default arithmetic -- a latency-bound call
        _step("beam_1", "beam", 1, "pbd"),
        # compliant beams, a small parameter sweep
        _step("beam_xpbd_64", "beam", 64, "xpbd"),
        # one organ at full resolution, stepped interactively or in an evaluation
        _step("liver_1", "ellipsoid", 1, "neo", tets=46640),
        # a few of them side by side, with the fast arithmetic
        _step("liver_fast_16", "ellipsoid", 16, "neo", tets=46640, arithmetic="fast"),
        # a small training batch of mixed meshes, default arithmetic
        _step("mixed_64", "mixed", 64, "neo", lo=500, hi=20000, pool=16),
        # training batches that fill the GPU, both arithmetics
        _step("mixed_512", "mixed", 512, "neo", lo=500, hi=20000, pool=32),
        _step("mixed_fast_512", "mixed", 512, "neo", lo=500, hi=20000, pool=32, arithmetic="fast"),
        # the reference-shaped step (one launch per reference kernel), as a user runs it
        # who wants the reference's own launch structure
        _step("plain_16", "mixed", 16, "neo", lo=500, hi=20000, pool=16, form="plain"),
        # one environment's image: the latency of an observation
        _observe("observe_1", 1, 5000, 5000, 1, 128, "vertex_color"),
        # the images of a training batch
        _observe("observe_256", 256, 500, 20000, 32, 128, "vertex_color"),
        # large textured images with a rigid table under the organ (the renderer's default
        # resolution and shading), for display or video
        _observe("observe_texture_8", 8, 2000, 20000, 4, 512, "texture", rigid=True),
        # a training loop's whole step
        {"name": "rl_256", "path": "rl", "envs": 256, "lo": 500, "hi": 20000, "pool": 32, "resolution": 128,
         "shading": "vertex_color", "arithmetic": "fast", "substeps": 8, "iterations": 10},
    ]


def _step(name, scene, envs, material, tets=800, lo=0, hi=0, pool=1, arithmetic="reference", form="batched",
          substeps=8, iterations=10):
    return {"name": name, "path": "step", "scene": scene, "envs": envs, "material": material, "tets": tets, "lo": lo,
            "hi": hi, "pool": pool, "arithmetic": arithmetic, "form": form, "substeps": substeps,
            "iterations": iterations}


def _observe(name, envs, lo, hi, pool, resolution, shading, rigid=False):
    return {"name": name, "path": "observe", "envs": envs, "lo": lo, "hi": hi, "pool": pool, "resolution": resolution,
            "shading": shading, "rigid": rigid}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "uniform", "mixed", "mixed", "plain", "observe", "observe", "rl"])
    arithmetic = rng.choice(["reference", "fast"])
    substeps, iterations = rng.choice([(8, 10), (8, 10), (8, 1), (4, 20), (16, 5)])
    if kind in ("one", "uniform"):
        tets = _log(rng, 100, 46640)
        envs = 1 if kind == "one" else max(2, min(512, _log(rng, 2, 500000 // tets + 2)))
        material = rng.choice(["neo", "neo", "neo", "pbd", "xpbd"])
        c = _step("", "ellipsoid", envs, material, tets=tets, arithmetic=arithmetic, substeps=substeps,
                  iterations=iterations)
    elif kind == "mixed":
        c = _step("", "mixed", _log(rng, 3, 480), "neo", lo=500, hi=_log(rng, 2000, 20000), pool=rng.randint(3, 24),
                  arithmetic=arithmetic, substeps=substeps, iterations=iterations)
    elif kind == "plain":
        c = _step("", "mixed", _log(rng, 1, 24), rng.choice(["neo", "pbd"]), lo=500, hi=20000, pool=rng.randint(1, 12),
                  form="plain", iterations=rng.choice([1, 5, 10]))
    elif kind == "observe":
        res = rng.choice([16, 50, 64, 100, 128, 128, 200, 256, 512])
        envs = max(1, min(300, _log(rng, 1, 4000000 // (res * res))))
        shading = rng.choice(["texture", "texture", "vertex_color", "grayscale", "normal", "depth"])
        hi = _log(rng, 600, 46640) if envs < 8 else _log(rng, 600, 20000)
        c = _observe("", envs, 500, hi, rng.randint(1, 16), res, shading, rigid=rng.random() < 0.5)
    else:
        c = {"name": "", "path": "rl", "envs": _log(rng, 2, 240), "lo": 500, "hi": _log(rng, 1000, 20000),
             "pool": rng.randint(1, 16), "resolution": rng.choice([64, 100, 128]), "shading": "vertex_color",
             "arithmetic": arithmetic, "substeps": 8, "iterations": 10}
    del c["name"]
    return c


# ------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _mesh(scene, tets, seed, texture=False, rigid=False):
    if scene == "beam":
        m = mg.beam(jitter=0.0)
    elif tets >= 46640:
        m = mg.ellipsoid(seed=seed)
    else:
        m = mg.ellipsoid_for_tets(tets, seed=seed)
    if texture:
        m = mg.add_texture(m, size=256, seed=seed)
    if rigid:
        lo, hi = m["vertex"].min(axis=0) - 2.0, m["vertex"].max(axis=0) + 2.0
        m = mg.with_rigids(m, [mg.rigid_box([lo[0], lo[1] - 0.5, lo[2]], [hi[0], lo[1], hi[2]])])
    return m


def _pool(case):
    """The case's distinct meshes: tet counts at the middles of ``pool`` equal parts of
    log [lo, hi], so that every seed has the same amount of work."""
    if case["path"] == "step" and case["scene"] != "mixed":
        return [_mesh(case["scene"], case["tets"], 0)]
    n, lo, hi = case["pool"], case["lo"], case["hi"]
    texture, rigid = case.get("shading") == "texture", bool(case.get("rigid", False))
    return [_mesh("ellipsoid", int(round(lo * (hi / lo) ** ((k + 0.5) / n))), k, texture, rigid) for k in range(n)]


def _env_meshes(case, rng):
    pool = _pool(case)
    return [pool[k % len(pool)] for k in rng.permutation(case["envs"])]


def _moving_state(model, meshes, rng):
    """Smoothly deformed positions (a few mm, fixed vertices in place) with a little noise,
    and smooth velocities of a few cm/s, as float32 arrays over all environments."""
    xs, vs = [], []
    for m in meshes:
        p = m["vertex"].astype(np.float64)
        free = (m["inverse_mass"] > 0)[:, None]
        k = rng.uniform(-0.5, 0.5, size=(2, 3, 3))
        ph = rng.uniform(0.0, 2.0 * math.pi, size=(2, 3))
        wave = [np.sin(p @ k[i].T + ph[i]) for i in range(2)]
        d = 0.2 * wave[0] + rng.normal(scale=0.01, size=p.shape)
        xs.append(p + d * free)
        vs.append(3.0 * wave[1] * free)
    x = torch.as_tensor(np.concatenate(xs).astype(np.float32), device=model.device)
    v = torch.as_tensor(np.concatenate(vs).astype(np.float32), device=model.device)
    return x, v


def _model(case, rng):
    """The model in its mid-episode state, its meshes, that state, and (for the paths that
    make images) the BVH a program builds once, at rest."""
    meshes = _env_meshes(case, rng)
    if case["path"] == "step" and case["material"] != "neo":
        m, _ = sc.beam_model(DEVICE, case["envs"], xpbd=case["material"] == "xpbd", mesh=meshes[0]) \
            if case["scene"] == "beam" else _pbd_model(case, meshes)
        m.simSubsteps, m.simConstraints = case["substeps"], case["iterations"]
        m.simDt = (1.0 / m.simFrameRate) / m.simSubsteps
    else:
        m, _ = sc.liver_model(DEVICE, case["envs"], meshes=meshes, substeps=case.get("substeps", 8),
                              iterations=case.get("iterations", 10))
    bvh = SimBVH(DEVICE, m) if case["path"] != "step" else None
    if m.hasInstrumentKinematics:
        shift = rng.uniform(-0.2, 0.2, size=(case["envs"], 3)) * np.array([1.0, 0.5, 1.0])
        m.moveTool(torch.as_tensor(shift.astype(np.float32), device=m.device))
        m.setEffectorInitialPosition()
    x, v = _moving_state(m, meshes, rng)
    m.vertex.copy_(x)
    m.velocity.copy_(v)
    m.initialVertex.copy_(x)
    if m.constraintFlags & L.DRAG and case["path"] != "observe":
        m.graspNearest(torch.ones(case["envs"], dtype=torch.int32, device=m.device), radius=0.8)
    m.transformSimMeshData()
    m.transformSimLaparoscopeMeshData()
    return m, meshes, x, v, bvh


def _pbd_model(case, meshes):
    flags = L.REFERENCE_STEP
    if case["material"] == "xpbd":
        flags = (flags & ~(L.DISTANCE | L.VOLUME)) | L.DISTANCE_XPBD | L.VOLUME_XPBD
    m, _ = sc.liver_model(DEVICE, case["envs"], meshes=meshes, distanceCompliance=1e-6, volumeComplianceXPBD=0.0)
    m.constraintFlags = flags
    return m, meshes


def _renderer(case, m, meshes, rng):
    ap = sc.fov_aperture(60.0)
    r = WarpRaycastRendererDO(DEVICE, m, resolution=case["resolution"], mode="headless", verticalAperture=ap,
                              horizontalAperture=ap, lightPos=(0.3, 1.0, 0.5), lightIntensity=0.8,
                              render_mode=SHADINGS[case["shading"]])
    pos, rot = sc.env_cameras(meshes, seed=int(rng.integers(1 << 30)))
    r.setCameras(pos, rot)
    return r


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    m, meshes, x, v, bvh = _model(case, rng)
    s = {"case": case, "model": m, "x": x, "v": v, "bvh": bvh}
    if case["path"] != "observe":
        batched = case.get("form", "batched") == "batched"
        s["integrator"] = SimIntegratorDO(DEVICE, batched=batched, arithmetic=case["arithmetic"] if batched else "reference")
        if batched:
            s["integrator"].plan(m)
    if case["path"] != "step":
        s["renderer"] = _renderer(case, m, meshes, rng)
    if case["path"] == "rl":
        d = rng.normal(size=(case["envs"], 3))
        d *= 0.05 / np.linalg.norm(d, axis=1, keepdims=True)
        s["action"] = torch.as_tensor(d.astype(np.float32), device=DEVICE)
        s["graph"] = Graph(lambda: _rl_step(s), prepare=lambda: s["renderer"]._desc(m))
    return s


# ---------------------------------------------------------------------------- one pass
def _restore(s):
    s["model"].vertex.copy_(s["x"])
    s["model"].velocity.copy_(s["v"])
    s["model"].resetCollisionInfo()


def _rl_step(s):
    m = s["model"]
    _restore(s)
    m.laparoscopeXForm.copy_(m.laparoscopeInitialXForm)
    m.applyCartesianActionsInWorkspace(s["action"])
    s["integrator"].stepModel(m)
    s["bvh"].refitBVH()
    s["renderer"].renderNew(s["bvh"], m)


def run(s):
    m, path = s["model"], s["case"]["path"]
    if path == "step":
        _restore(s)
        s["integrator"].stepModel(m)
        out = {"vertex": m.vertex, "velocity": m.velocity, "points": m.allVisPoint}
        if s["case"]["form"] == "batched":
            # the reference-shaped form's float atomics add in another order each time, which
            # can turn a touching triangle's contact on or off
            out["contacts"] = m.laparoscopeInCollision
        return out
    if path == "observe":
        s["bvh"].refitBVH()
        pixels = s["renderer"].renderNew(s["bvh"], m)
        return {"pixels": pixels, "depth": s["renderer"].depthImages(), "box_low": s["bvh"].aabbMin,
                "box_high": s["bvh"].aabbMax}
    s["graph"]()
    return {"vertex": m.vertex, "velocity": m.velocity, "effector": m.getLaparoscopePositionsTensor(),
            "contacts": m.laparoscopeInCollision, "pixels": s["renderer"].pixels, "depth": s["renderer"].depth}


def work(case):
    pool = _pool(case)
    V = E = T = F = P = 0.0
    for m in pool:
        V += len(m["vertex"])
        E += len(m["edge"])
        T += len(m["tetrahedron"])
        F += len(m["triangle"])
        P += len(m["point_to_vertex"])
    k = case["envs"] / len(pool)
    V, E, T, F, P = V * k, E * k, T * k, F * k, P * k
    nbytes = flops = 0.0
    if case["path"] != "observe":
        neo = case.get("material", "neo") == "neo"
        # state in and out, constraint tables once
        nbytes += V * (24 + 4 + 24) + E * 12 + T * (20 + (36 if neo else 0)) + F * 12 + P * 12
        flops += case["substeps"] * (case["iterations"] * (T * (130 + (260 if neo else 0)) + E * 35 + V * 9 + F * 6) + V * 25)
    if case["path"] != "step":
        rays = 4.0 * case["resolution"] ** 2 * case["envs"]
        # points, faces and normals once, the boxes of a binary tree of half the faces, the
        # images; a ray's direction, the path down to one leaf, one hit and its shading
        nbytes += P * 36 + F * (12 + 24) + rays / 4 * 16
        flops += F * 30 + rays * (60 + 25 * math.log2(max(2.0, F / case["envs"])) + 100)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------- the same in 64 bits (torch)
EPS = 2.220446049250313e-16
MOST_PAIRS = 3.0e10  # ray-triangle pairs a 64-bit image is made for


def exact(case, seed):
    if case["path"] == "rl":
        return None  # its two halves have values of their own in the other cases
    rng = np.random.Generator(np.random.PCG64(int(seed)))
    if case["path"] == "observe":
        meshes = _env_meshes(case, np.random.Generator(np.random.PCG64(int(seed))))
        faces = sum(len(m["vis_face"]) for m in meshes) + 500 * len(meshes)
        if 4.0 * case["resolution"] ** 2 * faces > MOST_PAIRS:
            return None
        m, meshes, _, _, _ = _model(case, rng)
        r = _renderer(case, m, meshes, rng)
        pixels, depth = _images64(case, m, r)
        return {"pixels": pixels, "depth": depth, "box_low": None, "box_high": None}
    m, _, x, v, _ = _model(case, rng)
    x, v = _step64(m, x.double(), v.double())
    points = m.allVisPoint.double().clone()
    map_ = m.pointToVertex.long().view(-1, 2)
    points[map_[:, 0]] = x[map_[:, 1]]
    out = {"vertex": x, "velocity": v, "points": points}
    if case["form"] == "batched":
        out["contacts"] = None
    return out


def _dot(a, b):
    return (a * b).sum(dim=-1, keepdim=True)


def _unit(a):
    n = a.norm(dim=-1, keepdim=True)
    return torch.where(n > 0, a / n.clamp_min(1e-300), torch.zeros_like(a))


def _f32(v):
    return float(np.float32(v))


def _step64(m, x, v):
    fl = m.constraintFlags
    inv = m.inverseMass.double().unsqueeze(1)
    tet = m.tetrahedron.long().view(-1, 4)
    edge = m.edge.long().view(-1, 2)
    rest = m.tetrahedronRestVolume.double().unsqueeze(1)
    signed = m.tetrahedronRestVolumeSigned.double().unsqueeze(1)
    D = m.tetrahedronDmInv.double().view(-1, 3, 3)
    L0 = m.edgeRestLength.double().unsqueeze(1)
    tri, env = m.triangle.long().view(-1, 3), m.triToEnv.long()
    drag = m.activeDragConstraint.double().unsqueeze(1)
    base, tip, rad = m.laparoscopeBase.double(), m.laparoscopeTip.double(), m.laparoscopeRadius.double()
    dt = _f32(m.simDt)
    g = torch.tensor([_f32(c) for c in m.gravity], dtype=torch.float64, device=x.device)
    damp = 1.0 - _f32(m.velocityDampening)
    volc, devc = _f32(m.globalVolumeComplianceNeoHookean), _f32(m.gloabalDeviatoricComplianceNeoHookean)
    a_dist = _f32(_f32(m.distanceComplianceXPBD) / (dt * dt))
    a_vol = _f32(_f32(m.volumeComplianceXPBD) / (dt * dt))
    mt, me = inv[tet], inv[edge]                    # [T, 4, 1], [E, 2, 1]
    grasp = 0.5 * _f32(m.globalKsDrag) * drag
    grasp_at = tip.view(-1, 4, 3)[:, 2][m.vertexToEnv.long()]
    for _ in range(m.simSubsteps):
        vel = torch.where(inv < EPS, torch.zeros_like(v), v + g * inv * dt * damp)
        xp = x + vel * dt
        lam_t, lam_e = torch.zeros_like(rest), torch.zeros_like(L0)
        for _ in range(m.simConstraints):
            dp = torch.zeros_like(xp)
            n = torch.zeros_like(inv)

            def add(ids, d, on):
                for k in range(ids.shape[1]):
                    dp.index_add_(0, ids[:, k], torch.where(on, d[:, k], torch.zeros_like(d[:, k])))
                    n.index_add_(0, ids[:, k], on.double())

            if fl & (L.VOLUME | L.VOLUME_XPBD | L.NEOHOOKEAN):
                pa = xp[tet[:, 0]]
                p1, p2, p3 = xp[tet[:, 1]] - pa, xp[tet[:, 2]] - pa, xp[tet[:, 3]] - pa
                q1, q2, q3 = torch.linalg.cross(p2, p3), torch.linalg.cross(p3, p1), torch.linalg.cross(p1, p2)
                q = torch.stack([-q1 - q2 - q3, q1, q2, q3], dim=1)
                w = (mt * _dot(q, q)).sum(dim=1)
                six = _dot(q3, p3)
                if fl & L.VOLUME:
                    dl = -_f32(m.globalKsVolume) * (rest - six.abs() / 6.0) / w
                    add(tet, q * mt * dl.unsqueeze(1), w.abs() >= EPS)
                if fl & L.VOLUME_XPBD:
                    dl = -(six / 6.0 - signed + a_vol * lam_t) / (w + a_vol)
                    on = w.abs() >= EPS
                    lam_t = torch.where(on, lam_t + dl, lam_t)
                    add(tet, q * mt * dl.unsqueeze(1), on)
                if fl & L.NEOHOOKEAN:
                    F = torch.stack([p1, p2, p3], dim=2) @ D                 # columns f0 f1 f2
                    f = [F[:, :, k] for k in range(3)]
                    c = torch.stack([torch.linalg.cross(f[1], f[2]), torch.linalg.cross(f[2], f[0]),
                                     torch.linalg.cross(f[0], f[1])], dim=2)
                    G = (c @ D.transpose(1, 2)).transpose(1, 2)              # rows g1 g2 g3
                    G = torch.cat([-G.sum(dim=1, keepdim=True), G], dim=1)
                    wh = (mt * _dot(G, G)).sum(dim=1)
                    C = _dot(f[0], c[:, :, 0]) - 1.0 - (1.0 / devc) / (1.0 / volc)
                    d = G * mt * (-C / (wh + volc / dt / dt / rest)).unsqueeze(1)
                    rs = F.flatten(1).norm(dim=1).view(-1, 1)
                    H = (F @ D.transpose(1, 2)).transpose(1, 2) / rs.unsqueeze(2)
                    H = torch.cat([-H.sum(dim=1, keepdim=True), H], dim=1)
                    wd = (mt * _dot(H, H)).sum(dim=1)
                    d = d + H * mt * (-rs / (wd + devc / dt / dt / rest)).unsqueeze(1)
                    add(tet, d, (wh >= EPS) & (wd >= EPS))
            if fl & (L.DISTANCE | L.DISTANCE_XPBD):
                r = xp[edge[:, 1]] - xp[edge[:, 0]]
                length = r.norm(dim=1, keepdim=True)
                w = me.sum(dim=1)
                on = (length >= EPS) & (w >= EPS) & (L0 >= EPS)
                C = length - L0
                if fl & L.DISTANCE:
                    d = -C * (r / length) * _f32(m.globalKsDistance) / w
                    add(edge, torch.stack([-d, d], dim=1) * me, on)
                if fl & L.DISTANCE_XPBD:
                    dl = -(C + a_dist * lam_e) / (w + a_dist)
                    lam_e = torch.where(on, lam_e + dl, lam_e)
                    d = dl * (r / length)
                    add(edge, torch.stack([-d, d], dim=1) * me, on)
            xp = xp + torch.where(n > 0, dp / n.clamp_min(1.0), torch.zeros_like(dp))
            if fl & L.DRAG:
                xp = xp - (xp - grasp_at) * grasp
            if fl & L.COLLIDE and len(tri):
                out = torch.zeros_like(xp)
                p = [xp[tri[:, k]] for k in range(3)]
                for i in range(3):
                    resp = _capsule64(p, tip[4 * env + i], base[4 * env + i], rad[4 * env + i].unsqueeze(1),
                                      _f32(m.globalKsContact))
                    for k in range(3):
                        out.index_add_(0, tri[:, k], resp[k])
                xp = xp - torch.where(inv > 0, out, torch.zeros_like(out))
        xp = torch.stack([xp[:, 0], xp[:, 1].clamp_min(_f32(m.groundLevel)), xp[:, 2]], dim=1)
        v = (xp - x) / dt
        x = xp
    return x, v


def _closest64(a, b, c, p):
    """Barycentric coordinates of the triangle's point nearest to p (region by region)."""
    ab, ac = b - a, c - a
    d1, d2 = _dot(ab, p - a), _dot(ac, p - a)
    d3, d4 = _dot(ab, p - b), _dot(ac, p - b)
    d5, d6 = _dot(ab, p - c), _dot(ac, p - c)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    one, zero = torch.ones_like(d1), torch.zeros_like(d1)
    s = va + vb + vc
    bary = torch.cat([1.0 - vb / s - vc / s, vb / s, vc / s], dim=1)

    def put(on, x, y, z):
        nonlocal bary
        bary = torch.where(on, torch.cat([x, y, z], dim=1), bary)

    t = (d4 - d3) / ((d4 - d3) + (d5 - d6))
    put((va <= 0) & (d4 >= d3) & (d5 >= d6), zero, t, 1.0 - t)  # the reference's order of the pair
    t = d2 / (d2 - d6)
    put((vb <= 0) & (d2 >= 0) & (d6 <= 0), 1.0 - t, zero, t)
    put((d6 >= 0) & (d5 <= d6), zero, zero, one)
    t = d1 / (d1 - d3)
    put((vc <= 0) & (d1 >= 0) & (d3 <= 0), 1.0 - t, t, zero)
    put((d3 >= 0) & (d4 <= d3), zero, one, zero)
    put((d1 <= 0) & (d2 <= 0), one, zero, zero)
    return bary


def _capsule64(p, tip, base, radius, ks):
    pa, pb, pc = p
    n = _unit(torch.linalg.cross(pb - pa, pc - pa))
    centre = (pa + pb + pc) * _f32(0.3333)
    axis = _unit(tip - base)
    a, b = base + axis * radius, tip - axis * radius
    denom = _dot(n, axis)
    line = base + axis * (_dot(n, centre - base) / denom)
    ref = _closest64(pa, pb, pc, line)              # a barycentric triple, used as a point
    d = b - a
    t = (_dot(d, ref - a) / _dot(d, d)).clamp(0.0, 1.0)
    t = torch.where(d.norm(dim=1, keepdim=True) < EPS, torch.full_like(t, 0.5), t)
    s = a + d * t
    w = _closest64(pa, pb, pc, s)
    sv = s - (pa * w[:, 0:1] + pb * w[:, 1:2] + pc * w[:, 2:3])
    dist = sv.norm(dim=1, keepdim=True)
    pv = (radius / dist - 1.0) * sv
    sq = _dot(w, w)
    resp = _unit(pv) * (pv.norm(dim=1, keepdim=True) / sq) * ks
    on = (denom.abs() >= EPS) & (sq >= EPS) & (dist <= radius)
    return [torch.where(on, resp * w[:, k:k + 1], torch.zeros_like(resp)) for k in range(3)]


def _images64(case, m, r):
    R, N = case["resolution"], case["envs"]
    W = 2 * R
    pts, faces = m.allVisPoint.double(), m.allVisFace.long().view(-1, 3)
    P = [pts[faces[:, k]] for k in range(3)]
    nsum = torch.zeros_like(pts)
    cr = torch.linalg.cross(P[1] - P[0], P[2] - P[0])
    for k in range(3):
        nsum.index_add_(0, faces[:, k], cr)
    normal = _unit(nsum)
    color = m.allVisPointColor.double()
    et = torch.arange(W * W, device=pts.device)
    sx = 2.0 * (et % W).double() / W - 1.0
    sy = 2.0 * (W - torch.div(et, W, rounding_mode="floor")).double() / W - 1.0
    tan, aspect = _f32(r.camera_tan), _f32(r.camera_aspect)
    local = torch.stack([sx * tan * aspect, sy * tan, -torch.ones_like(sx)], dim=1)
    pixels = torch.zeros(N, R, R, 3, dtype=torch.float64, device=pts.device)
    depth = torch.zeros(N, R, R, dtype=torch.float64, device=pts.device)
    lights, power = r.lightDir.double(), r.lightIntensity.double()
    for e in range(N):
        f0, f1 = int(m.envVisFaceStart[e]), int(m.envVisFaceStart[e + 1])
        q, ro = r.cameraRotT[e].double(), r.cameraPosT[e].double()
        u, c = q[:3], 2.0 * q[3] * q[3] - 1.0
        rd = local * c + u * (2.0 * (local @ u)).unsqueeze(1) + \
            torch.linalg.cross(u.expand_as(local), local) * (2.0 * q[3])
        rd = _unit(rd)
        a = P[0][f0:f1]
        ab, ac = P[1][f0:f1] - a, P[2][f0:f1] - a
        # det = rd.(ac x ab), u det = rd.(ac x (ro - a)), v det = rd.((ro - a) x ab): products of
        # the rays with three vectors per face
        tv = ro - a
        qv = torch.linalg.cross(tv, ab)
        mats = [torch.linalg.cross(ac, ab).t(), torch.linalg.cross(ac, tv).t(), qv.t()]
        td = _dot(ac, qv).t()
        best = torch.full((W * W,), 1e6, dtype=torch.float64, device=pts.device)
        hit = torch.zeros(W * W, dtype=torch.long, device=pts.device)
        chunk = max(1, 20000000 // max(1, f1 - f0))
        for k in range(0, W * W, chunk):
            d = rd[k:k + chunk]
            det = d @ mats[0]
            uu, vv = (d @ mats[1]) / det, (d @ mats[2]) / det
            t = td / det
            ok = (det.abs() >= 1e-4) & (uu >= 0) & (uu <= 1) & (vv >= 0) & (uu + vv <= 1) & (t > 0)
            t = torch.where(ok, t, torch.full_like(t, 1e6))
            best[k:k + chunk], hit[k:k + chunk] = t.min(dim=1)
        img = torch.zeros(W * W, 3, dtype=torch.float64, device=pts.device)
        dep = torch.zeros(W * W, dtype=torch.float64, device=pts.device)
        on = best < 1e6
        f, t, d = f0 + hit[on], best[on], rd[on]
        if len(f):
            p = ro + t.unsqueeze(1) * d
            A, B, C = P[0][f], P[1][f], P[2][f]
            area = torch.linalg.cross(B - A, C - A).norm(dim=1, keepdim=True)
            w = torch.linalg.cross(B - A, p - A).norm(dim=1, keepdim=True) / area
            v = torch.linalg.cross(p - A, C - A).norm(dim=1, keepdim=True) / area
            b = torch.cat([1.0 - w - v, v, w], dim=1)
            n = sum(b[:, k:k + 1] * normal[faces[f, k]] for k in range(3))
            if case["shading"] == "normal":
                col = n * 0.5 + 0.5
            elif case["shading"] == "depth":
                col = (t / 50.0).unsqueeze(1).expand(-1, 3)
            else:
                if case["shading"] == "grayscale":
                    albedo = torch.ones_like(n)
                else:
                    albedo = sum(color[faces[f, k]] for k in range(3)) / 3.0
                    if case["shading"] == "texture" and m.hasTextures:
                        albedo = _texels64(m, e, f - f0, b, albedo)
                lam = (power * (n @ lights.t()).view(-1, 1, len(lights))).clamp_min(0.0).sum(dim=2)
                col = lam * albedo
            img[on] = col.clamp_max(1.0)
            dep[on] = (t / 50.0).clamp_max(1.0)
        pixels[e] = img.view(R, 2, R, 2, 3).sum(dim=(1, 3)) / 4.0
        depth[e] = dep.view(R, 2, R, 2).sum(dim=(1, 3)) / 4.0
    return pixels, depth


def _texels64(m, e, lf, b, albedo):
    first, count = (int(v) for v in m.host["envObjects"].reshape(-1, 2)[e])
    objects = m.host["objectTexture"].reshape(-1, 5)[first:first + count]
    tex, idx = m.textureT.double().view(-1, 3), m.texIndicesT.long()
    coords = m.texCoordsT.double().view(-1, 2)
    for k, (lo, t0, S, c0, i0) in enumerate(objects.tolist()):
        hi = objects[k + 1][0] if k + 1 < count else 1 << 40
        on = (lf >= lo) & (lf < hi)
        if S == 0 or not bool(on.any()):
            continue
        ti = idx[i0 + 3 * (lf[on] - lo).unsqueeze(1) + torch.arange(3, device=lf.device)]
        uv = (b[on].unsqueeze(2) * coords[c0 + ti]).sum(dim=1)
        fx, fy = uv[:, 0] * (S - 1), (1.0 - uv[:, 1]) * (S - 1)
        x0, y0 = fx.long(), fy.long()
        ax, ay = (fx - x0).unsqueeze(1), (fy - y0).unsqueeze(1)

        def at(x, y):
            return tex[t0 + y.clamp(0, S - 1) + x.clamp(0, S - 1) * S]

        low = (1 - ax) * at(x0, y0) + ax * at(x0 + 1, y0)
        high = (1 - ax) * at(x0, y0 + 1) + ax * at(x0 + 1, y0 + 1)
        albedo = albedo.clone()
        albedo[on] = (1 - ay) * low + ay * high
    return albedo
