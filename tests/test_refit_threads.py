"""Refits of a small and of a large batch from two host threads at a time, each on its own
stream: every launch succeeds, and the boxes are those of a refit alone."""

import ctypes as C
import threading

import pytest
import torch

from ffsrl import SimBVH, _lib as L, meshgen as mg, scenarios as sc

pytestmark = pytest.mark.gpu


def test_two_threads(gpu):
    mesh = mg.ellipsoid_for_tets(800, seed=3)
    jobs = []
    for envs in (1, 200):  # on both sides of the number of SMs
        m, _ = sc.liver_model("cuda:0", envs, meshes=[mesh] * envs)
        bvh = SimBVH("cuda:0", m)
        torch.cuda.synchronize()
        jobs.append((m, bvh, bvh.aabbMin.clone(), torch.cuda.Stream()))
    status = [set(), set()]
    start = threading.Barrier(2)

    def refit(k):
        m, bvh, _, stream = jobs[k]
        start.wait()
        for _ in range(5000):
            status[k].add(L.lib().ffsrl_bvh_refit_fused(C.byref(bvh.desc), L.ptr(m.allVisPoint), L.ptr(m.allVisFace),
                                                        stream.cuda_stream))

    threads = [threading.Thread(target=refit, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [{L.OK}, {L.OK}]
    for _, bvh, want, _ in jobs:
        assert torch.equal(bvh.aabbMin, want)
