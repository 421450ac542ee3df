"""A server's small meshes take the general build (its slots share the GPU with each other): what rays hit
on meshes of 1 to 2,049 triangles, and the nodes they visit, are the oracle's."""
import time

import numpy as np
import pytest

from bvh_gb300 import meshgen, _capi as C
from bvh_gb300.serve import Server

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 33, 512, 513, 2047, 2048, 2049]


def test_small_meshes_served(gpu, oracle_lib):
    server = Server(slots=4)
    meshes = [meshgen.uniform_small(n, seed=61) for n in SIZES]
    rays, hits, done = [], [], {}
    for k, m in enumerate(meshes):
        ro, rd = meshgen.sphere_rays(m, 2048, seed=62)
        rays.append((ro, rd))
        hits.append([np.zeros(2048, np.float32)] + [np.zeros(2048, np.int32) for _ in range(4)])
        server.submit(k, m.arrays(), [ro[:, j].copy() for j in range(3)] + [rd[:, j].copy() for j in range(3)], hits[k])
    deadline = time.time() + 60
    while len(done) < len(SIZES) and time.time() < deadline:
        for r in server.poll(64, 50):
            done[r["tag"]] = r["status"]
    server.close()
    assert done == {k: C.BVH_OK for k in range(len(SIZES))}
    for k, m in enumerate(meshes):
        nodes, _, _ = oracle_lib.lbvh(m.arrays(), 30)
        exp = oracle_lib.trace(nodes, m.arrays(), *rays[k])
        assert np.array_equal(hits[k][0].view(np.uint32), exp[0].view(np.uint32)), SIZES[k]
        assert np.array_equal(hits[k][1], exp[1]), SIZES[k]
        assert np.array_equal(hits[k][2], exp[2]), SIZES[k]
