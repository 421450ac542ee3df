"""Batched builds read four triangles at a time where the arrays allow it: items that begin and end off a
multiple of four, or at the edges of an item of 4,096, and arrays that are not 16-byte aligned (which are
read one float at a time) give the trees of the meshes built alone, bit for bit."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from bvh_gb300.builders import TriangleMesh
from tests.gpu_util import build, stream

pytestmark = pytest.mark.gpu

COUNTS = {
    "offsets 0 to 3 mod 4": [1, 1, 1, 1, 2, 3, 5, 7, 4, 6, 9, 11, 13, 64, 63, 65, 255, 258],
    "item edges": [4095, 1, 4096, 4097, 3, 8191, 2, 8193, 12290],
    "one mesh": [16385],
}


@pytest.mark.parametrize("shifted", [None, 0, 8], ids=["aligned", "first array off", "last array off"])
@pytest.mark.parametrize("kind", list(COUNTS))
def test_batched_loads(gpu, oracle_lib, kind, shifted):
    from oracle import oracle as O
    counts = COUNTS[kind]
    mesh, offsets = meshgen.batch(counts, seed=23)
    n = int(offsets[-1])
    ts = []
    for k, a in enumerate(mesh.arrays()):
        t = gpu.empty(n + 4, dtype=gpu.float32, device="cuda")
        t = t[1:n + 1] if k == shifted else t[:n]
        t.copy_(gpu.from_numpy(np.ascontiguousarray(a, np.float32)))
        ts.append(t)
    ctx, single = Context(0), Context(0)
    tree = ctx.build_batched([t.data_ptr() for t in ts], offsets, ctx.params(C.ALGO_LBVH), stream(gpu))
    ctx.sync()
    nodes, idx = ctx.download(tree, stream(gpu))
    for m in range(len(counts)):
        a, b = int(offsets[m]), int(offsets[m + 1])
        sub = TriangleMesh(*[x[a:b] for x in mesh.arrays()])
        sn, si, _, _ = build(single, gpu, sub, single.params(C.ALGO_LBVH))
        assert np.array_equal(idx[a:b], si), m
        assert O.node_fields_equal(nodes[2 * a - m: 2 * b - m - 1], sn), m
    single.close()
    ctx.close()
