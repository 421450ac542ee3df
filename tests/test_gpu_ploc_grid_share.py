"""PLOC's cooperative iterations on part of the GPU: the fewest blocks, a half of them (both ends of its range),
and all, at small and large radii; several builds at once in streams of their own.  Trees equal the oracle's."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build, to_device

pytestmark = pytest.mark.gpu


def _sizes():
    """n per block 512 at r = 25, on 152 multiprocessors: 16, 17, 76, 77 -> 76, 121 -> 76, 122, 152 blocks."""
    return [8_192, 8_193, 38_912, 38_913, 61_952, 61_953, 77_824, 77_825]


@pytest.mark.parametrize("n,radius", [(n, 25) for n in _sizes()] + [(20_000, 1), (20_000, 100), (20_000, 128), (12_801, 100)])
def test_ploc_grid_share(gpu, oracle_lib, n, radius):
    ctx = Context(0)
    m = meshgen.uniform_small(n, seed=71)
    nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_PLOC, ploc_radius=radius))
    onodes, oidx, it, cs, rc = oracle_lib.ploc(m.arrays(), radius)
    assert rc == 0 and np.array_equal(idx, oidx) and oracle_lib.node_fields_equal(nodes, onodes)
    t = ctx.last_timing()
    assert t.ploc_iterations == it and t.ploc_cluster_sum == cs
    ctx.close()


def test_ploc_grids_side_by_side(gpu, oracle_lib):
    sizes = [9_000, 20_000, 30_000, 60_000]
    ctxs = [Context(0) for _ in sizes]
    streams = [gpu.cuda.Stream() for _ in sizes]
    meshes = [meshgen.uniform_small(n, seed=72) for n in sizes]
    inputs = [to_device(gpu, m.arrays()) for m in meshes]
    gpu.cuda.synchronize()
    for _ in range(3):
        trees = [c.build_device(p[1], n, c.params(C.ALGO_PLOC), s.cuda_stream)
                 for c, p, n, s in zip(ctxs, inputs, sizes, streams)]
    for c, tree, m, s in zip(ctxs, trees, meshes, streams):
        c.sync()
        nodes, idx = c.download(tree, s.cuda_stream)
        onodes, oidx, _, _, _ = oracle_lib.ploc(m.arrays(), 25)
        assert np.array_equal(idx, oidx) and oracle_lib.node_fields_equal(nodes, onodes)
        c.close()
