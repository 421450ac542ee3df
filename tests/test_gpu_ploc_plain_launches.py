"""PLOC without its cooperative kernel: small builds stay in the loop graph and the one-block tail (so those of
the tail alone can be captured), larger radii hand over to the tail as early; trees equal the oracle's."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build, stream, to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,radius", [(2, 25), (500, 25), (501, 25), (1_999, 25), (2_001, 25), (20_011, 25), (65_535, 25),
                                      (65_536, 25), (3_000, 128), (3_000, 129), (20_000, 200), (2_000, 512)])
@pytest.mark.parametrize("no_cooperative", [True, False])
def test_trees(gpu, oracle_lib, n, radius, no_cooperative):
    ctx = Context(0)
    m = meshgen.uniform_small(n, seed=95)
    nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_PLOC, ploc_radius=radius, no_cooperative=no_cooperative))
    on, oi, it, cs, rc = oracle_lib.ploc(m.arrays(), radius)
    assert rc == 0 and np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    t = ctx.last_timing()
    assert t.ploc_iterations == it and t.ploc_cluster_sum == cs
    ctx.close()


@pytest.mark.parametrize("no_cooperative", [True, False])
@pytest.mark.parametrize("n", [400, 1_000, 1_999])
def test_captured(gpu, oracle_lib, n, no_cooperative):
    ctx = Context(0)
    m = meshgen.uniform_small(n, seed=96)
    ts, ptrs = to_device(gpu, m.arrays())
    p = ctx.params(C.ALGO_PLOC, no_cooperative=no_cooperative)
    ctx.build_device(ptrs, n, p, stream(gpu))
    ctx.sync()
    g = gpu.cuda.CUDAGraph()
    with gpu.cuda.graph(g):
        tree = ctx.build_device(ptrs, n, p, stream(gpu))
    g.replay()
    gpu.cuda.synchronize()
    nodes, idx = ctx.download(tree, stream(gpu))
    on, oi, _, _, _ = oracle_lib.ploc(m.arrays(), 25)
    assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    ctx.close()
