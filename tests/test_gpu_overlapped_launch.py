"""Builds whose kernels start early (programmatic dependent launch) and report through page-locked memory:
back-to-back builds, builds replayed from a captured graph, and the stage times."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import to_device, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n,bits", [(5000, 30), (70_001, 63), (1_300_003, 60)])
def test_back_to_back_and_captured_builds(ctx, gpu, oracle_lib, n, bits):
    """Fifty builds of alternating meshes without a wait between them, then a captured one replayed: the
    last mesh's tree every time, equal to the oracle's."""
    a, b = meshgen.clustered(n, seed=1), meshgen.uniform_small(n // 2, seed=2)
    ta, pa = to_device(gpu, a.arrays())
    tb, pb = to_device(gpu, b.arrays())
    p = ctx.params(C.ALGO_LBVH, morton_bits=bits)
    want, widx, _ = oracle_lib.lbvh(a.arrays(), bits)
    for k in range(50):
        ctx.build_device(pb, b.size(), p, stream(gpu))
        tree = ctx.build_device(pa, n, p, stream(gpu))
    ctx.sync()
    nodes, idx = ctx.download(tree, stream(gpu))
    assert np.array_equal(idx, widx) and oracle_lib.node_fields_equal(nodes, want)
    g = gpu.cuda.CUDAGraph()
    with gpu.cuda.graph(g):
        tree = ctx.build_device(pa, n, p, stream(gpu))
    for _ in range(3):
        g.replay()
    gpu.cuda.synchronize()
    nodes, idx = ctx.download(tree, stream(gpu))
    assert np.array_equal(idx, widx) and oracle_lib.node_fields_equal(nodes, want)


@pytest.mark.parametrize("algo,kw", [(C.ALGO_LBVH, dict(morton_bits=63)), (C.ALGO_LBVH_PLUS, {}), (C.ALGO_PLOC, {})])
def test_stage_times(ctx, gpu, algo, kw):
    m = meshgen.clustered(300_000, seed=3)
    _, ptrs = to_device(gpu, m.arrays())
    for _ in range(3):
        ctx.build_device(ptrs, m.size(), ctx.params(algo, **kw), stream(gpu))
    t = ctx.last_timing()
    stages = [t.bounds_ms, t.morton_ms, t.sort_ms, t.emit_ms] + ([] if algo == C.ALGO_LBVH else [t.optimize_ms])
    assert all(s > 0 for s in stages)
    assert sum(stages) <= t.total_ms * 1.01 + 0.01
