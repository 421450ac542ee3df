"""Builds that replay a graph after other builds of the same context have grown its buffers a little at a time, so
that some buffers come back where they were and others do not: the trees are the oracle's."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build, stream, to_device

pytestmark = pytest.mark.gpu


def _grow(ctx, gpu, n, algo=C.ALGO_LBVH):
    build(ctx, gpu, meshgen.uniform_small(n, seed=60), ctx.params(algo, ploc_radius=10))


@pytest.mark.parametrize("rounds", [1, 3])
def test_lbvh_plus(gpu, oracle_lib, rounds):
    ctx = Context(0)
    mesh = meshgen.clustered(40_000, seed=61)
    on, oi = oracle_lib.lbvh_plus(mesh.arrays(), 60, rounds)
    p = ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=rounds)
    for step in (0, 100, 1, 2_000, 7, 500_000):
        if step:
            _grow(ctx, gpu, 40_000 + step)
        nodes, idx, _, _ = build(ctx, gpu, mesh, p)
        assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    ctx.close()


def test_ploc_loop(gpu, oracle_lib):
    ctx = Context(0)
    mesh = meshgen.clustered(20_000, seed=62)
    radius = 200  # (above the cooperative kernel's: the loop graph runs)
    on, oi, _, _, rc = oracle_lib.ploc(mesh.arrays(), radius)
    assert rc == 0
    for step, algo in ((0, C.ALGO_LBVH), (100, C.ALGO_LBVH), (150, C.ALGO_PLOC), (2_000, C.ALGO_LBVH), (400_000, C.ALGO_PLOC)):
        if step:
            _grow(ctx, gpu, 20_000 + step, algo)
        nodes, idx, _, _ = build(ctx, gpu, mesh, ctx.params(C.ALGO_PLOC, ploc_radius=radius))
        assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    ctx.close()


@pytest.mark.parametrize("algo", [C.ALGO_LBVH, C.ALGO_PLOC])
def test_batch_graph(gpu, oracle_lib, algo):
    ctx = Context(0)
    parts = [meshgen.uniform_small(n, seed=63 + k) for k, n in enumerate((3_000, 70, 9_001, 1, 2_500, 400))]
    off = np.concatenate([[0], np.cumsum([p.size() for p in parts])]).astype(np.int64)
    ts, ptrs = to_device(gpu, [np.concatenate([p.arrays()[k] for p in parts]) for k in range(9)])
    expected = [oracle_lib.lbvh(p.arrays(), 30)[:2] if algo == C.ALGO_LBVH else oracle_lib.ploc(p.arrays(), 10)[:2]
                for p in parts]
    n = int(off[-1])
    # a larger plain build, a larger PLOC build, a batch of more triangles and meshes, between replays of one graph
    for step in (None, 100, -100, 300_000, "batch", None):
        if step == "batch":
            more = meshgen.uniform_small(2 * n, seed=64)
            mt, mptrs = to_device(gpu, more.arrays())
            cut = np.linspace(0, 2 * n, 4_001).astype(np.int64)
            ctx.build_batched(mptrs, cut, ctx.params(C.ALGO_LBVH), stream(gpu))
            ctx.sync()
        elif step:
            _grow(ctx, gpu, n + abs(step), C.ALGO_LBVH if step > 0 else C.ALGO_PLOC)
        tree = ctx.build_batched(ptrs, off, ctx.params(algo, ploc_radius=10), stream(gpu), use_graph=True)
        ctx.sync()
        nodes, idx = ctx.download(tree, stream(gpu))
        for k, (on, oi) in enumerate(expected):
            a = 2 * off[k] - k
            assert np.array_equal(idx[off[k]:off[k + 1]], oi)
            assert oracle_lib.node_fields_equal(nodes[a:a + len(on)], on)
    ctx.close()
