"""Nodes above the tiles tell their siblings that they are done through their own padding: trees whose levels
pass through it (ends of tiles, long chains, ties, the change of the in-tile limit at 2,000,000) equal the
oracle's bit for bit, and the padding is 0 again afterwards, build after build in one context."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from bvh_gb300.builders import TriangleMesh
from tests import meshes as M
from tests.gpu_util import build, to_device, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


def _padding(nodes):
    w = np.ascontiguousarray(nodes).view(np.uint32).reshape(-1, 12)
    return w[:, [3, 7]]


MESHES = {
    "uniform": lambda n: meshgen.uniform_small(n, seed=41),
    "chains": lambda n: M.dense_cell(n),  # most codes equal: levels of one leaf each
    "identical": lambda n: M.identical(n),
}


@pytest.mark.parametrize("algo,bits", [(C.ALGO_LBVH, 30), (C.ALGO_LBVH, 63), (C.ALGO_LBVH_PLUS, 60)])
@pytest.mark.parametrize("kind,n", [(k, n) for k in MESHES for n in (2049, 2560, 2561, 70_001)] +
                         [("uniform", 1_999_999), ("uniform", 2_000_001)])
def test_emission_messages(ctx, gpu, oracle_lib, algo, bits, kind, n):
    mesh = MESHES[kind](n)
    p = ctx.params(algo, morton_bits=bits)
    if algo == C.ALGO_LBVH:
        on, oi, _ = oracle_lib.lbvh(mesh.arrays(), bits)
    else:
        if n > 100_000:
            pytest.skip("the emission is the same")
        on = None
    first = None
    for _ in range(2):
        nodes, idx, _, _ = build(ctx, gpu, mesh, p)
        assert not _padding(nodes).any()
        if on is not None:
            assert np.array_equal(idx, oi)
            assert oracle_lib.node_fields_equal(nodes, on)
        elif first is not None:
            assert np.array_equal(idx, first[1]) and oracle_lib.node_fields_equal(nodes, first[0])
        first = (nodes, idx)


def test_emission_messages_of_batches(ctx, gpu):
    parts = [meshgen.uniform_small(30_001, seed=42), M.dense_cell(9_000), M.identical(700), meshgen.uniform_small(513, seed=43)]
    off = np.concatenate([[0], np.cumsum([p.size() for p in parts])]).astype(np.int64)
    ts, ptrs = to_device(gpu, [np.concatenate([p.arrays()[k] for p in parts]) for k in range(9)])
    for _ in range(2):
        tree = ctx.build_batched(ptrs, off, ctx.params(C.ALGO_LBVH), stream(gpu))
        ctx.sync()
        nodes, _ = ctx.download(tree, stream(gpu))
        assert not _padding(nodes).any()
