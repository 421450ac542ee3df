"""Emission does not trust what the node memory held before a build: a caller's memory whose padding looks like a
finished node's, a context's 65,536th build and its neighbours, and builds that follow others whose sort
kept its data elsewhere."""
import ctypes

import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests import meshes as M
from tests.gpu_util import build, stream, to_device

pytestmark = pytest.mark.gpu


def _words(kind, total):
    w = np.zeros((total, 12), np.uint32)
    rng = np.random.default_rng(5)
    if kind == "builds":  # every node says that it is written, by some build
        k = rng.integers(1, 200, total).astype(np.uint32)
        w[:, 3], w[:, 7] = 64 * k, (k + 1) << 16
    elif kind == "ones":
        w[:] = 0xFFFFFFFF
    else:
        w[:] = rng.integers(0, 1 << 32, (total, 12), dtype=np.uint64).astype(np.uint32)
    return w


@pytest.mark.parametrize("kind", ["builds", "ones", "random"])
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("shape,n", [("uniform", 2_049), ("uniform", 70_001), ("chains", 9_001), ("identical", 5_000)])
def test_callers_memory(gpu, oracle_lib, kind, bits, shape, n):
    mesh = {"uniform": lambda: meshgen.uniform_small(n, seed=51), "chains": lambda: M.dense_cell(n),
            "identical": lambda: M.identical(n)}[shape]()
    ts, ptrs = to_device(gpu, mesh.arrays())
    on, oi, _ = oracle_lib.lbvh(mesh.arrays(), bits)
    nodes = gpu.from_numpy(_words(kind, 2 * n - 1).view(np.int32)).cuda()
    idx = gpu.empty(n, dtype=gpu.int32, device="cuda")
    gpu.cuda.synchronize()
    m = C.mesh_struct(ptrs, n)
    lib = C.load_library()
    for _ in range(3):
        C.check(lib.bvh_build_lbvh_static(ctypes.byref(m), bits, ctypes.c_void_p(nodes.data_ptr()),
                                          ctypes.c_void_p(idx.data_ptr()), ctypes.c_void_p(stream(gpu))), "static")
        gpu.cuda.synchronize()
        got = np.ascontiguousarray(nodes.cpu().numpy())
        assert not got.view(np.uint32).reshape(-1, 12)[:, [3, 7]].any()
        assert np.array_equal(idx.cpu().numpy().view(np.uint32), oi)
        assert oracle_lib.node_fields_equal(got.view(C.NODE_DTYPE).reshape(-1), on)


def test_build_65536(gpu, oracle_lib):
    """The builds around the 65,536th of one context, where a 16-bit count of builds is 0."""
    ctx = Context(0)
    small, big = meshgen.uniform_small(8, seed=52), meshgen.uniform_small(30_001, seed=53)
    ctx.reserve(big.size(), C.ALGO_LBVH_PLUS)
    ts, ptrs = to_device(gpu, small.arrays())
    p = ctx.params(C.ALGO_LBVH)
    expected = {bits: oracle_lib.lbvh(big.arrays(), bits)[:2] for bits in (30, 63)}
    for k in range(65_536 - 4):
        ctx.build_device(ptrs, small.size(), p, stream(gpu))
    ctx.sync()
    for k in range(4):
        for bits in (30, 63):
            nodes, idx, _, _ = build(ctx, gpu, big, ctx.params(C.ALGO_LBVH, morton_bits=bits))
            assert np.array_equal(idx, expected[bits][1]) and oracle_lib.node_fields_equal(nodes, expected[bits][0])
    on, oi = oracle_lib.lbvh_plus(big.arrays(), 60, 2)
    nodes, idx, _, _ = build(ctx, gpu, big, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=2))
    assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    ctx.close()


def test_builds_after_one_another(gpu, oracle_lib):
    """Long runs of equal codes (their low bits go through two buffers), batches with more meshes than their keys
    have room for, PLOC and LBVH+, in turn over the same memory and with sizes that move the leaves."""
    ctx = Context(0)
    ctx.reserve(90_000, C.ALGO_PLOC)
    parts = [M.identical(9_000), meshgen.uniform_small(20_001, seed=54), M.dense_cell(5_003), M.identical(1),
             M.identical(700), meshgen.uniform_small(513, seed=55)]
    off = np.concatenate([[0], np.cumsum([p.size() for p in parts])]).astype(np.int64)
    bt, bptrs = to_device(gpu, [np.concatenate([p.arrays()[k] for p in parts]) for k in range(9)])
    singles = [M.identical(30_000), M.dense_cell(40_001), meshgen.uniform_small(70_001, seed=56), M.identical(2_049)]
    for mesh in singles:
        for bits in (63, 60, 30):
            nodes, idx, _, _ = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH, morton_bits=bits))
            on, oi, _ = oracle_lib.lbvh(mesh.arrays(), bits)
            assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
            assert not _padding(nodes).any()
        for algo in (C.ALGO_LBVH, C.ALGO_PLOC):
            tree = ctx.build_batched(bptrs, off, ctx.params(algo, ploc_radius=10), stream(gpu))
            ctx.sync()
            nodes, idx = ctx.download(tree, stream(gpu))
            assert not _padding(nodes).any()
            for k, p in enumerate(parts):
                if algo == C.ALGO_LBVH:
                    on, oi, _ = oracle_lib.lbvh(p.arrays(), 30)
                else:
                    on, oi, _, _, _ = oracle_lib.ploc(p.arrays(), 10)
                a = 2 * off[k] - k
                assert np.array_equal(idx[off[k]:off[k + 1]], oi)
                assert oracle_lib.node_fields_equal(nodes[a:a + len(on)], on)
    ctx.close()


def _padding(nodes):
    return np.ascontiguousarray(nodes).view(np.uint32).reshape(-1, 12)[:, [3, 7]]
