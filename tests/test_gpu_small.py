"""Meshes of at most 2,048 triangles, which one block builds, against the oracle: every size at which its
shape changes, all code widths and algorithms, and inputs that make its special cases."""
import numpy as np
import pytest

from bvh_gb300 import Context, LBVHBuilder, TriangleMesh, meshgen, _capi as C
from tests.gpu_util import build, to_device, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


def _odd_mesh(kind, n):
    m = meshgen.clustered(n, seed=n)
    a = [x.copy() for x in m.arrays()]
    if kind == "identical":  # every code equal: the tie rule alone makes the tree
        a = [np.full_like(x, x[0]) for x in a]
    elif kind == "flat":  # no extent on one axis
        for k in (2, 5, 8):
            a[k][:] = 1.5
    elif kind == "nan":
        a[0][::7] = np.nan
        for k in range(9):
            a[k][n // 2] = np.nan
    elif kind == "inf":
        a[3][::11] = np.inf
        a[7][::13] = -np.inf
    elif kind == "negative":
        a = [-1e4 * x for x in a]
    return TriangleMesh(*a)


def _equal(O, got, want):
    return O.node_fields_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("bits", [30, 60, 63])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 255, 257, 1023, 1024, 1025, 1999, 2047, 2048, 2049])
def test_lbvh_sizes(ctx, gpu, oracle_lib, n, bits):
    m = meshgen.clustered(n, seed=n)
    nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_LBVH, morton_bits=bits))
    want = oracle_lib.lbvh(m.arrays(), bits)
    assert _equal(oracle_lib, (nodes, idx), want)


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("kind", ["identical", "flat", "nan", "inf", "negative"])
def test_lbvh_inputs(ctx, gpu, oracle_lib, kind, bits):
    m = _odd_mesh(kind, 1500)
    big = TriangleMesh(*[np.concatenate([a, a]) for a in m.arrays()])  # 3,000: the general kernels
    for mesh in (m, big):
        nodes, idx, _, _ = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH, morton_bits=bits))
        want = oracle_lib.lbvh(mesh.arrays(), bits)
        assert np.array_equal(idx, want[1])
        for f in ("min", "max", "left", "right"):
            assert np.array_equal(nodes[f], want[0][f], equal_nan=f in ("min", "max"))


@pytest.mark.parametrize("n", [1, 2, 3, 100, 1024, 1025, 2048])
def test_plus_and_ploc(ctx, gpu, oracle_lib, n):
    m = meshgen.clustered(n, seed=n + 1)
    for bits in (30, 60):
        nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=bits, treelet_rounds=2))
        assert _equal(oracle_lib, (nodes, idx), oracle_lib.lbvh_plus(m.arrays(), bits, 2))
    nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_PLOC, ploc_radius=25))
    want = oracle_lib.ploc(m.arrays(), 25)
    assert _equal(oracle_lib, (nodes, idx), want[:2])


def test_between_larger_builds_and_unaligned(ctx, gpu, oracle_lib):
    """Small builds share a workspace (epoch, status, buffers) with larger ones; rows of one array."""
    big, small = meshgen.clustered(50_000, seed=5), meshgen.uniform_small(1001, seed=6)
    rows = gpu.from_numpy(np.stack(small.arrays())).cuda()
    pb = to_device(gpu, big.arrays())
    for bits in (30, 63, 60):
        for algo in (C.ALGO_LBVH, C.ALGO_LBVH_PLUS):
            p = ctx.params(algo, morton_bits=bits)
            for mesh, ptrs in ((big, pb[1]), (small, [rows[k].data_ptr() for k in range(9)])) * 2:
                tree = ctx.build_device(ptrs, mesh.size(), p, stream(gpu))
                got = ctx.download(tree, stream(gpu))
                want = (oracle_lib.lbvh(mesh.arrays(), bits) if algo == C.ALGO_LBVH
                        else oracle_lib.lbvh_plus(mesh.arrays(), bits, 1))
                assert _equal(oracle_lib, got, want)
    t = ctx.last_timing()
    assert t.total_ms > 0


def test_host_builder(gpu, oracle_lib):
    b = LBVHBuilder(morton_bits=63)
    for n in (2048, 2049, 5, 1):
        m = meshgen.clustered(n, seed=n)
        b.build(m)
        assert _equal(oracle_lib, (b.getNodes(), b.getIndices()), oracle_lib.lbvh(m.arrays(), 63))
        assert b.getLastBuildTimeMS() > 0


@pytest.mark.parametrize("n,bits", [(1000, 30), (2000, 63)])
def test_first_build_captured(gpu, oracle_lib, n, bits):
    """A context whose first build of its kind is recorded into a graph."""
    c = Context(0)
    m = meshgen.clustered(n, seed=n)
    _, ptrs = to_device(gpu, m.arrays())
    p = c.params(C.ALGO_LBVH, morton_bits=bits)
    c.reserve(n)
    gpu.cuda.synchronize()
    g = gpu.cuda.CUDAGraph()
    with gpu.cuda.graph(g):
        tree = c.build_device(ptrs, n, p, stream(gpu))
    g.replay()
    gpu.cuda.synchronize()
    assert _equal(oracle_lib, c.download(tree, stream(gpu)), oracle_lib.lbvh(m.arrays(), bits))
    del g
    c.close()
