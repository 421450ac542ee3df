"""The packed traversal (traces of 16,384 rays or more) against the oracle and against the plain kernel,
which smaller traces take: the same hits and counters bit for bit on every tree the plain one accepts."""
import numpy as np
import pytest

from bvh_gb300 import Context, auto_camera, meshgen, _capi as C
from tests.gpu_util import build, to_device, stream

pytestmark = pytest.mark.gpu
NR = 16384  # the fewest rays that are traced packed


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


def _trace(ctx, gpu, nodes_ptr, n_nodes, mts, n_tris, rays, step):
    """Traces `rays` (n, 6) in calls of `step` rays; the five hit arrays as numpy."""
    n = rays.shape[0]
    dev = [gpu.from_numpy(np.ascontiguousarray(rays[:, k])).cuda() for k in range(6)]
    out = [gpu.full((n,), -7, dtype=gpu.float32 if k == 0 else gpu.int32, device="cuda") for k in range(5)]
    for b in range(0, n, step):
        ctx.trace(nodes_ptr, n_nodes, mts, n_tris, [t[b:].data_ptr() for t in dev], min(step, n - b),
                  [t[b:].data_ptr() for t in out], stream(gpu))
    gpu.cuda.synchronize()
    return [o.cpu().numpy().view(np.uint32) for o in out]


def _check(ctx, gpu, O, nodes, mesh, rays):
    dn = gpu.from_numpy(np.ascontiguousarray(nodes).view(np.uint8).reshape(-1)).cuda()
    ts, ptrs = to_device(gpu, mesh.arrays())
    packed = _trace(ctx, gpu, dn.data_ptr(), len(nodes), ptrs, mesh.size(), rays, len(rays))
    plain = _trace(ctx, gpu, dn.data_ptr(), len(nodes), ptrs, mesh.size(), rays, NR - 1)
    for a, b in zip(packed, plain):
        assert np.array_equal(a, b)
    k = min(len(rays), 2000)
    want = O.trace(nodes, mesh.arrays(), rays[:k, :3], rays[:k, 3:])
    for a, e in zip(packed, want):
        assert np.array_equal(a[:k], e.view(np.uint32))
    return packed


def _rays(mesh, n, seed):
    o, d = meshgen.sphere_rays(mesh, n, seed)
    d[:7] = [[1, 0, 0], [0, -1, 0], [0, 0, 1], [1e-7, 1, 0], [-1, 1e-9, 0], [0, 0, 0], [1, 1, 1]]
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("n", [2, 3, 9, 257, 30001])
@pytest.mark.parametrize("rays", [NR, NR + 1, 20011])
def test_sizes(ctx, gpu, oracle_lib, n, rays):
    m = meshgen.clustered(n, seed=n)
    nodes, _, _ = oracle_lib.lbvh(m.arrays(), 30)
    _check(ctx, gpu, oracle_lib, nodes, m, _rays(m, rays, 5))


def _chain(n, turn):
    """A tree of n leaves and depth n - 1: every inner node has one leaf and the rest of the chain, which is
    the left child where turn(i).  Every box is the whole scene, so every path is walked."""
    nodes = np.zeros(2 * n - 1, C.NODE_DTYPE)
    nodes["min"], nodes["max"] = -1.0, 2.0
    leaf = n - 1 + np.arange(n)
    for i in range(n - 1):
        rest = i + 1 if i + 1 < n - 1 else leaf[n - 1]
        nodes[i]["left"], nodes[i]["right"] = (rest, leaf[i]) if turn(i) else (leaf[i], rest)
    nodes["left"][leaf] = (np.arange(n) | 0x80000000).astype(np.uint32).view(np.int32)
    nodes["right"][leaf] = -1
    return nodes


@pytest.mark.parametrize("turn", [lambda i: True, lambda i: False, lambda i: i % 3 != 0, lambda i: i < 127,
                                  lambda i: i < 128], ids=["left", "right", "mixed", "left127", "left128"])
def test_deeper_than_the_stack(ctx, gpu, oracle_lib, turn):
    """Depth 399: the reference's 128-entry stack drops children, and the same ones are dropped here."""
    m = meshgen.uniform_small(400, seed=3)
    _check(ctx, gpu, oracle_lib, _chain(400, turn), m, _rays(m, NR, 6))


def test_odd_trees(ctx, gpu, oracle_lib):
    """Children outside the array, leaves without a triangle, NaN and infinite boxes."""
    m = meshgen.clustered(3000, seed=8)
    nodes, _, _ = oracle_lib.lbvh(m.arrays(), 30)
    g = np.random.Generator(np.random.PCG64(1))
    inner = g.permutation(np.arange(1, 2999))[:120]
    nodes["left"][inner[:20]] = 1 << 30
    nodes["right"][inner[20:40]] = -5
    nodes["right"][inner[40:60]] = 1 << 29
    nodes["min"][inner[60:80]] = np.nan
    nodes["max"][inner[80:100]] = np.inf
    nodes["min"][inner[90:110]] = -np.inf
    leaves = 2999 + g.permutation(3000)[:50]
    nodes["left"][leaves] = (np.arange(50) * 100 + 2990 | 0x80000000).astype(np.uint32).view(np.int32)
    _check(ctx, gpu, oracle_lib, nodes, m, _rays(m, NR, 7))


@pytest.mark.parametrize("w,h", [(128, 128), (129, 131), (641, 27), (3, 7001)])
def test_pinhole_pixels(ctx, gpu, w, h):
    """Odd image sizes: the image traced at once against its rays traced in small calls."""
    from bvh_gb300.builders import pinhole_rays
    m = meshgen.clustered(20000, seed=9)
    nodes, _, tree, ts = build(ctx, gpu, m, ctx.params(C.ALGO_PLOC))
    ptrs = [t.data_ptr() for t in ts]
    cam = auto_camera(nodes[0])
    n = w * h
    out = [gpu.full((n,), -7, dtype=gpu.float32 if k == 0 else gpu.int32, device="cuda") for k in range(5)]
    ctx.trace_pinhole(tree.nodes, tree.n_nodes, ptrs, m.size(), cam, w, h, [t.data_ptr() for t in out], stream(gpu))
    rays = [gpu.empty(n, device="cuda") for _ in range(6)]
    pinhole_rays(cam, w, h, [t.data_ptr() for t in rays], stream(gpu))
    gpu.cuda.synchronize()
    plain = _trace(ctx, gpu, tree.nodes, tree.n_nodes, ptrs, m.size(), gpu.stack(rays, 1).cpu().numpy(), NR - 1)
    for a, b in zip(out, plain):
        assert np.array_equal(a.cpu().numpy().view(np.uint32), b)


def test_streams_and_capture(ctx, gpu):
    """Two streams at once on one context, and a trace inside a captured graph, give the same hits."""
    m = meshgen.clustered(20000, seed=10)
    _, _, tree, ts = build(ctx, gpu, m, ctx.params(C.ALGO_LBVH))
    ptrs = [t.data_ptr() for t in ts]
    rays = [gpu.from_numpy(np.ascontiguousarray(a)).cuda() for a in _rays(m, 50000, 8).T]
    rp = [t.data_ptr() for t in rays]

    def out():
        return [gpu.full((50000,), -7, dtype=gpu.float32 if k == 0 else gpu.int32, device="cuda") for k in range(5)]

    want, a, b, c = out(), out(), out(), out()
    gpu.cuda.synchronize()
    ctx.trace(tree.nodes, tree.n_nodes, ptrs, m.size(), rp, 50000, [t.data_ptr() for t in want], stream(gpu))
    gpu.cuda.synchronize()
    s1, s2 = gpu.cuda.Stream(), gpu.cuda.Stream()
    for _ in range(3):
        for s, o in ((s1, a), (s2, b)):
            ctx.trace(tree.nodes, tree.n_nodes, ptrs, m.size(), rp, 50000, [t.data_ptr() for t in o], s.cuda_stream)
    g = gpu.cuda.CUDAGraph()
    gpu.cuda.synchronize()
    with gpu.cuda.graph(g):
        ctx.trace(tree.nodes, tree.n_nodes, ptrs, m.size(), rp, 50000, [t.data_ptr() for t in c], stream(gpu))
    g.replay()
    gpu.cuda.synchronize()
    for o in (a, b, c):
        assert all(gpu.equal(x.view(gpu.int32), y.view(gpu.int32)) for x, y in zip(o, want))
