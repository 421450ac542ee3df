"""PLOC's neighbour search while many clusters live: both forms (radii below 32 and from 32 on), at the
radii where a distance's last group is whole, ragged or one pair, with equal areas in every window
and with areas near the ends of the range, against the oracle, bit for bit."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from bvh_gb300.builders import TriangleMesh
from tests.gpu_util import build, to_device, stream

pytestmark = pytest.mark.gpu

N = 330_001  # above the 311,296 clusters that the one-launch form takes, with a ragged last tile


def _lattice(n, scale):
    """Unit right triangles on a cubic lattice: most areas in a window are equal."""
    side = int(np.ceil(n ** (1 / 3)))
    k = np.arange(n)
    p = np.stack([k % side, k // side % side, k // (side * side)], 1).astype(np.float32)
    e = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 1]], np.float32)
    v = [(p + e[j]) * np.float32(scale) for j in range(3)]
    return TriangleMesh(*[np.ascontiguousarray(v[j][:, a]) for j in range(3) for a in range(3)])


MESHES = {
    "random": lambda n: meshgen.uniform_small(n, seed=31),
    "lattice": lambda n: _lattice(n, 1.0),
    "lattice 1e16": lambda n: _lattice(n, 2.0 ** 53),  # areas to 1e36
    "lattice 1e-21": lambda n: _lattice(n, 2.0 ** -70),  # areas of neighbours are denormal
}


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind,radius", [("random", r) for r in (1, 2, 3, 4, 5, 6, 7, 8, 25, 31, 32, 33, 34, 35, 127, 128)] +
                         [("lattice", r) for r in (3, 25, 31, 32, 100)] +
                         [(k, r) for k in ("lattice 1e16", "lattice 1e-21") for r in (25, 32)])
def test_ploc_search(ctx, gpu, oracle_lib, kind, radius):
    m = MESHES[kind](N)
    nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_PLOC, ploc_radius=radius))
    onodes, oidx, it, cs, rc = oracle_lib.ploc(m.arrays(), radius)
    assert rc == 0
    assert np.array_equal(idx, oidx)
    assert oracle_lib.node_fields_equal(nodes, onodes)
    t = ctx.last_timing()
    assert t.ploc_iterations == it and t.ploc_cluster_sum == cs


@pytest.mark.parametrize("radius", [5, 25, 31, 32, 50, 128])
def test_ploc_search_stops_at_mesh_ends(ctx, gpu, oracle_lib, radius):
    parts = [MESHES["random"](20_001), _lattice(9_999, 1.0), MESHES["random"](5), _lattice(30_000, 1.0)]
    off = np.concatenate([[0], np.cumsum([p.size() for p in parts])]).astype(np.int64)
    ts, ptrs = to_device(gpu, [np.concatenate([p.arrays()[k] for p in parts]) for k in range(9)])
    tree = ctx.build_batched(ptrs, off, ctx.params(C.ALGO_PLOC, ploc_radius=radius), stream(gpu))
    ctx.sync()
    nodes, idx = ctx.download(tree, stream(gpu))
    for k, p in enumerate(parts):
        onodes, oidx, _, _, rc = oracle_lib.ploc(p.arrays(), radius)
        assert rc == 0
        a, b = int(off[k]), int(off[k + 1])
        assert np.array_equal(idx[a:b], oidx), k
        assert oracle_lib.node_fields_equal(nodes[2 * a - k: 2 * b - k - 1], onodes), k
