"""LBVH+ where boxes are not tame (NaN, infinite or huge coordinates, which the passes refit) and at the edge
of it, over several passes and all routes through the heights, against the oracle."""
import numpy as np
import pytest

from bvh_gb300 import Context, TriangleMesh, meshgen, _capi as C
from tests.gpu_util import to_device, stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


def _mesh(kind, n):
    m = meshgen.clustered(n, seed=n + 7) if kind != "strands" else meshgen.strands(n // 50, 50, seed=n)
    a = [x.copy() for x in m.arrays()]
    if kind == "edge":  # the largest coordinate that is still tame, and one just above
        for k in range(9):
            a[k] *= np.float32(1e13) / np.float32(2)
        a[0][n // 2] = np.float32(1e13)
    elif kind == "above":
        a[0][n // 2] = np.nextafter(np.float32(1e13), np.float32(2e13))
    elif kind == "huge":  # areas up to 1e28, just below the subset DP's infinity
        for k in range(9):
            a[k] *= np.float32(1e14)
    elif kind == "overflow":  # costs past that infinity: such a treelet stays as it is
        for k in range(9):
            a[k] *= np.float32(1e18)
    elif kind == "nan":
        for k in range(9):
            a[k][::97] = np.nan
        a[4][::31] = np.nan
    elif kind == "inf":
        a[2][5::101] = np.inf
        a[6][7::203] = -np.inf
    elif kind == "identical":
        a = [np.full_like(x, x[0]) for x in a]
    return TriangleMesh(*a)


@pytest.mark.parametrize("n", [3, 40, 2000, 6001, 60_003])
@pytest.mark.parametrize("kind", ["tame", "strands", "identical", "edge", "above", "huge", "nan"])
def test_passes(ctx, gpu, oracle_lib, kind, n):
    m = _mesh(kind, max(n, 50) if kind == "strands" else n)
    _, ptrs = to_device(gpu, m.arrays())
    for rounds in (1, 2, 3):
        want, widx = oracle_lib.lbvh_plus(m.arrays(), 60, rounds)
        for kw in (dict(), dict(host_loops=True), dict(no_cooperative=True)):
            tree = ctx.build_device(ptrs, m.size(), ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=rounds, **kw),
                                    stream(gpu))
            nodes, idx = ctx.download(tree, stream(gpu))
            assert np.array_equal(idx, widx)
            for f in ("min", "max", "left", "right"):
                assert np.array_equal(nodes[f], want[f], equal_nan=f in ("min", "max")), (rounds, kw, f)


@pytest.mark.parametrize("n", [3, 2000, 60_003])
@pytest.mark.parametrize("kind", ["overflow", "inf"])
def test_costs_past_infinity(ctx, gpu, kind, n):
    """The oracle, like the reference, has no answer where no split is below infinity; the routes through the
    heights agree on it, and every box is the union of its children's."""
    m = _mesh(kind, n)
    _, ptrs = to_device(gpu, m.arrays())
    got = []
    for kw in (dict(), dict(host_loops=True), dict(no_cooperative=True)):
        tree = ctx.build_device(ptrs, n, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=2, **kw), stream(gpu))
        got.append(ctx.download(tree, stream(gpu)))
    for nodes, idx in got[1:]:
        assert np.array_equal(idx, got[0][1])
        assert all(np.array_equal(nodes[f], got[0][0][f]) for f in ("min", "max", "left", "right"))
    nodes = got[0][0]
    inner = nodes[: n - 1]
    l, r = nodes[inner["left"]], nodes[inner["right"]]
    assert np.array_equal(inner["min"], np.minimum(l["min"], r["min"]))
    assert np.array_equal(inner["max"], np.maximum(l["max"], r["max"]))
