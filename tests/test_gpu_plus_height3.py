"""LBVH+ passes around the sizes where the way of the first heights changes: height 3 in one launch of the general DP
or one per treelet size, early or plain launches.  Each equals the oracle, bit for bit."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build

pytestmark = pytest.mark.gpu


def _edge(ctx):
    """The largest n whose height 3 takes the general DP: eight triangles for each of its lanes."""
    import torch
    return 8 * 32 * 8 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("at,rounds", [("edge - 1", 1), ("edge + 8", 1), ("edge - 1", 2), ("edge + 8", 2)])
def test_height_three(gpu, oracle_lib, at, rounds):
    ctx = Context(0)
    n = _edge(ctx) + (8 if "+" in at else -1)
    mesh = meshgen.uniform_small(n, seed=51)
    nodes, idx, _, _ = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=rounds))
    on, oi = oracle_lib.lbvh_plus(mesh.arrays(), 60, rounds)[:2]
    assert np.array_equal(idx, oi)
    assert oracle_lib.node_fields_equal(nodes, on)
    ctx.close()


@pytest.mark.parametrize("n", [1_999_999, 2_000_000])
def test_launches(gpu, oracle_lib, n):
    ctx = Context(0)
    mesh = meshgen.uniform_small(n, seed=52)
    nodes, idx, _, _ = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60))
    on, oi = oracle_lib.lbvh_plus(mesh.arrays(), 60, 1)[:2]
    assert np.array_equal(idx, oi)
    assert oracle_lib.node_fields_equal(nodes, on)
    ctx.close()
