"""Emission's wait for an announced node gives up and reports it; the tree it leaves cannot be walked into what is
missing, no treelet pass follows its links, and builds afterwards are whole."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [1, 2, 5_000])
def test_emission_gives_up(gpu, oracle_lib, polls):
    lib = C.load_library()
    for _ in range(2):  # (the second run starts from what the first one left)
        assert lib.bvh_selftest_bounded_wait(0, polls) == C.BVH_ERR_TIMEOUT
    ctx = Context(0)
    m = meshgen.uniform_small(9_001, seed=81)
    for rounds in (1, 3):
        nodes, idx, _, _ = build(ctx, gpu, m, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60, treelet_rounds=rounds))
        on, oi = oracle_lib.lbvh_plus(m.arrays(), 60, rounds)
        assert np.array_equal(idx, oi) and oracle_lib.node_fields_equal(nodes, on)
    ctx.close()
