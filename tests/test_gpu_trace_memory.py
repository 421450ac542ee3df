"""The scratch of large traces is counted, kept for the next ones, and given back: on request, and by itself once
the traces have become smaller."""
import numpy as np
import pytest

from bvh_gb300 import Context, meshgen, _capi as C
from tests.gpu_util import build, stream

pytestmark = pytest.mark.gpu
NR = 65_536
PIECE = 33 << 20  # the allocator's unit, and what lies beside the records


def _tracer(gpu, ctx, n):
    mesh = meshgen.uniform_small(n, seed=91)
    _, _, tree, ts = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH))
    nodes = gpu.empty(48 * tree.n_nodes, dtype=gpu.uint8, device="cuda")  # (a later build of the context reuses its own)
    host, _ = ctx.download(tree, stream(gpu))
    nodes.copy_(gpu.from_numpy(np.ascontiguousarray(host).view(np.uint8).reshape(-1).copy()))
    o, d = meshgen.sphere_rays(mesh, NR, 5)
    rays = [gpu.from_numpy(np.ascontiguousarray(a)).cuda() for a in np.concatenate([o, d], 1).astype(np.float32).T]
    out = [gpu.full((NR,), -7, dtype=gpu.float32 if k == 0 else gpu.int32, device="cuda") for k in range(5)]
    keep = (ts, nodes, rays, out)

    def run(k=1):
        for _ in range(k):
            ctx.trace(nodes.data_ptr(), tree.n_nodes, [t.data_ptr() for t in ts], n, [r.data_ptr() for r in rays], NR,
                      [t.data_ptr() for t in out], stream(gpu))
        gpu.cuda.synchronize()
        return [t.clone() for t in keep[3]]

    return run


def test_counted_and_given_back(gpu):
    ctx = Context(0)
    n = 500_000
    big, small = _tracer(gpu, ctx, n), _tracer(gpu, ctx, 20_000)
    records = 64 * (3 * n - 1)
    without = ctx.device_bytes()
    want = big()
    held = ctx.device_bytes()
    assert without + records <= held < without + records + PIECE
    big(3)
    assert ctx.device_bytes() == held  # kept, not added to
    free = gpu.cuda.mem_get_info()[0]
    ctx.trim()
    assert ctx.device_bytes() == without
    assert gpu.cuda.mem_get_info()[0] >= free + records - (4 << 20)
    assert all(gpu.equal(a, b) for a, b in zip(big(), want))
    assert ctx.device_bytes() == held
    first = small()
    assert ctx.device_bytes() == held  # one small trace among large ones gives nothing back
    small(32)
    assert ctx.device_bytes() <= without + PIECE
    assert all(gpu.equal(a, b) for a, b in zip(small(), first))
    assert all(gpu.equal(a, b) for a, b in zip(big(), want))
    ctx.trim()
    ctx.trim()
    assert ctx.device_bytes() == without
    ctx.close()


def test_buffers_are_counted(gpu):
    """What a context holds covers its result and input buffers and grows with each kind of build."""
    ctx = Context(0)
    n = 200_000
    m = meshgen.uniform_small(n, seed=92)
    before = ctx.device_bytes()
    build(ctx, gpu, m, ctx.params(C.ALGO_LBVH_PLUS, morton_bits=60))
    lbvh = ctx.device_bytes()
    assert lbvh - before >= n * (96 + 32 + 24 + 8 + 2)  # nodes, boxes, keys and values, rendezvous words, two byte arrays
    build(ctx, gpu, m, ctx.params(C.ALGO_PLOC))
    assert ctx.device_bytes() - lbvh >= n * (64 + 12)
    ctx.close()
