"""Large traces of which few rays, or none, enter the scene: whether the tree is repacked for them or walked as it
is, the hits and counters are the oracle's, bit for bit."""
import numpy as np
import pytest

from bvh_gb300 import Context, auto_camera, meshgen, _capi as C
from tests.gpu_util import build, stream
from tests.test_gpu_trace_packed import NR, _chain, _check, _rays, _trace

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    c = Context(0)
    yield c
    c.close()


def _some(mesh, n, enter, seed=11):
    """Rays that point away from the scene but for those of the index array `enter`."""
    rays = _rays(mesh, n, seed)
    o, d = rays[:, :3], rays[:, 3:]
    away = np.ones(n, bool)
    away[enter] = False
    d[:7] = d[7]  # (no special directions)
    o[:7] = o[7]
    center = o.mean(0)
    d[away] = o[away] - center
    return rays


@pytest.mark.parametrize("nr", [NR, 20_011, 70_000])
@pytest.mark.parametrize("enter", ["none", "first", "last", "one", "few", "half", "all"])
@pytest.mark.parametrize("n", [2, 300, 20_011])
def test_few_rays_enter(ctx, gpu, oracle_lib, nr, enter, n):
    mesh = meshgen.clustered(n, seed=82)
    nodes, _, _ = oracle_lib.lbvh(mesh.arrays(), 30)
    g = np.random.Generator(np.random.PCG64(nr))
    idx = {"none": [], "first": [0], "last": [nr - 1], "one": [nr // 3], "few": g.choice(nr, 9, False),
           "half": np.arange(nr // 2), "all": np.arange(nr)}[enter]
    rays = _some(mesh, nr, idx)
    got = _check(ctx, gpu, oracle_lib, nodes, mesh, rays)
    if enter in ("one", "few"):  # (_check's oracle sees the first 2,000 rays: these as well)
        want = oracle_lib.trace(nodes, mesh.arrays(), rays[idx, :3], rays[idx, 3:])
        for a, e in zip(got, want):
            assert np.array_equal(a[idx], e.view(np.uint32))
    if enter == "none":
        assert (got[2] == 1).all() and (got[1] == np.uint32(0xFFFFFFFF)).all()


def test_walked_as_it_is_below_the_stack(ctx, gpu, oracle_lib):
    """Depth 399 with one entering ray in 16,384: dropped pushes without records."""
    mesh = meshgen.uniform_small(400, seed=3)
    for turn in (lambda i: True, lambda i: False, lambda i: i % 3 != 0, lambda i: i < 128):
        nodes = _chain(400, turn)
        for k in (5, 9_000):
            rays = _rays(mesh, NR, 6)
            rays[:, :3] = 50.0
            rays[:, 3:] = np.array([0.6, 0.64, 0.48], np.float32)
            rays[k] = _rays(mesh, NR, 6)[k]
            _check(ctx, gpu, oracle_lib, nodes, mesh, rays)


@pytest.mark.parametrize("w,h", [(256, 256), (641, 27), (3, 7001)])
@pytest.mark.parametrize("view", ["away", "corner"])
def test_images(ctx, gpu, w, h, view):
    from bvh_gb300.builders import pinhole_rays
    mesh = meshgen.clustered(20_000, seed=83)
    nodes, _, tree, ts = build(ctx, gpu, mesh, ctx.params(C.ALGO_LBVH))
    ptrs = [t.data_ptr() for t in ts]
    cam = auto_camera(nodes[0])
    for k in range(3):
        if view == "away":
            cam.look_at[k] = 2 * cam.eye[k] - cam.look_at[k]
        else:
            cam.look_at[k] += (1.9, -0.6, 1.1)[k]
    n = w * h
    out = [gpu.full((n,), -7, dtype=gpu.float32 if k == 0 else gpu.int32, device="cuda") for k in range(5)]
    ctx.trace_pinhole(tree.nodes, tree.n_nodes, ptrs, mesh.size(), cam, w, h, [t.data_ptr() for t in out], stream(gpu))
    rays = [gpu.empty(n, device="cuda") for _ in range(6)]
    pinhole_rays(cam, w, h, [t.data_ptr() for t in rays], stream(gpu))
    gpu.cuda.synchronize()
    plain = _trace(ctx, gpu, tree.nodes, tree.n_nodes, ptrs, mesh.size(), gpu.stack(rays, 1).cpu().numpy(), NR - 1)
    for a, b in zip(out, plain):
        assert np.array_equal(a.cpu().numpy().view(np.uint32), b)
    if view == "away":
        assert int(out[2].max()) == 1
