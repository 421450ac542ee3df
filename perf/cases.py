"""The work this library does for its users, as cases that can be timed.

A case is a dict of plain values; `prepare` makes what a program holds before the call (device
arrays, a context, a tree to trace), `run` makes one pass through the public entry points.  Four
kinds, each with the sizes its callers have:

  build    one mesh, device in, device tree out (Context.build_device): LBVH, LBVH+ or PLOC, from
           a served request's 1,000 triangles to the 10,000,000 of a large scene
  host     one mesh through the builder interface, host arrays in and out (LBVHBuilder.build)
  batch    many meshes of uneven size in one call (Context.build_batched), as for per-object trees
  rays     closest hits of explicit rays against a tree in hand (Context.trace)
  render   one image: primary rays, traversal and shading (Context.trace_pinhole, Context.shade)

Meshes follow bvh_gb300.meshgen's distributions, drawn on the device so that they are quick to
make: uniform small triangles, 64 Gaussian clusters, a displaced icosphere, thin strands.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import bvh_gb300
from bvh_gb300 import _capi as C

_ALGO = {"lbvh": C.ALGO_LBVH, "lbvhplus": C.ALGO_LBVH_PLUS, "ploc": C.ALGO_PLOC}


def _case(kind, mesh="uniform", n=0, algo="lbvh", bits=30, rounds=1, radius=25, packed=False, **more):
    return dict(kind=kind, mesh=mesh, n=n, algo=algo, bits=bits, rounds=rounds, radius=radius, packed=packed, **more)


def listed():
    return [
        # the smallest mesh a served build+trace request carries: launches and latency
        dict(_case("build", "clustered", 1000), name="lbvh30_1k"),
        # a plain LBVH of an ordinary object, rebuilt every frame
        dict(_case("build", "uniform", 100_000), name="lbvh30_100k"),
        # a whole large scene with long Morton codes
        dict(_case("build", "clustered", 10_000_000, bits=63), name="lbvh63_10m"),
        # the drop-in builder call: host arrays up, tree and indices down, a ragged size
        dict(_case("host", "uniform", 1_000_003), name="lbvh30_host_1m"),
        # LBVH+ as its builder runs it (60-bit, one pass), on nine rows of one upload buffer; with an
        # odd size those rows are not 16-byte aligned
        dict(_case("build", "clustered", 200_003, "lbvhplus", 60, packed=True), name="lbvhplus_200k"),
        # LBVH+ with three restructuring passes on a large scene, for a tree that is traced a lot
        dict(_case("build", "clustered", 10_000_000, "lbvhplus", 60, rounds=3), name="lbvhplus3_10m"),
        # PLOC of one object of a game-sized scene, a ragged size
        dict(_case("build", "strands", 20_011, "ploc"), name="ploc25_20k"),
        # PLOC of a whole large scene, default radius
        dict(_case("build", "clustered", 10_000_000, "ploc"), name="ploc25_10m"),
        # PLOC with the widest radius in use, on a closed surface
        dict(_case("build", "icosphere", 1_310_720, "ploc", radius=100), name="ploc100_1m"),
        # one tree per object for a scene of 1,024 objects of 64 to 262,144 triangles
        dict(_case("batch", meshes=1024), name="batch_lbvh30_1024"),
        # incoherent rays against thin geometry: tree quality as it is measured, 1M rays
        dict(_case("rays", "strands", 2_000_000, "lbvhplus", 60, rays=1_000_000), name="rays_strands_1m"),
        # a full-HD image of the large scene: coherent primary rays and diffuse shading
        dict(_case("render", "clustered", 10_000_000, bits=63, width=1920, height=1080), name="render_1080p"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_tree(rng, lo, hi):
    """A mesh and the algorithm that builds its tree."""
    mesh = rng.choice(("uniform", "clustered", "clustered", "strands", "icosphere"))
    n = 20 * 4 ** rng.randint(3, 8) if mesh == "icosphere" else _log_int(rng, lo, hi)
    algo = rng.choice(("lbvh", "lbvh", "lbvhplus", "ploc"))
    bits = rng.choice((30, 60, 63)) if algo == "lbvh" else 60 if algo == "lbvhplus" else 30
    return _case("build", mesh, min(n, hi), algo, bits, rng.choice((1, 1, 3)), rng.choice((10, 25, 25, 100)),
                 rng.random() < 0.25)


def draw(rng):
    kind = rng.choice(("build",) * 5 + ("host", "batch", "rays", "render"))
    if kind == "build":
        return _draw_tree(rng, 1000, 10_000_000)
    if kind == "host":
        c = _draw_tree(rng, 1000, 1_000_003)
        return dict(c, kind="host", mesh="uniform" if c["mesh"] == "icosphere" else c["mesh"], algo="lbvh",
                    bits=rng.choice((30, 60, 63)))
    if kind == "batch":
        return _case("batch", algo=rng.choice(("lbvh", "lbvh", "ploc")), meshes=_log_int(rng, 32, 1024))
    if kind == "rays":
        c = _draw_tree(rng, 1000, 2_000_000)
        if c["mesh"] == "strands":  # a plain LBVH of strands is not what its users trace
            c = dict(c, algo="lbvhplus", bits=60, rounds=1)
        return dict(c, kind="rays", rays=_log_int(rng, 16_384, 1_000_000))
    c = _draw_tree(rng, 1000, 10_000_000)
    if c["mesh"] == "strands":
        c = dict(c, mesh="clustered")
    w = _log_int(rng, 160, 1920)
    return dict(c, kind="render", width=w, height=max(1, w * 9 // 16))


# ---- inputs ---------------------------------------------------------------------------------
def _dirs(g, n):
    d = torch.randn((n, 3), generator=g, device="cuda")
    return d / d.norm(dim=1, keepdim=True).clamp_min(1e-20)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _uniform(n, g):
    c = _rand(g, n, 3)
    return [c + (_rand(g, n, 3) - 0.5) * 0.01 for _ in range(3)]


def _clustered(n, g):
    means = _rand(g, 64, 3)
    c = means[torch.randint(0, 64, (n,), generator=g, device="cuda")]
    c = c + torch.randn((n, 3), generator=g, device="cuda") * 0.02
    edge = torch.exp(_rand(g, n, 1) * math.log(1e2) + math.log(1e-4))
    return [c + _dirs(g, n) * edge for _ in range(3)]


def _strands(n, g, segments=100):
    s = (n + segments - 1) // segments
    start = _rand(g, s, 1, 3)
    p = start + torch.cumsum(_dirs(g, s * segments).view(s, segments, 3) * 0.01, 1)
    p = torch.cat([start, p], 1).abs()
    p = torch.where(p > 1, 2 - p, p).clamp(0, 1)
    a, b = p[:, :-1].reshape(-1, 3)[:n], p[:, 1:].reshape(-1, 3)[:n]
    side = torch.linalg.cross(b - a, _dirs(g, n))
    return [a, b, a + side / side.norm(dim=1, keepdim=True).clamp_min(1e-20) * 1e-4]


def _icosphere(n, g):
    t = (1 + 5 ** 0.5) / 2
    v = torch.tensor([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t],
                      [0, 1, -t], [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]], dtype=torch.float64, device="cuda")
    f = torch.tensor([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4],
                      [11, 10, 2], [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8],
                      [3, 8, 9], [4, 9, 5], [2, 4, 11], [6, 2, 10], [8, 6, 7], [9, 8, 1]], device="cuda")
    tri = (v / v.norm(dim=1, keepdim=True))[f]
    while tri.shape[0] < n:
        a, b, c = tri.unbind(1)
        ab, bc, ca = ((x / x.norm(dim=1, keepdim=True)) for x in (a + b, b + c, c + a))
        tri = torch.stack([torch.stack(q, 1) for q in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))], 1)
        tri = tri.reshape(-1, 3, 3)
    r = 1.0
    for octave in range(4):  # smooth radial displacement, the same for shared corners
        k = _dirs(g, 1).double()[0] * 4 * 2 ** octave
        r = r + 0.025 * 0.5 ** octave * torch.sin((tri * k).sum(-1, keepdim=True) * math.pi)
    return [x.contiguous() for x in (tri[:n] * r).float().unbind(1)]


_MESHES = {"uniform": _uniform, "clustered": _clustered, "strands": _strands, "icosphere": _icosphere}


def _counts(case):
    """A batch's layout belongs to its case; the seed draws the geometry in it."""
    g = np.random.default_rng(case["meshes"])
    return np.exp(g.uniform(math.log(64), math.log(262_144), case["meshes"])).astype(np.int64)


def _soa(case, seed):
    """The nine device arrays of a case, as rows of one (9, n) tensor or each on its own."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "batch":
        counts = torch.from_numpy(_counts(case)).cuda()
        v = _uniform(int(counts.sum()), g)
        scale = torch.repeat_interleave(torch.exp((_rand(g, len(counts), 1) * 2 - 1) * math.log(10)), counts, 0)
        shift = torch.repeat_interleave(_rand(g, len(counts), 3) * 20 - 10, counts, 0)
        v = [x * scale + shift for x in v]
    else:
        v = _MESHES[case["mesh"]](case["n"], g)
    rows = [v[k // 3][:, k % 3] for k in range(9)]
    return list(torch.stack(rows)) if case["packed"] else [r.contiguous() for r in rows]


def _params(ctx, case):
    return ctx.params(_ALGO[case["algo"]], morton_bits=case["bits"], treelet_rounds=case["rounds"],
                      ploc_radius=case["radius"])


class _Device:
    """A device allocation of a context as torch sees it; it keeps the context, which owns the memory."""

    def __init__(self, ctx, ptr, shape, typestr):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _tree_views(ctx, tree):
    """min, max, (left, right) and the sorted triangle indices of a device tree, without a copy."""
    nodes = torch.as_tensor(_Device(ctx, tree.nodes, (tree.n_nodes, 12), "<f4"), device="cuda")
    index = torch.as_tensor(_Device(ctx, tree.indices, (tree.n_prims,), "<i4"), device="cuda")
    return {"min": nodes[:, 0:3], "max": nodes[:, 4:7], "children": nodes.view(torch.int32)[:, 8:10],
            "indices": index}


def _rays(case, soa, seed):
    """Origins on a sphere around the scene, directions towards points inside its box."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    lo = torch.stack([torch.stack([soa[k].min() for k in (a, a + 3, a + 6)]).min() for a in range(3)])
    hi = torch.stack([torch.stack([soa[k].max() for k in (a, a + 3, a + 6)]).max() for a in range(3)])
    o = (lo + hi) / 2 + _dirs(g, case["rays"]) * (1.5 * (hi - lo).norm() / 2)
    d = lo + _rand(g, case["rays"], 3) * (hi - lo) - o
    d = d / d.norm(dim=1, keepdim=True)
    return [x[:, k].contiguous() for x in (o, d) for k in range(3)]


def prepare(case, seed):
    soa = _soa(case, seed)
    st = {"case": case, "n": soa[0].shape[0]}
    if case["kind"] == "host":
        st["builder"] = bvh_gb300.LBVHBuilder(morton_bits=case["bits"])
        st["mesh"] = bvh_gb300.TriangleMesh(*[a.cpu().numpy() for a in soa])
        return st
    ctx = bvh_gb300.Context(0)
    stream = torch.cuda.current_stream().cuda_stream
    st.update(ctx=ctx, soa=soa, ptrs=[a.data_ptr() for a in soa], stream=stream, params=_params(ctx, case), views={})
    ctx.reserve(st["n"], _ALGO[case["algo"]])
    if case["kind"] == "batch":
        st["offsets"] = np.concatenate([[0], np.cumsum(_counts(case))]).astype(np.uint32)
    if case["kind"] in ("rays", "render"):
        st["tree"] = tree = ctx.build_device(st["ptrs"], st["n"], st["params"], stream)
        ctx.sync()
        count = case["rays"] if case["kind"] == "rays" else case["width"] * case["height"]
        hits = [torch.empty(count, dtype=torch.float32 if k == 0 else torch.int32, device="cuda") for k in range(5)]
        st["hits"] = dict(zip(("t", "prim", "nodes_visited", "aabb_tests", "tri_tests"), hits))
        st["hit_ptrs"] = [h.data_ptr() for h in hits]
        if case["kind"] == "rays":
            st["rays"] = _rays(case, soa, seed)
            st["ray_ptrs"] = [r.data_ptr() for r in st["rays"]]
        else:
            root = torch.as_tensor(_Device(ctx, tree.nodes, (12,), "<f4"), device="cuda").cpu().numpy()
            st["camera"] = bvh_gb300.auto_camera(root.view(C.NODE_DTYPE)[0])
            st["diag"] = float(np.linalg.norm(root[4:7] - root[0:3]))
            st["rgb"] = torch.empty(3 * count, device="cuda")
    return st


# ---- one pass -------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "host":
        b = st["builder"]
        b.build(st["mesh"])
        nodes = b.getNodes()
        return {"min": nodes["min"], "max": nodes["max"], "left": nodes["left"], "right": nodes["right"],
                "indices": b.getIndices()}
    ctx = st["ctx"]
    if kind in ("build", "batch"):
        if kind == "build":
            tree = ctx.build_device(st["ptrs"], st["n"], st["params"], st["stream"])
        else:
            tree = ctx.build_batched(st["ptrs"], st["offsets"], st["params"], st["stream"])
        key = (tree.nodes, tree.indices)
        if key not in st["views"]:  # a program maps the context's buffers once, not on every build
            st["views"] = {key: _tree_views(ctx, tree)}
        return st["views"][key]
    tree = st["tree"]
    if kind == "rays":
        ctx.trace(tree.nodes, tree.n_nodes, st["ptrs"], st["n"], st["ray_ptrs"], case["rays"], st["hit_ptrs"],
                  st["stream"])
        return st["hits"]
    ctx.trace_pinhole(tree.nodes, tree.n_nodes, st["ptrs"], st["n"], st["camera"], case["width"], case["height"],
                      st["hit_ptrs"], st["stream"])
    ctx.shade(st["ptrs"], st["n"], st["camera"], case["width"], case["height"], st["hit_ptrs"], 2, st["diag"],
              (0.267261, 0.801784, 0.534522), st["rgb"].data_ptr(), st["stream"])
    return dict(st["hits"], rgb=st["rgb"])


# ---- what a pass cannot do without ----------------------------------------------------------
def work(case):
    """Input read once, output written once.  Arithmetic: 30 operations per triangle for its box,
    centroid and code and 6 per merged box; PLOC adds 14 per pair of the first search and its halving
    successors (a union's area and a compare); LBVH+ adds, per inner node and pass, the areas of a
    7-leaf treelet's 127 subsets (14 each) and a cost and compare for each of their 966 splits; a ray
    two box tests of 20 operations per level of its tree and one triangle test of 60."""
    kind = case["kind"]
    n = case["n"] if kind != "batch" else int(_counts(case).sum())
    if kind in ("rays", "render"):
        count = case["rays"] if kind == "rays" else case["width"] * case["height"]
        depth = math.ceil(math.log2(max(n, 2)))
        tree = min(96 * n + 36 * n, count * (2 * depth * 48 + 36))
        return {"bytes": tree + count * ((24 + 20) if kind == "rays" else (20 + 12)),
                "flops": count * (2 * depth * 20 + 60)}
    flops = 36 * n
    if case["algo"] == "ploc":
        flops += 2 * n * case["radius"] * 14
    if case["algo"] == "lbvhplus":
        flops += case["rounds"] * n * (127 * 14 + 966 * 2)
    return {"bytes": (36 + 96 + 4) * n, "flops": flops}


# ---- the same in plain torch ----------------------------------------------------------------
def _spread(v, bits):
    out = torch.zeros_like(v)
    for b in range(bits):
        out |= ((v >> b) & 1) << (3 * b)
    return out


def _bit_length(x):
    out = torch.zeros_like(x)
    for s in (32, 16, 8, 4, 2, 1):
        big = (x >> s) > 0
        out += big * s
        x = torch.where(big, x >> s, x)
    return out + (x > 0)


def _exact_lbvh(soa, offsets, bits):
    """The linear BVH of each mesh [offsets[m], offsets[m+1]): Morton order, the radix tree over it and
    its boxes.  The Morton grid is defined on 32-bit arithmetic, so codes are made in it; what is
    computed from them (orders, ranges, minima and maxima) is exact."""
    n = soa[0].shape[0]
    off = torch.as_tensor(np.asarray(offsets, np.int64), device="cuda")
    count = off[1:] - off[:-1]
    mesh = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    start = off[mesh]
    lo = torch.stack([torch.minimum(torch.minimum(soa[a], soa[a + 3]), soa[a + 6]) for a in range(3)])
    hi = torch.stack([torch.maximum(torch.maximum(soa[a], soa[a + 3]), soa[a + 6]) for a in range(3)])
    code = torch.zeros(n, dtype=torch.int64, device="cuda")
    per = bits // 3
    for a in range(3):
        mn = torch.empty(len(count), device="cuda").scatter_reduce(0, mesh, lo[a], "amin", include_self=False)
        mx = torch.empty(len(count), device="cuda").scatter_reduce(0, mesh, hi[a], "amax", include_self=False)
        ext = torch.where(mx - mn > 1e-6, mx - mn, torch.ones_like(mn))
        x = ((lo[a] + hi[a]) * 0.5 - mn[mesh]) / ext[mesh]
        x = (x * float(2 ** per)).clamp(0.0, float(2 ** per - 1)).to(torch.int64)
        code |= _spread(x, per) << (2 - a if bits == 30 else a)
    order = torch.sort(code, stable=True).indices
    order = order[torch.sort(mesh[order], stable=True).indices]
    code, index = code[order], (order - start[order])
    # how unlike neighbours k and k + 1 are: the highest bit their codes (or, for equal codes, their
    # indices) differ in; across meshes, more than anything
    step = torch.where(code[1:] == code[:-1], _bit_length(index[1:] ^ index[:-1]),
                       _bit_length(code[1:] ^ code[:-1]) + 32)
    step = torch.where(mesh[1:] == mesh[:-1], step, torch.full_like(step, 200))
    wall = torch.full((1,), 200, dtype=torch.int64, device="cuda")
    step = torch.cat([wall, step, wall])  # step[k + 1] lies between sorted positions k and k + 1
    at = torch.arange(n, device="cuda")
    first = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    last = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    for v in torch.unique(step).tolist():
        if v == 200:
            continue
        walls = torch.nonzero(step > v).flatten()
        here = torch.nonzero(step == v).flatten()
        k = torch.searchsorted(walls, here)  # the node split at `here` lies between the walls around it
        first[here] = walls[k - 1]
        last[here] = walls[k] - 1
    k = torch.nonzero(step[1:n] < 200).flatten() + 1  # inner nodes by the wall they straddle
    f, l, split, m = first[k], last[k], k - 1, mesh[k]
    base, o = 2 * off[m] - m, off[m]
    left_side = step[l + 1] < step[f]
    root = (step[l + 1] == 200) & (step[f] == 200)
    row = base + torch.where(root, 0, torch.where(left_side, l, f) - o)
    leaf_row = 2 * start - mesh + count[mesh] - 1 + (at - start)
    children = torch.full((2 * n - len(count), 2), -1, dtype=torch.int64, device="cuda")
    children[leaf_row, 0] = index - 2 ** 31
    children[row, 0] = torch.where(f == split, count[m] - 1, 0) + split - o
    children[row, 1] = torch.where(l == split + 1, count[m] - 1, 0) + split + 1 - o
    out = {}
    size = _bit_length(l - f + 1) - 1
    for name, box, op in (("min", lo, torch.minimum), ("max", hi, torch.maximum)):
        res = torch.empty((children.shape[0], 3), dtype=torch.float64, device="cuda")
        for a in range(3):
            table = box[a][order].double()
            res[leaf_row, a] = table
            for j in range(int(size.max()) + 1 if len(size) else 0):
                if j:
                    h = 1 << (j - 1)
                    table = torch.cat([op(table[:-h], table[h:]), table[-h:]])
                sel = torch.nonzero(size == j).flatten()
                res[row[sel], a] = op(table[f[sel]], table[l[sel] + 1 - (1 << j)])
        out[name] = res
    return out, children, index


def _exact_rays(case, seed):
    """Closest hits by testing every triangle, in 64 bits."""
    soa = _soa(case, seed)
    rays = [r.double() for r in _rays(case, soa, seed)]
    v = [torch.stack([x.double() for x in soa[3 * k:3 * k + 3]], -1) for k in range(3)]
    e1, e2 = v[1] - v[0], v[2] - v[0]
    best = torch.full((case["rays"],), 1e30, dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // case["n"])
    for b in range(0, case["rays"], step):
        o = torch.stack([r[b:b + step] for r in rays[:3]], -1)[:, None]
        d = torch.stack([r[b:b + step] for r in rays[3:]], -1)[:, None]
        p = torch.linalg.cross(d.expand(-1, case["n"], -1), e2[None].expand(d.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        t0 = o - v[0]
        u = (t0 * p).sum(-1) / det
        q = torch.linalg.cross(t0, e1[None].expand_as(t0))
        w = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (det.abs() >= 1e-6) & (u >= -1e-5) & (u <= 1.00001) & (w >= -1e-5) & (u + w <= 1.00001) & (t >= 1e-6)
        best[b:b + step] = torch.where(ok, t, 1e30).min(1).values
    return best


def exact(case, seed):
    """Trees of plain LBVH builds, and hit distances where every ray can be tested against every
    triangle.  PLOC's and LBVH+'s topology follows from comparing 32-bit areas and has no value of its
    own in 64 bits."""
    if case["kind"] == "rays" and case["rays"] * case["n"] <= 5_000_000_000:
        return {"t": _exact_rays(case, seed), "prim": None, "nodes_visited": None, "aabb_tests": None,
                "tri_tests": None}
    if case["algo"] != "lbvh" or case["kind"] in ("rays", "render"):
        return None
    soa = _soa(case, seed)
    n = soa[0].shape[0]
    offsets = [0, n]
    if case["kind"] == "batch":
        offsets = np.concatenate([[0], np.cumsum(_counts(case))])
    box, children, index = _exact_lbvh(soa, offsets, case["bits"])
    if case["kind"] == "host":
        return {"min": box["min"], "max": box["max"], "left": children[:, 0], "right": children[:, 1],
                "indices": index}
    return {"min": box["min"], "max": box["max"], "children": children, "indices": index}
