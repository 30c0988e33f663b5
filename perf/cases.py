"""The work that programs have this framework do, as cases that can be timed.

Every case goes through the public Python binding (a thin layer over the C ABI of include/cstone_gb300.h):

- "pipeline": one whole pass, keys -> sort -> gather -> leaf build -> link -> geometry [-> halos] -> neighbours;
- "steps":    one incremental time step of a moving, periodic set (graph replay, updateOctree from the last tree);
- "batch":    many independent uneven sets in one call;
- "host":     a whole pass from pinned host arrays with the neighbour lists returned to the host as CSR;
- "stages":   the drop-in stage calls one after the other, as a code that replaces the reference's calls one by one;
- "sort":     the stable key/index sort alone;
- "clusters": cluster-pair lists and an SPH density over them;
- "lists":    stored neighbour rows and an SPH density over them;
- "sources":  the tree operations of a gravity solver: counts and mass centres swept upwards, target groups.
"""
import math
import os
import sys
import types

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("cornerstone-octree_gb300"))
import cstone_gb300 as cs  # noqa: E402

DEV = "cuda:0"


def listed():
    return [
        # a small request of the served stream (its sizes begin at 2^12): launches and latency
        dict(name="pipeline small", kind="pipeline", n=4096, dist="uniform", coord=64, key=64, curve="hilbert",
             bucket=64, k=100, ngmax=200, halos=False, periodic=False),
        # a clustered FP32 set of odd size with the coarse 32-bit Morton keys, one of a per-set loop
        dict(name="pipeline f32 odd", kind="pipeline", n=120007, dist="plummer", coord=32, key=32, curve="morton",
             bucket=16, k=60, ngmax=100, halos=True, periodic=False),
        # the plain single-set build: 2^20 FP64 particles uniform in [-1, 1]^3, bucket 64, ngmax 150
        dict(name="pipeline uniform 1M", kind="pipeline", n=1 << 20, dist="uniform", coord=64, key=64,
             curve="hilbert", bucket=64, k=92, ngmax=150, halos=False, periodic=False),
        # the headline: the clustered full path with halos of the first quarter of the key space
        dict(name="pipeline plummer 16M", kind="pipeline", n=1 << 24, dist="plummer", coord=64, key=64,
             curve="hilbert", bucket=64, k=100, ngmax=200, halos=True, periodic=False),
        # time steps of a periodic FP32 box: Morton64, bucket 32, h = 1.2 spacings, noise of 0.1 spacings per step
        dict(name="steps 32M", kind="steps", n=1 << 25, ngmax=150, bucket=32),
        # uneven independent FP32 sets, log-uniform sizes, uniform and Plummer, about 60 neighbours
        dict(name="batch 128 sets", kind="batch", sets=128, ngmax=100),
        # a host program's pass: inputs copied in, lists copied out
        dict(name="host lists 500k", kind="host", n=500009, k=100, ngmax=200),
        # stage calls with double coordinates and float h, as the reference's <double, float> instantiations
        dict(name="stages 200k", kind="stages", n=200003, k=100, ngmax=150, bucket=64),
        # a particle reorder by 32-bit keys
        dict(name="sort u32 20M", kind="sort", n=20000003, key=32),
        # neighbour-list consumers
        dict(name="clusters f64 250k", kind="clusters", n=250001, coord=64, k=100),
        dict(name="lists f32 200k", kind="lists", n=200001, coord=32, k=60, ngmax=128),
        # gravity sources over a clustered set
        dict(name="sources 4M", kind="sources", n=4000037, coord=64, bucket=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pipeline"] * 4 + ["steps", "batch", "host", "stages", "sort", "clusters", "lists", "sources"])
    if kind == "pipeline":
        coord, dist = rng.choice([64, 64, 32]), rng.choice(["uniform", "plummer"])
        key = 64 if coord == 64 else rng.choice([64, 32])
        # 32-bit keys have ten levels only: dense cores need the small sets
        most = (1 << 17 if key == 32 else 1 << 20 if coord == 32 else 12000000) if dist == "plummer" else \
            (1 << 22 if key == 32 else 12000000)
        n = _log(rng, 4096, most)
        k = rng.choice([60, 92, 100])
        return dict(kind=kind, n=n, dist=dist, coord=coord, key=key, curve=rng.choice(["hilbert", "morton"]),
                    bucket=rng.choice([16, 32, 64]), k=k, ngmax=rng.choice([k + k // 2, 2 * k]),
                    halos=rng.random() < 0.5, periodic=dist == "uniform" and rng.random() < 0.3)
    if kind == "steps":
        return dict(kind=kind, n=_log(rng, 1 << 17, 1 << 25), ngmax=rng.choice([100, 150]),
                    bucket=rng.choice([32, 64]))
    if kind == "batch":
        return dict(kind=kind, sets=_log(rng, 4, 128), ngmax=100)
    if kind == "host":
        return dict(kind=kind, n=_log(rng, 1 << 14, 500009), k=rng.choice([60, 100]), ngmax=200)
    if kind == "stages":
        return dict(kind=kind, n=_log(rng, 1 << 12, 1 << 20), k=100, ngmax=150, bucket=rng.choice([16, 64]))
    if kind == "sort":
        return dict(kind=kind, n=_log(rng, 1 << 12, 20000003), key=rng.choice([32, 64]))
    if kind == "clusters":
        return dict(kind=kind, n=_log(rng, 1 << 14, 250001), coord=rng.choice([64, 32]), k=rng.choice([60, 100]))
    if kind == "lists":
        return dict(kind=kind, n=_log(rng, 1 << 14, 200001), coord=rng.choice([64, 32]), k=60, ngmax=128)
    return dict(kind=kind, n=_log(rng, 1 << 14, 4000037), coord=rng.choice([64, 32]), bucket=rng.choice([16, 64]))


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------

def _plummer(g, n):
    """scale radius 1, truncated at r = 100: positions and radii, FP64"""
    top = (1.0 + 1e-4) ** -1.5  # mass fraction within r = 100
    u = torch.rand(3, n, generator=g, device=DEV, dtype=torch.float64)
    r = 1.0 / torch.sqrt((u[0] * top).clamp_min(1e-300) ** (-2.0 / 3.0) - 1.0)
    z = (1.0 - 2.0 * u[1]) * r
    rho = torch.sqrt((r * r - z * z).clamp_min(0.0))
    phi = 2.0 * math.pi * u[2]
    return rho * torch.cos(phi), rho * torch.sin(phi), z, r


def _particles(g, n, dist, coord, k, side=2.0):
    """x, y, z, h (about k neighbours within 2 h) and the box's corners"""
    dt = torch.float64 if coord == 64 else torch.float32
    if dist == "uniform":
        x, y, z = (torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * side - side / 2 for _ in range(3))
        h = torch.full((n,), 0.5 * (3 * k * side ** 3 / (4 * math.pi * n)) ** (1 / 3), device=DEV, dtype=dt)
        return x.to(dt), y.to(dt), z.to(dt), h, (-side / 2,) * 3, (side / 2,) * 3
    x, y, z, r = _plummer(g, n)
    density = n * 3 / (4 * math.pi) * (1 + r * r) ** -2.5
    h = torch.minimum(0.5 * (3 * k / (4 * math.pi * density)) ** (1 / 3), 0.3 * r.clamp_min(1.0))
    x, y, z, h = x.to(dt), y.to(dt), z.to(dt), h.to(dt)
    return x, y, z, h, tuple(float(a.min()) for a in (x, y, z)), tuple(float(a.max()) for a in (x, y, z))


def _sorted_set(x, y, z, h, box, coord, bucket):
    """a program's tree and SFC-ordered particles, as owned tensors"""
    p = cs.Pipeline(coord, 64, cs.HILBERT, bucket, 0, 1.0, 1.0, False, False)
    r = p.run(x, y, z, h, box)
    o = {k: v.clone() for k, v in p.outputs().items()}
    torch.cuda.synchronize()
    o["tree"] = types.SimpleNamespace(num_leaves=r.num_leaves, num_nodes=r.num_nodes,
                                      child_offsets=o["child_offsets"], parents=o["parents"],
                                      internal_to_leaf=o["internal_to_leaf"])
    return o


def _tree_arrays(n, bucket, coord, key, halos=False):
    """a program's own arrays for a tree, of a capacity that does not depend on the particles (zero beyond the tree)"""
    L = 16 * (n // bucket) + 4096
    N = L + L // 7 + 1
    ct, kt = torch.float64 if coord == 64 else torch.float32, cs.key_dtype(key)
    shapes = dict(leaves=(L + 1, kt), counts=(L, torch.int32), prefixes=(N, kt), child_offsets=(N, torch.int32),
                  centers=((N, 3), ct), sizes=((N, 3), ct))
    if halos:
        shapes["halo_flags"] = (N, torch.uint8)
    return {k: torch.zeros(shape, dtype=dt, device=DEV) for k, (shape, dt) in shapes.items()}


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind, s = case["kind"], dict(case)
    if kind == "pipeline":
        x, y, z, h, lo, hi = _particles(g, case["n"], case["dist"], case["coord"], case["k"])
        s["in"] = (x, y, z, h)
        s["box"] = cs.make_box(lo, hi, cs.PERIODIC if case["periodic"] else cs.OPEN)
        top = 1 << (30 if case["key"] == 32 else 63)
        s["focus"] = (0, top // 4) if case["halos"] else (0, 0)
        s["pipe"] = cs.Pipeline(case["coord"], case["key"], cs.HILBERT if case["curve"] == "hilbert" else cs.MORTON,
                                case["bucket"], case["ngmax"], 1.0, 1.0, case["halos"], True)
        # the object's buffers are sized by its first run; the rows' unused tails are zero
        s["pipe"].run(*s["in"], s["box"], s["focus"])
        s["pipe"].outputs()["neighbors"].zero_()
        s["own"] = _tree_arrays(case["n"], case["bucket"], case["coord"], case["key"], case["halos"])
    elif kind == "steps":
        n, spacing = case["n"], case["n"] ** (-1.0 / 3)
        a = torch.rand(3, n, generator=g, device=DEV)
        b = a + torch.randn(3, n, generator=g, device=DEV) * (0.1 * spacing)
        b -= torch.floor(b)
        b[b >= 1.0] = 0.0
        s["h"] = torch.full((n,), 1.2 * spacing, device=DEV)
        s["at"], s["sets"] = 0, (a, b)
        s["box"] = cs.make_box(0.0, 1.0, cs.PERIODIC)
        s["pipe"] = cs.Pipeline(32, 64, cs.MORTON, case["bucket"], case["ngmax"], 1.0, 1.0, False, True)
        # the first step builds from the root; the next ones capture the two graphs of the leaf arrays' ping-pong
        for k in (0, 1, 0, 1):
            s["pipe"].step(*s["sets"][k], s["h"], s["box"], True)
        s["pipe"].outputs()["neighbors"].zero_()
        s["own"] = _tree_arrays(n, case["bucket"], 32, 64)
    elif kind == "batch":
        # the sets' sizes belong to the case: spread evenly over the logarithm, with a jitter, in random order
        rng = np.random.default_rng(case["sets"])
        u = (np.arange(case["sets"]) + rng.random(case["sets"])) / case["sets"]
        sizes = rng.permutation(np.floor(2.0 ** (10 + 10 * u)).astype(int))
        parts, boxes, s["buckets"] = [], [], [int(b) for b in rng.choice([16, 32, 64], case["sets"])]
        for k, n in enumerate(sizes):
            if k % 2 == 0:
                x, y, z, h, lo, hi = _particles(g, int(n), "uniform", 32, 60, 1.0)
            else:
                x, y, z, _, lo, hi = _particles(g, int(n), "plummer", 32, 60)
                # one h per set: about 60 neighbours at the mean density within the half-mass radius
                half = 1.0 / math.sqrt(0.5 ** (-2.0 / 3.0) - 1.0)
                h = torch.full((int(n),), 0.5 * (60 * 2 / n) ** (1 / 3) * half, device=DEV)
            parts.append((x, y, z, h))
            boxes.append(cs.make_box(lo, hi))
        s["in"] = [torch.cat([p[c] for p in parts]) for c in range(4)]
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)])
        s["boxes"] = boxes
        s["batch"] = cs.Batch(32, cs.MORTON, case["ngmax"])
        s["batch"].run(*s["in"], s["offsets"], s["boxes"], s["buckets"])
        s["batch"].outputs()["neighbors"].zero_()
        s["own"] = _tree_arrays(int(sizes.sum()) + 64 * case["sets"], 16, 32, 64)
        del s["own"]["child_offsets"]
    elif kind == "host":
        n = case["n"]
        x, y, z, h, lo, hi = _particles(g, n, "plummer", 64, case["k"])
        s["box"] = cs.make_box(lo, hi)
        s["pipe"] = cs.Pipeline(64, 64, cs.HILBERT, 64, case["ngmax"], 1.0, 1.0, True, True)
        s["in"] = [a.cpu().pin_memory() for a in (x, y, z, h)]
        s["out"] = dict(offsets=torch.zeros(n + 1, dtype=torch.int64).pin_memory(),
                        list=torch.zeros(n * (case["k"] + case["k"] // 4), dtype=torch.int32).pin_memory(),
                        counts=torch.zeros(n, dtype=torch.int32).pin_memory(),
                        flags=torch.zeros(n // 2 + 8192, dtype=torch.uint8).pin_memory())
        s["pipe"].run_host_csr(*s["in"], s["box"], (0, 1 << 61), *s["out"].values())
    elif kind == "stages":
        x, y, z, h, lo, hi = _particles(g, case["n"], "plummer", 64, case["k"])
        s["in"], s["box"] = (x, y, z, h.float()), cs.make_box(lo, hi)
        s["rows"] = (torch.zeros((case["n"], case["ngmax"]), dtype=torch.int32, device=DEV),
                     torch.zeros(case["n"], dtype=torch.int32, device=DEV))
        s["own"] = _tree_arrays(case["n"], case["bucket"], 64, 64, True)
    elif kind == "sort":
        bits, dt = (30, torch.int32) if case["key"] == 32 else (63, torch.int64)
        s["keys"] = torch.randint(0, (1 << bits) - 1, (case["n"],), generator=g, device=DEV, dtype=dt)
    elif kind in ("clusters", "lists"):
        x, y, z, h, lo, hi = _particles(g, case["n"], "uniform", case["coord"], case["k"])
        s["box"] = cs.make_box(lo, hi)
        s.update(_sorted_set(x, y, z, h, s["box"], case["coord"], 64))
        s["m"] = torch.rand(case["n"], generator=g, device=DEV, dtype=x.dtype) + 0.5
        if kind == "lists":
            s["rows"] = (torch.zeros((case["n"], case["ngmax"]), dtype=torch.int32, device=DEV),
                         torch.zeros(case["n"], dtype=torch.int32, device=DEV))
    else:
        x, y, z, h, lo, hi = _particles(g, case["n"], "plummer", case["coord"], 100)
        s["box"] = cs.make_box(lo, hi)
        s.update(_sorted_set(x, y, z, h, s["box"], case["coord"], case["bucket"]))
        s["m"] = torch.rand(case["n"], generator=g, device=DEV, dtype=x.dtype) + 0.5
        s["l2i"] = s["leaf_to_internal"][s["tree"].num_nodes - s["tree"].num_leaves:]
        # of a capacity that does not depend on the particles
        N = 18 * (case["n"] // case["bucket"]) + 8192
        s["node_counts"] = torch.zeros(N, dtype=torch.int32, device=DEV)
        s["node_centers"] = torch.zeros((N, 4), dtype=x.dtype, device=DEV)
        s["groups"] = torch.zeros(2 * (case["n"] // 64 + 2), dtype=torch.int32, device=DEV)
    return s


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------

PER_PARTICLE = ("sorted_keys", "order", "x", "y", "z", "h", "neighbors", "neighbor_counts")


def _keep(own, tree):
    """the tree into the program's own arrays"""
    for k, a in own.items():
        a[:tree[k].shape[0]].copy_(tree[k])
    return own


def _outputs(owner, own):
    """the object's results: views of its device memory per particle (which hold the object while any of them is
    held), and the tree"""
    o = owner.outputs()
    got = {k: o[k] for k in PER_PARTICLE if k in o}
    for a in got.values():
        a.owner = owner
    return {**got, **_keep(own, o)}


def run(s):
    kind = s["kind"]
    if kind == "pipeline":
        s["pipe"].run(*s["in"], s["box"], s["focus"])
        return _outputs(s["pipe"], s["own"])
    if kind == "steps":
        s["pipe"].step(*s["sets"][s["at"]], s["h"], s["box"], True)
        s["at"] ^= 1
        return _outputs(s["pipe"], s["own"])
    if kind == "batch":
        s["batch"].run(*s["in"], s["offsets"], s["boxes"], s["buckets"])
        return _outputs(s["batch"], s["own"])
    if kind == "host":
        o = s["out"]
        s["pipe"].run_host_csr(*s["in"], s["box"], (0, 1 << 61), o["offsets"], o["list"], o["counts"], o["flags"])
        return o
    if kind == "stages":
        x, y, z, h = s["in"]
        keys, order = cs.sort_pairs(cs.sfc_keys(x, y, z, s["box"]))
        x, y, z, h = (cs.gather(order, a) for a in (x, y, z, h))
        leaves, counts, layout, _ = cs.compute_octree(keys, s["bucket"])
        t = cs.build_octree(leaves)
        centers, sizes = cs.geo_centers(t.prefixes, s["box"])
        l2i = t.leaf_to_internal[t.num_internal:]
        last = t.num_leaves // 4
        sc, ss = cs.search_boxes(x, y, z, h, layout, 0, last, 2.0, l2i, centers)
        flags = cs.find_halos(t, centers, sizes, sc, ss, s["box"], 0, last)
        nb, nc = cs.find_neighbors(x, y, z, h, 0, s["n"], s["box"], t, layout, centers, sizes, s["ngmax"],
                                   out=s["rows"])
        tree = dict(leaves=leaves, counts=counts, prefixes=t.prefixes, child_offsets=t.child_offsets[:t.num_nodes],
                    centers=centers, sizes=sizes, halo_flags=flags)
        return dict(keys=keys, order=order, x=x, y=y, z=z, h=h, neighbors=nb, neighbor_counts=nc,
                    **_keep(s["own"], tree))
    if kind == "sort":
        return cs.sort_pairs(s["keys"].clone())
    if kind == "clusters":
        p = [s[c] for c in "xyzh"]
        lists, counts = cs.cluster_nblist(*p, s["box"], s["tree"], s["layout"], s["centers"], s["sizes"], 64, 512)
        return dict(counts=counts, rho=cs.ijloop_density_clusters(*p, s["m"], lists, counts))
    if kind == "lists":
        p = [s[c] for c in "xyzh"]
        nb, nc = cs.find_neighbors(*p, 0, s["n"], s["box"], s["tree"], s["layout"], s["centers"], s["sizes"],
                                   s["ngmax"], out=s["rows"])
        return dict(neighbors=nb, counts=nc, rho=cs.ijloop_density_list(*p, s["m"], s["box"], nb, nc))
    p, nc, cen = [s[c] for c in "xyz"], s["node_counts"], s["node_centers"]
    nc[s["l2i"].long()] = s["counts"]
    cs.upsweep_sum(s["child_offsets"], nc, s["parents"])
    cs.leaf_source_centers(*p, s["m"], s["l2i"], s["layout"], cen)
    cs.upsweep_source_centers(s["child_offsets"], cen, s["parents"])
    groups = cs.group_splits(0, s["n"], *p, s["h"], s["leaves"], s["layout"], s["box"], 64, 8.0)
    s["groups"][:groups.numel()].copy_(groups)
    return dict(node_counts=nc, centers=cen, groups=s["groups"])


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and its values in 64 bits
# ---------------------------------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = int(case["sets"] * 1023 * 1024 / (10 * math.log(2)))  # the mean of the log-uniform sizes
        return dict(bytes=n * (16 + 16 + 4 + 4 + 4 * 60), flops=8 * n * 60)
    n, t = case["n"], case.get("coord", 64) // 8
    if kind == "pipeline":
        # x, y, z, h in and sorted out, keys, order, counts, rows; the tree is small beside them
        return dict(bytes=n * (8 * t + case["key"] // 8 + 8 + 4 * case["k"]), flops=8 * n * case["k"])
    if kind == "steps":
        return dict(bytes=n * (32 + 8 + 8 + 4 * 57), flops=8 * n * 57)
    if kind == "host":
        return dict(bytes=n * (32 + 8 + 4 + 4 * case["k"]), flops=8 * n * case["k"])
    if kind == "stages":
        return dict(bytes=n * (28 + 28 + 8 + 8 + 4 * case["k"]), flops=8 * n * case["k"])
    if kind == "sort":
        return dict(bytes=n * (2 * case["key"] // 8 + 4), flops=0)
    if kind == "clusters":
        return dict(bytes=n * 6 * t, flops=20 * n * case["k"])
    if kind == "lists":
        return dict(bytes=n * (6 * t + 4 + 4 * case["k"]), flops=20 * n * case["k"])
    return dict(bytes=n * 5 * t, flops=8 * n)


def _density(s):
    """rho_i = h_i^-3 sum of m_j w(|x_i - x_j| / h_i) over |x_i - x_j| < 2 h_i, i itself among the j"""
    x = torch.stack([s[c].double() for c in "xyz"], 1)
    h, m, n = s["h"].double(), s["m"].double(), s["n"]
    # particles in cells of the largest 2 h; a cell's particles meet those of the 27 cells around it
    lo, edge = x.min(0).values, float(2 * h.max()) * (1 + 1e-9)
    c = ((x - lo) / edge).long()
    dims = c.max(0).values + 3
    ident = ((c[:, 0] + 1) * dims[1] + c[:, 1] + 1) * dims[2] + c[:, 2] + 1
    ident, order = torch.sort(ident)
    x, h2, m2 = x[order], h[order], m[order]
    rho = torch.zeros(n, dtype=torch.float64, device=x.device)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                other = ident + (dx * dims[1] + dy) * dims[2] + dz
                first, last = torch.searchsorted(ident, other), torch.searchsorted(ident, other, right=True)
                for k in range(int((last - first).max())):
                    j = (first + k).clamp_max(n - 1)
                    q = (x - x[j]).square().sum(1).sqrt() / h2
                    w = torch.where(q < 1, 1 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2 - q) ** 3)
                    rho += torch.where((first + k < last) & (q < 2), m2[j] * w, torch.zeros_like(w))
    out = torch.empty_like(rho)
    out[order] = rho / h2 ** 3
    return out


def _centers(s):
    """mass centres (x, y, z, mass) of every node: leaves from their particles, nodes from their eight children"""
    layout, m = s["layout"].long(), s["m"].double()
    leaf = torch.repeat_interleave(torch.arange(layout.numel() - 1, device=layout.device), layout.diff())
    per = torch.stack([s[c].double() * m for c in "xyz"] + [m], 1)
    nodes = torch.zeros_like(s["node_centers"], dtype=torch.float64)
    nodes[s["l2i"].long()] = torch.zeros((layout.numel() - 1, 4), dtype=torch.float64,
                                         device=layout.device).index_add_(0, leaf, per)
    child, ranges = s["child_offsets"].long(), s["level_range"].tolist()
    for level in range(len(ranges) - 2, -1, -1):
        at = torch.arange(ranges[level], max(ranges[level], ranges[level + 1]), device=layout.device)
        at = at[child[at] > 0]
        if at.numel():
            nodes[at] = nodes[child[at][:, None] + torch.arange(8, device=layout.device)].sum(1)
    nodes[:, :3] /= torch.where(nodes[:, 3:] > 0, nodes[:, 3:], torch.ones_like(nodes[:, 3:]))
    return nodes


def exact(case, seed):
    kind = case["kind"]
    if kind == "clusters":
        return dict(counts=None, rho=_density(prepare(case, seed)))
    if kind == "lists":
        return dict(neighbors=None, counts=None, rho=_density(prepare(case, seed)))
    if kind == "sources":
        return dict(node_counts=None, centers=_centers(prepare(case, seed)), groups=None)
    # the others return whole numbers, copies of their inputs and box corners of the tree that they built
    return None
