"""GPU parity of the tiled neighbour search (32 targets x 32 candidates per tensor-core tile) at the places where it can
go wrong: sets that end inside a warp or a tile, rows that fill up inside a tile, targets too spread or with radii too
different for a tile, particles at one point or exactly at the radius, sets far from the origin, coarse keys (most
particles outside their leaf's box) and cell radii below and above the search radius. Counts and lists equal the oracle's
exactly; the smaller groups of the tuning take the other kernel and must agree too."""
import numpy as np
import pytest
import torch

from gpu_util import neighbor_lists_equal, to_dev, u32, uniform

pytestmark = pytest.mark.gpu


def _check(cs, O, x, y, z, h, bucket, ngmax, kind=1, bits=64, ext=1.0, lo=None, hi=None, bnd=0):
    lo = lo if lo is not None else [float(a.min()) - 1e-3 for a in (x, y, z)]
    hi = hi if hi is not None else [float(a.max()) + 1e-3 for a in (x, y, z)]
    ref = O.pipeline(x, y, z, h, O.make_box(lo, hi, bnd), bucket, ngmax, kind, bits, ext)
    p = cs.Pipeline(64 if x.dtype == np.float64 else 32, bits, kind, bucket, ngmax, ext, 1.0, False, True)
    t = to_dev(x, y, z, h)
    for group in (32, 16):
        p.set_tuning(group, 7)
        p.run(*t, cs.make_box(lo, hi, bnd))
        out = p.outputs()
        torch.cuda.synchronize()
        neighbor_lists_equal(u32(out["neighbors"]).reshape(-1, ngmax), u32(out["neighbor_counts"]), ref["nb"], ref["nc"],
                             ngmax)
    return ref["nc"]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 96, 97, 500, 4100])
def test_sizes_around_warps_and_tiles(cs, O, n, dtype):
    x, y, z = uniform(O, 100 + n, n, -1.0, 1.0, dtype)
    h = np.full(n, 0.5 * (3 * 40 * 8 / (4 * np.pi * max(n, 60))) ** (1 / 3), dtype)
    _check(cs, O, x, y, z, h, 8, 64)


@pytest.mark.parametrize("ngmax", [1, 7, 32, 33])
def test_rows_that_fill_up(cs, O, ngmax):
    x, y, z = uniform(O, 5, 1500, -1.0, 1.0)
    nc = _check(cs, O, x, y, z, np.full(1500, 0.25), 16, ngmax)
    assert nc.max() > ngmax
    assert _check(cs, O, x, y, z, np.full(1500, 4.0), 16, ngmax).min() == 1499  # everything is a neighbour


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_radii_and_spreads_beyond_a_tile(cs, O, dtype):
    rng = np.random.default_rng(3)
    n = 6000
    x, y, z = uniform(O, 7, n, -1.0, 1.0, dtype)
    h = (0.05 * 10.0 ** rng.uniform(-2.5, 0.5, n)).astype(dtype)
    h[::97] = 0.0
    _check(cs, O, x, y, z, h, 16, 100)
    # clumps far apart along a Morton curve, radii of the clumps' size
    c = rng.integers(0, 40, n)
    centres = rng.uniform(-50.0, 50.0, (3, 40))
    x, y, z = ((centres[k][c] + rng.normal(0, 0.01, n)).astype(dtype) for k in range(3))
    _check(cs, O, x, y, z, np.full(n, 0.004, dtype), 16, 100, kind=0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_coincident_particles_and_pairs_at_the_radius(cs, O, dtype):
    rng = np.random.default_rng(4)
    pts = rng.uniform(-1.0, 1.0, (5, 3))
    x, y, z = (pts[rng.integers(0, 5, 700)][:, k].astype(dtype) for k in range(3))
    _check(cs, O, x, y, z, np.full(700, 1e-3, dtype), 64, 200)
    # a lattice whose spacing is the radius, and one whose face diagonal nearly is (strict <)
    g = np.arange(16) / 8.0
    x, y, z = (a.reshape(-1).astype(dtype) for a in np.meshgrid(g, g, g, indexing="ij"))
    for r in (0.125, np.nextafter(dtype(0.125), dtype(1)), 0.125 * np.sqrt(2.0), 0.25):
        _check(cs, O, x, y, z, np.full(x.size, dtype(r) / dtype(2), dtype), 16, 64, lo=(0, 0, 0), hi=(2, 2, 2))


@pytest.mark.parametrize("offset", [1e3, 1e6, -3e8])
def test_sets_far_from_the_origin(cs, O, offset):
    x, y, z = uniform(O, 9, 3000, 0.0, 1.0)
    h = np.full(3000, 0.06)
    _check(cs, O, x + offset, y - offset, z + 2 * offset, h, 16, 100)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("ext", [0.8, 1.0, 1.3])
def test_coarse_keys_and_cell_radii(cs, O, kind, ext):
    n = 30000
    x, y, z = (a.astype(np.float32) for a in O.plummer(31, n))
    lo, hi = [float(a.min()) for a in (x, y, z)], [float(a.max()) for a in (x, y, z)]
    _check(cs, O, x, y, z, np.full(n, 0.06, np.float32), 16, 100, kind, 32, ext, lo, hi)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bnd", [1, (1, 0, 0), (0, 1, 1)])
@pytest.mark.parametrize("reach", [0.01, 0.05, 0.11, 0.3])
def test_periodic_boundaries(cs, O, reach, bnd, dtype):
    """Spheres across faces, edges and corners: folded tiles for the small ones, the path kernel for warps that reach too
    far for one image, both in the larger ones. A part of the particles sits on the faces."""
    n = 8000
    x, y, z = uniform(O, 41, n, -1.0, 2.0, dtype)
    x[::50], y[7::50], z[9::50], x[11::50] = -1, 2, -1, 2
    h = (3.0 * reach / 2 * (0.2 + 0.8 * O.philox_uniform(42, 0, n, 0.0, 1.0))).astype(dtype)
    for kind, bits in ((1, 64), (0, 64)) + (((0, 32),) if dtype == np.float32 else ()):
        _check(cs, O, x, y, z, h, 16, 300, kind, bits, 1.0, (-1.0,) * 3, (2.0,) * 3, bnd)
    # a set in the corners of a box far from the origin: the period is large against the radii
    c = (O.philox_uniform(43, 0, 3 * n, 0.0, 1.0).reshape(3, n) - 0.5) * 0.4
    x, y, z = (np.where(v < 0, v + 1000.0, v).astype(dtype) for v in c)
    _check(cs, O, x, y, z, np.full(n, reach * 0.2, dtype), 16, 300, 1, 64, 1.0, (0.0,) * 3, (1000.0,) * 3, bnd)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("first,last", [(0, 33), (37, 6990), (1000, 1001), (6999, 7000)])
@pytest.mark.parametrize("reach", [0.05, 0.3])
def test_periodic_ranges_with_stale_counts(cs, O, reach, first, last, dtype):
    """Which blocks of 32 the periodic kernels serve is marked in the counts: ranges that begin and end inside a block,
    into count arrays full of that mark."""
    n = 7000
    x, y, z = uniform(O, 51, n, -1.0, 1.0, dtype)
    obox, box = O.make_box(-1.0, 1.0, 1), cs.make_box(-1.0, 1.0, 1)
    ref = O.pipeline(x, y, z, np.full(n, reach, dtype), obox, 16, 1, 1, 64, with_neighbors=False)
    leaves = torch.from_numpy(ref["leaves"].view(np.int64)).cuda()
    o = cs.build_octree(leaves)
    t = to_dev(ref["x"], ref["y"], ref["z"], ref["h"])
    c, s = cs.geo_centers(o.prefixes, box, t[0].dtype, 1)
    out = (torch.full((last - first, 100), -1, dtype=torch.int32, device="cuda"),
           torch.full((last - first,), -1, dtype=torch.int32, device="cuda"))
    rnb, rnc = O.find_neighbors(ref["x"], ref["y"], ref["z"], ref["h"], first, last, obox, ref["tree"], ref["layout"],
                                ref["centers"], ref["sizes"], 100)
    cs.find_neighbors(*t, first, last, box, o, torch.from_numpy(ref["layout"].view(np.int32)).cuda(), c, s, 100, out=out)
    torch.cuda.synchronize()
    neighbor_lists_equal(u32(out[0]).reshape(-1, 100), u32(out[1]), rnb, rnc, 100)
