"""GPU parity of the tiled neighbour search where the search radius is small against the coordinates' rounding: FP32 sets
whose radius is a few spacings of their coordinates, a dense core in a wide box, the same across a periodic face, and
batched sets of very different scales. The path-safe threshold is below zero there, so that no pair is decided by the tile
itself. Counts and lists equal the oracle's exactly."""
import numpy as np
import pytest
import torch

from gpu_util import neighbor_lists_equal, to_dev, u32, uniform
from test_gpu_batch import check_set, run_batch

pytestmark = pytest.mark.gpu


def _check(cs, O, x, y, z, h, lo, hi, bnd=0, ngmax=100):
    ref = O.pipeline(x, y, z, h, O.make_box(lo, hi, bnd), 16, ngmax)
    assert ref["nc"].mean() > 5  # the case is about pairs
    p = cs.Pipeline(64 if x.dtype == np.float64 else 32, 64, 1, 16, ngmax, 1.0, 1.0, False, True)
    t = to_dev(x, y, z, h)
    for group in (32, 16):
        p.set_tuning(group, 7)
        p.run(*t, cs.make_box(lo, hi, bnd))
        out = p.outputs()
        torch.cuda.synchronize()
        neighbor_lists_equal(u32(out["neighbors"]).reshape(-1, ngmax), u32(out["neighbor_counts"]), ref["nb"], ref["nc"],
                             ngmax)


@pytest.mark.parametrize("ulps", [2, 5, 10, 30, 100])
@pytest.mark.parametrize("offset", [1e3, 1e5, 1e6])
def test_radii_of_a_few_spacings(cs, O, offset, ulps):
    n = 3000
    r = ulps * float(np.spacing(np.float32(offset)))
    side = r * (4 * np.pi * n / (3 * 40)) ** (1 / 3)
    x, y, z = uniform(O, 61, n, 0.0, side)
    x, y, z = ((v + o).astype(np.float32) for v, o in ((x, offset), (y, -offset), (z, 0.5 * offset)))
    lo, hi = [float(a.min()) for a in (x, y, z)], [float(a.max()) for a in (x, y, z)]
    _check(cs, O, x, y, z, np.full(n, r / 2, np.float32), lo, hi)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("radius", [1e-7, 1e-6, 1e-5])
def test_a_dense_core_in_a_wide_box(cs, O, radius, dtype):
    n, wide = 4000, 2e3
    r = radius * wide
    x, y, z = uniform(O, 62, n, -3.0 * r, 3.0 * r)
    u, v, w = uniform(O, 63, n, -wide / 2, wide / 2)
    few = np.arange(n) % 16 == 0
    x, y, z = (np.where(few, a, b).astype(dtype) for a, b in ((u, x), (v, y), (w, z)))
    _check(cs, O, x, y, z, np.full(n, r / 2, dtype), (-wide / 2,) * 3, (wide / 2,) * 3, 0, 400)


@pytest.mark.parametrize("ulps", [2, 5, 20])
@pytest.mark.parametrize("bnd", [1, (1, 0, 0)])
def test_small_radii_across_a_periodic_face(cs, O, bnd, ulps):
    n, at, side = 4000, 1e5, 16.0
    r = ulps * float(np.spacing(np.float32(at)))
    c = uniform(O, 64, n, -3.0 * r, 3.0 * r)
    x, y, z = (np.where(v < 0, v + side, v) for v in c)
    x, y, z = ((v + at).astype(np.float32) for v in (x, y, z))
    _check(cs, O, x, y, z, np.full(n, r / 2, np.float32), (at,) * 3, (at + side,) * 3, bnd, 200)


def test_batched_sets_of_different_scales(cs, O):
    rng = np.random.default_rng(65)
    sets = []
    for n, scale in ((4096, 0.01), (700, 3e3), (1000, 1e-4), (2000, 1.0)):
        x, y, z = (rng.uniform(0.0, scale, n).astype(np.float32) for _ in range(3))
        h = np.full(n, 0.5 * scale * (3 * 40 / (4 * np.pi * n)) ** (1 / 3), np.float32)
        sets.append(dict(x=x, y=y, z=z, h=h, lo=(0.0,) * 3, hi=(scale,) * 3, bucket=16))
    _, out, offsets = run_batch(cs, sets, 32, cs.MORTON, 100)
    for j, s in enumerate(sets):
        check_set(O, out, offsets, j, s, 0, 100)
