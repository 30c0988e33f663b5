"""GPU parity of the neighbour search in periodic boxes with particles above the box (moved, not yet wrapped): their keys
are those of the last cells, a target whose sphere crosses a boundary meets them folded, any other target where they are.
Cell radii below and above the search radius. Counts and lists equal the oracle's exactly."""
import numpy as np
import pytest
import torch

from gpu_util import neighbor_lists_equal, to_dev, u32, uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("bnd", [1, (1, 0, 0), (0, 1, 1)])
@pytest.mark.parametrize("ext", [0.8, 1.0, 1.5, 3.0])
@pytest.mark.parametrize("part", [0.02, 0.5])
def test_particles_above_a_periodic_box(cs, O, part, ext, bnd, dtype):
    n, ngmax = 8000, 200
    rng = np.random.default_rng(82)
    # about the corners of the box, dense enough for warps whose targets fold to one image; a part stays unwrapped
    x, y, z = (np.where((c < 0) | (rng.random(n) < part), c + 1, c).astype(dtype)
               for c in uniform(O, 81, n, -0.15, 0.15))
    h = (0.01 + 0.01 * rng.random(n)).astype(dtype)
    for kind, bits in ((1, 64), (0, 64)) + (((0, 32),) if dtype == np.float32 else ()):
        ref = O.pipeline(x, y, z, h, O.make_box(0.0, 1.0, bnd), 16, ngmax, kind, bits, ext)
        p = cs.Pipeline(64 if dtype == np.float64 else 32, bits, kind, 16, ngmax, ext, 1.0, False, True)
        t = to_dev(x, y, z, h)
        for group in (32, 16):
            p.set_tuning(group, 7)
            p.run(*t, cs.make_box(0.0, 1.0, bnd))
            out = p.outputs()
            torch.cuda.synchronize()
            neighbor_lists_equal(u32(out["neighbors"]).reshape(-1, ngmax), u32(out["neighbor_counts"]), ref["nb"],
                                 ref["nc"], ngmax)


@pytest.mark.parametrize("ext", [1.0, 3.0])
def test_particles_on_the_far_face_of_a_distant_box(cs, O, ext):
    """FP32, spacings far larger than the box's own rounding: spheres that reach the lower face only by less than half a
    spacing (their targets do not cross it) and particles exactly on the upper face, one period away."""
    n, ngmax, lo, hi = 4000, 300, 1e5, 1e5 + 16
    u = float(np.spacing(np.float32(lo)))
    rng = np.random.default_rng(83)
    x, y, z = (np.where(c < 0, c + hi, c + lo).astype(np.float32) for c in uniform(O, 84, n, -1.5, 1.5))
    h = (0.5 * u * rng.uniform(80.0, 150.0, n)).astype(np.float32)
    k = np.arange(0, 1200, 2)
    for v in (y, z):
        v[k] = v[k + 1] = (lo + u * rng.integers(160, 190, k.size)).astype(np.float32)
    x[k], x[k + 1], h[k + 1] = hi, lo + 150 * u, 0.5 * 150.3 * u
    ref = O.pipeline(x, y, z, h, O.make_box(lo, hi, 1), 16, ngmax, 1, 64, ext)
    p = cs.Pipeline(32, 64, 1, 16, ngmax, ext, 1.0, False, True)
    p.run(*to_dev(x, y, z, h), cs.make_box(lo, hi, 1))
    out = p.outputs()
    torch.cuda.synchronize()
    neighbor_lists_equal(u32(out["neighbors"]).reshape(-1, ngmax), u32(out["neighbor_counts"]), ref["nb"], ref["nc"], ngmax)
