"""GPU parity of the tree operations at their kernels' edges: target groups whose cuts sit at the criterion (the FP32
screen must leave them to FP64), far from the origin and with tiny and zero h; leaf centres over leaves of 0 to 70
particles with zero and negative masses; upsweeps of a whole tree. Equal to the oracle bit for bit."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("size", [32, 64])
@pytest.mark.parametrize("case", ["criterion", "offset", "tiny"])
def test_group_splits_at_the_criterion(cs, O, case, size, dtype):
    rng = np.random.default_rng(size)
    n = 3001
    x, y, z = (a.astype(dtype) for a in O.plummer(11, n, 10.0))
    h = (0.02 + 0.2 * rng.random(n)).astype(dtype)
    if case == "offset":
        x, y, z = x + dtype(1000), y - dtype(1000), z + dtype(3000)
    if case == "tiny":
        x, y, z, h = x * dtype(1e-12), y * dtype(1e-12), z * dtype(1e-12), h * dtype(1e-12)
        h[::7] = 0
    lo, hi = [float(a.min()) for a in (x, y, z)], [float(a.max()) for a in (x, y, z)]
    ref = O.pipeline(x, y, z, h, O.make_box(lo, hi), 16, 1, with_neighbors=False)
    x, y, z, h = (np.array(ref[c]) for c in "xyzh")
    if case == "criterion":
        # h such that 2 h / (shortest edge) is the distance to the next particle in the unit box, some ulps about it
        ext = [dtype(b) - dtype(a) for a, b in zip(lo, hi)]
        d = np.sqrt(sum((np.diff(a) * (dtype(1) / e)) ** 2 for a, e in zip((x, y, z), ext)))
        h[:-1] = 0.5 * d * min(ext)
        for k in range(1, 6):
            h[k::6] = np.nextafter(h[k::6], dtype(0) if k % 2 else dtype(np.inf))
    first, last = 5, n - 7
    for tol in (0.5, 8.0):
        want = O.group_splits(first, last, x, y, z, h, ref["leaves"], ref["layout"], lo, hi, size, tol)
        t = to_dev(x, y, z, h)
        got = cs.group_splits(first, last, *t, torch.from_numpy(ref["leaves"].view(np.int64)).cuda(),
                              torch.from_numpy(ref["layout"].view(np.int32)).cuda(), cs.make_box(lo, hi), size, tol)
        assert np.array_equal(u32(got), want)


@pytest.mark.parametrize("dtype,mtype", [(np.float64, np.float64), (np.float64, np.float32), (np.float32, np.float32)])
def test_source_centers_over_uneven_leaves(cs, O, dtype, mtype):
    rng = np.random.default_rng(2)
    sizes = np.concatenate([np.arange(71), rng.integers(0, 70, 930)])
    layout = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    n, L = int(layout[-1]), sizes.size
    x, y, z = (rng.normal(0, 1, n).astype(dtype) for _ in range(3))
    m = rng.normal(0, 1, n).astype(mtype)
    m[int(layout[40]):int(layout[41])] = 0
    l2i = rng.permutation(L + 5)[:L].astype(np.int32)
    want = O.leaf_mass_centers(x, y, z, m, l2i, layout, L + 5)
    got = torch.zeros((L + 5, 4), dtype=torch.float64 if dtype == np.float64 else torch.float32, device="cuda")
    cs.leaf_source_centers(*to_dev(x, y, z, m, l2i, layout.view(np.int32)), got)
    assert np.array_equal(got.cpu().numpy()[l2i], np.asarray(want).reshape(-1, 4)[l2i])
