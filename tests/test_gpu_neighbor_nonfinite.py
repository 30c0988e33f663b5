"""GPU parity of the neighbour search with targets and candidates whose coordinates are not finite, in open and periodic
boxes: they have no neighbours, and the targets that share their warps keep all of theirs. Smoothing lengths of zero,
infinity and NaN among ordinary ones. Counts and lists equal the oracle's exactly."""
import numpy as np
import pytest
import torch

from gpu_util import neighbor_lists_equal, to_dev, u32, uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("spread,bnd", [(1.0, 0), (1.0, 1), (0.1, 1)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("axis", [0, 2, 3])
def test_values_that_are_not_finite(cs, O, axis, value, spread, bnd, dtype):
    n, ngmax = 3000, 80
    obox, box = O.make_box(-1.0, 1.0, bnd), cs.make_box(-1.0, 1.0, bnd)
    x, y, z = uniform(O, 71, n, -spread, spread, dtype)
    if spread < 1.0:  # about the corners of the box: warps at the faces whose targets fold to one image
        x, y, z = (np.where(v < 0, v + dtype(1), v - dtype(1)) for v in (x, y, z))
    ref = O.pipeline(x, y, z, np.full(n, 0.1 * spread, dtype), obox, 16, 1, with_neighbors=False)
    a = [ref[c].copy() for c in "xyzh"]
    # the first target of a warp, inner ones, two of one warp, the last one of all
    a[axis][[0, 32, 77, 500, 501, 1024, 1600, 2048, n - 1]] = value
    a[3][[40, 900]] = 0
    rnb, rnc = O.find_neighbors(*a, 0, n, obox, ref["tree"], ref["layout"], ref["centers"], ref["sizes"], ngmax)
    o = cs.build_octree(torch.from_numpy(ref["leaves"].view(np.int64)).cuda())
    t = to_dev(*a)
    c, s = to_dev(ref["centers"], ref["sizes"])
    nb, nc = cs.find_neighbors(*t, 0, n, box, o, torch.from_numpy(ref["layout"].view(np.int32)).cuda(), c, s, ngmax)
    torch.cuda.synchronize()
    neighbor_lists_equal(u32(nb).reshape(-1, ngmax), u32(nc), rnb, rnc, ngmax)
