"""GPU parity of the halo traversals that are handed on in pieces: a few focus leaves whose search boxes hold most of the
tree (every pass takes part), many of them at once (the lists of the later passes overflow and the rest is walked in
place), through the pipeline's scratch memory and through the stage call's own, and the stage call inside a graph
capture (no scratch memory). Flags equal the oracle's exactly."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,hmax,last", [(3000, 2.0, 1 << 61), (60000, 1.0, 1 << 57), (60000, 0.2, 1 << 61),
                                         (40000, 4.0, 3 << 61)])
def test_long_traversals(cs, O, n, hmax, last, dtype):
    rng = np.random.default_rng(n)
    x, y, z = (a.astype(dtype) for a in O.plummer(17, n, 10.0))
    lo, hi = [float(a.min()) for a in (x, y, z)], [float(a.max()) for a in (x, y, z)]
    h = (0.01 + hmax * rng.random(n) ** 8).astype(dtype)
    obox, box = O.make_box(lo, hi), cs.make_box(lo, hi)
    ref = O.pipeline(x, y, z, h, obox, 8, 1, with_neighbors=False)
    tree, leaves = ref["tree"], ref["leaves"]
    first, end = 0, int(np.searchsorted(leaves, np.uint64(last)))
    l2i = tree.leaf_to_internal[tree.num_internal:]
    sc, ss = O.search_boxes(ref["x"], ref["y"], ref["z"], ref["h"], ref["layout"], first, end, 2.0, l2i, ref["centers"])
    want = O.find_halos(tree, ref["centers"], ref["sizes"], sc, ss, obox, first, end)
    p = cs.Pipeline(64 if dtype == np.float64 else 32, 64, cs.HILBERT, 8, 1, 1.0, 1.0, True, False)
    p.run(*to_dev(x, y, z, h), box, (0, last))
    out = p.outputs()
    torch.cuda.synchronize()
    assert np.array_equal(out["halo_flags"].cpu().numpy(), want)
    o = cs.build_octree(torch.from_numpy(leaves.view(np.int64)).cuda())
    c, s = cs.geo_centers(o.prefixes, box, torch.float64 if dtype == np.float64 else torch.float32)
    tsc, tss = to_dev(sc, ss)
    flags = cs.find_halos(o, c, s, tsc, tss, box, first, end)
    torch.cuda.synchronize()
    assert np.array_equal(flags.cpu().numpy(), want)
    graph, flags = torch.cuda.CUDAGraph(), torch.zeros_like(flags)
    with torch.cuda.graph(graph):
        cs.find_halos(o, c, s, tsc, tss, box, first, end, flags)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(flags.cpu().numpy(), want)
