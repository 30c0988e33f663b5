"""GPU parity of the octree linkage at the edges of its tiles of 1024 leaves: one node more or less than a tile, several
tiles, and trees that reach the deepest level along one path or at the ends of the curve. Equal to the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import keys_u

pytestmark = pytest.mark.gpu


def _tree(rng, splits, bits, where):
    """cornerstone array of a root split `splits` times: at random leaves, or always at the first, last or a fixed key"""
    max_level = 21 if bits == 64 else 10
    leaves = [(0, 8**max_level)]
    fixed = int(rng.integers(0, 8**max_level))
    for _ in range(splits):
        open_ = [i for i, (a, w) in enumerate(leaves) if w > 1]
        if where == "first":
            i = open_[0]
        elif where == "last":
            i = open_[-1]
        elif where == "path":
            i = next((i for i in open_ if leaves[i][0] <= fixed < sum(leaves[i])), open_[len(open_) // 2])
        else:
            i = open_[int(rng.integers(0, len(open_)))]
        a, w = leaves[i]
        leaves[i:i + 1] = [(a + k * (w // 8), w // 8) for k in range(8)]
    return np.array([a for a, _ in leaves] + [8**max_level], np.uint64 if bits == 64 else np.uint32)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("where", ["random", "first", "last", "path"])
@pytest.mark.parametrize("splits", [0, 1, 21, 146, 147, 292, 293, 439, 900])
def test_link_at_tile_edges(cs, O, splits, where, bits):
    leaves = _tree(np.random.default_rng(splits), splits, bits, where)
    assert leaves.size - 1 == 7 * splits + 1
    ref = O.build_octree(leaves, bits)
    o = cs.build_octree(torch.from_numpy(leaves.view(np.int64 if bits == 64 else np.int32)).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(keys_u(o.prefixes), ref.prefixes)
    assert np.array_equal(o.child_offsets[: o.num_nodes].cpu().numpy(), ref.child_offsets)
    groups = (o.num_nodes - 1) // 8  # a single leaf has no sibling group, its one slot is never written
    assert np.array_equal(o.parents.cpu().numpy()[:groups], ref.parents[:groups])
    assert np.array_equal(o.level_range.cpu().numpy(), ref.level_range)
    assert np.array_equal(o.internal_to_leaf.cpu().numpy(), ref.internal_to_leaf)
    assert np.array_equal(o.leaf_to_internal.cpu().numpy(), ref.leaf_to_internal)
