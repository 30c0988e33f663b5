"""The one-block sort of up to 8192 keys and the tiled sort just above it: sizes around its warps and its end, keys of all
ones (the padding's value), partial bit ranges, given values and 0..n-1. Stable: equal to numpy's stable argsort."""
import numpy as np
import pytest
import torch

from gpu_util import keys_u, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [2, 33, 255, 256, 257, 2047, 2048, 2049, 4097, 7937, 8191, 8192, 8193, 12289])
def test_small_sorts(cs, n, bits):
    rng = np.random.default_rng(n)
    ut, st = (np.uint32, np.int32) if bits == 32 else (np.uint64, np.int64)
    for kind, (b0, b1) in (("random", (0, bits)), ("ones", (0, bits)), ("few", (3, bits - 5)), ("random", (bits - 9, bits))):
        k = rng.integers(0, np.iinfo(ut).max, n, dtype=ut, endpoint=True)
        if kind == "ones":
            k[rng.random(n) < 0.7] = np.iinfo(ut).max
        if kind == "few":
            k = (k % ut(5)) << ut(bits // 2)
        vals = rng.integers(0, 1 << 31, n).astype(np.int32)
        order = np.argsort((k >> ut(b0)) & ut((1 << (b1 - b0)) - 1), kind="stable")
        for v in (None, vals):
            dk = torch.from_numpy(k.view(st).copy()).cuda()
            dv = None if v is None else torch.from_numpy(v.copy()).cuda()
            sk, sv = cs.sort_pairs(dk, dv, b0, b1, iota=v is None)
            assert np.array_equal(keys_u(sk), k[order].astype(np.uint64))
            assert np.array_equal(u32(sv), order.astype(np.uint32) if v is None else vals[order].view(np.uint32))
