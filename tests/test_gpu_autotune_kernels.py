"""The autotuner runs each traversal kernel once: candidates that differ in a field that no kernel reads share its time,
and among them the first one is kept."""
import numpy as np
import pytest
import torch

from gpu_util import to_dev, uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_candidates_of_one_kernel_share_its_time(cs, O, dtype):
    n = 60000
    p = cs.Pipeline(64 if dtype == np.float64 else 32, 64, cs.HILBERT, 64, 100, 1.0, 1.0, False, True)
    p.run(*to_dev(*uniform(O, 91, n, 0.0, 1.0, dtype), np.full(n, 0.5 * (90 / (4 * np.pi * n)) ** (1 / 3), dtype)),
          cs.make_box(0.0, 1.0))
    r = p.autotune(3)
    torch.cuda.synchronize()
    times = {}
    for c, ms in r["tried"][:-2]:  # the last two are the sort's tile shapes
        times.setdefault(c["nb_group"], []).append(ms)
    assert sorted(times) == [8, 16, 32] and all(len(set(t)) == 1 for t in times.values())
    assert r["best"]["nb_by_target_cost"] == 7
