"""Two balance-function contexts of different grids in one process: the kernel's
shared memory is set for the largest grid, not for the last context made."""
import numpy as np
import pytest

from hadronic_afterburner_toolkit_gb300 import bf

pytestmark = pytest.mark.gpu


def test_small_grid_made_after_a_large_one():
    rng = np.random.default_rng(1)
    off = np.array([0, 200])
    lists = [(off, rng.uniform(-3.0, 3.0, 200), rng.normal(0.0, 1.0, 200))]
    jobs = [(0, 0, 0, 0, 0, 0, 0.0)]
    large = bf.BfEngine(600, 2.0)
    small = bf.BfEngine(11, 2.0)
    for b in (large, small, large):
        b.reset()
        b.bin(lists, jobs)
    # wide y bins hold the narrow ones' pairs, but for those past the range
    assert abs(large.hist(0).sum() - small.hist(0).sum()) < 0.1 * small.hist(0).sum()
    assert small.hist(0).sum() > 10000
    large.close()
    small.close()
