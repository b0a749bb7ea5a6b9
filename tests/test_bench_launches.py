"""bench.py's count of kernels in a trace of the hole: the path kernel and the areas,
and three kernels for every piece of rays that is ordered."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("rays,kernels", [(1, 2), ((1 << 21) - 1, 2), (1 << 21, 5), (10_000_000, 5), (1 << 25, 5),
                                          ((1 << 25) + 1, 8), (400_000_000, 2 + 3 * 12), (1 << 29, 2 + 3 * 16),
                                          ((1 << 29) + 1, 3 + 3 * (9 + 8))])  # 2^28 + 1 and 2^28 rays
def test_launches_per_step(rays, kernels):
    import bench
    assert bench.launches_per_step(rays) == kernels
