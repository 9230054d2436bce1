"""bench.py's work model: the windows per seed counted on the host are those that the kernel's diagnostics
form counts on the whole workloads (COLLATZ_RANGE_STATS: 4 869 798 755 windows of 2 608 524 069 seeds at 2^40,
10 538 229 063 of 5 401 515 694 at 2^60).  The sample's mean lies within 3 standard errors: a seed's
windows have a standard deviation of at most 1.6."""
import math

import pytest


@pytest.mark.parametrize("offset,size,k,want", [(1 << 40, 1 << 38, 24, 4869798755 / 2608524069),
                                                (1 << 60, 1 << 40, 34, 10538229063 / 5401515694)])
def test_windows_per_seed(offset, size, k, want):
    import bench
    n = 3000
    assert abs(bench.windows_per_seed(offset, size, k, n) - want) < 3 * 1.6 / math.sqrt(n)
