"""The bench's achieved operation rate: its survivors over the time of every kernel that reads survivors (those of the rest
list come by the shared-prime kernels, after the persistent one)."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def test_rate_counts_the_time_of_all_survivors():
    import bench
    # 24 operations for each of 10^9 survivors in 90 + 10 ms
    assert bench.achieved_gops(10 ** 9, 90.0, 10.0) == pytest.approx(240.0)
