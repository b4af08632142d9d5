"""What bench.py's roofline counts for a transport kernel: the records it reads and
writes and the steps it makes (CPU only)."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("ms,kernel,steps,records", [([3.0, 2.0, 1.0], 0, 70, 30), ([1.0, 2.0, 1.5], 1, 24, 12),
                                                     ([1.0, 1.2, 1.5], 2, 9, 7)])
def test_steps_and_bytes_are_the_kernels_own(ms, kernel, steps, records):
    import bench
    st = {"transport_ms": ms, "step_launches": [4, 4, 0], "transport_steps": [70, 40, 9], "booked_steps": 16,
          "transport_read": [20, 8, 4], "transport_written": [10, 4, 3], "bytes_per_track": 96}
    assert bench.dominant_kernel(st) == (kernel, max(1, [4, 4, 0][kernel]), ms[kernel], steps, records, 96 * records)
