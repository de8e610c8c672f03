"""Host arithmetic of the benchmark line."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench


def test_butterfly_peak_follows_the_primes_not_their_number():
    probe = (0.0, 0.0, 1.0, 2.0)
    for widths, sets, peak in (([2], [0], 1.0), ([2], [3], 2.0), ([3], [1], 2.0), ([4], [0], 2.0),
                               ([2, 2, 3, 3], [0, 3, 1, 1], 1.75)):
        assert bench.butterfly_peak(np.array(widths), np.array(sets), probe) == peak
