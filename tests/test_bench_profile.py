"""The bench line's measured traffic comes from the committed profile of the
dominant kernel: the file has to be there, and the block-step kernel's say no
less than the three fields read once."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_profiles_of_the_dominant_kernels_are_found():
    for kernel in ("STEP", "E", "H"):
        traffic, path = bench.profile_traffic(kernel)
        assert traffic is not None, path
    assert bench.profile_traffic("STEP")[0] >= 2048 * 2048 * 12
