"""CPU: shared arrays of field elements are declared on 16-byte boundaries.
The kernels read and write them as 16-byte vectors, while the element type
has a 32-bit word's alignment, so nothing but the declaration secures it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_gpu_b200", "csrc")


def test_shared_elements_are_aligned():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        for line in open(path):
            if re.search(r"__shared__\s.*\bfe\s+\w+\[", line):
                found.append((os.path.basename(path), line.strip(), "__align__(16)" in line))
    assert found
    assert all(ok for _, _, ok in found), [f for f in found if not f[2]]
