"""Rules on how many blocks fit the device ask it for its SMs: the sources name
no count of their own, which a partition of the GPU would not have."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pascal_poisson_fft_b200", "csrc")


def test_no_literal_sm_count():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for line in open(path):
            code = line.split("//")[0]
            assert not re.search(r"\b14[78]L?\b", code), (path, line)
