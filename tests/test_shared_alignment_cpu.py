"""Dynamic shared memory follows a kernel's static shared variables, so the
compiler aligns it to its element type alone.  Kernels copy into it and read
from it 16 bytes at a time: every dynamic array asks for 16 bytes."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_dynamic_shared_arrays_ask_for_16_bytes():
    found = 0
    for path in glob.glob(os.path.join(ROOT, "tart-gnss_b200", "csrc", "*.cu*")):
        for line in open(path):
            if re.search(r"extern\s+__shared__", line):
                found += 1
                m = re.search(r"__align__\((\d+)\)", line)
                assert m and int(m.group(1)) % 16 == 0, (os.path.basename(path), line.strip())
    assert found >= 8
