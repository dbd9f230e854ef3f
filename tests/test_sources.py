"""Properties of the kernels' sources that no run shows."""
import glob
import os
import re

from icpp_2020_parhde_gb300 import build


def test_dynamic_shared_memory_is_declared_aligned():
    """A dynamic shared array follows the kernel's static ones; copies and vector accesses of 16 bytes into it are only
    right when the declaration asks for that alignment."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(build.CSRC, "*.cu"))):
        for line in open(path):
            m = re.match(r"\s*extern __shared__ (.*);", line)
            if m:
                seen += 1
                a = re.match(r"__align__\((\d+)\)", m.group(1))
                assert a and int(a.group(1)) % 16 == 0, "%s: %s" % (os.path.basename(path), line.strip())
    assert seen >= 20
