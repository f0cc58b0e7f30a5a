"""Every dynamic shared-memory array of the kernels is declared with the 16-byte alignment that the
vector accesses (and, with them, the sizes the layouts are rounded to) rely on."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "bernsteinbasis.jl_gb300", "csrc")


def test_dynamic_shared_arrays_are_aligned():
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as fh:
            for line in re.findall(r"extern __shared__[^;]*;", fh.read()):
                found += 1
                assert "__align__(16)" in line or "__align__(1024)" in line, (path, line)
    assert found >= 10
