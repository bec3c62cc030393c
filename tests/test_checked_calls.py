"""Device copies, fills and allocations of the library are checked: none stands as a
statement of its own, its status dropped."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200", "csrc")


def test_no_status_of_a_copy_fill_or_allocation_is_dropped():
    dropped = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        # the statement begins with the call, or with a condition's closing bracket before it
        for m in re.finditer(r"(?:[;{}]|\) )\s*(cuda(?:Memcpy|Memset|Malloc)\w*)\((?=[^;]*\);)", code):
            dropped.append((os.path.basename(path), m.group(1), code[:m.start(1)].count("\n") + 1))
    assert not dropped
