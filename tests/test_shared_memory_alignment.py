"""CPU check of the kernels' dynamic shared memory: an array that FP64 or
vector values are carved from declares the alignment they need (a block's
static shared variables may end at any word, and a misaligned FP64 access
faults)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imaging_fcs_1_52_gb300", "csrc")
DECL = re.compile(r"extern\s+__shared__\s+(?:__align__\((\d+)\)\s+)?([\w ]+?)\s+(\w+)\[\]")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_dynamic_shared_arrays_declare_eight_bytes(path):
    for align, typ, name in DECL.findall(open(path).read()):
        assert typ == "double" or int(align or 0) >= 8, f"{typ} {name}[]"
