"""CPU: the lanes that a warp-wide operation waits for are known beforehand.

A vote or reduction waits for every lane that its mask names.  A mask read from
__activemask() in divergent code names the lanes that happen to run together
just then, and nothing makes them arrive together; a warp's operations take a
mask that holds by the kernel's structure.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "recon-scanner_gb300", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


@pytest.mark.parametrize("name", FILES)
def test_no_mask_of_the_moment(name):
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
    assert "__activemask" not in src and "activemask.b32" not in src
