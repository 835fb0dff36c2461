"""Device memory is allocated in one place.  The pool of the stateless entry
points keeps memory between calls; an allocation that fails must take it back
before it gives up, so the library's only cudaMalloc calls are those of
device_malloc, which does."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxelsim_fea_b200", "csrc")


def test_every_device_allocation_can_take_the_pool_back():
    found = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        with open(path) as f:
            src = re.sub(r"//[^\n]*|\"(?:[^\"\\\n]|\\.)*\"", "", f.read())
        n = len(re.findall(r"\bcuda(?:Malloc|MallocAsync|MallocManaged|MallocPitch)\s*\(", src))
        if n:
            found[os.path.basename(path)] = n
    assert found == {"vf_workspace.cu": 2}, found
