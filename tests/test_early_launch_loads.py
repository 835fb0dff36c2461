"""Kernels that start before their predecessor ends (those that call
pdl_enter) read what it writes through plain pointers only.  The read-only data
path (const __restrict__ parameters, __ldg) is specified for data that nobody
writes while the kernel exists; an early kernel exists while its predecessor
still writes.  Read from the sources: in each such kernel every
const __restrict__ pointer and every __ldg names set-up data -- operators,
masks, diagonals, index tables -- and waits before its first statement."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voxelsim_fea_b200", "csrc")
SETUP = {"stc", "sqd", "minv", "minvc", "mask", "cm", "fm", "E", "MU", "store", "Sinv", "perm", "Ainv"}
# local names of set-up data: rows of an inverse, the diagonal as vectors, the separators' blocks
LOCAL = {"row", "mv", "W", "am", "E", "MU"}


def _early_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__", src):
            start = src.index("{", m.end())
            depth, i = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            head, body = src[m.end():start], src[start + 1:i - 1]
            if "pdl_enter()" in body:
                yield os.path.basename(path), re.findall(r"(\w+)\s*\(", head)[-1], head, body


def test_early_kernels_read_dependent_data_through_plain_pointers():
    seen, wrong = 0, []
    for name, kernel, head, body in _early_kernels():
        seen += 1
        if not body.lstrip().startswith("pdl_enter();"):
            wrong.append((name, kernel, "does not wait first"))
        for text in (head, body):
            for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", text):
                if p not in SETUP:
                    wrong.append((name, kernel, "const __restrict__ " + p))
        for p in re.findall(r"__ldg\(\s*\(?(?:\([^()]*\))?\s*([\w.]+)", body):
            if p not in SETUP | LOCAL | {"a.mask"}:
                wrong.append((name, kernel, "__ldg of " + p))
    assert seen >= 25
    assert not wrong, wrong
