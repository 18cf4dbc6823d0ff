"""A block-wide barrier under a condition needs one that every thread of the
block decides alike: made of the kernel's arguments (A., E., S., D., g., apply) alone."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpumetropolis_b200", "csrc")


def test_conditional_barriers_depend_on_arguments_only():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for cond in re.findall(r"\bif\s*\(([^;{}]*?)\)\s*\{?\s*__syncthreads\b", text):
            seen += 1
            names = re.findall(r"[A-Za-z_]\w*(?:\.\w+)*", cond)
            assert all(re.fullmatch(r"[AESDg]\.\w+|apply", n) for n in names), (path, cond)
    assert seen
